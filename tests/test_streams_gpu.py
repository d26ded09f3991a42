"""Calls from many threads at once, more of them than streams are kept for later calls, with the
cached memory and idle streams given back in between: every result is exact."""
import json
import os
import threading

import numpy as np
import pytest

from conftest import GOLDEN_DIR

pytestmark = pytest.mark.gpu
KAT = {int(k): v for k, v in json.load(open(os.path.join(GOLDEN_DIR, "ref_vectors.json")))["kat_counts"].items()}


def test_concurrent_calls_and_trim(nqb):
    boards = nqb.sample_boards(11, 500, 8, 12, 2, 5)
    want, _ = nqb.solve_batch(boards, form=nqb.FORM_BATCHED)
    model = nqb.Model(seed=3)
    predicted = model.predict(boards)
    bad = []

    def work(k):
        for i in range(6):
            if nqb.count(10 + (k + i) % 5, 3, form=(k + i) & 1) != KAT[10 + (k + i) % 5]:
                bad.append(("count", k, i))
            if k % 3 == 0 and not np.array_equal(nqb.solve_batch(boards, form=nqb.FORM_BATCHED)[0], want):
                bad.append(("batch", k, i))
            if k % 3 == 1 and not np.array_equal(model.predict(boards), predicted):
                bad.append(("predict", k, i))
            if k == 5:
                nqb.trim_device_memory(0)

    for _ in range(2):
        threads = [threading.Thread(target=work, args=(k,)) for k in range(24)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        nqb.trim_device_memory(0)
        nqb.trim_device_memory(0)
    model.close()
    assert not bad
