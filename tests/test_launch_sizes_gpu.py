"""Launches of one kernel with deep and with shallow stacks from several threads at once: the
shared memory a launch needs (above 48 KB from 13 stack rows on with 256 threads) must not depend on
what another thread's launch of the same kernel asked for a moment before."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
THREADS, LAUNCHES = 8, 400


@pytest.mark.parametrize("form", ["plain", "batched"])
def test_deep_and_shallow_launches_at_once(nqb, form):
    torch = pytest.importorskip("torch")
    pool = nqb.generate_pool(8, 2)
    want, st = nqb.solve_states(pool)
    items = torch.from_numpy(pool.view(np.uint8).copy()).cuda()
    failed, results = [], [None] * THREADS
    gate = threading.Barrier(THREADS)

    def work(k):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            out = torch.zeros((LAUNCHES, 4), dtype=torch.int64, device="cuda")
            scratch = torch.zeros((LAUNCHES, 64), dtype=torch.uint8, device="cuda")  # queue words, no steal ring
        stream.synchronize()
        gate.wait()
        depth = 30 if k % 2 else 6  # rows of the stack: 124 KB or 28 KB a block of 256 threads
        for i in range(LAUNCHES):
            try:
                if form == "plain":
                    nqb.plain_launch(items.data_ptr(), len(pool), out[i].data_ptr(), block_size=256, stack_depth=depth,
                                     stream=stream.cuda_stream)
                else:
                    nqb.batched_launch_ex(items.data_ptr(), len(pool), scratch[i].data_ptr(), 64, out[i].data_ptr(),
                                          block_size=256, stack_depth=depth, stream=stream.cuda_stream)
            except nqb.NQBError as e:
                failed.append((k, i, e.status))
                break
        stream.synchronize()
        results[k] = out.cpu().numpy()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(THREADS)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
    for r in results:
        assert (r == [want, st["nodes"], 0, 0]).all()
