"""Device memory of the split of small launches (refine.cu): the smallest calls take little of it,
pools built without read-backs fit the room that their estimate gives them, and a call whose levels
do not fit, or that finds no memory for them at all, still gives the same results (the checked
build takes less room, or asks for more memory than there is, on request)."""
import os
import subprocess
import sys

import pytest

from conftest import ORACLE_DIR, PKG_DIR, ROOT

pytestmark = pytest.mark.gpu
CHECKED = os.path.join(PKG_DIR, "libnqb_checked.so")


@pytest.mark.parametrize("form", [0, 1])
def test_smallest_calls_take_little_memory(nqb, form):
    torch = pytest.importorskip("torch")
    boards = nqb.sample_boards(3, 16, 8, 12, 2, 5)
    for call in (lambda: nqb.count(8, 2, form=form), lambda: nqb.solve_batch(boards, form=form)):
        call()  # loads the kernels
        torch.cuda.synchronize()
        nqb.trim_device_memory(0)
        before = torch.cuda.mem_get_info()[0]
        call()
        # the pool maps memory in pieces of up to 32 MB; the split's buffers once took 102 MB here
        assert before - torch.cuda.mem_get_info()[0] <= 64 << 20


def small_pool(n, d):
    size = (n + 1) // 2
    for r in range(1, d):
        size *= n * (1.0 - r / n) ** 2.4
        if size > 0.8 * 3200000:
            return False
    return True


@pytest.mark.parametrize("n", [4, 5, 8, 11, 12, 13, 14, 15, 16, 17])
def test_estimated_room_holds_every_level(nqb, n):
    # a pool that did not fit would be built again level by level, in fewer counted launches
    for d in range(2, n):
        if not small_pool(n, d):
            continue
        st = nqb.count_ex(n, d)[1]
        split_levels = min(4, max(0, n - d - 8))
        assert st["kernel_launches"] == 1 + (d - 1) + split_levels + 1, (n, d)


SCRIPT = r"""
import os, sys, importlib.util
import numpy as np
spec = importlib.util.spec_from_file_location("nqb", sys.argv[1] + "/__init__.py")
nqb = importlib.util.module_from_spec(spec); spec.loader.exec_module(nqb)
sys.path.insert(0, sys.argv[2]); import nqo
boards = np.concatenate([nqb.sample_boards(5, 300, 8, 14, 1, 4), nqb.sample_boards(6, 40, 14, 16, 3, 6)])
want_boards, want_nodes = nqo.solve_states(boards)
each = [nqo.solve_states(boards[i:i + 1])[1] for i in range(len(boards))]
pools = [(8, 3), (10, 6), (12, 4), (12, 9), (13, 1), (14, 4), (15, 6), (16, 3), (16, 6), (17, 5)]
want = {}
for room in (None, 16, 100, 5000, 200000, 0):
    if room is not None:
        os.environ["NQB_SPLIT_ROOM"] = str(room)
    for n, d in pools:
        c, st = nqb.count_ex(n, d, count_unit_nodes=True)
        b, sb = nqb.count_ex(n, d, form=nqb.FORM_BATCHED)
        got = (c, st["nodes"], st["unit_nodes"], st["states"])
        if room is None:
            want[n, d] = got
        assert got == want[n, d] and (b, sb["nodes"], sb["states"]) == (c, st["nodes"], st["states"]), (room, n, d)
        if room == 0:
            assert st["kernel_launches"] == sb["kernel_launches"] == 1, (n, d)  # no split
    for form in (0, 1):
        got, st = nqb.solve_batch(boards, form=form)
        assert np.array_equal(got, want_boards) and st["nodes"] == want_nodes, (room, form)
    nodes, counts = nqb.record_nodes(boards)
    assert np.array_equal(counts, want_boards) and list(nodes) == each, room
print("all equal", nqb.LIB_PATH)
"""


def test_levels_that_do_not_fit():
    env = dict(os.environ, NQB_LIBRARY=CHECKED)
    env.pop("NQB_SPLIT_ROOM", None)
    p = subprocess.run([sys.executable, "-c", SCRIPT, PKG_DIR, ORACLE_DIR], capture_output=True, text=True, env=env,
                       timeout=1200, cwd=ROOT)
    assert p.returncode == 0, p.stderr[-3000:]
    assert p.stdout.split() == ["all", "equal", CHECKED]
