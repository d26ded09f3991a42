"""One to a few boards, on both sides of the free columns from which the batched form gives a split
batch the whole GPU: counts and nodes of each board against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# free columns 12 to 16: the split's four levels leave items of 8 to 12
@pytest.mark.parametrize("n,d", [(20, 8), (22, 9), (22, 8), (14, 0), (24, 9), (28, 13), (16, 1), (28, 12)])
@pytest.mark.parametrize("boards", [1, 3, 17])
def test_few_boards(nqb, nqo, n, d, boards):
    if d == 0:
        b = np.zeros(boards, dtype=nqb.STATE_DTYPE)
        b["n"], b["weight"] = n, 1
        b, boards = b[:1], 1
    else:
        boards = min(boards, 3) if (n, d) in [(16, 1), (28, 12)] else boards
        b = nqb.sample_boards(10 * n + d, boards, n, n, d, d)
    want, nodes = nqo.solve_states(b)
    for block in (64, 128, 256):
        got, st = nqb.solve_batch(b, form=nqb.FORM_BATCHED, block_size=block)
        assert np.array_equal(got, want) and st["nodes"] == nodes, block
    per_nodes, counts = nqb.record_nodes(b)
    assert np.array_equal(counts, want) and int(per_nodes.sum()) == nodes
