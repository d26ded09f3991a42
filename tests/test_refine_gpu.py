"""Items split before a launch that has few of them (refine.cu), against the oracle: launches
around the limits of the split (free columns at, below and above the least that is split),
boards of very different sizes in one batch, boards that the split makes vanish, and the node
totals per board."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def board_set(nqb, kind):
    if kind == "around the least split":  # 7, 8 and 9 free columns
        return np.concatenate([nqb.sample_boards(s, 40, n, n, d, d) for s, (n, d) in
                               enumerate([(8, 1), (9, 1), (9, 2), (12, 4), (12, 3), (16, 9)])])
    if kind == "uneven":
        big = np.zeros(3, dtype=nqb.STATE_DTYPE)
        big["n"], big["weight"] = [12, 11, 13], [2, 1, 2]
        return np.concatenate([big[:1], nqb.sample_boards(7, 300, 4, 13, 1, 3), big[1:]])
    if kind == "vanishing":  # every column but the outer ones attacked in the rows to come
        b = nqb.sample_boards(3, 64, 14, 14, 4, 4)
        b["ldiag"][::2] |= (1 << 14) - 2
        b["rdiag"][1::4] |= (1 << 14) - 1
        return b
    return nqb.sample_boards(31, 64, 31, 31, 24, 29)  # the widest board


@pytest.mark.parametrize("kind", ["around the least split", "uneven", "vanishing", "widest"])
def test_few_boards_match_oracle(nqb, nqo, kind):
    boards = board_set(nqb, kind)
    want, nodes = nqo.solve_states(boards)
    for form in (nqb.FORM_PLAIN, nqb.FORM_BATCHED):
        got, st = nqb.solve_batch(boards, form=form)
        assert np.array_equal(got, want) and st["nodes"] == nodes, form
    per_nodes, counts = nqb.record_nodes(boards)
    each = [nqo.solve_states(boards[i:i + 1])[1] for i in range(len(boards))]
    assert np.array_equal(counts, want) and list(per_nodes) == each


@pytest.mark.parametrize("n,d", [(9, 1), (10, 2), (12, 2), (13, 3), (14, 3)])
def test_shallow_pools_keep_counts_nodes_and_unit_nodes(nqb, nqo, n, d):
    want = nqo.replay_pool(n, d) if d > 1 else None
    c, st = nqb.count_ex(n, d, count_unit_nodes=True)
    b, sb = nqb.count_ex(n, d, form=nqb.FORM_BATCHED)
    assert c == b and st["nodes"] == sb["nodes"] and st["states"] == sb["states"]
    if want:
        assert (c, st["nodes"], st["unit_nodes"]) == (want["count"], want["nodes"], want["unit"])
