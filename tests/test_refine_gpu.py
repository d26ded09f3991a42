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


@pytest.mark.parametrize("n", [4, 5, 6, 7, 8, 11])
def test_every_pool_depth_of_small_boards(nqb, nqo, n):
    # the pool built without read-backs: each depth's size, and the count below it
    for d in range(1, n):
        for form in (nqb.FORM_PLAIN, nqb.FORM_BATCHED):
            c, st = nqb.count_ex(n, d, form=form)
            assert st["states"] == nqb.pool_size(n, d), (n, d, form)
            want = nqb.generate_pool(n, d)
            total, nodes = nqo.solve_states(want) if len(want) else (np.zeros(1, dtype=np.uint64), 0)
            assert c == int(np.sum(total)) and st["nodes"] == nodes, (n, d, form)


def test_pools_around_the_buffers_size(nqb):
    # the largest pools built without read-backs and the smallest built with them
    for n, d in [(17, 6), (17, 7), (18, 6), (15, 7), (15, 9), (16, 7), (16, 8), (16, 15)]:
        c, st = nqb.count_ex(n, d, form=nqb.FORM_BATCHED)
        assert st["states"] == nqb.pool_size(n, d)
        assert c == {15: 2279184, 16: 14772512, 17: 95815104, 18: 666090624}[n]
