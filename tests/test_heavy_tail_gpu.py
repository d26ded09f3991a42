"""Queues of many small boards with a few large ones at their end: the rest of the GPU takes rows of
the large ones over, and every board's count and nodes stay exact, for FIFO batches and for plans."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def queue(nqb, nqo):
    small = nqb.sample_boards(21, 1200, 8, 11, 2, 5)
    small = small[np.random.default_rng(1).integers(0, len(small), 700000)]
    large = np.concatenate([nqb.sample_boards(22, 1, 17, 17, 2, 2), nqb.sample_boards(23, 1, 20, 20, 5, 5)])
    kinds, at = np.unique(np.concatenate([small, large]), return_inverse=True)
    counts, _ = nqo.solve_states(kinds)
    nodes = np.array([nqo.solve_states(kinds[i:i + 1])[1] for i in range(len(kinds))], dtype=np.uint64)
    return np.concatenate([small, large]), np.asarray(counts)[at], nodes[at]


@pytest.mark.parametrize("few", [False, True])  # both cadences: many items a lane, and few
def test_batch(nqb, queue, few):
    boards, want, nodes = (v[-60000:] if few else v for v in queue)
    for block in (64, 128, 256):
        got, st = nqb.solve_batch(boards, form=nqb.FORM_BATCHED, block_size=block)
        assert np.array_equal(got, want) and st["nodes"] == int(nodes.sum())


def test_nodes_of_each_board(nqb, queue):
    boards, want, nodes = queue
    got_nodes, got = nqb.record_nodes(boards)
    assert np.array_equal(got, want) and np.array_equal(got_nodes, nodes)


def test_plan(nqb, queue):
    boards, want, nodes = queue
    plan = nqb.BatchPlan(boards)
    for _ in range(2):
        got, st = plan.run()
        assert np.array_equal(got, want) and st["nodes"] == int(nodes.sum())
    plan.close()
