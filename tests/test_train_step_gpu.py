"""The fused training step against the float64 restatement at the edges of its tiles: less than a
row tile, one row more or less, and more tiles than the GPU has SMs (a block's gradients then
add up over several tiles)."""
import numpy as np
import pytest

import mlp_ref

pytestmark = pytest.mark.gpu
BLOCKS = {"W1": (mlp_ref.KW1, mlp_ref.KB1), "b1": (mlp_ref.KB1, mlp_ref.KW2), "W2": (mlp_ref.KW2, mlp_ref.KB2),
          "b2": (mlp_ref.KB2, mlp_ref.KW3), "w3": (mlp_ref.KW3, mlp_ref.KB3), "b3": (mlp_ref.KB3, mlp_ref.NPARAMS)}


def make(nqb, rows, seed):
    rng = np.random.default_rng(seed)
    boards = nqb.sample_boards(seed, rows, 12, 20, 2, 8)
    m = nqb.Model(seed=seed)
    p = m.get_params()
    p[mlp_ref.KB1:mlp_ref.KW2] = rng.normal(0, 0.1, mlp_ref.H)
    p[mlp_ref.KB2:mlp_ref.KW3] = rng.normal(0, 0.1, mlp_ref.H)
    p[mlp_ref.KB3] = 2.0
    m.set_params(p)
    return m, p, boards, rng.normal(10, 4, rows).astype(np.float32)


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 1000, 20000])
def test_gradients_at_tile_edges(nqb, rows):
    m, p, boards, t = make(nqb, rows, rows)
    loss, g = m.loss_grad(boards, t)
    m.close()
    want_loss, want = mlp_ref.loss_grad(p.astype(np.float64), mlp_ref.features(boards), t.astype(np.float64))
    # the restatement rounds to fp16 at the same points; what is left is fp32 accumulation
    # (2^-24 x sqrt(K) per sum) and operands that land on the other side of an fp16 rounding
    # (2^-11 of themselves, a few in a thousand of them)
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    for name, (a, b) in BLOCKS.items():
        assert np.linalg.norm(g[a:b] - want[a:b]) <= 1e-4 * np.linalg.norm(want[a:b]) + 1e-12, (name, rows)


def test_training_is_reproducible_and_masks_the_last_tile(nqb):
    m, p, boards, t = make(nqb, 1500, 5)
    runs = []
    for _ in range(2):
        m.set_params(p)
        losses = m.train(boards, t, epochs=3, batch=400, lr=1e-3)  # 400, 400, 400, 300: ragged tiles
        runs.append((losses, m.get_params()))
    m.close()
    assert np.array_equal(runs[0][0], runs[1][0]) and np.array_equal(runs[0][1], runs[1][1])
    assert runs[0][0][2] < runs[0][0][0]
