"""The inference kernel at the edges of its row tiles and of its grid, against the float64
restatement with the same fp16 rounding points."""
import numpy as np
import pytest

import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 127, 128, 129, 2 * 148 * 128 + 1])
def test_predictions_at_tile_edges(nqb, rows):
    m = nqb.Model(seed=rows)
    p = m.get_params()
    rng = np.random.default_rng(rows)
    p[mlp_ref.KB1:mlp_ref.KW2] = rng.normal(0, 0.1, mlp_ref.H)
    p[mlp_ref.KB2:mlp_ref.KW3] = rng.normal(0, 0.1, mlp_ref.H)
    p[mlp_ref.KB3] = 1.5
    m.set_params(p)
    boards = nqb.sample_boards(rows, rows, 8, 31, 1, 7)
    got = m.predict(boards)
    assert np.array_equal(got, m.predict(boards))
    m.close()
    want, _ = mlp_ref.forward(p.astype(np.float64), mlp_ref.features(boards))
    # one hidden unit on the other side of an fp16 rounding moves a row by 2^-11 |h w3|, below 1e-3
    assert np.max(np.abs(got - want)) < 1e-3
    assert np.linalg.norm(got - want) < 1e-4 * np.linalg.norm(want)
