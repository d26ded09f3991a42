"""What the times of nqb_stats stand for: gen_ms ends with the pool, before its items are split
further, and h2d_ms with the copy, before the states are looked over on the device."""
import pytest

pytestmark = pytest.mark.gpu


def least(call, field, runs=40):
    call()
    return min(call()[1][field] for _ in range(runs))


@pytest.mark.parametrize("form", [0, 1])
def test_pool_generation_ends_with_the_pool(nqb, form):
    # depth 1: one small kernel makes the pool and four levels split it; depth 5: five kernels
    one = least(lambda: nqb.count_ex(16, 1, form=form), "gen_ms")
    five = least(lambda: nqb.count_ex(16, 5, form=form), "gen_ms")
    assert 0 < one < 0.4 * five


@pytest.mark.parametrize("form", [0, 1])
def test_copy_time_ends_with_the_copy(nqb, form):
    # from 8192 states on a kernel and a read-back (25 us) follow the copy
    states = nqb.sample_boards(4, 8192, 8, 9, 3, 5)
    host = least(lambda: nqb.solve_states(states[:8191], form=form), "h2d_ms")
    device = least(lambda: nqb.solve_states(states, form=form), "h2d_ms")
    assert 0 < device < host + 0.010
