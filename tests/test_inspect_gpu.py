"""Large host arrays are looked over on the device: states the kernels do not accept are refused
wherever they stand, around the size from which the device does it; the widest and the emptiest
boards give the stack depth."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [8191, 8192, 8193, 20011])
@pytest.mark.parametrize("form", [0, 1])
def test_bad_states_are_refused(nqb, count, form):
    good = nqb.sample_boards(5, count, 6, 8, 3, 5)
    want, st = nqb.solve_batch(good, form=form)
    for at in (0, count // 2, count - 1):
        for field, value in (("n", 0), ("n", 32), ("n", 255), ("flags", 1), ("cols", 1 << 8)):
            bad = good.copy()
            bad[field][at] = value
            for call in (lambda: nqb.solve_batch(bad, form=form), lambda: nqb.solve_states(bad, form=form)):
                with pytest.raises(nqb.NQBError) as e:
                    call()
                assert e.value.status == nqb.E_INVALID
    got, st2 = nqb.solve_batch(good, form=form)
    assert np.array_equal(got, want) and st2["nodes"] == st["nodes"]


def test_one_deep_board_among_many(nqb, nqo):
    boards = nqb.sample_boards(6, 9000, 6, 8, 3, 5)
    boards[4321] = (0, 0, 0, 0, 12, 2, 0)  # an empty 12 x 12 board needs the deepest stack
    boards[17] = nqb.sample_boards(8, 1, 31, 31, 28, 28)[0]
    boards[8999] = (255, 0, 0, 8, 8, 1, 0)  # a complete board
    want, nodes = nqo.solve_states(boards)
    for form in (0, 1):
        got, st = nqb.solve_batch(boards, form=form)
        assert np.array_equal(got, want) and st["nodes"] == nodes
