"""A call that really runs out of device memory fails by itself: the calls after it on the same
thread do not report its error again."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", [0, 1])
def test_calls_after_a_failed_allocation(nqb, form):
    one = nqb.generate_pool(8, 2)[:1].copy()
    total = ctypes.c_uint64(7)
    # 16 TB of states: the device buffer is refused before any state is read
    st = nqb.lib().nqb_solve_states(one.ctypes.data_as(ctypes.c_void_p), 1 << 40, None, ctypes.byref(total), None)
    assert st == nqb.E_NOMEM and total.value == 0
    assert nqb.count(8, 2, form=form) == 92
    boards = nqb.sample_boards(1, 20, 8, 9, 2, 3)
    want, _ = nqb.solve_batch(boards, form=form)
    st = nqb.lib().nqb_solve_states(one.ctypes.data_as(ctypes.c_void_p), 1 << 40, None, ctypes.byref(total), None)
    assert st == nqb.E_NOMEM
    assert np.array_equal(nqb.solve_batch(boards, form=form)[0], want)
