"""Positions outside [-L, 2L) are refused however far out they are: also where x / dx overflows FP32."""
import pytest

import tild
from helpers import small_diblock

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("far", [1e3, 3e9, 3e38, -3e38])
def test_far_positions_are_refused(order, far):
    s = small_diblock(3, order)  # node spacing 0.5
    for axis in range(3):
        x = s.x.copy()
        x[5, axis] = far
        with tild.Context(s) as c:
            c.set_state(x)
            with pytest.raises(tild.TildError) as e:
                c.forces()
        assert e.value.status == tild.ERR_BAD_INPUT
