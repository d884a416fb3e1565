"""The gather that starts while the grid passes end (order <= 1, small systems)."""
import numpy as np
import pytest

import tild
from helpers import charged_system, small_diblock

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ahead", [0, 1])
@pytest.mark.parametrize("system", [lambda: small_diblock(3, 1), lambda: small_diblock(2, 0), lambda: charged_system()],
                         ids=["3d", "2d", "charged"])
def test_small_systems_beside_padding(system, ahead):
    """In a slot with blocks of padding alone, launched, captured and replayed, with sorts and stepping calls
    between: the steps of the system alone, one per call."""
    s = system()
    with tild.Batch([s], capacity=[s.ns + 2000]) as b, tild.Context(s) as c:
        for run in (b, c):
            t = run.get_tune()
            t.spread_ahead = ahead
            run.set_tune(t)
        for n in (1, 5, 64, 64, 3):
            b.step(n)
            for _ in range(n):
                c.step(1)
        assert all(np.array_equal(u, v) for u, v in zip(b.get_state(0), c.get_state()))
        assert np.array_equal(b.density(0), c.density())
