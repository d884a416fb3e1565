"""Stop steps at, below and above the step counter of a system that is active."""
import numpy as np
import pytest

import tild
from helpers import charged_system, small_diblock

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots", [False, True])
@pytest.mark.parametrize("n", [1, 5, 64])
@pytest.mark.parametrize("offset", [-30, -1, 0, 1, 2, 40, 200])
def test_stop_relative_to_the_step_counter(slots, n, offset):
    """A counter never runs backwards: a system takes the steps up to its stop, and one that is active at or
    past it takes one step and leaves the active set; either way it is where that many steps bring it."""
    systems = [small_diblock(3, 1, seed=3), charged_system()]
    cap = [s.ns for s in systems] if slots else None
    with tild.Batch(systems, capacity=cap) as B, tild.Batch(systems, capacity=cap) as R:
        for b in (B, R):
            b.step(40)
        B.set_stop(1, 40 + offset)
        B.step(n)
        moved = min(n, max(offset, 1))
        for _ in range(moved):
            R.step(1)
        assert B.step_count(1) == 40 + moved == R.step_count(1)
        assert B.active(1) == (moved < offset)
        assert np.array_equal(B.get_state(1)[0], R.get_state(1)[0])
        B.step(n)
        if moved >= offset:
            assert B.step_count(1) == 40 + moved
            assert np.array_equal(B.get_state(1)[0], R.get_state(1)[0])
        assert B.step_count(0) == 40 + 2 * n


def test_step_counter_set_past_the_stop():
    s = small_diblock(3, 1)
    with tild.Batch([s], capacity=[s.ns]) as B:
        B.set_stop(0, 20)
        B.set_step(0, 50)
        B.step(8)
        assert B.step_count(0) == 51 and not B.active(0)
