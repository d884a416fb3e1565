"""Force evaluations of large systems keep their beads in sorted order (tild_run_forces)."""
import ctypes

import numpy as np
import pytest

import tild
from helpers import small_diblock

pytestmark = pytest.mark.gpu


def test_a_new_topology_is_sorted_at_its_first_evaluation():
    """It puts the beads back in the caller's order: the next evaluation sorts, which shows as launches."""
    s = small_diblock(3, 3, nx=(40, 40, 40), box=(20.0, 20.0, 20.0), n_chains=5200, N=20, seed=9)
    with tild.Batch([s]) as b:
        def launches():
            n = ctypes.c_int64()
            tild.lib().tild_kernel_launches(b._h, ctypes.byref(n))
            return n.value

        def evaluation():
            b.set_state(0, s.x)
            n0 = launches()
            f = b.forces(0)
            return launches() - n0, f

        first, f0 = evaluation()
        second, f1 = evaluation()
        assert first > second
        b.set_topology(0, s)
        third, f2 = evaluation()
        assert third == first
        assert np.array_equal(f0, f1) and np.array_equal(f0, f2)
