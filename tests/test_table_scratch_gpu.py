"""Table builds above 2^18 points transform half of a style's virial kernels at a time."""
import numpy as np
import pytest

import oracle
import tild
from helpers import ENERGY_RTOL, small_diblock
from tild_serve import device_free_bytes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [(64, 64, 64), (65, 63, 65)], ids=["whole", "halves"])
def test_virials_on_both_sides_of_the_line(nx):
    s = small_diblock(3, 1, nx=nx, box=tuple(0.5 * n for n in nx), n_chains=1200)
    o = oracle.Oracle(s)
    o.forces(s.x, 0)
    oo = o.observables(s.x)
    with tild.Context(s) as c:
        og = c.observables()
    assert og["upe"] == pytest.approx(oo["upe"], rel=ENERGY_RTOL)
    scale = np.abs(oo["style_virial"]).max()
    np.testing.assert_allclose(og["style_virial"], oo["style_virial"], rtol=ENERGY_RTOL, atol=1e-5 * scale)


def test_scratch_stays_below_the_fields():
    """A 96^3 system of two types: 192 bytes a point of densities, spectra, fields and tables, and at most as much
    again of table scratch and transform work areas (371 MB with whole styles at a time)."""
    s = small_diblock(3, 1, nx=(96, 96, 96), box=(48.0, 48.0, 48.0), n_chains=200)
    with tild.Context(s):       # the transforms' modules are loaded
        pass
    free = device_free_bytes(0)
    with tild.Context(s) as c:
        c.sync()
        assert free - device_free_bytes(0) < 2 * 192 * 96 ** 3
