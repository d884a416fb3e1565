"""Settings that differ from the defaults of order >= 2 in 3D (the brick layout of the field), the library
transforms beside the own passes, and the stencil's divisions at orders 2 to 4."""
import numpy as np
import pytest

import oracle
import tild
from helpers import FORCE_RTOL, erf_system, rel_l2, small_diblock
from tild import Style

pytestmark = pytest.mark.gpu


def _run(s, tune, steps=70):
    with tild.Context(s) as c:
        t = c.get_tune()
        for k, v in tune.items():
            setattr(t, k, v)
        c.set_tune(t)
        c.step(steps)
        return c.get_state()


LINEAR = {"field_layout": tild.FIELD_LINEAR}


@pytest.mark.parametrize("order", [2, 3, 4])
@pytest.mark.parametrize("tune", [
    LINEAR,
    {**LINEAR, "gather_mode": tild.GATHER_BOX},
    {**LINEAR, "gather_mode": tild.GATHER_BOX, "gather_cap": 1024},   # most chunks fall back to global reads
    {**LINEAR, "spread_ahead": 1},
    {**LINEAR, "spread_cap": 12288},
    {"spread_ahead": 1, "spread_cap": 12288},
])
def test_linear_layout_and_box_gather_against_the_default(order, tune):
    s = small_diblock(3, order, nx=(20, 18, 16), box=(10.0, 9.0, 8.0), n_chains=150, N=10, seed=31)
    with tild.Context(s) as c:
        assert c.get_tune().field_layout == tild.FIELD_BRICK
    for a, b in zip(_run(s, {}), _run(s, tune)):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("order", [2, 3, 4])
def test_box_gather_forces_match_the_oracle(order):
    s = small_diblock(3, order, nx=(20, 18, 16), box=(10.0, 9.0, 8.0), n_chains=150, N=10, seed=31)
    with tild.Context(s) as c:
        t = c.get_tune()
        t.field_layout, t.gather_mode = tild.FIELD_LINEAR, tild.GATHER_BOX
        c.set_tune(t)
        fg = c.forces()
    assert rel_l2(fg, oracle.Oracle(s).forces(s.x, 0)) < FORCE_RTOL


CASES = {
    "diblock3d_p1": lambda: small_diblock(3, 1),
    "diblock3d_p3": lambda: small_diblock(3, 3, nx=(18, 16, 20), box=(9.0, 8.0, 10.0)),
    "diblock3d_p2_odd": lambda: small_diblock(3, 2, nx=(15, 17, 19), box=(7.5, 8.5, 9.5)),
    "diblock2d_p3": lambda: small_diblock(2, 3, nx=(21, 24)),
    "gaussian_erf_p3": lambda: erf_system(tild.STYLE_GAUSSIAN_ERF),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_library_transforms_paired_and_per_channel_and_own_passes(name):
    """Plain batches keep the library transforms, paired (complex) or, beside a fieldphase style, per channel;
    a single system takes the own passes: the same densities, forces and energies to FP32 rounding."""
    s, other = CASES[name](), CASES[name]()
    field = CASES[name]()
    field.styles = field.styles + [Style(tild.STYLE_FIELDPHASE, 0, 1, 0.0, phase=0, dir=0, n_periods=1)]
    got = []
    for systems in ([s, other], [field, other]):
        with tild.Batch(systems) as B:
            got.append((B.forces(0), B.density(0), B.observables(0)["upe"]))
    with tild.Context(s) as c:
        got.append((c.forces(), c.density(), c.observables()["upe"]))
    for f, rho, e in got[1:]:
        assert rel_l2(f, got[0][0]) < 1e-6
        assert np.array_equal(rho, got[0][1])
        assert e == pytest.approx(got[0][2], rel=1e-6)


@pytest.mark.parametrize("order", [2, 3, 4])
def test_weight_divisions_are_correctly_rounded(order):
    """Offsets of k / 32 node spacings make every polynomial of the weights exact in FP32, fused or not, so that the
    divisions by 48 (order 3), 96, 192 and 384 (order 4) are all that rounds: the FP32 quotients, bit for bit."""
    nx, dx = (16, 18, 20), np.float32(0.5)
    box = tuple(0.5 * n for n in nx)
    k = np.arange(-16, 17) if order % 2 == 0 else np.arange(-16, 16)   # the nearest node, or the cell
    off = np.stack(np.meshgrid(k, k, k, indexing="ij"), -1).reshape(-1, 3) / 32.0
    if order % 2 == 0:
        off = off[(off < 0.5).all(1)]
    rng = np.random.default_rng(8)
    cell = np.stack([rng.integers(1, n - 1, len(off)) for n in nx], 1)
    x = ((cell + off + (0.0 if order % 2 == 0 else 0.5)) * 0.5).astype(np.float32)
    n = len(x)
    z = np.zeros((n, 3), np.int32)
    s = tild.System(dim=3, nx=nx, box=box, types=np.zeros(n, np.int32), x=x, n_bonds=np.zeros(n, np.int32), bonded_to=z,
                    bond_type=z, ntypes=1, styles=[Style(tild.STYLE_GAUSSIAN, 0, 0, 1.0, 0.7)], pmeorder=order)
    with tild.Context(s) as c:
        inds, w = c.stencil()
    f, t = np.float32, off
    if order == 2:
        W = [f(0.125 - 0.5 * t + 0.5 * t**2), f(0.75 - t**2), f(0.125 + 0.5 * t + 0.5 * t**2)]
    elif order == 3:
        W = [f(1 - 6 * t + 12 * t**2 - 8 * t**3) / f(48), f(23 - 30 * t - 12 * t**2 + 24 * t**3) / f(48),
             f(23 + 30 * t - 12 * t**2 - 24 * t**3) / f(48), f(1 + 6 * t + 12 * t**2 + 8 * t**3) / f(48)]
    else:   # the stencil's cube is the square's square
        W = [f(1 - 8 * t + 24 * t**2 - 32 * t**4 + 16 * t**4) / f(384),
             f(19 - 44 * t + 24 * t**2 + 16 * t**4 - 16 * t**4) / f(96), f(115 - 120 * t**2 + 48 * t**4) / f(192),
             f(19 + 44 * t + 24 * t**2 - 16 * t**4 - 16 * t**4) / f(96),
             f(1 + 8 * t + 24 * t**2 + 32 * t**4 + 16 * t**4) / f(384)]
    gvol = dx * dx * dx
    j = 0
    for a in np.ndindex(*([order + 1] * 3)):
        i = [(cell[:, d] - order // 2 + a[d]) % nx[d] for d in range(3)]
        assert np.array_equal(inds[:, j], i[0] + (i[1] + i[2] * nx[1]) * nx[0])
        assert np.array_equal(w[:, j], W[a[0]][:, 0] * W[a[1]][:, 1] * W[a[2]][:, 2] / gvol)
        j += 1
