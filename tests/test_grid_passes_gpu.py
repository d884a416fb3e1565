"""The grid passes (tild_fft.cu) at the edges of their radices, tiles and channel counts: forces
against the FP64 oracle at the FP32 tolerance of the parity tests."""
import numpy as np
import pytest

import oracle
import tild
import tild_systems as ts
from helpers import FORCE_RTOL, rel_l2
from tild import Style

pytestmark = pytest.mark.gpu


def _system(nx, ntypes=2, charged=False, seed=3, ramp=None):
    dim = len(nx)
    rng = np.random.default_rng(seed)
    box = tuple(0.5 * n for n in nx)
    chains, N = 60, 8
    ns = chains * N
    x = ts.random_walk_chains(rng, chains, N, box, dim)
    types = rng.integers(0, ntypes, ns).astype(np.int32)
    styles = [Style(tild.STYLE_GAUSSIAN, a, b, 1.0 + 0.3 * a + 0.7 * b, 0.7) for a in range(ntypes) for b in range(a, ntypes)]
    if ramp == "alone":      # the only style of its pair of types
        styles[0].ramp, styles[0].final_prefactor = True, 3.0
    elif ramp == "beside":   # beside a constant style of the same types
        styles.append(Style(tild.STYLE_GAUSSIAN_ERF, 0, 0, 2.0, 0.5, 0.6, ramp=True, final_prefactor=5.0))
    nb, bt, by = ts.topology_from_bonds(ns, ts.linear_bonds(chains, N))
    q = rng.choice([-1.0, 0.0, 1.0], ns).astype(np.float32) if charged else None
    return tild.System(dim=dim, nx=tuple(nx) + (1,) * (3 - dim), box=box + (1.0,) * (3 - dim), types=types, x=x, n_bonds=nb,
                       bonded_to=bt, bond_type=by, ntypes=ntypes, styles=styles, pmeorder=1, charges=q, bjerrum=1.0,
                       smearing=0.5, max_steps=100)


SHAPES = [
    (16, 16, 16), (13, 14, 15), (9, 11, 12), (5, 6, 7),       # one radix per stage, tiles larger than the grid
    (17, 8, 8), (8, 17, 8), (8, 8, 17),                       # a prime edge per axis
    (34, 38, 46), (29, 31, 37),                               # direct second stages after a radix, and alone
    (127, 6, 5), (4, 256, 3), (6, 5, 128), (256, 3, 4),       # the longest lines
    (33, 52, 75), (20, 18, 22),
    (25, 12, 10), (12, 125, 10),                              # 125 = 5 x 25 stays with the library
    (40, 40), (21, 24), (256, 9), (9, 256), (101, 12), (12, 101),
]


@pytest.mark.parametrize("nx", SHAPES, ids=lambda v: "x".join(map(str, v)))
def test_forces_over_grid_shapes(nx):
    s = _system(nx)
    with tild.Context(s) as c:
        fg = c.forces()
        rho = c.density()
    assert rel_l2(fg, oracle.Oracle(s).forces(s.x, 0)) < FORCE_RTOL
    # every bead is spread once: the integral of a type's density is its number of beads
    vol = np.prod([0.5] * len(nx))
    counts = np.bincount(s.types, minlength=2)
    assert np.allclose(rho.astype(np.float64).sum(1) * vol, counts, rtol=1e-5)


@pytest.mark.parametrize("ntypes,charged", [(1, False), (1, True), (2, True), (3, False), (3, True), (4, True), (5, False), (7, True)])
def test_forces_over_channel_counts(ntypes, charged):
    s = _system((18, 15, 16), ntypes, charged)
    with tild.Context(s) as c:
        fg = c.forces()
        c.forces()
        again = c.forces()
    assert rel_l2(fg, oracle.Oracle(s).forces(s.x, 0)) < FORCE_RTOL
    assert np.array_equal(fg, again)


@pytest.mark.parametrize("ramp", ["alone", "beside"])
@pytest.mark.parametrize("ntypes", [1, 2])
def test_ramped_multipliers(ramp, ntypes):
    s = _system((16, 12, 18), ntypes, ramp=ramp)
    with tild.Context(s) as c:
        c.set_step(40)
        fg = c.forces()
    assert rel_l2(fg, oracle.Oracle(s).forces(s.x, 40)) < FORCE_RTOL


def test_densities_belong_to_the_last_step_of_a_call():
    """Only the last step of a call stores the densities: they are those of one step per call."""
    s = _system((20, 18, 16))
    with tild.Context(s) as a, tild.Context(s) as b:
        a.step(45)
        for _ in range(45):
            b.step(1)
        assert np.array_equal(a.density(), b.density())
        oa, ob = a.observables(), b.observables()
        assert oa["upe"] == ob["upe"] and np.array_equal(oa["ptens"], ob["ptens"])


@pytest.mark.parametrize("order", [0, 1])
def test_stencil_divisions_are_correctly_rounded(order):
    """Indices and weights with node spacings that are no binary fractions: the FP32 division results."""
    nx, box = (23, 37, 41), (7.3, 11.1, 13.7)
    s = _system(nx)
    rng = np.random.default_rng(8)
    L = np.array(box, np.float32)
    dx = L / np.array(nx, np.float32)
    x = (rng.random((20000, 3)) * L).astype(np.float32)
    x[:3000] = (rng.integers(0, 23, (3000, 3)) * dx).astype(np.float32)   # on or next to node planes
    x = np.minimum(x, L)
    n = len(x)
    z = np.zeros((n, 3), np.int32)
    s = tild.System(dim=3, nx=nx, box=box, types=np.zeros(n, np.int32), x=x, n_bonds=np.zeros(n, np.int32), bonded_to=z,
                    bond_type=z, ntypes=1, styles=[Style(tild.STYLE_GAUSSIAN, 0, 0, 1.0, 0.7)], pmeorder=order)
    with tild.Context(s) as c:
        inds, w = c.stencil()
    gi = ((x + np.float32(0.5) * dx) / dx if order == 0 else x / dx).astype(np.int64)
    if order == 0:
        W = [[np.ones(n, np.float32)] for _ in range(3)]
    else:  # x - (gi + 0.5) dx is one fused operation on the device: exact in double, then rounded
        gdx = (x.astype(np.float64) - (gi + 0.5) * dx.astype(np.float64)).astype(np.float32)
        sx = gdx / dx
        W = [[np.float32(0.5) - sx[:, d], np.float32(0.5) + sx[:, d]] for d in range(3)]
    gvol = np.float32(dx[0] * dx[1]) * dx[2]
    k = 0
    for a in np.ndindex(*([order + 1] * 3)):
        i = [(gi[:, d] + a[d]) % nx[d] for d in range(3)]
        assert np.array_equal(inds[:, k], i[0] + (i[1] + i[2] * nx[1]) * nx[0])
        assert np.array_equal(w[:, k], W[0][a[0]] * W[1][a[1]] * W[2][a[2]] / gvol)
        k += 1


def test_slot_batch_mixes_passes_and_library_shapes():
    """Shapes that take the passes, shapes that do not, and an inactive system, in one slot batch."""
    systems = [_system(nx, seed=k) for k, nx in enumerate([(16, 18, 20), (12, 125, 10), (60, 9, 50), (29, 12, 10)])]
    with tild.Batch(systems, capacity=[s.ns + 300 for s in systems]) as B:
        fb = [B.forces(i) for i in range(len(systems))]
        B.set_active(2, False)
        x2 = B.get_state(2)[0]
        B.step(19)
        assert np.array_equal(x2, B.get_state(2)[0])
        rho = [B.density(i) for i in range(len(systems))]
        upe = [B.observables(i)["upe"] for i in range(len(systems))]
    for i, s in enumerate(systems):
        assert rel_l2(fb[i], oracle.Oracle(s).forces(s.x, 0)) < FORCE_RTOL, i
        counts = np.bincount(s.types, minlength=2)
        assert np.allclose(rho[i].astype(np.float64).sum(1) * 0.125, counts, rtol=1e-5)
        assert np.isfinite(upe[i])
