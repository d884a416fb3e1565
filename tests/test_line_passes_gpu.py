"""The passes over grid lines of planes too large for one block (more than 2,304 points), and the plane
kernels' wider launches: forces against the FP64 oracle for every variant of the y and inverse passes."""
import numpy as np
import pytest

import oracle
import tild
import tild_systems as ts
from helpers import FORCE_RTOL, rel_l2
from tild import Style

pytestmark = pytest.mark.gpu


def _system(nx, ntypes=2, order=1, seed=3, per_node=0.02):
    rng = np.random.default_rng(seed)
    box = tuple(0.5 * n for n in nx)
    chains = max(60, int(per_node * np.prod(nx)) // 8)
    ns = 8 * chains
    nb, bt, by = ts.topology_from_bonds(ns, ts.linear_bonds(chains, 8))
    styles = [Style(tild.STYLE_GAUSSIAN, a, b, 1.0 + 0.3 * a + 0.7 * b, 0.7) for a in range(ntypes) for b in range(a, ntypes)]
    return tild.System(dim=3, nx=tuple(nx), box=box, types=rng.integers(0, ntypes, ns).astype(np.int32),
                       x=ts.random_walk_chains(rng, chains, 8, box, 3), n_bonds=nb, bonded_to=bt, bond_type=by,
                       ntypes=ntypes, styles=styles, pmeorder=order, max_steps=100)


# 16 columns per block from 303,104 points over all pairs (16 x 32 x 592), 8 below; a prime factor above 16 of
# an axis takes the direct transform
LINE_SHAPES = [
    (50, 49, 12), (64, 61, 8), (61, 64, 8), (64, 40, 29), (128, 20, 10),   # 8 columns: regular, direct y, x, z
    (68, 64, 72), (64, 68, 72), (68, 68, 68), (68, 61, 76), (61, 60, 86),  # 16 columns: 4 x 17, direct y, direct x
    (256, 16, 17), (16, 256, 19), (12, 254, 24),
]


@pytest.mark.parametrize("ntypes", [1, 2, 3])
@pytest.mark.parametrize("nx", LINE_SHAPES, ids=lambda v: "x".join(map(str, v)))
def test_forces_of_line_passes(nx, ntypes):
    s = _system(nx, ntypes)
    with tild.Context(s) as c:
        fg = c.forces()
        rho = c.density()
        c.step(3)
        moved = c.get_state()[0]
    assert rel_l2(fg, oracle.Oracle(s).forces(s.x, 0)) < FORCE_RTOL
    assert np.allclose(rho.astype(np.float64).sum(1) * 0.125, np.bincount(s.types, minlength=ntypes), rtol=1e-5)
    assert np.isfinite(moved).all()


@pytest.mark.parametrize("ntypes", [2, 3])
@pytest.mark.parametrize("nx", [(29, 31, 104), (40, 40, 100), (17, 48, 128)], ids=lambda v: "x".join(map(str, v)))
def test_forces_of_many_planes(nx, ntypes):
    """More than 296 fields of planes: 256 threads per plane in the inverse, direct and regular."""
    s = _system(nx, ntypes)
    with tild.Context(s) as c:
        fg = c.forces()
    assert rel_l2(fg, oracle.Oracle(s).forces(s.x, 0)) < FORCE_RTOL


@pytest.mark.parametrize("order", [2, 3, 4])
@pytest.mark.parametrize("layout", [tild.FIELD_LINEAR, tild.FIELD_BRICK])
def test_nodes_of_both_layouts(layout, order):
    """Line passes and plane passes write the linear and the brick layout of the field."""
    for nx in ((70, 50, 9), (21, 18, 22)):
        s = _system(nx, 2, order)
        with tild.Context(s) as c:
            t = c.get_tune()
            t.field_layout = layout
            c.set_tune(t)
            fg = c.forces()
        assert rel_l2(fg, oracle.Oracle(s).forces(s.x, 0)) < FORCE_RTOL, nx


def test_slots_of_line_and_plane_shapes():
    """Slots whose shapes all go by lines because one of them is too large for planes."""
    systems = [_system(nx, seed=k) for k, nx in enumerate([(60, 50, 8), (16, 18, 20), (29, 12, 10)])]
    with tild.Batch(systems, capacity=[s.ns + 300 for s in systems]) as B:
        fb = [B.forces(i) for i in range(3)]
    for i, s in enumerate(systems):
        assert rel_l2(fb[i], oracle.Oracle(s).forces(s.x, 0)) < FORCE_RTOL, i
