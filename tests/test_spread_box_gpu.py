"""The default shared box of the spread, and its sums when chunks overflow it."""
import numpy as np
import pytest

import tild
import tild_systems as ts
from tild import Style

pytestmark = pytest.mark.gpu


def _system(order, ntypes, per_channel, edge=32):
    rng = np.random.default_rng(4)
    box = (edge / 2.0,) * 3
    chains = int(per_channel * ntypes * edge ** 3) // 8
    ns = 8 * chains
    nb, bt, by = ts.topology_from_bonds(ns, ts.linear_bonds(chains, 8))
    return tild.System(dim=3, nx=(edge,) * 3, box=box, types=rng.integers(0, ntypes, ns).astype(np.int32),
                       x=ts.random_walk_chains(rng, chains, 8, box, 3), n_bonds=nb, bonded_to=bt, bond_type=by,
                       ntypes=ntypes, styles=[Style(tild.STYLE_GAUSSIAN, 0, 0, 1.0, 0.7)], pmeorder=order, max_steps=100)


@pytest.mark.parametrize("order,ntypes,per_channel,cap", [
    (2, 2, 1.0, 6144), (2, 8, 0.56, 6144), (2, 12, 0.56, 12288),
    (3, 2, 0.65, 6144), (3, 4, 1.0, 6144), (3, 4, 0.6, 12288), (3, 8, 0.56, 12288), (3, 1, 0.56, 12288),
    (3, 2, 0.5, 12288), (4, 2, 1.0, 12288)])
def test_default_box_holds_the_chunks(order, ntypes, per_channel, cap):
    s = _system(order, ntypes, per_channel)
    rho = []
    for mode in (tild.SPREAD_TILED, tild.SPREAD_DIRECT):
        with tild.Context(s) as c:
            t = c.get_tune()
            assert t.spread_cap == cap
            t.spread_mode = mode
            c.set_tune(t)
            c.step(2)
            rho.append(c.density())
    assert np.array_equal(rho[0], rho[1])
