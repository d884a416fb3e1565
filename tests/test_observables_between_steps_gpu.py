"""Observables and S(k) read between stepping calls belong to the last force evaluation, whether the
steps ran as launches, as a freshly captured graph or as a replayed one."""
import numpy as np
import pytest

import tild
from helpers import charged_system, small_diblock

pytestmark = pytest.mark.gpu

CASES = {
    "paired_p1": lambda: small_diblock(3, 1),
    "paired_p3": lambda: small_diblock(3, 3, nx=(18, 16, 20), box=(9.0, 8.0, 10.0)),
    "odd_channels_p1": lambda: charged_system(),
    "odd_channels_p3": lambda: charged_system(pmeorder=3),
    "film_p1": lambda: small_diblock(2, 1),
}


def numpy_sk(rho, s):
    """rho_k^2 of one density field over the full grid, rho_k with the 1 / M of the forward transform kept
    outside: the accumulator holds rho_k rho_k / M."""
    n = s.nx[:s.dim][::-1]
    rk = np.fft.fftn(rho.astype(np.float64).reshape(n))
    return (rk * rk).ravel() / rho.size


@pytest.mark.parametrize("name", sorted(CASES))
def test_records_after_replayed_graphs(name):
    """Four stepping calls of 64, the later ones replays alone, each with a record and an S(k) sample: the
    records of the same run made of single launches, and the samples of the densities."""
    s = CASES[name]()
    with tild.Context(s) as a, tild.Context(s) as b:
        acc = 0.0
        for _ in range(4):
            a.step(64)
            for _ in range(64):
                b.step(1)
            oa, ob = a.observables(), b.observables()
            a.sk_accumulate(0, 0)
            b.sk_accumulate(0, 0)
            acc = acc + numpy_sk(a.density()[0], s)
            assert np.array_equal(a.get_state()[0], b.get_state()[0])
            assert oa["upe"] == ob["upe"]
            assert np.array_equal(oa["ptens"], ob["ptens"])
            assert np.array_equal(oa["style_energy"], ob["style_energy"])
        (ka, na), (kb, nb) = a.sk_get(0), b.sk_get(0)
    assert na == nb == 4
    assert np.array_equal(ka, kb)
    # FP32 spectra against FP64 ones: an error of 2^-24 log2(M) of the field's norm in each mode is about
    # 1e-6 of a fluctuation mode, twice that in its square
    assert np.abs(ka - acc / 4)[1:].max() < 1e-5 * np.abs(acc / 4)[1:].max()


def test_slot_batch_records_after_replayed_graphs():
    """The same for slots: two shapes, one of them with an odd number of channels."""
    systems = [small_diblock(3, 1, seed=3), small_diblock(3, 1, seed=4), charged_system()]
    cap = [s.ns + 100 for s in systems]
    with tild.Batch(systems, capacity=cap) as A, tild.Batch(systems, capacity=cap) as B:
        for _ in range(4):
            A.step(64)
            for _ in range(64):
                B.step(1)
            for i in range(3):
                oa, ob = A.observables(i), B.observables(i)
                A.sk_accumulate(i, 0, 0)
                B.sk_accumulate(i, 0, 0)
                assert oa["upe"] == ob["upe"] and np.array_equal(oa["ptens"], ob["ptens"]), i
        for i in range(3):
            assert np.array_equal(A.sk_get(i, 0)[0], B.sk_get(i, 0)[0]), i


@pytest.mark.parametrize("read_between", [False, True])
@pytest.mark.parametrize("steps", [5, 64])
def test_a_shape_at_rest_keeps_its_record(steps, read_between):
    """A system whose whole shape takes no part in the steps keeps the energies, virials and S(k) of its
    last force evaluation, read before or not."""
    systems = [small_diblock(3, 1, seed=3), charged_system()]
    with tild.Batch(systems, capacity=[s.ns + 100 for s in systems]) as B:
        B.step(10)
        want = B.observables(1)
        B.sk_accumulate(1, 0, 0)
        sk = B.sk_get(1, 0)[0]
    with tild.Batch(systems, capacity=[s.ns + 100 for s in systems]) as B:
        B.step(10)
        if read_between:
            B.observables(1)
        B.set_active(1, False)
        for _ in range(3):
            B.step(steps)
            got = B.observables(1)
            assert got["upe"] - got["ubond"] == pytest.approx(want["upe"] - want["ubond"], rel=1e-12)
            assert np.array_equal(got["style_virial"], want["style_virial"])
        B.sk_accumulate(1, 0, 0)
        assert np.array_equal(B.sk_get(1, 0)[0], sk)
        B.set_active(1, True)       # and moves on from there
        B.step(steps)
        moved = B.observables(1)
    assert moved["upe"] != want["upe"]
