"""Temperatures the generated right-hand side covers (mechgen.temperature_range): its
exponential has no overflow handling, so every argument and every partial product
of species exponentials has to stay within e^+-690."""
from types import SimpleNamespace

import numpy as np
import pytest

from pelelmex_b200 import mechanism as M, mechgen


def _flat(g, products, troe=None, flags=1):
    """One reaction of the last species to `products` [(species, nu)]; g/RT of the
    species are constants."""
    n = len(g)
    nasa = np.zeros((n, 15))
    nasa[:, 0] = 1000.0
    nasa[:, 7] = nasa[:, 14] = -np.asarray(g, float)  # g/RT = -a6
    sp, nu = -np.ones((1, 8), np.int32), np.zeros((1, 8), np.int32)
    sp[0, 0], nu[0, 0] = n - 1, 1
    for i, (k, v) in enumerate(products):
        sp[0, 4 + i], nu[0, 4 + i] = k, v
    z = np.zeros((1, 3))
    a = dict(nasa=nasa, sp=sp, nu=nu, arr=z, arr_lo=z, arr_rev=z, rtype=np.array([3 if troe else 0]),
             rflags=np.array([flags]), troe=np.array([troe or (0.0, 1.0, 1.0, 0.0)]))
    return SimpleNamespace(arrays=a, n_species=n, n_reactions=1)


def test_partial_products_are_bounded():
    # e^400 e^400 e^-400: the whole product is small enough, its first two factors are not
    assert mechgen.temperature_range(_flat([400.0, -400.0, 0.0], [(0, 2), (1, 1)])) == (1000.0, 1000.0)
    assert mechgen.temperature_range(_flat([300.0, -400.0, 0.0], [(0, 2), (1, 1)])) == (50.0, 20000.0)
    # the last factors: 680 and two powers of ln(Ru T / 1 atm), 11.3 at 1000 K
    assert mechgen.temperature_range(_flat([340.0, 0.0], [(0, 2), (1, 1)])) == (1000.0, 1000.0)


@pytest.mark.parametrize("troe,flags,want", [
    ((0.5, -2.0, 1e3, 0.0), 1, (50.0, 1350.0)),   # -T / T3 <= 690
    ((0.5, 1e3, -2.0, 0.0), 1, (50.0, 1350.0)),   # -T / T1 <= 690
    ((0.5, 1e3, 1e3, -4e5), 5, (580.0, 20000.0)),   # -T2 / T <= 690
    ((0.5, 1e3, 1e3, -4e5), 1, (50.0, 20000.0)),   # no T2 in this form
    ((0.5, 1e-3, 1e3, 1e9), 5, (50.0, 20000.0)),   # underflows only
])
def test_troe_arguments_are_bounded(troe, flags, want):
    assert mechgen.temperature_range(_flat([0.0, 0.0], [(0, 1)], troe, flags)) == want


RANGES = {"synth_h2_9": (95.0, 17900.0), "synth_ch4_21": (140.0, 17350.0), "synth_c12_53": (180.0, 12550.0)}


@pytest.mark.parametrize("name", RANGES)
def test_bundled_mechanisms(name):
    assert mechgen.temperature_range(M.flatten(M.builtin(name))) == RANGES[name]


@pytest.mark.gpu
@pytest.mark.parametrize("name", RANGES)
def test_rates_at_the_ends_of_the_range(name, oracle_mod):
    """Rates just inside and outside the range, by warp and by thread, against the
    oracle: sums of products of 64-bit terms whose exponents reach 690, each with a
    relative error of as many round-offs, 1e-11 of the largest in all."""
    from test_round_kernels import _dev, _field, torch
    from pelelmex_b200.reactor import ReactorB200
    lo, hi = RANGES[name]
    mech, orc = M.builtin(name), oracle_mod.Oracle(M.flatten(M.builtin(name)))
    r = ReactorB200(name).init()
    for n in (9, 40000):
        f = _field(name, n)
        T = np.resize(np.array([lo - 10.0, lo + 1.0, lo + 10.0, 300.0, 9000.0, hi - 100.0, hi - 1.0, hi + 100.0]), n)
        rhoH = f.rhoY.sum(axis=0) * M.mix_h_mass(mech, T, (f.rhoY / f.rhoY.sum(axis=0)).T)
        Tg = _dev(T)
        w = r.inst_rr(_dev(f.rhoY * 1e3), _dev(rhoH * 0.1), Tg).cpu().numpy()
        Tg = Tg.cpu().numpy()
        assert np.abs(Tg / T - 1.0).max() < 1e-10 and torch.isfinite(torch.tensor(w)).all()
        for c in range(min(n, 16)):
            ref = orc.wdot(Tg[c], f.rhoY[:, c] / mech.mw()) * mech.mw() * 1e3
            assert np.abs(w[:, c] - ref).max() <= 1e-11 * np.abs(ref).max() + 1e-290
    r.close()


@pytest.mark.gpu
def test_react_of_a_hot_cell_by_warp_and_by_thread(oracle_mod):
    """A cell that starts above 8000 K (a failed step's state, say) beside flame cells:
    the same bits in a small and a large batch, and the oracle's result."""
    from test_gpu_parity import T_RTOL, run_gpu
    from test_round_kernels import _field
    f = _field("synth_ch4_21", 20000)
    f.T[7] = 9500.0
    a = run_gpu("synth_ch4_21", f, kernel="rounds")
    s = f.subset(np.arange(16))
    b = run_gpu("synth_ch4_21", s, kernel="rounds")
    assert (a["status"] == 0).all()
    assert np.array_equal(a["T"][:16], b["T"]) and np.array_equal(a["rhoY"][:, :16], b["rhoY"])
    o = oracle_mod.Oracle(M.flatten(M.builtin("synth_ch4_21"))).react(s.rhoY, s.frhoY, s.T, s.rhoH, s.frhoH, s.dt, rtol=1e-8,
                                                                     atol=1e-12, max_order=5)
    assert o["nfail"] == 0 and (np.abs(b["T"] / o["T"] - 1.0) <= T_RTOL).all()
