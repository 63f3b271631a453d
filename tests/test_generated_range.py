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
    assert mechgen.temperature_range(_flat([300.0, -400.0, 0.0], [(0, 2), (1, 1)])) == (150.0, 8000.0)
    # the last factors: 680 and two powers of ln(Ru T / 1 atm), 11.3 at 1000 K
    assert mechgen.temperature_range(_flat([340.0, 0.0], [(0, 2), (1, 1)])) == (1000.0, 1000.0)


@pytest.mark.parametrize("troe,flags,want", [
    ((0.5, -2.0, 1e3, 0.0), 1, (150.0, 1350.0)),   # -T / T3 <= 690
    ((0.5, 1e3, -2.0, 0.0), 1, (150.0, 1350.0)),   # -T / T1 <= 690
    ((0.5, 1e3, 1e3, -4e5), 5, (580.0, 8000.0)),   # -T2 / T <= 690
    ((0.5, 1e3, 1e3, -4e5), 1, (150.0, 8000.0)),   # no T2 in this form
    ((0.5, 1e-3, 1e3, 1e9), 5, (150.0, 8000.0)),   # underflows only
])
def test_troe_arguments_are_bounded(troe, flags, want):
    assert mechgen.temperature_range(_flat([0.0, 0.0], [(0, 1)], troe, flags)) == want


@pytest.mark.parametrize("name,lo", [("synth_h2_9", 150.0), ("synth_ch4_21", 150.0), ("synth_c12_53", 180.0)])
def test_bundled_mechanisms(name, lo):
    assert mechgen.temperature_range(M.flatten(M.builtin(name))) == (lo, 8000.0)
