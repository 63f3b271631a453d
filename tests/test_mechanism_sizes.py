"""Mechanisms of one species count and different numbers of reactions: reactors of
two of them used in turn in one process, and one whose reactions' derivatives do
not fit the Jacobian kernel's shared memory.  The long mechanisms are the bundled
ones with every reaction written `times` over and its rate divided by that, so
their solution is the plain one's."""
import copy

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pelelmex_b200 import mechanism as M, workloads as W  # noqa: E402
from pelelmex_b200.reactor import ReactorB200  # noqa: E402
from test_gpu_parity import DEV, T_RTOL, Y_ATOL, _dev  # noqa: E402


def _repeated(name, times):
    mech = copy.deepcopy(M.builtin(name))
    div = lambda a: a if a is None else (a[0] / times, a[1], a[2])  # noqa: E731
    for r in mech.reactions:
        r.arr, r.arr_lo, r.arr_rev = div(r.arr), div(r.arr_lo), div(r.arr_rev)
    mech.reactions = [r for r in mech.reactions for _ in range(times)]
    mech.name = f"{name}_x{times}"
    return mech


def _field(name, n):
    mech = M.builtin(name)
    if name == "synth_h2_9":
        return W.premixed_h2(mech, edge=48, cells=np.arange(n), dt=3e-7)
    if name == "synth_ch4_21":
        return W.flame_ch4(mech, cells=W.sample_cells(128 ** 3, n, seed=5), dt=1e-6)
    return W.c12_flame_grf(mech, edge=64, cells=W.sample_cells(64 ** 3, n, seed=5), dt=1e-7)


def _reactor(mech, lu_fp64=False, rtol=1e-8, atol=1e-12):
    return ReactorB200(mech, rtol=rtol, atol=atol, max_order=5, lu_fp64=lu_fp64, kernel="rounds").init()


def _react(r, f):
    a = [_dev(v) for v in (f.rhoY, f.frhoY, f.T, f.rhoH, f.frhoH)]
    _, _, st = r.react_flat(*a, torch.zeros(f.ncells, dtype=torch.float64, device=DEV), dt_react=f.dt, stats=True)
    return a[0].cpu().numpy(), a[2].cpu().numpy(), st


# shared memory of a CTA of the Jacobian kernel: 85, 86 and 78 KB for the long
# mechanism, 12, 38 and 40 KB for the plain one
@pytest.mark.parametrize("name,times", [("synth_h2_9", 20), ("synth_ch4_21", 4), ("synth_c12_53", 4)])
def test_reactors_of_two_mechanisms_in_turn(name, times):
    f = _field(name, 65)
    a, b = _reactor(_repeated(name, times)), _reactor(M.builtin(name))
    first = _react(a, f)
    plain = _react(b, f)
    again = _react(a, f)
    assert np.array_equal(first[0], again[0]) and np.array_equal(first[1], again[1])
    assert np.abs(first[1] - plain[1]).max() <= T_RTOL * plain[1].max()
    a.close()
    b.close()

# above 100 KB a CTA the derivatives go to device memory
@pytest.mark.parametrize("name,times", [("synth_h2_9", 28), ("synth_ch4_21", 6), ("synth_c12_53", 8)])
@pytest.mark.parametrize("lu_fp64", [False, True])
def test_derivatives_in_device_memory(name, times, lu_fp64):
    f = _field(name, 300)
    a, b = _reactor(_repeated(name, times), lu_fp64), _reactor(M.builtin(name), lu_fp64)
    (y, T, st), (yp, Tp, sp) = _react(a, f), _react(b, f)
    assert st["n_failed"] == 0 and sp["n_failed"] == 0
    assert np.abs(T - Tp).max() <= T_RTOL * Tp.min()
    rho, err = f.rhoY.sum(axis=0), Y_ATOL
    if name == "synth_c12_53":
        # step decisions that flip at round-off move a cell by the integrator's own
        # error, which is that of the plain mechanism against a tight solve
        c = _reactor(M.builtin(name), True, 1e-12, 1e-20)
        yt = _react(c, f)[0]
        c.close()
        err, yp = 3.0 * (np.abs(yp - yt).max(axis=0) / rho).max() + 1e-9, yt
    assert (np.abs(y - yp).max(axis=0) / rho).max() <= err
    # a wrong Jacobian costs Newton iterations first; step decisions that flip at
    # round-off move the counts of the 53-species field by a few per cent
    for k in ("nst", "nfe", "nje", "nlu"):
        assert abs(st[k] - sp[k]) <= (3e-2 if name == "synth_c12_53" else 2e-3) * sp[k] + 2, k
    a.close()
    b.close()
