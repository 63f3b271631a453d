"""The Jacobian kernel's table (csrc/jac_table.h) against the sums written out:
with made-up derivatives of every reaction's rate, each entry of d(wdot)/d(C, T)
must be the sum of net stoichiometry times derivative."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from pelelmex_b200 import mechanism as M

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("jt") / "libjt.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(ROOT / "pelelmex_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "jac_table_c.cpp"), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def _ip(a):
    return a.ctypes.data_as(ctypes.c_void_p)


@pytest.mark.parametrize("name", ["synth_h2_9", "synth_ch4_21", "synth_c12_53"])
def test_entries_are_the_written_out_sums(lib, name):
    f = M.flatten(M.builtin(name))
    a, N, R = f.arrays, f.n_species, f.n_reactions
    sp = np.ascontiguousarray(np.asarray(a["sp"], np.int32).reshape(R, 8).T)
    sgn = np.where(np.arange(8) < 4, -1, 1)[:, None]
    nu = np.ascontiguousarray(np.where(sp >= 0, np.asarray(a["nu"], np.int32).reshape(R, 8).T * sgn, 0).astype(np.int32))
    rtype = np.ascontiguousarray(a["rtype"], np.int32)
    eptr, esp = np.ascontiguousarray(a["eff_ptr"], np.int32), np.ascontiguousarray(a["eff_sp"], np.int32)
    em1 = np.ascontiguousarray(np.asarray(a["eff_val"], np.float64) - 1.0)
    ld = (N + 1) | 1
    nd = ctypes.c_int()
    args = (N, R, _ip(rtype), _ip(sp), _ip(nu), _ip(eptr), _ip(esp), _ip(em1), ld)
    assert lib.jac_table_apply(*args, None, ctypes.byref(nd), None) == 0
    D = np.random.default_rng(3).normal(size=nd.value)
    out = np.empty((N + 1) * ld + 2 * N)
    assert lib.jac_table_apply(*args, _ip(D), ctypes.byref(nd), _ip(out)) == 0
    ref, u, w, p = np.zeros((N + 1, N)), np.zeros(N), np.zeros(N), 0
    for j in range(R):
        slots = [s for s in range(8) if sp[s, j] >= 0]
        net = np.zeros(N)
        for s in slots:
            net[sp[s, j]] += nu[s, j]
        for s in slots:
            ref[sp[s, j]] += net * D[p]
            p += 1
        ref[N] += net * D[p]
        w += net * D[p + 1]
        p += 2
        if rtype[j]:
            u += net * D[p]
            for q in range(eptr[j], eptr[j + 1]):
                ref[esp[q]] += net * em1[q] * D[p]
            p += 1
    assert p == nd.value
    got = out[:(N + 1) * ld].reshape(N + 1, ld)[:, :N]
    # sums of at most a few hundred terms of order one, in another order
    assert np.abs(got - ref).max() < 1e-12 and np.abs(out[(N + 1) * ld:] - np.concatenate([u, w])).max() < 1e-12
