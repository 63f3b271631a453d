"""The round integrator's register inverses (csrc/gj_inverse.cuh) by a warp on the
CPU whose lanes run one after another between warp-wide operations, in several
orders: whatever the order, the inverse must be the one of the matrix."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parent.parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = tmp_path_factory.mktemp("gj") / "libgj.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-fno-strict-aliasing", "-w", "-shared", "-fPIC", "-I",
                    str(ROOT / "pelelmex_b200" / "csrc"), "-I", str(ROOT / "tests" / "cpp"),
                    str(ROOT / "tests" / "cpp" / "gj_inverse_c.cpp"), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


def _invert(lib, J, dsc, gamma, fp64, order):
    n = J.shape[0]
    J, dsc, out = np.ascontiguousarray(J), np.ascontiguousarray(dsc), np.empty((n, n))
    p = lambda a: a.ctypes.data_as(ctypes.c_void_p)  # noqa: E731
    return lib.gj_invert(n, fp64, p(J), p(dsc), ctypes.c_double(gamma), order, p(out)), out


@pytest.mark.parametrize("n,fp64", [(10, 1), (22, 1), (10, 0), (22, 0), (54, 0)])
@pytest.mark.parametrize("order", [0, 1, 2, 3])
def test_inverse_in_every_lane_order(lib, n, fp64, order):
    rng = np.random.default_rng(10 * n + order)
    J = rng.normal(size=(n, n)) / np.sqrt(n)
    dsc = np.ones(n) if fp64 else np.exp(rng.uniform(-3.0, 3.0, n))
    A = dsc[:, None] * (np.eye(n) - 1.7 * J) / dsc
    ier, out = _invert(lib, J, dsc, 1.7, fp64, order)
    ref = np.linalg.inv(A)
    # Gauss-Jordan with partial pivoting: n growth factors of at most n on the
    # round-off of the data, amplified by the condition number
    bound = n * n * np.linalg.cond(A, np.inf) * (2.0 ** -53 if fp64 else 2.0 ** -24) * np.abs(ref).max()
    assert ier == 0 and np.abs(out - ref).max() <= bound


@pytest.mark.parametrize("n,fp64", [(10, 1), (22, 1), (22, 0), (54, 0)])
def test_singular_matrix_is_reported(lib, n, fp64):
    J = np.zeros((n, n))
    J[3, 3] = 0.5  # row 3 of I - 2 J vanishes
    assert _invert(lib, J, np.ones(n), 2.0, fp64, 0)[0] > 0
