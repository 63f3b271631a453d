"""T from (h, Y) and production rates of a cell do not depend on how many cells are
evaluated with it: T and rates by one launch of a warp per cell, T by thread and
rates by warp, and both by thread give the same bits."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pelelmex_b200 import mechanism as M  # noqa: E402
from pelelmex_b200.reactor import ReactorB200  # noqa: E402
from test_gpu_parity import _dev  # noqa: E402
from test_round_kernels import _field  # noqa: E402


# one launch up to `lim` cells; rates by thread above 9472 cells (37888 with 53 species)
@pytest.mark.parametrize("name,lim,big", [("synth_h2_9", 4096, 20000), ("synth_ch4_21", 4096, 20000),
                                          ("synth_c12_53", 2048, 40000)])
def test_cell_is_independent_of_its_batch(name, lim, big):
    f = _field(name, big)
    T = np.resize(np.array([0.9, 1.0, 1.1]), big) * f.T  # first guess
    ends = np.array([60.0, 94.0, 96.0, 139.0, 141.0, 179.0, 181.0, 12500.0, 12600.0, 17300.0, 17400.0, 17850.0, 18000.0])
    T[:ends.size] = ends  # around the ends of the generated code's temperatures
    state = np.where(np.arange(big) < ends.size, T, f.T)
    rhoH = f.rhoY.sum(axis=0) * M.mix_h_mass(M.builtin(name), state, (f.rhoY / f.rhoY.sum(axis=0)).T)
    r = ReactorB200(name).init()
    ref = {}
    for n in (big, lim + 1, lim, 33, 1):
        rhoY, h = _dev(f.rhoY[:, :n] * 1e3), _dev(rhoH[:n] * 0.1)
        Tr, Tt = _dev(T[:n]), _dev(T[:n])
        w = r.inst_rr(rhoY, h, Tr)
        r.t_from_hy(rhoY, h, Tt)
        assert torch.equal(Tr, Tt)
        ref = ref or {"T": Tr, "w": w}
        assert torch.equal(Tr, ref["T"][:n]) and torch.equal(w, ref["w"][:, :n])
    r.close()
