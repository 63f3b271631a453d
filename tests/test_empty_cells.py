"""Temperature and rates of a cell without mass (a covered one, say): undefined, not
a number that looks like a result, and the cells beside it are as without it."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pelelmex_b200 import mechanism as M  # noqa: E402
from pelelmex_b200.reactor import ReactorB200  # noqa: E402
from test_gpu_parity import _dev  # noqa: E402
from test_round_kernels import _field  # noqa: E402


# rates by warp and, above 9472 (37888 with 53 species) cells, by thread
@pytest.mark.parametrize("name,n", [("synth_h2_9", 5), ("synth_ch4_21", 130), ("synth_c12_53", 130), ("synth_ch4_21", 12000)])
def test_cell_without_mass(name, n):
    f = _field(name, n)
    Y, empty = f.rhoY / f.rhoY.sum(axis=0), n // 2
    rhoY = f.rhoY * 1e3
    rhoH = f.rhoY.sum(axis=0) * M.mix_h_mass(M.builtin(name), f.T, Y.T) * 0.1
    r = ReactorB200(name).init()
    full, Tf = _dev(rhoY), _dev(f.T)
    wf = r.inst_rr(full, _dev(rhoH), Tf)
    rhoY[:, empty] = 0.0
    for h in (0.0, 1.0e5, -1.0e5):
        rhoH[empty] = h
        Te, Tt = _dev(f.T), _dev(f.T)
        we = r.inst_rr(_dev(rhoY), _dev(rhoH), Te)
        r.t_from_hy(_dev(rhoY), _dev(rhoH), Tt)
        keep = torch.arange(n, device=Te.device) != empty
        assert torch.isnan(Te[empty]) and torch.isnan(Tt[empty])
        assert torch.equal(Te[keep], Tf[keep]) and torch.equal(we[:, keep], wf[:, keep])
    r.close()
