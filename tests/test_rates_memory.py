"""Device memory that the kernels of the rates and right-hand sides take beside the
caller's arrays: local memory is set aside for every thread the GPU can hold, so an
array of a cell's size in one of them costs hundreds of megabytes."""
import subprocess
import sys
from pathlib import Path

import pytest

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

SCRIPT = """
import torch
from pelelmex_b200.reactor import ReactorB200
r = ReactorB200({name!r}).init()
free = []
for n in (64, 60000):
    rhoY = torch.full((r.N, n), 1e-2, dtype=torch.float64, device="cuda:0")
    T = torch.full((n,), 1200.0, dtype=torch.float64, device="cuda:0")
    h = torch.full((n,), 1e6, dtype=torch.float64, device="cuda:0")
    torch.empty_like(rhoY)
    torch.cuda.synchronize()
    free.append(torch.cuda.mem_get_info()[0])
    r.inst_rr(rhoY, h, T)
    torch.cuda.synchronize()
    free.append(torch.cuda.mem_get_info()[0])
print((free[0] - free[1] + free[2] - free[3]) >> 20)
"""


# 148 SMs of 2048 threads: 1 KB a thread, code and spills included, is 296 MB
@pytest.mark.parametrize("name", ["synth_h2_9", "synth_ch4_21", "synth_c12_53"])
def test_rates_take_little_memory(name):
    out = subprocess.run([sys.executable, "-c", SCRIPT.format(name=name)], cwd=ROOT, capture_output=True, text=True, check=True)
    assert int(out.stdout.split()[-1]) <= 296
