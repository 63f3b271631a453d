"""The rule that splits K over a cluster (csrc/split_rule.h) against what both sides
took on a B200 of 148 SMs, and the GEMM on both sides of its line."""
import ctypes
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent

# (M, N, K, us a GEMM with whole tiles, us with K split): launches in a row from a graph
MEASURED = [
    (128, 16, 1024, 28.0, 6.5), (128, 80, 16384, 507.5, 33.7), (256, 256, 16384, 806.5, 44.2), (1024, 512, 1088, 60.8, 25.2),
    (2048, 80, 1088, 37.9, 19.9), (2048, 512, 1024, 57.9, 39.9), (3072, 256, 1024, 57.8, 30.4), (3072, 512, 1088, 61.0, 70.9),
    (3072, 512, 2048, 108.0, 81.6), (4096, 80, 1024, 36.0, 29.8), (4096, 256, 1024, 57.7, 39.8), (4096, 512, 1024, 58.0, 77.7),
    (4096, 512, 1088, 61.4, 93.9), (4096, 512, 4096, 208.3, 167.2), (4096, 512, 16384, 1042.1, 528.1),
    (6144, 80, 1024, 36.2, 40.6), (6144, 80, 1088, 38.1, 50.3), (6144, 80, 2048, 67.8, 61.0), (6144, 128, 1024, 41.3, 30.3),
    (6144, 256, 1088, 61.1, 71.0), (6144, 256, 2048, 108.8, 81.7), (8192, 48, 1088, 34.4, 23.0), (8192, 80, 1024, 36.2, 53.9),
    (8192, 80, 2048, 67.9, 82.2), (8192, 80, 4096, 130.9, 141.0), (8192, 80, 16384, 656.8, 489.3), (8192, 128, 1088, 44.5, 48.0),
    (8192, 128, 2048, 77.7, 55.1), (8192, 256, 1024, 58.1, 77.7), (8192, 256, 1088, 61.4, 93.8), (8192, 256, 4096, 211.2, 167.3),
    (9344, 16, 1088, 30.2, 19.7), (9344, 64, 1024, 33.9, 27.7), (9344, 80, 4096, 131.4, 160.6), (9344, 128, 1024, 41.8, 48.2),
    (9344, 128, 1088, 44.9, 58.2), (9344, 128, 2048, 77.6, 67.1), (9344, 256, 1024, 58.2, 88.2), (9344, 256, 2048, 108.7, 122.1),
    (9344, 256, 16384, 1007.3, 594.2),
]


@pytest.fixture(scope="module")
def pays(tmp_path_factory):
    so = tmp_path_factory.mktemp("sr") / "libsr.so"
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(ROOT / "pelelmex_b200" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "split_rule_c.cpp"), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so)).split_pays


@pytest.mark.parametrize("M,N,K,whole,split", MEASURED)
def test_the_faster_side_is_taken(pays, M, N, K, whole, split):
    assert bool(pays(M, N, K, 148)) == (split < whole)


def test_short_ragged_or_many_tiles_are_not_split(pays):
    assert not pays(128, 16, 960, 148) and not pays(128, 16, 1040, 148) and not pays(128 * 74, 256, 16384, 148)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K", [(8192, 128, 1024), (8192, 128, 1088), (6144, 80, 1088), (6144, 80, 2048),
                                   (4096, 512, 1024), (3072, 512, 2048), (9344, 256, 1088), (9344, 256, 4096)])
def test_gemm_on_both_sides_of_the_line(M, N, K):
    torch = pytest.importorskip("torch")
    from pelelmex_b200.surrogate import gemm
    g = torch.Generator(device="cuda:0").manual_seed(K)
    A = torch.randn((M, K), device="cuda:0", generator=g).to(torch.bfloat16)
    B = torch.randn((N, K), device="cuda:0", generator=g).to(torch.bfloat16)
    C = torch.full((M, N), 7.0, device="cuda:0")
    gemm(A, B, C)
    ref = A.double() @ B.double().T
    # one FP32 rounding of the running sum per 16 products, then 8 partial sums:
    # each at most 2^-23 of the sum of magnitudes
    bound = (K / 16 + 8) * 2.0 ** -23 * (A.double().abs() @ B.double().abs().T)
    assert ((C.double() - ref).abs() <= bound).all()
