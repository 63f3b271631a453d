"""GEMMs with few tiles and a long K (the weight gradients), which a cluster of
CTAs shares: edges of the K ranges (fewer chunks than an even split, last CTAs
without any), N tiles of 16 to 64, partial output columns, the same bits twice."""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pelelmex_b200.surrogate import gemm  # noqa: E402

DEV = "cuda:0"


# K = 1024: 2 chunks of 64 for each of 8 CTAs; 1088: 17 chunks, so 3 for the
# first five, 2 for the sixth and none for the last two; 16384: the training batch
@pytest.mark.parametrize("M,N,K,n_valid", [(128, 16, 1024, 0), (256, 32, 1088, 22), (128, 48, 1216, 0),
                                           (256, 256, 1024, 0), (256, 80, 2112, 70), (256, 512, 4096, 0),
                                           (256, 256, 16384, 0), (128, 256, 16384, 255)])
def test_split_k_matches_fp64(M, N, K, n_valid):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    A = torch.randn((M, K), device=DEV, generator=g).to(torch.bfloat16)
    B = torch.randn((N, K), device=DEV, generator=g).to(torch.bfloat16)
    bias = torch.randn(N, device=DEV, generator=g)
    err = torch.zeros(1, dtype=torch.int32, device=DEV)
    C = torch.full((M, N), 7.0, device=DEV)
    gemm(A, B, C, bias, n_valid=n_valid, err=err)
    again = torch.full((M, N), 7.0, device=DEV)
    gemm(A, B, again, bias, n_valid=n_valid, err=err)
    nv = n_valid or N
    ref = A.double() @ B.double().T + bias.double()
    # one FP32 rounding of the running sum per 16 products, then 8 partial sums
    # and the bias: each at most 2^-23 of the sum of magnitudes
    bound = (K / 16 + 9) * 2.0 ** -23 * (A.double().abs() @ B.double().abs().T + bias.double().abs())
    assert int(err.item()) == 0
    assert ((C.double() - ref).abs() <= bound)[:, :nv].all()
    assert (C[:, nv:] == 7.0).all() and torch.equal(C, again)
