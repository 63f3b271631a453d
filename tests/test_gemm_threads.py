"""GEMMs of different shapes from several threads, each on a stream of its own: a
call's launch must not depend on what another thread launches in between."""
import threading

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from pelelmex_b200.surrogate import gemm  # noqa: E402

DEV = "cuda:0"


# split K with N tiles of 16 and 64; one tile at a time with 32 and 512 columns;
# weights resident in shared memory, 48 and 256 columns
@pytest.mark.parametrize("shapes", [[(128, 16, 1024), (128, 64, 1024)], [(128, 32, 320), (128, 512, 512)],
                                    [(128, 48, 64), (128, 256, 256)]])
def test_shapes_from_two_threads(shapes):
    errors = []

    def work(M, N, K, seed):
        try:
            g = torch.Generator(device=DEV).manual_seed(seed)
            A = torch.randn((M, K), device=DEV, generator=g).to(torch.bfloat16)
            B = torch.randn((N, K), device=DEV, generator=g).to(torch.bfloat16)
            first, C = torch.empty((M, N), device=DEV), torch.empty((M, N), device=DEV)
            with torch.cuda.stream(torch.cuda.Stream(DEV)):
                torch.cuda.current_stream().wait_stream(torch.cuda.default_stream())
                gemm(A, B, first)
                for _ in range(1500):
                    gemm(A, B, C)
                torch.cuda.current_stream().synchronize()
            ref = A.double() @ B.double().T
            # FP32 sums of K products: each partial sum rounded, 2^-23 of the magnitudes
            bound = K * 2.0 ** -23 * (A.double().abs() @ B.double().abs().T)
            assert ((C.double() - ref).abs() <= bound).all() and torch.equal(C, first)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(*s, i)) for i, s in enumerate(shapes * 2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
