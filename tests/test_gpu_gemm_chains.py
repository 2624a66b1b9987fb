"""The FP64 GEMM's long sums (Grams and updates of tall blocks) run in chains of
at most 256 terms: equal terms whose running sum rounds the same way every time, against
the exact sum.  A chain of n terms may be off by n u: 256 of them, at most 64
chains in a K slice here and at most 128 slices."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,upper,slices", [(64, 64, 262144, 1, 64), (16, 16, 262147, 1, 64), (40, 7, 100001, 0, 16),
                                                (30, 30, 3000, 0, 0), (128, 130, 5000, 0, 0)])
def test_equal_terms(gpu_lib, M, N, K, upper, slices):
    import torch

    L = gpu_lib
    t = 1.0 + 2.0 ** -42 - 2.0 ** -48
    A = torch.ones(M, K, dtype=torch.float64, device="cuda")  # column-major K x M
    B = torch.full((N, K), t, dtype=torch.float64, device="cuda")
    C = torch.zeros(N, M, dtype=torch.float64, device="cuda")
    part = torch.empty(max(1, slices * M * N), dtype=torch.float64, device="cuda")
    assert L.prim_gemm(M, N, K, A, K, 1, 0, B, K, 0, 0, C, M, 1.0, 0.0, 0, 0, upper, part if slices else None,
                       slices * M * N) == 0
    torch.cuda.synchronize()
    got = C.cpu()
    if upper:
        got = got[torch.tril(torch.ones(N, M, dtype=torch.bool))]  # the stored rows are columns
    # K t exactly: K whole, K (2^-42 - 2^-48) below an ulp of it or exact
    err = ((got - K) - K * (2.0 ** -42 - 2.0 ** -48)).abs().max().item()
    assert err <= (256 + 64 + 128) * 2.0 ** -53 * K
