"""The FP64 GEMM's tiles (16, 32 and 64 wide), K splits and mask ranges at
their edges, against numpy: what a mask leaves out is never read into the
product (it holds NaN here).  An entry's error is at most (K + 2) u times the
product of the absolute values (any summation order), u = 2^-53; numpy's own
product has the same bound."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _stored(rng, r, c, mask):
    """A stored operand and its value: NaN where the mask does not read."""
    X = rng.standard_normal((r, c))
    i, j = np.indices((r, c))
    unread = {0: np.zeros((r, c), bool), 1: i <= j, 2: i > j, 3: i < j, 4: i >= j}[mask]
    S = np.asfortranarray(np.where(unread, np.nan, X))
    V = np.where(unread, 0.0, X)
    if mask in (1, 4):
        V[np.arange(min(r, c)), np.arange(min(r, c))] = 1.0
    return S, V


@pytest.mark.parametrize("M,N,K", [(15, 17, 16), (16, 16, 32), (33, 31, 65), (64, 1, 63), (1, 65, 700),
                                   (17, 130, 2049), (128, 350, 128), (640, 640, 33)])
@pytest.mark.parametrize("ta,tb,ma,mb", [(0, 0, 0, 0), (1, 0, 1, 0), (0, 1, 1, 1), (1, 1, 2, 2), (0, 0, 3, 4),
                                         (1, 0, 4, 3), (0, 0, 2, 2)])
def test_gemm_edges(gpu_lib, M, N, K, ta, tb, ma, mb):
    import torch

    L = gpu_lib
    rng = np.random.default_rng([M, N, K, ta, tb, ma, mb])
    As, A = _stored(rng, *((K, M) if ta else (M, K)), ma)
    Bs, B = _stored(rng, *((N, K) if tb else (K, N)), mb)
    A, B = (A.T if ta else A), (B.T if tb else B)
    ref, mag = A @ B, np.abs(A) @ np.abs(B)
    dA, dB, dC = L.to_device_colmajor(As), L.to_device_colmajor(Bs), L.colmajor(M, N, fill=7.0)
    part = torch.empty(8 * M * N, dtype=torch.float64, device="cuda")
    for plen in (0, part.numel()):
        for upper in (0, 1):
            dC.fill_(7.0)
            L.prim_gemm(M, N, K, dA, As.shape[0], ta, ma, dB, Bs.shape[0], tb, mb, dC, M, 1.0, 0.0, 0, 0, upper,
                        part, plen)
            torch.cuda.synchronize()
            got = L.from_device(dC)
            keep = np.triu(np.ones((M, N), bool)) if upper else np.ones((M, N), bool)
            assert np.all(np.abs(got - ref)[keep] <= 2 * (K + 2) * U * mag[keep]), (plen, upper)
            assert np.all(got[~keep] == 7.0), (plen, upper)
