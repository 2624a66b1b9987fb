"""Block reflectors of up to 64 columns (the product's K slices are added up and
multiplied by T in one launch) and of 65 (a reduction and a product), against
numpy in extended precision.  An entry's error is at most (m + 2 k + 8) u times
the same expression of absolute values; what T's lower part holds is not read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (40, 1, 3), (129, 33, 16), (700, 2, 31), (700, 65, 32), (1413, 153, 33),
                                   (2000, 305, 63), (900, 457, 64), (900, 700, 64), (900, 40, 65)])
@pytest.mark.parametrize("room", [0, 1])
def test_block_reflector(gpu_lib, m, n, k, room):
    import torch

    L = gpu_lib
    rng = np.random.default_rng([m, n, k])
    V = np.tril(rng.standard_normal((m, k)), -1)
    V[np.arange(k), np.arange(k)] = 1.0
    Tu = np.triu(rng.standard_normal((k, k)))
    C = rng.standard_normal((m, n))
    stored = np.where(np.tril(np.ones((m, k)), -1) > 0, V, np.nan)  # R's place is not read
    A = np.asfortranarray(np.hstack([stored, C]))
    T = np.asfortranarray(np.where(np.triu(np.ones((k, k))) > 0, Tu, np.nan))
    dA, dT = L.to_device_colmajor(A), L.to_device_colmajor(T)
    lw = L.query_dormqrf_w03(m, n, k, 0, k, k, None, m, None, k, None, -1) + room * 16 * k * n
    dW = torch.empty(lw, dtype=torch.float64, device="cuda")
    assert L.dormqrf_w03(m, n, k, 0, k, k, dA, m, dT, k, dW, lw) == 0
    torch.cuda.synchronize()
    x = np.longdouble
    bound = (m + 2 * k + 8) * U
    ref = C - V.astype(x) @ (Tu.T.astype(x) @ (V.T.astype(x) @ C.astype(x)))
    mag = np.abs(C) + np.abs(V) @ (np.abs(Tu.T) @ (np.abs(V.T) @ np.abs(C)))
    got = L.from_device(dA)
    assert np.all(np.abs(got[:, k:] - ref) <= bound * mag)
    assert np.array_equal(got[:, :k], stored, equal_nan=True)
    if m == k:
        return
    Q = np.asfortranarray(np.vstack([np.full((k, n), np.nan), C[k:]]))  # its top counts as zeros
    dQ = L.to_device_colmajor(Q)
    dV = L.to_device_colmajor(np.asfortranarray(stored))
    lw = L.query_dormqrbz_w03(m, n, k, 0, 0, k, None, m, None, m, None, k, None, -1) + room * 16 * k * n
    dW = torch.empty(lw, dtype=torch.float64, device="cuda")
    assert L.dormqrbz_w03(m, n, k, 0, 0, k, dV, m, dQ, m, dT, k, dW, lw) == 0
    torch.cuda.synchronize()
    X = np.vstack([np.zeros((k, n)), C[k:]])
    ref = X - V.astype(x) @ (Tu.astype(x) @ (V.T.astype(x) @ X.astype(x)))
    mag = np.abs(X) + np.abs(V) @ (np.abs(Tu) @ (np.abs(V.T) @ np.abs(X)))
    assert np.all(np.abs(L.from_device(dQ) - ref) <= bound * mag)
