"""The small triangular kernels of the reconstruction (N <= 64) at the edges of
their two-values-per-lane split, against numpy: errors within 8 n u of the
condition-free bounds (backward error of a triangular solve, of Cholesky and of
LU without pivoting on a matrix whose pivots are at least 1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("N", [1, 2, 31, 32, 33, 63, 64])
def test_triangular_solves(gpu_lib, N):
    import torch

    L = gpu_lib
    rng = np.random.default_rng(N)
    M = 2049 + 131
    Uu = np.asfortranarray(np.triu(rng.standard_normal((N, N)), 1) + np.diag(rng.uniform(1, 2, N) * rng.choice([-1, 1], N)))
    B = np.asfortranarray(rng.standard_normal((M, N)))
    S = rng.choice([-1.0, 1.0], N)
    dB, dU = L.to_device_colmajor(B), L.to_device_colmajor(Uu)
    for alpha in (1.0, -0.5):
        dB.copy_(L.to_device_colmajor(B))
        L.prim_trsm_right_upper(M, N, alpha, dU, N, dB, M, torch.from_numpy(S).cuda())
        torch.cuda.synchronize()
        X = L.from_device(dB)
        assert np.all(np.abs(X @ Uu - alpha * B * S) <= 8 * N * U * (np.abs(X) @ np.abs(Uu) + np.abs(B)))
    Lo = np.asfortranarray(np.tril(rng.standard_normal((N, N)), -1) + np.eye(N))
    C = np.asfortranarray(rng.standard_normal((N, 9)))
    dC = L.to_device_colmajor(C)
    L.prim_trsm_left_lower_unit(N, 9, L.to_device_colmajor(Lo), N, dC, N)
    torch.cuda.synchronize()
    X = L.from_device(dC)
    assert np.all(np.abs(Lo @ X - C) <= 8 * N * U * (np.abs(Lo) @ np.abs(X) + np.abs(C)))
    C = np.asfortranarray(np.triu(rng.standard_normal((N, N))))
    dC = L.to_device_colmajor(C)
    L.prim_trsm_right_lower_unit_trans(N, N, -1.0, L.to_device_colmajor(Lo), N, dC, N)
    torch.cuda.synchronize()
    X = L.from_device(dC)
    assert np.all(np.abs(X @ Lo.T + C) <= 8 * N * U * (np.abs(X) @ np.abs(Lo.T) + np.abs(C)))


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 32, 33, 63, 64])
def test_cholesky_and_sign_lu(gpu_lib, n):
    import torch

    L = gpu_lib
    rng = np.random.default_rng(n)
    X = rng.standard_normal((3 * n, n))
    G = np.asfortranarray(X.T @ X)
    low = np.asfortranarray(np.triu(G) + np.tril(np.full((n, n), 9.0), -1))
    dG = L.to_device_colmajor(low)
    L.prim_potrf_upper(n, dG, n)
    torch.cuda.synchronize()
    got = L.from_device(dG)
    R = np.triu(got)
    assert np.array_equal(np.tril(got, -1), np.tril(low, -1))
    assert np.all(np.abs(R.T @ R - G) <= 8 * n * U * (np.abs(R.T) @ np.abs(R)))
    assert L.gpu_status() == 0
    # a non-positive pivot: rows above it are the factor, the rest is untouched
    bad = n // 2
    H = low.copy(order="F")
    H[bad, bad] -= 2 * G[bad, bad]
    dH = L.to_device_colmajor(H)
    L.prim_potrf_upper(n, dH, n)
    torch.cuda.synchronize()
    got = L.from_device(dH)
    assert L.gpu_status() & 1
    L.gpu_clear_status()
    assert np.array_equal(got[:bad], L.from_device(dG)[:bad]) and got[bad, bad] <= 0.0
    assert np.array_equal(got[bad + 1:], H[bad + 1:]) and np.array_equal(got[bad, :bad], H[bad, :bad])
    assert np.array_equal(got[bad, bad + 1:], H[bad, bad + 1:])
    # LU of T S - I
    Q, _ = np.linalg.qr(rng.standard_normal((2 * n + 3, n)))
    T = np.asfortranarray(Q[:n])
    dT, dS = L.to_device_colmajor(T), torch.zeros(n, dtype=torch.float64, device="cuda")
    L.prim_lu_sign(n, dT, n, dS)
    torch.cuda.synchronize()
    got, Sg = L.from_device(dT), dS.cpu().numpy()
    Lf, Uf = np.tril(got, -1) + np.eye(n), np.triu(got)
    assert set(np.unique(Sg)) <= {-1.0, 1.0} and np.all(np.diag(Uf) <= -1.0)
    assert np.all(np.abs(Lf @ Uf - (T * Sg - np.eye(n))) <= 8 * n * U * (np.abs(Lf) @ np.abs(Uf)))
