"""Quotients that leave the FP64 range in the kernels that multiply by a
reciprocal and correct by the residual: an overflow is an infinity, as a division
gives it, and what is finite is unaffected."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _same(got, exp, tol):
    """The same infinities and NaNs, finite entries within tol of the largest."""
    assert np.array_equal(np.isnan(got), np.isnan(exp))
    inf, fin = np.isinf(exp), np.isfinite(exp)
    assert np.array_equal(np.isinf(got), inf) and np.array_equal(got[inf], exp[inf])
    assert np.all(np.abs(got[fin] - exp[fin]) <= tol * np.abs(exp[fin]).max(initial=0.0))


@pytest.mark.parametrize("n", [1, 3, 33, 64])
def test_triangular_solve_of_many_rows(gpu_lib, n):
    """x U = b row by row in divisions: 2^600 / 2^-600 and an infinite b."""
    import torch

    L = gpu_lib
    m = 5000
    rng = np.random.default_rng(n)
    U = np.asfortranarray(np.triu(rng.uniform(-1.0, 1.0, (n, n)), 1) / n + np.diag(rng.uniform(1.0, 2.0, n)))
    U[n - 1, n - 1] = -(2.0 ** -600)
    B = rng.uniform(1.0, 2.0, (m, n)) * np.where(rng.random((m, n)) < 0.5, -1.0, 1.0)
    B[::7, n - 1] *= 2.0 ** 600
    B[1, 0], B[2, n // 2], B[3, n - 1] = np.inf, -np.inf, np.nan
    B = np.asfortranarray(B)
    X = B.copy()
    with np.errstate(all="ignore"):
        for c in range(n):
            for p in range(c):
                X[:, c] -= X[:, p] * U[p, c]
            X[:, c] /= U[c, c]
    assert np.isinf(X[::7, n - 1]).any()
    dU, dB = L.to_device_colmajor(U), L.to_device_colmajor(B)
    assert L.prim_trsm_right_upper(m, n, 1.0, dU, n, dB, m, None) == 0
    torch.cuda.synchronize()
    # n products and a quotient of entries of one size, each rounded once
    _same(L.from_device(dB), X, 4 * n * 2.0 ** -53)


@pytest.mark.parametrize("n", [1, 2, 33, 40])
def test_batched_back_substitution(gpu_lib, n):
    """R x = y with x_n = 2^600 / 2^-600, A its own R (nothing below a diagonal)."""
    import torch

    L = gpu_lib
    R = np.diag(np.arange(1.0, n + 1.0))
    R[n - 1, n - 1] = 2.0 ** -600
    R[: n - 1, n - 1] = np.where(np.arange(n - 1) % 3 == 0, -2.0, 0.5)
    b = np.arange(2.0, n + 2.0)[:, None]
    b[n - 1] = 2.0 ** 600
    x = b.copy()
    with np.errstate(all="ignore"):
        for k in range(n - 1, -1, -1):  # column by column, as BLAS solves it
            x[k] /= R[k, k]
            x[:k, 0] -= R[:k, k] * x[k, 0]
    assert np.isinf(x[n - 1])
    dA, dB = L.to_device_colmajor(np.asfortranarray(R)), L.to_device_colmajor(np.asfortranarray(b))
    nb = L.lib().lila_query_dgels_batched(1)
    work = torch.empty(nb, dtype=torch.uint8, device="cuda")
    info = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    assert L.dgels_batched_prepare(1, [n], [n], 1, [dA], [n], [dB], [n], work, nb) == 0
    assert L.dgels_batched_run(1, 1, work, info) == 0
    torch.cuda.synchronize()
    assert info.item() == 0
    assert np.array_equal(L.from_device(dB), x, equal_nan=True)


@pytest.mark.parametrize("n,k", [(1, 0), (2, 0), (33, 5), (64, 31), (64, 63), (70, 5)])
def test_cholesky_with_an_infinite_pivot(gpu_lib, n, k):
    """An infinite diagonal entry is a positive pivot: its row is zero right of
    the root, the rows below go on, and nothing breaks down."""
    import torch

    L = gpu_lib
    rng = np.random.default_rng(n + k)
    X = rng.standard_normal((n, 2 * n))
    A = np.asfortranarray(X @ X.T)
    A[k, k] = np.inf
    R = np.triu(A)
    for j in range(n):
        R[j, j] = np.sqrt(R[j, j])
        R[j, j + 1:] /= R[j, j]
        for r in range(j + 1, n):
            R[r, r:] -= R[j, r] * R[j, r:]
    assert np.isfinite(np.delete(R.diagonal(), k)).all()
    dA = L.to_device_colmajor(A)
    L.gpu_clear_status()
    assert L.prim_potrf_upper(n, dA, n) == 0
    torch.cuda.synchronize()
    assert L.gpu_status() == 0
    # n products and a quotient per entry; the matrix is well conditioned
    _same(np.triu(L.from_device(dA)), R, 64 * n * 2.0 ** -53)


@pytest.mark.parametrize("n", [4, 64, 70])
@pytest.mark.parametrize("lower", [0, 1])
def test_sign_lu_with_large_entries(gpu_lib, n, lower):
    """The sign of a column is the one for which |s t - 1| as FP64 rounds it is not
    the smaller, also where t is so large that both sides round alike."""
    import torch

    L = gpu_lib
    rng = np.random.default_rng(n + lower)
    d = rng.uniform(-1.0, 1.0, n)
    big = [2.0 ** 60, -(2.0 ** 60), 2.0 ** 53 + 4, 2.0 ** 53 + 2, 2.0 ** 53, 2.0 ** 53 - 1, 1e300, np.inf, -np.inf,
           2.0 ** -54, 2.0 ** -54 * (1 + 2.0 ** -52), -(2.0 ** -54)]
    d[: len(big)] = big[:n]
    # nothing is subtracted: the strict triangle is quotients, or stays
    W = rng.uniform(-1.0, 1.0, (n, n))
    T = np.asfortranarray((np.tril(W, -1) if lower else np.triu(W, 1)) + np.diag(d))
    if lower:
        T[n - 1, 0] = np.inf
    E, S = T.copy(order="F"), np.zeros(n)
    with np.errstate(all="ignore"):
        for k in range(n):
            S[k] = -1.0 if abs(1.0 - E[k, k]) < abs(1.0 + E[k, k]) else 1.0
            E[:, k] *= S[k]
            E[k, k] -= 1.0
            E[k + 1:, k] /= E[k, k]
            E[k + 1:, k + 1:] -= np.outer(E[k + 1:, k], E[k, k + 1:])
    dT, dS = L.to_device_colmajor(T), torch.zeros(n, dtype=torch.float64, device="cuda")
    assert L.prim_lu_sign(n, dT, n, dS) == 0
    torch.cuda.synchronize()
    assert np.array_equal(dS.cpu().numpy(), S)
    got = L.from_device(dT)
    assert np.array_equal(np.isnan(got), np.isnan(E))
    # one quotient per entry
    ok = ~np.isnan(E)
    with np.errstate(invalid="ignore"):
        assert np.all((got[ok] == E[ok]) | (np.abs(got[ok] - E[ok]) <= 4 * 2.0 ** -53 * np.abs(E[ok])))
