"""What a triangular mask leaves out is not multiplied where whole K steps fall to
it: a NaN opposite those zeros stays where it is (as in BLAS' triangular products),
and one that meets a stored entry spreads."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_masked_product(gpu_lib):
    import torch

    L = gpu_lib
    n, c = 300, 9
    rng = np.random.default_rng(0)
    A = np.asfortranarray(rng.standard_normal((n, n)))
    B = np.asfortranarray(rng.standard_normal((n, c)))
    B[5, 2], B[290, 4] = np.nan, np.inf
    dA, dB, dC = L.to_device_colmajor(A), L.to_device_colmajor(B), L.colmajor(n, c, fill=0.0)
    assert L.prim_gemm(n, c, n, dA, n, 0, 2, dB, n, 0, 0, dC, n, 1.0, 0.0, 0, 0, 0, None, 0) == 0
    torch.cuda.synchronize()
    got = L.from_device(dC)
    # an upper triangle's row r takes the rows of B from r on
    assert np.isnan(got[:6, 2]).all() and not np.isfinite(got[:291, 4]).any()
    clean = [j for j in range(c) if j not in (2, 4)]
    exp = np.triu(A) @ B[:, clean]
    assert np.abs(got[:, clean] - exp).max() <= 4 * n * 2.0 ** -53 * (np.abs(np.triu(A)) @ np.abs(B[:, clean])).max()
    # past the tile of row 5 nothing meets it
    exp = np.triu(A)[64:] @ np.where(np.isnan(B[:, 2]), 0.0, B[:, 2])
    assert np.abs(got[64:, 2] - exp).max() <= 4 * n * 2.0 ** -53 * np.abs(A).max() * np.nansum(np.abs(B[:, 2]))


@pytest.mark.parametrize("n", [6, 64])
def test_solve_with_an_upper_triangle(gpu_lib, n):
    """X L^T = B, B upper triangular: row r of X depends on L's columns from r on."""
    import torch

    L = gpu_lib
    rng = np.random.default_rng(n)
    Lo = np.asfortranarray(np.tril(rng.uniform(-1, 1, (n, n)) / n, -1) + np.eye(n))
    B = np.asfortranarray(np.triu(rng.uniform(1, 2, (n, n))))
    p = n // 2
    X = B.copy()
    for c in range(n):
        for q in range(c):
            X[:, c] -= X[:, q] * Lo[c, q]
    Ln = Lo.copy(order="F")
    Ln[n - 1, p] = np.nan
    dL, dB = L.to_device_colmajor(Ln), L.to_device_colmajor(B)
    assert L.prim_trsm_right_lower_unit_trans(n, n, 1.0, dL, n, dB, n) == 0
    torch.cuda.synchronize()
    got = L.from_device(dB)
    hit = np.zeros((n, n), dtype=bool)
    hit[: p + 1, n - 1] = True  # rows whose X(:, p) is stored
    assert np.array_equal(np.isnan(got), hit)
    assert np.abs(got[~hit] - X[~hit]).max() <= 4 * n * 2.0 ** -53 * np.abs(X).max()
