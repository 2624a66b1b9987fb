"""Householder QR of a matrix held in one CTA (V, R, T tiles and explicit Q in
one launch) and the one-CTA panel behind dgeqr3, against the oracle's
recursive driver and dgeqr3, at the suite's elementwise tolerance; columns
scaled by powers of two whose squares leave the FP64 range against the same
matrix unscaled (V, T and Q do not change, R's columns scale)."""
import numpy as np
import pytest

import lila_cases as C

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,ii,mt,leaf,panel,nx", [
    (2, 2, 0, 1, 1, 1, 2), (9, 3, 2, 4, 1, 1, 5), (17, 17, 0, 17, 0, 0, 4), (33, 16, 1, 5, 1, 0, 3),
    (40, 33, 7, 64, 1, 1, 8), (150, 65, 3, 16, 1, 1, 8), (300, 64, 0, 4, 0, 1, 64), (128, 128, 0, 7, 1, 1, 200),
    (110, 100, 10, 96, 1, 1, 4)])
def test_one_launch_qr_against_oracle(gpu_lib, oracle_lib, m, n, ii, mt, leaf, panel, nx):
    L = gpu_lib
    before = L.launch_count()
    out = C.run_gpu(L, "recursive", m, n, ii, mt, leaf, panel, nx, lda=m + 3, ldq=m + 1, seed=m + n)
    assert L.launch_count() - before == 1
    ref = C.run_cpu(oracle_lib, "recursive", m, n, ii, mt, leaf, panel, nx, lda=m + 3, ldq=m + 1, seed=m + n)
    err = C.compare_factor(out, ref, m, n, ii, mt)
    assert max(err.values()) < C.TOL, err
    # what the routine does not define keeps its contents
    M = C.tile_mask(n, ii, mt)
    assert np.array_equal(out[1][~M], ref[1][~M] * 0 + 7.0)
    assert np.array_equal(out[0][:, :ii], ref[0][:, :ii]) and np.array_equal(out[0][m:], ref[0][m:])
    assert np.array_equal(out[2][:ii], ref[2][:ii])
    outv = C.run_gpu_vq(L, "recursive", m, n, ii, mt, leaf, panel, max(2, nx), seed=m + n)
    refv = C.run_cpu_vq(oracle_lib, "recursive", m, n, ii, mt, leaf, panel, max(2, nx), seed=m + n)
    err = C.compare_factor(outv, refv, m, n, ii, mt)
    assert max(err.values()) < C.TOL, err


@pytest.mark.parametrize("m,n", [(2, 2), (64, 64), (200, 37), (255, 63), (300, 200)])
def test_dgeqr3_small_and_near_square(gpu_lib, oracle_lib, m, n):
    L = gpu_lib
    A = np.asfortranarray(np.random.default_rng(m * n).standard_normal((m, n)))
    if n > 5:
        A[:, 3] = 0.0
    Ao, To = A.copy(order="F"), np.asfortranarray(np.zeros((n, n)))
    oracle_lib.dgeqr3(m, n, Ao, m, To, n)
    dA, dT = L.to_device_colmajor(A), L.colmajor(n, n, fill=0.0)
    assert L.dgeqr3(m, n, dA, m, dT, n) == 0
    assert C.max_rel(L.from_device(dA), Ao) < C.TOL
    assert C.max_rel(np.triu(L.from_device(dT)), np.triu(To)) < C.TOL


@pytest.mark.parametrize("power", [600, -600, -1040])
def test_extreme_column_scales(gpu_lib, oracle_lib, power):
    L = gpu_lib
    m, n = 90, 12
    A = np.asfortranarray(np.round(np.random.default_rng(5).standard_normal((m, n)) * 64) / 64)
    Ao, To = A.copy(order="F"), np.asfortranarray(np.zeros((n, n)))
    oracle_lib.dgeqr3(m, n, Ao, m, To, n)
    k = np.where(np.arange(n) % 3 == 1, power, 0)
    As = np.asfortranarray(np.ldexp(A, k[None, :]))
    dA, dT = L.to_device_colmajor(As), L.colmajor(n, n, fill=0.0)
    assert L.dgeqr3(m, n, dA, m, dT, n) == 0
    got = L.from_device(dA)
    V, Vo = np.tril(got, -1), np.tril(Ao, -1)
    R, Ro = np.triu(got[:n]), np.triu(Ao[:n])
    # a scaled column whose updates stay above the subnormals keeps every bit it
    # has; below them its entries are rounded to multiples of 2^-1074
    tol = C.TOL if power > -1000 else 64 * 2.0 ** (-1074 - power)
    assert C.max_rel(V, Vo) < tol
    assert np.all(np.abs(np.ldexp(R, -k[None, :]) - Ro) < tol * 8 * m)
    assert C.max_rel(np.triu(L.from_device(dT)), np.triu(To)) < tol
