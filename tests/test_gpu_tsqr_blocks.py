"""The TSQR tree's block kernels at every split of a block over lanes (4, 8 or
16 lanes per column, 32 or 64 rows per lane), with short last blocks, against
the oracle's Householder QR after sign normalisation (the suite's 1e-12), and
columns scaled by powers of two whose squares leave the FP64 range."""
import numpy as np
import pytest

import lila_cases as C
from test_gpu_tsqr import run_tsqr

pytestmark = pytest.mark.gpu


def _householder(oracle_lib, A):
    m, n = A.shape
    Ah, Th = A.copy(order="F"), np.asfortranarray(np.zeros((16, n)))
    Qh = np.asfortranarray(np.zeros((m, n)))
    w = np.zeros(8 * m * 16 + 4 * n * n)
    oracle_lib.dgeqrf_w03_recursive(C.lparam(1, 1, 16), m, n, 0, 16, Ah, m, Th, 16, Qh, m, w, w.size)
    return np.triu(Ah[:n]), Qh


@pytest.mark.parametrize("m,n,mb,arity", [(513, 1, 16, 2), (700, 7, 100, 16), (1025, 16, 256, 16), (2600, 32, 256, 16),
                                          (3073, 32, 256, 4), (1301, 90, 130, 2), (1561, 52, 256, 5), (641, 64, 64, 4),
                                          (90, 64, 64, 2)])
def test_block_shapes(gpu_lib, oracle_lib, m, n, mb, arity):
    L = gpu_lib
    A = np.asfortranarray(np.random.default_rng([m, n]).standard_normal((m, n)))
    dA, _, dQ = run_tsqr(L, A, 16, mb, arity)
    Rg, Qg = np.triu(L.from_device(dA)[:n]), L.from_device(dQ)
    Rh, Qh = _householder(oracle_lib, A)
    sg, sh = np.sign(np.diag(Rg)), np.sign(np.diag(Rh))
    assert C.max_rel(Rg * sg[:, None], Rh * sh[:, None]) < 1e-12
    assert C.max_rel(Qg * sg[None, :], Qh * sh[None, :]) < 1e-12


@pytest.mark.parametrize("power", [600, -600])
def test_extreme_column_scales(gpu_lib, power):
    L = gpu_lib
    m, n = 900, 24
    A = np.asfortranarray(np.random.default_rng(3).standard_normal((m, n)))
    k = np.where(np.arange(n) % 4 == 1, power, 0)
    Q0 = L.from_device(run_tsqr(L, A, 8, 128, 4)[2])
    dA, _, dQ = run_tsqr(L, np.asfortranarray(np.ldexp(A, k[None, :])), 8, 128, 4)
    Q1, R1 = L.from_device(dQ), np.triu(L.from_device(dA)[:n])
    assert C.max_rel(Q1, Q0) < 1e-12
    assert C.max_rel(Q1 @ np.ldexp(R1, -k[None, :]), A) < 1e-12
