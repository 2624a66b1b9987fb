"""The cooperative Householder panel on columns whose squares leave the FP64
range: scaled by powers of two, V and T are those of the unscaled matrix (against
the oracle's dgeqr3) and R's columns scale.  Zero columns among them are taken
twice too."""
import numpy as np
import pytest

import lila_cases as C

pytestmark = pytest.mark.gpu


def _panel(L, A):
    import torch

    m, n = A.shape
    dA, dT = L.to_device_colmajor(A), L.colmajor(n, n, fill=0.0)
    L.trace(True)
    assert L.dgeqr3(m, n, dA, m, dT, n) == 0
    torch.cuda.synchronize()
    tr = L.trace_summary()
    L.trace(False)
    assert "panel_coop" in tr, tr
    return L.from_device(dA), np.triu(L.from_device(dT))


@pytest.mark.parametrize("m,n", [(256, 2), (260, 10), (1000, 20), (300, 33), (4000, 64), (40001, 64)])
@pytest.mark.parametrize("power,every", [(600, 3), (-600, 3), (-600, 1), (-1040, 3), (1000, 1)])
def test_extreme_column_scales(gpu_lib, oracle_lib, m, n, power, every):
    L = gpu_lib
    A = np.asfortranarray(np.round(np.random.default_rng(m + n).standard_normal((m, n)) * 64) / 64)
    Ao, To = A.copy(order="F"), np.asfortranarray(np.zeros((n, n)))
    oracle_lib.dgeqr3(m, n, Ao, m, To, n)
    k = np.where(np.arange(n) % every == every - 1, power, 0)
    got, T = _panel(L, np.asfortranarray(np.ldexp(A, k[None, :])))
    V, Vo = np.tril(got, -1), np.tril(Ao, -1)
    R, Ro = np.ldexp(np.triu(got[:n]), -k[None, :]), np.triu(Ao[:n])
    # a scaled column whose updates stay above the subnormals keeps every bit it
    # has; below them its entries are rounded to multiples of 2^-1074 at every one
    # of up to n updates
    tol = C.TOL if power > -1000 else n * 2.0 ** (-1074 - power)
    assert C.max_rel(V, Vo) < tol
    assert C.max_rel(R, Ro) < tol
    assert C.max_rel(T, np.triu(To)) < tol


def test_zero_and_one_sided_columns(gpu_lib, oracle_lib):
    """A zero column (tau 0), one whose entries below the pivot vanish beside it
    when squared, and a panel of zeros."""
    L = gpu_lib
    m, n = 700, 24
    rng = np.random.default_rng(3)
    A = rng.standard_normal((m, n))
    A[:, 5] = 0.0
    A[:, 0] *= 2.0 ** -600
    A[0, 0] = 1.0
    A = np.asfortranarray(A)
    Ao, To = A.copy(order="F"), np.asfortranarray(np.zeros((n, n)))
    oracle_lib.dgeqr3(m, n, Ao, m, To, n)
    got, T = _panel(L, A)
    assert C.max_rel(got[1:, 0], Ao[1:, 0]) < C.TOL
    assert C.max_rel(got, Ao) < C.TOL and C.max_rel(T, np.triu(To)) < C.TOL
    got, T = _panel(L, np.asfortranarray(np.zeros((m, n))))
    assert not got.any() and not T.any()
