"""Split-precision products whose operands are both split beforehand and that need
no K slices (the persistent kernel): the bits of the tiles' own splitting, in every
form of the epilogue, from half a K stage to several windows of tensor memory, and
with operands that are not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

M, N = 2900, 2850  # ragged tiles; 2^27 multiply-adds from K = 17 on
ST_NONFINITE = 4


def _both(L, K, ta, tb, ma, mb, alpha, beta, zero_rows, add_diag, upper_only, spoil=None):
    import torch

    g = torch.Generator(device="cuda")
    g.manual_seed(K)
    # column-major: a (cols, rows) row-major tensor
    A = torch.randn((M, K) if ta else (K, M), generator=g, dtype=torch.float64, device="cuda")
    A *= torch.pow(10.0, 8.0 * torch.rand((A.shape[0], 1), generator=g, dtype=torch.float64, device="cuda") - 4.0)
    B = torch.randn((K, N) if tb else (N, K), generator=g, dtype=torch.float64, device="cuda")
    C0 = torch.randn(N, M, generator=g, dtype=torch.float64, device="cuda")
    if spoil:
        spoil(A, B)
    up = lambda x, b: (x + b - 1) // b * b  # noqa: E731
    room = 2 * up(K, 32) * (up(M, 128) + up(N, 64)) + 2 * (M + N) + 64
    out, st = [], []
    for plen in (0, room):
        part = torch.zeros(max(plen, 1), dtype=torch.float64, device="cuda")
        C = C0.clone()
        L.gpu_clear_status()
        L.trace(True)
        assert L.prim_ozgemm(M, N, K, A, A.shape[1], ta, ma, B, B.shape[1], tb, mb, C, M, alpha, beta, zero_rows,
                             add_diag, upper_only, part if plen else None, plen) == 0
        torch.cuda.synchronize()
        tr = L.trace_summary()
        L.trace(False)
        assert ("ozgemm_pre_split" in tr) == bool(plen) and "splitk_reduce" not in tr, tr
        out.append(C)
        st.append(L.gpu_status())
    L.gpu_clear_status()
    return A, B, C0, out, st


@pytest.mark.parametrize("K", [17, 33, 128, 129, 300])
@pytest.mark.parametrize("alpha,beta,zero_rows,add_diag,upper_only",
                         [(1.0, 0.0, 0, 0, 0), (-1.0, 1.0, 5, 0, 0), (1.0, 1.0, 0, 0, 1), (0.5, 0.0, 0, 0, 0),
                          (-1.0, 0.25, 130, 0, 1), (1.0, 0.0, 0, 1, 0), (-2.0, 1.0, 3, 1, 1)])
def test_epilogues(gpu_lib, K, alpha, beta, zero_rows, add_diag, upper_only):
    import torch

    A, B, C0, out, st = _both(gpu_lib, K, 1, 0, 0, 0, alpha, beta, zero_rows, add_diag, upper_only)
    assert st == [0, 0]
    assert torch.equal(out[0], out[1])
    # against the FP64 product, at the bound of test_gpu_ozgemm.py
    exp = alpha * (B @ A.t())
    a, b = A.abs(), B.abs()
    bound = abs(alpha) * 2.0 ** -50 * (b.sum(1)[:, None] * a.max(1).values[None, :] + b.max(1).values[:, None] * a.sum(1)[None, :])
    if add_diag:
        exp.diagonal().add_(1.0)
    keep = torch.ones(N, M, dtype=torch.bool, device="cuda")
    keep[:, :zero_rows] = False
    exp = exp + beta * C0 * keep
    bound += 2.0 ** -53 * (2.0 * K * abs(alpha) * (b @ a.t()) + 4.0 * exp.abs() + 4.0 * beta * C0.abs() + 4.0)
    if upper_only:
        low = torch.triu(torch.ones(N, M, dtype=torch.bool, device="cuda"), 1)  # row > column
        assert torch.equal(out[1][low], C0[low])
        exp, bound, got = exp[~low], bound[~low], out[1][~low]
    else:
        got = out[1]
    assert bool(((got - exp).abs() <= bound).all())


@pytest.mark.parametrize("ta,tb,ma,mb", [(0, 0, 1, 0), (0, 1, 2, 1), (1, 1, 3, 4)])
@pytest.mark.parametrize("K", [40, 200])
def test_transposes_and_masks(gpu_lib, K, ta, tb, ma, mb):
    import torch

    _, _, _, out, st = _both(gpu_lib, K, ta, tb, ma, mb, -1.0, 1.0, 2, 0, 0)
    assert st == [0, 0] and torch.equal(out[0], out[1])


@pytest.mark.parametrize("K", [64, 160])
def test_nonfinite_and_zero_operands(gpu_lib, K):
    """A row of op(A) with an infinity and a column of op(B) with a NaN give NaN
    there and a status; zero rows and columns give C."""
    import torch

    def spoil(A, B):
        A[7, 3] = np.inf
        B[1000, K - 1] = np.nan
        A[2899] = 0.0
        B[2849] = 0.0

    _, _, C0, out, st = _both(gpu_lib, K, 1, 0, 0, 0, -1.0, 1.0, 0, 0, 0, spoil)
    assert st[0] & ST_NONFINITE and st[0] == st[1]
    bad = torch.zeros(N, M, dtype=torch.bool, device="cuda")
    bad[:, 7] = True
    bad[1000] = True
    for C in out:
        assert torch.equal(torch.isnan(C), bad)
        assert torch.equal(C[:1000, 2899], C0[:1000, 2899]) and torch.equal(C[2849, 8:], C0[2849, 8:])
    assert torch.equal(torch.nan_to_num(out[0]), torch.nan_to_num(out[1]))
