"""Split-precision products whose K exceeds what one grid dimension counts in
steps (65,535 of 32 values for the digits, of 64 for the scales): operands split
beforehand give the bits of the tiles' own splitting, and no launch is refused."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [2097120, 2097121, 4194337])
def test_more_steps_than_a_grid_dimension(gpu_lib, K):
    import torch

    L = gpu_lib
    M, N = 16, 256
    g = torch.Generator(device="cuda")
    g.manual_seed(K)
    A = torch.randn(M, K, generator=g, dtype=torch.float64, device="cuda")  # column-major K x M
    B = torch.randn(N, K, generator=g, dtype=torch.float64, device="cuda")
    # room for op(A)'s digits and scales, none for K slices
    room = 2 * ((K + 31) // 32 * 32) * 128 + 64 * M // 2 + 64
    out = []
    L.gpu_clear_status()
    for plen in (0, room):
        part = torch.zeros(max(plen, 1), dtype=torch.float64, device="cuda")
        C = torch.zeros(N, M, dtype=torch.float64, device="cuda")
        L.trace(True)
        assert L.prim_ozgemm(M, N, K, A, K, 1, 0, B, K, 0, 0, C, M, 1.0, 0.0, 0, 0, 0, part if plen else None,
                             plen) == 0
        torch.cuda.synchronize()
        tr = L.trace_summary()
        L.trace(False)
        assert ("ozgemm_pre_split" in tr) == bool(plen), tr
        out.append(C)
    assert torch.equal(out[0], out[1])
    assert L.gpu_status() == 0
    # the bound of an entry plus the FP64 product's own rounding
    ref = B @ A.t()
    assert float((out[0] - ref).abs().max()) <= 2.0 ** -48 * 8 * K
