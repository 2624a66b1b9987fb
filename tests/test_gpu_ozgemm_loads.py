"""The split-precision GEMM's unmasked loads (16-byte, 8-byte and tested per
element) at the edges where one gives way to the next: odd leading dimensions,
masks whose zeros reach into a tile, ragged tiles and K steps; against the
oracle's double-double product within the bound of test_gpu_ozgemm.py."""
import pytest

from test_gpu_ozgemm import run_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(128, 64, 32), (129, 65, 33), (256, 192, 160), (131, 64, 257), (64, 320, 130)])
@pytest.mark.parametrize("ta,tb,ma,mb", [(0, 0, 1, 0), (1, 0, 1, 1), (0, 1, 2, 2), (1, 1, 3, 4), (0, 0, 4, 3),
                                         (1, 1, 0, 1)])
def test_loads_at_edges(gpu_lib, oracle_lib, M, N, K, ta, tb, ma, mb):
    run_case(gpu_lib, oracle_lib, M, N, K, ta, tb, ma, mb, -1.0, 1.0, zero_rows=min(3, M), seed=M + N + K)


@pytest.mark.parametrize("M,N,K", [(640, 520, 512), (1101, 300, 450), (128, 2500, 500), (2100, 70, 1000)])
@pytest.mark.parametrize("ta,tb,ma,mb", [(0, 0, 1, 0), (1, 0, 1, 0), (0, 1, 0, 1), (1, 1, 3, 4)])
def test_operands_split_beforehand(gpu_lib, M, N, K, ta, tb, ma, mb):
    """Operands split once for all tiles (scratch with room for their digits,
    none for K slices) give the bits of the tiles' own splitting."""
    import numpy as np
    import torch

    L = gpu_lib
    rng = np.random.default_rng([M, N, K])
    As = np.asfortranarray(rng.standard_normal((K, M) if ta else (M, K)) * 10.0 ** rng.uniform(-3, 3, (1, M if ta else K)))
    Bs = np.asfortranarray(rng.standard_normal((N, K) if tb else (K, N)))
    dA, dB = L.to_device_colmajor(As), L.to_device_colmajor(Bs)
    up = lambda x, b: (x + b - 1) // b * b  # noqa: E731
    reused = (up(M, 128) if N > 192 else 0) + (up(N, 64) if M > 384 else 0)
    room = 2 * up(K, 32) * reused + 2 * (M + N) + 64
    out = []
    for plen in (0, room):
        part = torch.zeros(max(plen, 1), dtype=torch.float64, device="cuda")
        dC = L.colmajor(M, N, fill=0.5)
        L.trace(True)
        assert L.prim_ozgemm(M, N, K, dA, As.shape[0], ta, ma, dB, Bs.shape[0], tb, mb, dC, M, -1.0, 1.0, 2, 0, 0,
                             part if plen else None, plen) == 0
        torch.cuda.synchronize()
        tr = L.trace_summary()
        L.trace(False)
        assert ("ozgemm_pre_split" in tr) == bool(plen), tr
        out.append(L.from_device(dC))
    assert np.array_equal(out[0], out[1])
    assert L.gpu_status() == 0
