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
