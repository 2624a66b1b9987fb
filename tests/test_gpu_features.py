"""The selector's features at the edges of their size classes, row chunks and
panels, against the oracle.  Columns of norm near one, condition at most 10:
the condition estimate's relative error is below 100 n^2 2^-53 (FP32 rounding of
the output decides), a pivot's in FP32 below (m + n + 10) 2^-24 kappa^2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 64, 65, 87, 88, 89, 96, 97, 121, 128])
def test_feature_edges(gpu_lib, n):
    import selector as S
    import torch

    L = gpu_lib
    rng = np.random.default_rng(n)
    ms = sorted({max(2 * n, m) for m in (1, 15, 16, 17, 63, 64, 65, 255, 256, 257, 1000)})
    A = []
    for m in ms:
        Q, _ = np.linalg.qr(rng.standard_normal((m, n)))
        V, _ = np.linalg.qr(rng.standard_normal((n, n)))
        A.append(np.asfortranarray((Q * np.geomspace(1, 0.1, n)) @ V.T))
    A.append(np.zeros((2 * n, n), order="F"))  # singular: no estimate, no FP32 factor
    ms.append(2 * n)
    B = [np.zeros((m, 4), order="F") for m in ms]
    dA, dB = [L.to_device_colmajor(a) for a in A], [L.to_device_colmajor(b) for b in B]
    h = L.GelsMixed(ms, [n] * len(ms), 4, dA, ms, dB, ms)
    F = torch.full((len(ms), 5), 7.0, dtype=torch.float32, device="cuda")
    assert h.features(F) == 0
    torch.cuda.synchronize()
    F = F.cpu().numpy().astype(np.float64)
    h.close()
    for t, (m, a) in enumerate(zip(ms, A)):
        fo = S.features(a)
        assert abs(F[t, 0] - np.log2(m) / 12) < 1e-6 and abs(F[t, 1] - np.log2(n) / 7) < 1e-6
        if t + 1 == len(ms):
            assert F[t, 3] == 2.0 and F[t, 4] == 2.0
            continue
        assert abs(F[t, 3] - fo[3]) < 1e-6, (m, F[t], fo)
        G = np.linalg.cholesky(a.T @ a).diagonal()
        rel = (m + n + 10) * 2.0 ** -24 * 100
        assert abs(F[t, 4] - np.log10(G.max() / G.min()) / 3) < rel / 3 + 1e-6, (m, F[t], fo)
        c = np.linalg.norm(a, axis=0)
        assert abs(F[t, 2] - np.log10(c.max() / c.min()) / 4) < (m + 2) * 2.0 ** -24 / 4 + 1e-6, (m, F[t], fo)
