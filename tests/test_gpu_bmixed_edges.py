"""The mixed least-squares variants at the edges of their Cholesky factors (size
classes, halves of the inverse, four substitution entries per lane).  For kappa =
10 a backward-stable solution is within 40 sqrt(m) n u (kappa + kappa^2 |r| /
(|A| |x|)) of the exact one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


@pytest.mark.parametrize("nrhs", [1, 8])
@pytest.mark.parametrize("variant", [0, 1])
def test_variants_at_size_edges(gpu_lib, variant, nrhs):
    import torch

    L = gpu_lib
    rng = np.random.default_rng([variant, nrhs])
    ns = [1, 2, 3, 4, 5, 15, 16, 17, 31, 32, 33, 47, 63, 64, 65, 95, 96, 97, 127, 128]
    ms = [max(2 * n, 64) + (n % 3) for n in ns]
    probs = []
    for m, n in zip(ms, ns):
        Q, _ = np.linalg.qr(rng.standard_normal((m, n)))
        V, _ = np.linalg.qr(rng.standard_normal((n, n)))
        A = np.asfortranarray((Q * np.geomspace(1, 0.1, n)) @ V.T)
        x = rng.standard_normal((n, nrhs))
        probs.append((A, np.asfortranarray(A @ x + 1e-3 * rng.standard_normal((m, nrhs)))))
    dA = [L.to_device_colmajor(a) for a, _ in probs]
    dB = [L.to_device_colmajor(b) for _, b in probs]
    h = L.GelsMixed(ms, ns, nrhs, dA, ms, dB, ms)
    fails, info, orth = h.run([variant] * len(ns))
    torch.cuda.synchronize()
    assert fails == 0 and np.all(np.asarray(info) == 0)
    for t, (A, b) in enumerate(probs):
        m, n = A.shape
        x = L.from_device(dB[t])[:n]
        ref = np.linalg.lstsq(A, b, rcond=None)[0]
        for j in range(nrhs):
            nx = np.linalg.norm(ref[:, j])
            lim = 40 * np.sqrt(m) * n * U * (10 + 100 * np.linalg.norm(b[:, j] - A @ ref[:, j]) / nx)
            assert np.linalg.norm(x[:, j] - ref[:, j]) <= lim * nx, (n, j)
    h.close()
