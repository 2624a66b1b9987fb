"""The batched FP64 least-squares solver's launches (a CTA per instance,
clusters of 8 or 4 CTAs for the large instances of a small batch) at the edges of panels, column
groups and row blocks, against the oracle's restatement of the reference
driver: V and R at the suite's elementwise tolerance, x within 64 kappa^2 u
(both are backward stable, the residual is not small; kappa from the singular
values)."""
import numpy as np
import pytest

import lila_cases as C

pytestmark = pytest.mark.gpu


def _solve(L, probs, nrhs, pad):
    import torch

    ld = [A.shape[0] + pad for A, _ in probs]
    dA, dB = [], []
    for (A, b), l in zip(probs, ld):
        dA.append(L.colmajor(l, A.shape[1], fill=3.0))
        dB.append(L.colmajor(l, nrhs, fill=3.0))
        dA[-1][: A.shape[0]].copy_(L.to_device_colmajor(A))
        dB[-1][: A.shape[0]].copy_(L.to_device_colmajor(b))
    ms, ns = [A.shape[0] for A, _ in probs], [A.shape[1] for A, _ in probs]
    nb = L.lib().lila_query_dgels_batched(len(probs))
    work = torch.empty(nb, dtype=torch.uint8, device="cuda")
    info = torch.full((len(probs),), -1, dtype=torch.int32, device="cuda")
    assert L.dgels_batched_prepare(len(probs), ms, ns, nrhs, dA, ld, dB, ld, work, nb) == 0
    L.trace(True)
    assert L.dgels_batched_run(len(probs), nrhs, work, info) == 0
    torch.cuda.synchronize()
    tr = L.trace_summary()
    L.trace(False)
    return [L.from_device(x) for x in dA], [L.from_device(x) for x in dB], info.cpu().numpy(), tr


SHAPES = [(1, 1), (8, 8), (9, 1), (17, 9), (33, 32), (64, 33), (300, 64), (257, 130), (520, 260), (2048, 8),
          (4097, 9), (1000, 128), (3001, 63)]


@pytest.mark.parametrize("nrhs,pad", [(1, 0), (4, 3), (8, 8)])
def test_routes_against_oracle(gpu_lib, oracle_lib, nrhs, pad):
    L = gpu_lib
    rng = np.random.default_rng(nrhs)
    probs = []
    for m, n in SHAPES:
        A = np.asfortranarray(rng.standard_normal((m, n)))
        probs.append((A, np.asfortranarray(rng.standard_normal((m, nrhs)))))
    gA, gB, info, _ = _solve(L, probs, nrhs, pad)
    for t, (A, b) in enumerate(probs):
        m, n = A.shape
        Ao, bo = A.copy(order="F"), b.copy(order="F")
        oracle_lib.ls_solve(m, n, nrhs, Ao, m, np.asfortranarray(np.zeros((n, n))), n, bo, m, np.zeros(n * nrhs))
        assert info[t] == 0
        assert C.max_rel(gA[t][:m], Ao) < C.TOL, (m, n)
        assert np.all(gA[t][m:] == 3.0) and np.all(gB[t][m:] == 3.0)
        kappa = np.linalg.cond(A)
        assert np.abs(gB[t][:n] - bo[:n]).max() / np.abs(bo[:n]).max() <= 64 * kappa * kappa * 2.0 ** -53 + 1e-13, (m, n)


@pytest.mark.parametrize("count", [3, 400, 1200])
def test_zero_and_extreme_columns(gpu_lib, count):
    """A zero column is reported, columns scaled by powers of two whose
    squares leave the FP64 range give the scaled solution (clusters of 8 for 3
    instances, of 4 for 400, one CTA each for 1,200)."""
    L = gpu_lib
    m, n, nrhs = 700, 40, 3
    rng = np.random.default_rng(9)
    A = np.asfortranarray(rng.standard_normal((m, n)))
    b = np.asfortranarray(rng.standard_normal((m, nrhs)))
    k = np.where(np.arange(n) % 5 == 2, 600, np.where(np.arange(n) % 5 == 3, -600, 0))
    Z = A.copy(order="F")
    Z[:, 17] = 0.0
    probs = [(A, b), (np.asfortranarray(np.ldexp(A, k[None, :])), b), (Z, b)] + [(A, b)] * (count - 3)
    gA, gB, info, _ = _solve(L, probs, nrhs, 0)
    assert info[0] == 0 and info[1] == 0 and info[2] == 18
    assert C.max_rel(np.tril(gA[1], -1), np.tril(gA[0], -1)) < C.TOL
    x0, x1 = gB[0][:n], np.ldexp(gB[1][:n], k[:, None])
    assert np.abs(x1 - x0).max() / np.abs(x0).max() < 64 * np.linalg.cond(A) ** 2 * 2.0 ** -53
    assert not np.isfinite(gB[2][:18]).any() and np.isfinite(gB[2][18:n]).all()
    for t in range(3, count):
        assert np.array_equal(gB[t], gB[3])
