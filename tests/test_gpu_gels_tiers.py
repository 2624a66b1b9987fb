"""The batched FP64 solver's three launches side by side, as they run untraced
(tracing records an event after each launch, which keeps them apart): every run
gives the bits of the traced one and the oracle's solutions, and the instances go
to the teams that the batch's work asks for."""
import numpy as np
import pytest

import lila_cases as C
from test_gpu_gels_routes import SHAPES

pytestmark = pytest.mark.gpu

# (m, n) of a batch, how many instances go to clusters of 8 and of 4 CTAs
BATCHES = {
    "all": (SHAPES, 6, 1),
    "eight": ([(700, 40)] * 3, 3, 0),
    "four": ([(700, 40)] * 400, 0, 400),
    "one": ([(700, 40)] * 1200, 0, 0),
    "mixed": ([(4096, 128)] * 2 + [(700, 40)] * 300 + [(300, 20)] * 500, 2, 300),
}


@pytest.mark.parametrize("batch", list(BATCHES))
def test_side_by_side(gpu_lib, oracle_lib, batch):
    import torch

    L = gpu_lib
    shapes, eight, four = BATCHES[batch]
    nrhs, count = 4, len(shapes)
    rng = np.random.default_rng(count)
    # a few distinct problems per shape, each checked against the oracle once
    made, probs = {}, []
    for t, s in enumerate(shapes):
        key = s + (t % 3,)
        if key not in made:
            made[key] = (np.asfortranarray(rng.standard_normal(s)), np.asfortranarray(rng.standard_normal((s[0], nrhs))))
        probs.append(key)
    src = {k: (L.to_device_colmajor(A), L.to_device_colmajor(b)) for k, (A, b) in made.items()}
    dA = [torch.empty_like(src[k][0]) for k in probs]
    dB = [torch.empty_like(src[k][1]) for k in probs]
    ms, ns = [s[0] for s in shapes], [s[1] for s in shapes]
    nb = L.lib().lila_query_dgels_batched(count)
    work = torch.empty(nb, dtype=torch.uint8, device="cuda")
    info = torch.full((count,), -1, dtype=torch.int32, device="cuda")
    assert L.dgels_batched_prepare(count, ms, ns, nrhs, dA, ms, dB, ms, work, nb) == 0
    # the bounds of the launches' instances behind their three counters
    bounds = work[12:28].view(torch.int32).tolist()
    assert bounds == [0, eight, eight + four, count]

    def run(traced):
        for k, a, b in zip(probs, dA, dB):
            a.copy_(src[k][0])
            b.copy_(src[k][1])
        info.fill_(-1)
        torch.cuda.synchronize()
        if traced:
            L.trace(True)
        assert L.dgels_batched_run(count, nrhs, work, info) == 0
        torch.cuda.synchronize()
        if traced:
            tr = L.trace_summary()
            L.trace(False)
            # both cluster launches were accepted
            assert tr["gels_batched_clusters"][0] == 2 and tr["gels_batched"][0] == 1, tr
        assert not info.any().item()
        return [x.clone() for x in dA], [x.clone() for x in dB]

    A1, B1 = run(True)
    for _ in range(4):
        A, B = run(False)
        assert all(torch.equal(x, y) for x, y in zip(A + B, A1 + B1))
    for k in made:
        t = probs.index(k)
        m, n = shapes[t]
        Ao, bo = made[k][0].copy(order="F"), made[k][1].copy(order="F")
        oracle_lib.ls_solve(m, n, nrhs, Ao, m, np.asfortranarray(np.zeros((n, n))), n, bo, m, np.zeros(n * nrhs))
        assert C.max_rel(L.from_device(A1[t]), Ao) < C.TOL, (m, n)
        kappa = np.linalg.cond(made[k][0])
        x = L.from_device(B1[t])[:n]
        assert np.abs(x - bo[:n]).max() / np.abs(bo[:n]).max() <= 64 * kappa * kappa * 2.0 ** -53 + 1e-13, (m, n)
