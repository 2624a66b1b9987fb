"""The work a user of lila_gb300 has it do, as timed cases.

A case is a dict of plain values.  Four families, by entry point:

  qr     lila_dgeqrf_w03_recursive (V, R, T and explicit Q of a general
         matrix), optionally followed by lila_dormqrf_z03 (Q^T C);
  apply  lila_dormqrf_w03: a block reflector applied to the columns beside it;
  tall   the tall-skinny leaves: Cholesky QR + reconstruction in FP64 (hr), the
         split-precision leaf (split, shift), the TSQR tree (tsqr);
  ls     batched least squares: the FP64 solver, the mixed variants with the
         caller's routes, and the learned selector.

Every factorization works in place, so a pass copies the caller's matrix into
the working buffer first, as a program that keeps its data does.
"""
import math

import numpy as np
import torch

import lila_gb300 as L

F64 = torch.float64


def listed():
    return [
        # the reference driver's default call (87 x 53, offset 6, tiles of 4 columns): launch latency
        {"name": "qr_87x53", "family": "qr", "m": 87, "n": 53, "i": 6, "mt": 4, "lda": 87, "ldq": 87, "leaf": 1,
         "panel": 1, "nx": 7, "precision": "fp64", "nrhs": 0, "decades": 0.0},
        # the reference's sweep shape: odd sizes, an offset, padded leading dimensions
        {"name": "qr_1413x692", "family": "qr", "m": 1413, "n": 692, "i": 97, "mt": 32, "lda": 1902, "ldq": 1809,
         "leaf": 1, "panel": 1, "nx": 64, "precision": "fp64", "nrhs": 0, "decades": 0.0},
        # a regression-sized dense problem: QR, explicit Q and Q^T applied to 64 right-hand sides
        {"name": "qr_4000x1000_qtc", "family": "qr", "m": 4000, "n": 1000, "i": 0, "mt": 256, "lda": 4000,
         "ldq": 4000, "leaf": 1, "panel": 1, "nx": 512, "precision": "fp64", "nrhs": 64, "decades": 0.0},
        # a large square matrix with graded columns, products on the tensor cores
        {"name": "qr_split_6000", "family": "qr", "m": 6000, "n": 6000, "i": 0, "mt": 128, "lda": 6000, "ldq": 6000,
         "leaf": 1, "panel": 1, "nx": 128, "precision": "split", "nrhs": 0, "decades": 6.0},
        # the trailing update that dominates a large factorization
        {"name": "apply_split_16384x8192", "family": "apply", "m": 16384, "n": 8192, "k": 128, "mt": 128,
         "precision": "split"},
        # a tall FP64 leaf (well-conditioned panels): Cholesky QR + reconstruction
        {"name": "tall_hr_262144x64", "family": "tall", "m": 262144, "n": 64, "mt": 64, "method": "hr",
         "log_kappa": 2.0},
        # a small tall leaf with an odd row count whose first pass the caller asks to be shifted
        {"name": "tall_shift_20001x48", "family": "tall", "m": 20001, "n": 48, "mt": 16, "method": "shift",
         "log_kappa": 3.0},
        # the headline: 4,194,304 x 64 on the tensor cores
        {"name": "tall_split_4194304x64", "family": "tall", "m": 4194304, "n": 64, "mt": 64, "method": "split",
         "log_kappa": 2.0},
        # the tree QR, for panels of unknown conditioning without split precision
        {"name": "tall_tsqr_131072x32", "family": "tall", "m": 131072, "n": 32, "mt": 32, "method": "tsqr",
         "log_kappa": 3.0},
        # uneven least squares, FP64 Householder in one persistent launch
        {"name": "ls_fp64_500", "family": "ls", "count": 500, "mmax": 4096, "nmax": 128, "nrhs": 4, "ld": 8,
         "solver": "fp64", "log_kappa": 4.0},
        # the same stream at serving size, routed by the caller's knowledge of the conditioning
        {"name": "ls_mixed_2000", "family": "ls", "count": 2000, "mmax": 4096, "nmax": 128, "nrhs": 4, "ld": 8,
         "solver": "mixed", "log_kappa": 4.0},
        # the learned selector: features, inference, routed solve
        {"name": "ls_learned_1000", "family": "ls", "count": 1000, "mmax": 4096, "nmax": 128, "nrhs": 4, "ld": 8,
         "solver": "learned", "log_kappa": 4.0},
    ]


def _between(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["qr", "qr", "qr_split", "apply", "hr", "shift", "split", "tsqr", "ls", "ls"])
    if kind == "qr":
        m = _between(rng, 64, 4000)
        n = _between(rng, 16, min(m - 1, 1000))
        i = rng.choice([0, 0, rng.randrange(0, max(1, min(100, m - n)))])
        return {"family": "qr", "m": m, "n": n, "i": i, "mt": _between(rng, 4, 256), "lda": m + rng.choice([0, 0, 3, 64]),
                "ldq": m + rng.choice([0, 0, 5, 32]), "leaf": rng.choice([0, 1, 1]), "panel": rng.choice([0, 1]),
                "nx": _between(rng, 8, 512), "precision": "fp64", "nrhs": rng.choice([0, 0, rng.randrange(1, 65)]),
                "decades": rng.choice([0.0, 6.0])}
    if kind == "qr_split":
        n = _between(rng, 1024, 5000)
        m = min(8192, int(n * rng.uniform(1.0, 1.6)))
        return {"family": "qr", "m": m, "n": n, "i": 0, "mt": rng.choice([64, 128]), "lda": m, "ldq": m, "leaf": 1,
                "panel": 1, "nx": rng.choice([64, 128, 256]), "precision": "split", "nrhs": 0, "decades": 6.0}
    if kind == "apply":
        k = _between(rng, 32, 256)
        n = _between(rng, 64, 8192)
        m = max(k + 1, _between(rng, 512, 16384))
        fp64 = m * n * k < 1 << 32 and rng.random() < 0.5
        return {"family": "apply", "m": m, "n": n, "k": k, "mt": rng.choice([32, 64, 128]),
                "precision": "fp64" if fp64 else "split"}
    if kind in ("hr", "shift", "split", "tsqr"):
        top = {"hr": 262144, "shift": 1048576, "split": 4194304, "tsqr": 131072}[kind]
        n = _between(rng, 8, 64)
        # a TSQR row block holds at most 16,384 entries
        if kind == "tsqr":
            n = min(n, 48)
        return {"family": "tall", "m": _between(rng, 10000, top), "n": n, "mt": rng.choice([16, 32, 64]),
                "method": kind, "log_kappa": rng.uniform(0.0, 2.0 if kind == "hr" else 4.0)}
    solver = rng.choice(["fp64", "mixed", "learned"])
    nmax = _between(rng, 16, 128)
    return {"family": "ls", "count": _between(rng, 60, {"fp64": 500, "mixed": 2000, "learned": 1000}[solver]),
            "mmax": _between(rng, 4 * nmax, 4096), "nmax": nmax, "nrhs": rng.randrange(1, 9), "ld": rng.choice([1, 8]),
            "solver": solver, "log_kappa": rng.uniform(1.0, 4.0)}


# ---------------------------------------------------------------------------
# inputs.  Matrices are kept as (columns, ld) row-major tensors: column-major
# storage, as the library takes it.
# ---------------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _randn(g, *shape):
    return torch.randn(shape, generator=g, dtype=F64, device="cuda")


def _zeros(*shape):
    return torch.zeros(shape, dtype=F64, device="cuda")


def _t_tiles(V, tau, i, mt):
    """T (n, mt) of the reflectors with unit lower V (n, m) and tau: the
    compact-WY factor D (I + striu(V^T V) D)^-1 of every tile of mt columns,
    tiles counted from the global column index."""
    n = V.shape[0]
    T = _zeros(n, mt)
    a = i
    while a < i + n:
        b = min((a // mt + 1) * mt, i + n)
        v, d = V[a - i:b - i], tau[a - i:b - i]
        S = torch.triu(v @ v.t(), 1)
        eye = torch.eye(b - a, dtype=F64, device="cuda")
        t = d[:, None] * torch.linalg.solve_triangular(eye + S * d[None, :], eye, upper=True)
        T[a - i:b - i, a % mt:a % mt + (b - a)] = t.t()
        a = b
    return T


def _householder(block):
    """LAPACK's Householder QR of a (n, m) column-major block in 64 bits:
    (V and R in one (n, m) block, V unit lower, tau, Q as (n, m))."""
    vr, tau = torch.geqrf(block.t())
    q = torch.linalg.householder_product(vr, tau)
    vr = vr.t().contiguous()
    V = torch.triu(vr, 1)
    V.diagonal().fill_(1.0)
    return vr, V, tau, q.t().contiguous()


def _qr_input(case, seed):
    g = _gen(seed)
    A0 = _randn(g, case["n"] + case["i"], case["lda"])
    if case["decades"]:
        j = torch.arange(case["n"] + case["i"], dtype=F64, device="cuda")
        A0 *= torch.pow(10.0, -case["decades"] * j / A0.shape[0])[:, None]
    return A0, _randn(g, case["nrhs"], case["m"])


def _tall_input(case, seed):
    """m x n with singular values log-spaced from about 1 to 1 / kappa."""
    m, n = case["m"], case["n"]
    g = _gen(seed)
    G = _randn(g, n, m)
    W, _ = torch.linalg.qr(_randn(g, n, n))
    sig = torch.pow(10.0, -case["log_kappa"] * torch.arange(n, dtype=F64, device="cuda") / max(1, n - 1))
    return (W * (sig / math.sqrt(m))[None, :]) @ G


def _apply_input(case, seed):
    g = _gen(seed)
    vr, V, tau, _ = _householder(_randn(g, case["k"], case["m"]))
    return vr, V, _t_tiles(V, tau, 0, case["mt"]), _randn(g, case["n"], case["m"])


def _ls_sizes(case):
    """m ~ U{max(2n, 64)..mmax}, n ~ U{4..nmax}, kappa log-uniform: the same
    shapes whatever the seed, as a stream of batches of one job has."""
    r = np.random.default_rng([case["count"], case["mmax"], case["nmax"]])
    n = r.integers(4, case["nmax"] + 1, case["count"])
    m = np.array([int(r.integers(min(max(2 * k, 64), case["mmax"]), case["mmax"] + 1)) for k in n])
    return m, n, r.uniform(0.0, case["log_kappa"], case["count"])


def _ls_chunks(case, seed, chunk=125):
    """The instances as zero-padded blocks (k, nmax, mmax): A^T = W diag(sigma) G
    with G Gaussian and W orthogonal (two reflections), b = A x + noise."""
    m, n, logk = _ls_sizes(case)
    g = _gen(seed)
    for c0 in range(0, case["count"], chunk):
        s = slice(c0, min(c0 + chunk, case["count"]))
        mt, nt = torch.as_tensor(m[s], device="cuda"), torch.as_tensor(n[s], device="cuda")
        mm, nn = int(m[s].max()), int(n[s].max())
        rows = (torch.arange(mm, device="cuda")[None, :] < mt[:, None]).to(F64)
        cols = (torch.arange(nn, device="cuda")[None, :] < nt[:, None]).to(F64)
        lk = torch.as_tensor(logk[s], device="cuda")
        sig = torch.pow(10.0, -lk[:, None] * torch.arange(nn, device="cuda") / (nt[:, None] - 1)) * cols
        A = _randn(g, len(mt), nn, mm) * (sig / torch.sqrt(mt[:, None].to(F64)))[:, :, None] * rows[:, None, :]
        for _ in range(2):
            w = _randn(g, len(mt), nn) * cols
            w = w / torch.linalg.vector_norm(w, dim=1, keepdim=True)
            A -= 2.0 * w[:, :, None] * torch.bmm(w[:, None, :], A)
        x = _randn(g, len(mt), case["nrhs"], nn) * cols[:, None, :]
        B = torch.bmm(x, A) + 1e-10 * _randn(g, len(mt), case["nrhs"], mm) * rows[:, None, :]
        yield s, m, n, A, B


def prepare(case, seed):
    s = {"case": case}
    fam = case["family"]
    if fam == "qr":
        m, n, i, mt = case["m"], case["n"], case["i"], case["mt"]
        s["A0"], s["C0"] = _qr_input(case, seed)
        s["lp"] = [0, case["leaf"], case["panel"], case["nx"]]
        s["A"], s["C"] = torch.empty_like(s["A0"]), torch.empty_like(s["C0"])
        s["T"], s["Q"] = _zeros(n + i, mt), _zeros(n + i, case["ldq"])
        lw = L.query_dgeqrf_w03_recursive(s["lp"], m, n, i, mt, None, case["lda"], None, mt, None, case["ldq"], None, -1)
        if case["nrhs"]:
            lw = max(lw, L.query_dormqrf_w03(m, case["nrhs"], n, i, 0, mt, None, case["lda"], None, mt, None, -1))
    elif fam == "apply":
        m, n, k, mt = case["m"], case["n"], case["k"], case["mt"]
        vr, _, s["T"], s["C0"] = _apply_input(case, seed)
        s["A"] = torch.cat([vr, s["C0"]])
        lw = L.query_dormqrf_w03(m, n, k, 0, k, mt, None, m, None, mt, None, -1)
    elif fam == "tall":
        m, n, mt = case["m"], case["n"], case["mt"]
        s["A0"] = _tall_input(case, seed)
        s["A"], s["T"], s["Q"] = torch.empty_like(s["A0"]), _zeros(n, mt), _zeros(n, m)
        if case["method"] == "hr":
            lw = L.query_dgeqrf_w03_mt_hr(m, n, 0, mt, None, m, None, mt, None, m, None, -1)
        elif case["method"] == "tsqr":
            lw = L.query_dgeqrf_w03_tsqr(0, 0, m, n, 0, mt)
        else:
            lw = L.query_dgeqrf_w03_mt_hr_mixed(m, n, 0, mt, None, m, None, mt, None, m, None, -1)
    else:
        return _prepare_ls(case, seed, s)
    s["lw"] = lw
    s["work"] = torch.empty(lw, dtype=F64, device="cuda")
    return s


def _prepare_ls(case, seed, s):
    count, nrhs, pad = case["count"], case["nrhs"], case["ld"]
    m, n, logk = _ls_sizes(case)
    ld = (m + pad - 1) // pad * pad
    off = np.concatenate([[0], np.cumsum(ld * n)])
    boff = np.concatenate([[0], np.cumsum(ld * nrhs)])
    A0, B0 = _zeros(int(off[-1])), _zeros(int(boff[-1]))
    for sl, _, _, A, B in _ls_chunks(case, seed):
        # pack: instance, column, row, each column ld long
        lds, ns = torch.as_tensor(ld[sl], device="cuda"), torch.as_tensor(n[sl], device="cuda")
        wide = max(A.shape[2], int(ld[sl].max()))
        keep_r = torch.arange(wide, device="cuda")[None, :] < lds[:, None]
        keep_c = torch.arange(A.shape[1], device="cuda")[None, :] < ns[:, None]
        A = torch.nn.functional.pad(A, (0, wide - A.shape[2]))
        B = torch.nn.functional.pad(B, (0, wide - B.shape[2]))
        A0[off[sl.start]:off[sl.stop]] = A[keep_c[:, :, None] & keep_r[:, None, :]]
        B0[boff[sl.start]:boff[sl.stop]] = B[keep_r[:, None, :].expand(-1, nrhs, -1)]
    s["A0"], s["B0"], s["A"], s["B"] = A0, B0, A0.clone(), B0.clone()
    aptr = [s["A"].data_ptr() + 8 * int(o) for o in off[:-1]]
    bptr = [s["B"].data_ptr() + 8 * int(o) for o in boff[:-1]]
    # where the solutions stand in B: rows 0..n-1 of every right-hand side, instance by instance
    at = [int(boff[t]) + int(ld[t]) * j for t in range(count) for j in range(nrhs)]
    k = torch.as_tensor(np.repeat(n, nrhs), device="cuda")
    start = torch.repeat_interleave(torch.as_tensor(at, device="cuda"), k)
    first = torch.repeat_interleave(torch.cumsum(k, 0) - k, k)
    s["at"] = start + torch.arange(len(start), device="cuda") - first
    mi, ni, li = [v.tolist() for v in (m, n, ld)]
    if case["solver"] == "fp64":
        nb = L.lib().lila_query_dgels_batched(count)
        s["work"] = torch.empty(nb, dtype=torch.uint8, device="cuda")
        s["info"] = torch.zeros(count, dtype=torch.int32, device="cuda")
        if L.dgels_batched_prepare(count, mi, ni, nrhs, aptr, li, bptr, li, s["work"], nb) != 0:
            raise RuntimeError("dgels_batched_prepare failed")
        return s
    s["h"] = L.GelsMixed(mi, ni, nrhs, aptr, li, bptr, li)
    if case["solver"] == "learned":
        from lila_gb300 import selector_train

        s["params"] = selector_train.load_params()
    else:
        # the caller's routes: Cholesky QR 2 for the better conditioned half, the shift for the rest, and the FP64
        # solver for one in ten
        s["route"] = [2 if t % 10 == 9 else int(logk[t] > case["log_kappa"] / 2) for t in range(count)]
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _ok(rc):
    if rc < 0:
        raise RuntimeError("return code %d" % rc)


def run(s):
    c = s["case"]
    if c["family"] == "qr":
        m, n, i, mt, lda, ldq = c["m"], c["n"], c["i"], c["mt"], c["lda"], c["ldq"]
        s["A"].copy_(s["A0"])
        if c["precision"] == "split":
            before = L.gpu_set_precision(1)
        _ok(L.dgeqrf_w03_recursive(s["lp"], m, n, i, mt, s["A"], lda, s["T"], mt, s["Q"], ldq, s["work"], s["lw"]))
        if c["precision"] == "split":
            L.gpu_set_precision(before)
        out = {"A": s["A"][i:, i:m], "T": s["T"][i:], "Q": s["Q"][i:, i:m]}
        if c["nrhs"]:
            s["C"].copy_(s["C0"])
            _ok(L.dormqrf_z03(m, c["nrhs"], n, i, 0, mt, s["A"], lda, s["T"], mt, s["C"], m, s["work"], s["lw"]))
            out["C"] = s["C"]
        return out
    if c["family"] == "apply":
        m, n, k, mt = c["m"], c["n"], c["k"], c["mt"]
        s["A"][k:].copy_(s["C0"])
        before = L.gpu_set_precision(1 if c["precision"] == "split" else 0)
        _ok(L.dormqrf_w03(m, n, k, 0, k, mt, s["A"], m, s["T"], mt, s["work"], s["lw"]))
        L.gpu_set_precision(before)
        return s["A"][k:]
    if c["family"] == "tall":
        m, n, mt = c["m"], c["n"], c["mt"]
        s["A"].copy_(s["A0"])
        a = (m, n, 0, mt, s["A"], m, s["T"], mt, s["Q"], m, s["work"], s["lw"])
        if c["method"] == "hr":
            _ok(L.dgeqrf_w03_mt_hr(*a))
        elif c["method"] == "tsqr":
            _ok(L.dgeqrf_w03_tsqr(0, 0, *a))
        elif c["method"] == "shift":
            _ok(L.dgeqrf_w03_mt_hr_mixed_v(2, *a))
        else:
            _ok(L.dgeqrf_w03_mt_hr_mixed(*a))
        return {"A": s["A"], "T": s["T"], "Q": s["Q"]}
    s["A"].copy_(s["A0"])
    s["B"].copy_(s["B0"])
    if c["solver"] == "fp64":
        _ok(L.dgels_batched_run(c["count"], c["nrhs"], s["work"], s["info"]))
        return {"x": s["B"][s["at"]], "info": s["info"]}
    if c["solver"] == "learned":
        rc, info, _, route = s["h"].solve(s["params"])
        _ok(rc)
        return {"x": s["B"][s["at"]], "info": np.array(info), "route": np.array(route)}
    rc, info, _ = s["h"].run(s["route"])
    _ok(rc)
    return {"x": s["B"][s["at"]], "info": np.array(info)}


# ---------------------------------------------------------------------------
# what a pass cannot do without, and what it returns in 64 bits
# ---------------------------------------------------------------------------
def work(case):
    if case["family"] == "qr":
        m, n, k = case["m"] - case["i"], case["n"], case["nrhs"]
        return {"bytes": 8.0 * (3 * m * n + n * min(n, case["mt"]) + 2 * m * k),
                "flops": 4.0 * m * n * n - 4.0 / 3.0 * n ** 3 + 4.0 * m * n * k - 2.0 * n * n * k}
    if case["family"] == "apply":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 8.0 * (2 * m * n + m * k), "flops": 4.0 * m * n * k - 2.0 * n * k * k}
    if case["family"] == "tall":
        m, n = case["m"], case["n"]
        return {"bytes": 24.0 * m * n, "flops": 4.0 * m * n * n - 4.0 / 3.0 * n ** 3}
    # mean sizes of the draw: n ~ U{4..nmax}, m ~ U{2n..mmax}
    n, k = (4 + case["nmax"]) / 2.0, case["nrhs"]
    m = (min(max(2 * n, 64), case["mmax"]) + case["mmax"]) / 2.0
    n2 = (case["nmax"] ** 2 + 4 * case["nmax"] + 16) / 3.0
    return {"bytes": case["count"] * 8.0 * (m * n + m * k + n * k),
            "flops": case["count"] * (2.0 * m * n2 - 2.0 / 3.0 * n * n2 + k * (4.0 * m * n - 2.0 * n2) + k * n2)}


def exact(case, seed):
    if case["family"] == "qr":
        A0, C0 = _qr_input(case, seed)
        i, m = case["i"], case["m"]
        vr, V, tau, Q = _householder(A0[i:, i:m])
        out = {"A": vr, "T": _t_tiles(V, tau, i, case["mt"]), "Q": Q}
        if case["nrhs"]:
            T = _t_tiles(V, tau, 0, case["n"])
            C = C0.clone()
            C[:, i:] -= ((C0[:, i:] @ V.t()) @ T.t()) @ V
            out["C"] = C
        return out
    if case["family"] == "apply":
        _, V, T, C = _apply_input(case, seed)
        for a in range(0, case["k"], case["mt"]):
            b = min(a + case["mt"], case["k"])
            t = T[a:b, :b - a]
            C = C - ((C @ V[a:b].t()) @ t.t()) @ V[a:b]
        return C
    if case["family"] == "tall":
        vr, V, tau, Q = _householder(_tall_input(case, seed))
        return {"A": vr, "T": _t_tiles(V, tau, 0, case["mt"]), "Q": Q}
    xs = []
    for s, _, n, A, B in _ls_chunks(case, seed):
        # Cholesky QR of the padded blocks (identity where there is no column), then refinement steps on the residual
        # that converge to rounding level
        nt = torch.as_tensor(n[s], device="cuda")
        pad = (torch.arange(A.shape[1], device="cuda")[None, :] >= nt[:, None]).to(F64)
        R = torch.linalg.cholesky(torch.bmm(A, A.transpose(1, 2)) + torch.diag_embed(pad))
        x = torch.zeros(B.shape[0], B.shape[1], A.shape[1], dtype=F64, device="cuda")
        for _ in range(4):
            r = B - torch.bmm(x, A)
            x = x + torch.cholesky_solve(torch.bmm(A, r.transpose(1, 2)), R).transpose(1, 2)
        keep = torch.arange(A.shape[1], device="cuda")[None, None, :] < nt[:, None, None]
        xs.append(x[keep.expand_as(x)])
    out = {"x": torch.cat(xs), "info": None}
    if case["solver"] == "learned":
        out["route"] = None
    return out
