"""Benchmark: tall-skinny QR through the lila C ABI on one GB300.

Workload: the tall-skinny Cholesky QR + Householder reconstruction leaf of
the w03 interface on A = U diag(sigma) V^T, m = 4,194,304, n = 64, mt = 32
(U = Q factor of a seeded Gaussian, V Haar-random, sigma log-spaced 1 ->
1/kappa, kappa cycled over 1e2, 1e6, 1e10, 1e14; synthetic, seeds 201/202).
One step = one factorization (V and S*R into A, T tiles, explicit Q*S) of a
fresh, already-resident copy of A; every copy is 2.1 GB, far larger than the
129 MB L2, so no L2 flush is needed between steps.

value: the split-precision leaf lila_dgeqrf_w03_mt_hr_mixed (FP64-grade
accuracy, checked per kappa), GFLOP/s credited with the Householder count
4mn^2 - 4/3 n^3 (lila-c/main_w03.c:200), plus matrices/s.  plain_fp64: the
reference-structured FP64 leaf lila_dgeqrf_w03_mt_hr on the same inputs.
e2e: the mixed call with the input copied from pinned host memory and V/R/Q
copied back inside the timed region; over a stream of matrices the copies of
neighbouring steps overlap the factorization on two copy streams.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
"""
import argparse
import gc
import json
import os
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
for _p in (ROOT, os.path.join(ROOT, "oracle")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

METRIC = "QR GFLOP/s & mats/s at FP64-grade accuracy: mixed vs plain FP64, 1 GB300"


# DRAM bytes of one k_ozaki_map launch per row of A (64 columns): the ncu
# capture of a 1,048,576 x 64 launch read 537.0 MB and wrote 485.3 MB; the
# kernel streams its rows once, so the traffic grows in proportion to m.
MAP_DRAM_BYTES_PER_ROW = (537.0e6 + 485.3e6) / 1048576


def credited_flops(m, n):
    return 4.0 * m * n * n - 4.0 / 3.0 * n ** 3


def load_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f), "measured"
    except OSError:
        return {"hbm_gbs": 6800.0, "bf16_tflops": 1900.0, "bf16_tflops_sustained": 1700.0}, "fallback"


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
_UV_CACHE = {}


def _uv_factors(m, n, seed_u, seed_v):
    """U = Q of a seeded m x n Gaussian, V Haar n x n (host numpy, computed once)."""
    import numpy as np

    key = (m, n, seed_u, seed_v)
    if key not in _UV_CACHE:
        rng = np.random.default_rng(seed_u)
        U, _ = np.linalg.qr(rng.standard_normal((m, n)))
        rv = np.random.default_rng(seed_v)
        V, Rv = np.linalg.qr(rv.standard_normal((n, n)))
        V = V * np.sign(np.diag(Rv))[None, :]
        _UV_CACHE[key] = (np.asfortranarray(U), V)
    return _UV_CACHE[key]


def make_tall_input_torch(m, n, kappa, seed_u=201, seed_v=202, device="cuda"):
    """A = U diag(sigma) V^T as a column-major device matrix (cuBLAS matmul only)."""
    import torch

    U_np, V_np = _uv_factors(m, n, seed_u, seed_v)
    U = torch.from_numpy(U_np.T.copy()).to(device).t()
    V = torch.from_numpy(V_np).to(device)
    sig = torch.tensor([kappa ** (-j / (n - 1)) for j in range(n)], dtype=torch.float64, device=device)
    A = (U * sig.unsqueeze(0)) @ V.t()
    out = torch.empty((n, m), dtype=torch.float64, device=device).t()
    out.copy_(A)
    del U, A
    return out


def make_tall_input_numpy(m, n, kappa, seed_u=201, seed_v=202):
    import numpy as np

    rng = np.random.default_rng(seed_u)
    U, _ = np.linalg.qr(rng.standard_normal((m, n)))
    rv = np.random.default_rng(seed_v)
    V, Rv = np.linalg.qr(rv.standard_normal((n, n)))
    V = V * np.sign(np.diag(Rv))[None, :]
    sig = np.array([kappa ** (-j / (n - 1)) for j in range(n)])
    return np.asfortranarray((U * sig[None, :]) @ V.T)


# ---------------------------------------------------------------------------
# clocks
# ---------------------------------------------------------------------------
class ClockSampler:
    """nvidia-smi samples every 100 ms from start() to stop(); stop(window)
    keeps the samples whose timestamps fall in the window (host wall-clock
    datetimes around the timed region), all of them if none does."""
    FIELDS = ("timestamp,index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index=0):
        self.proc = None
        self.lines = []
        self.gpu = gpu_index

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), "--query-gpu=" + self.FIELDS, "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self, window=None):
        import datetime as _dt

        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        samples = []
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 10:
                continue
            try:
                ts = _dt.datetime.strptime(parts[0], "%Y/%m/%d %H:%M:%S.%f")
                smv, smaxv = float(parts[2]), float(parts[3])
            except ValueError:
                continue
            samples.append((ts, smv, smaxv, {nm for nm, v in zip(names, parts[6:10]) if v.lower() == "active"}))
        if not samples:
            return None
        inside = samples
        where = "sampler run"
        if window is not None:
            pad = _dt.timedelta(milliseconds=50)
            sel = [x for x in samples if window[0] - pad <= x[0] <= window[1] + pad]
            if sel:
                inside, where = sel, "timed region"
        sm = sorted(x[1] for x in inside)
        reasons = set().union(*[x[3] for x in inside])
        return {"sm_mhz": sm[len(sm) // 2], "sm_max_mhz": max(x[2] for x in inside), "reasons": sorted(reasons),
                "samples": len(inside), "samples_from": where}


# ---------------------------------------------------------------------------
# CPU baseline and reference arm: the reference's algorithms restated in C
# (oracle/lila_oracle.c, pinned elementwise against the reference compiled
# from its own sources) on scipy's OpenBLAS, all host cores.  The compiled
# reference itself cannot run on the Arm GPU host (built here for x86-64, and
# its sources are not there); the restatement is its stand-in ("port").
# ---------------------------------------------------------------------------
CPU_HH = {"leaf": 1, "panel": 1, "mt": 200, "nx": 20}    # the reference's best family (FP64 Householder)
CPU_HR = {"leaf": 2, "panel": 0, "mt": 32, "nx": 64}     # its Cholesky QR + reconstruction leaf


def _cpu_lib():
    import oracle as O

    lib = O.load("oracle_ob")
    if lib is not None:
        return lib, "on scipy's OpenBLAS"
    return O.load("oracle"), "on its own BLAS loops (OpenMP)"


def _cpu_factor(lib, A0, fam):
    """One lila_dgeqrf_w03_recursive of the restatement with the family's
    leaf / panel / mt / nx; returns seconds and the outputs."""
    import numpy as np

    import oracle as O

    m, n = A0.shape
    lp = O.lila_param(fam["leaf"], fam["panel"], fam["nx"])
    lw = lib.query_dgeqrf_w03_recursive(lp, m, n, 0, fam["mt"]) + 4 * (m + n) + n * n
    A = A0.copy(order="F")
    T = np.zeros((fam["mt"], n), order="F")
    Q = np.zeros((m, n), order="F")
    W = np.zeros(lw)
    t0 = time.perf_counter()
    lib.dgeqrf_w03_recursive(lp, m, n, 0, fam["mt"], A, m, T, fam["mt"], Q, m, W, lw)
    t = time.perf_counter() - t0
    return t, A, Q


def _cpu_accuracy(A0, A, Q):
    import numpy as np

    n = A0.shape[1]
    R = np.triu(A[:n, :n])
    with np.errstate(all="ignore"):
        res = float(np.linalg.norm(Q @ R - A0) / np.linalg.norm(A0))
        orth = float(np.linalg.norm(np.eye(n) - Q.T @ Q))
    return res, orth


def cpu_baseline(m, n, kappa, reps=2):
    """The FP64 Householder leaf on one full-size matrix (1 warm-up + reps
    timed), beside the Cholesky QR + reconstruction leaf on the same matrix."""
    lib, how = _cpu_lib()
    A0 = make_tall_input_numpy(m, n, kappa)
    times = []
    for r in range(reps + 1):
        t, A, Q = _cpu_factor(lib, A0, CPU_HH)
        if r:
            times.append(t)
    t = sorted(times)[len(times) // 2]
    res, orth = _cpu_accuracy(A0, A, Q)
    th, Ah, Qh = _cpu_factor(lib, A0, CPU_HR)
    rh, oh = _cpu_accuracy(A0, Ah, Qh)
    cores = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else os.cpu_count()
    tol = 50 * n * 2.0 ** -53
    return {
        "value": credited_flops(m, n) / t / 1e9,
        "unit": "GFLOP/s",
        "cores": cores,
        "kind": "port",
        "sample": "the reference's FP64 Householder QR (lila_dgeqrf_w03_recursive, leaf 1, panel 1, mt 200, nx 20) "
                  "restated in C %s, one full %d x %d matrix at kappa %g, median of %d after 1 warm-up, "
                  "OPENBLAS threads %s" % (how, m, n, kappa, reps, os.environ.get("OPENBLAS_NUM_THREADS", cores)),
        "seconds_per_matrix": t,
        "accuracy": {"res": res, "orth": orth, "tol": tol, "meets_gate": res <= tol and orth <= tol},
        "cholqr_hr_leaf": {"gflops": credited_flops(m, n) / th / 1e9, "seconds": th, "res": rh, "orth": oh,
                           "meets_gate": rh <= tol and oh <= tol,
                           "call": "leaf 2 (lila_dgeqrf_w03_mt_hr), mt 32, nx 64"},
    }


# ---------------------------------------------------------------------------
# GPU arm
# ---------------------------------------------------------------------------
KAPPAS = (1e2, 1e6, 1e10, 1e14)


def _fro(torch, X):
    return float(torch.sqrt((X * X).sum()))


def _accuracy(torch, Af, Q, base, n):
    R = torch.triu(Af[:n, :n])
    res = _fro(torch, Q @ R - base) / _fro(torch, base)
    orth = _fro(torch, torch.eye(n, dtype=torch.float64, device="cuda") - Q.t() @ Q)
    return res, orth


def run_ours(args, rank, world):
    import torch

    import lila_gb300 as L

    torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", "0")))
    L.lib()
    L.prim_ozaki_map_path(args.map_path)
    m, n, mt = args.m, args.n, args.mt
    kappas = KAPPAS if args.kappa is None else (args.kappa,)
    bases = [make_tall_input_torch(m, n, k) for k in kappas]
    nk = len(kappas)
    T = L.colmajor(mt, n, fill=0.0)
    Q = L.colmajor(m, n, fill=0.0)
    lw_mixed = L.query_dgeqrf_w03_mt_hr_mixed(m, n, 0, mt, None, m, None, mt, None, m, None, -1)
    lw_plain = L.query_dgeqrf_w03_mt_hr(m, n, 0, mt, None, m, None, mt, None, m, None, -1)
    W = torch.empty(max(lw_mixed, lw_plain), dtype=torch.float64, device="cuda")
    stream = torch.cuda.current_stream()

    def fresh(count, start):
        out = []
        for s in range(count):
            b = torch.empty((n, m), dtype=torch.float64, device="cuda").t()
            b.copy_(bases[(start + s) % nk])
            out.append(b)
        return out

    def mixed(A):
        rc = L.dgeqrf_w03_mt_hr_mixed(m, n, 0, mt, A, m, T, mt, Q, m, W, lw_mixed)
        assert rc == 0, rc

    def plain(A):
        rc = L.dgeqrf_w03_mt_hr(m, n, 0, mt, A, m, T, mt, Q, m, W, lw_plain)
        assert rc == 0, rc

    # ---- mixed (headline): fresh resident copy of A per step, kappas cycled
    L.gpu_clear_status()
    bufs = fresh(args.warmup, 0)
    for b in bufs:
        mixed(b)
    del bufs
    # the clock sampler starts before the inputs are copied, so that it is
    # sampling when the timed region begins
    clocks = ClockSampler(int(os.environ.get("LOCAL_RANK", "0")))
    clocks.start()
    bufs = fresh(args.steps, 0)
    torch.cuda.synchronize()
    if world > 1:
        import torch.distributed as dist

        dist.barrier()
    L.trace(True)
    l0 = L.launch_count()
    evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
    torch.cuda.synchronize()
    import datetime as _dt

    gc.collect()
    gc.disable()
    w0 = _dt.datetime.now()
    evs[0].record(stream)
    for s in range(args.steps):
        mixed(bufs[s])
        evs[s + 1].record(stream)
    torch.cuda.synchronize()
    w1 = _dt.datetime.now()
    gc.enable()
    launches = L.launch_count() - l0
    trace = L.trace_summary()
    L.trace(False)
    clk = clocks.stop((w0, w1))
    ms = evs[0].elapsed_time(evs[-1]) / args.steps
    per_kappa_ms = {}
    for s in range(args.steps):
        per_kappa_ms.setdefault("%g" % kappas[s % nk], []).append(evs[s].elapsed_time(evs[s + 1]))
    if world > 1:
        import torch.distributed as dist

        t = torch.tensor([ms], dtype=torch.float64, device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    status_mixed = L.gpu_status()
    # accuracy of one factorization per kappa (FP64 torch products, reporting only)
    acc_mixed = {}
    for k, base in zip(kappas, bases):
        A1 = torch.empty((n, m), dtype=torch.float64, device="cuda").t()
        A1.copy_(base)
        mixed(A1)
        res, orth = _accuracy(torch, A1, Q, base, n)
        cres, corth = L.gpu_last_check()
        acc_mixed["%g" % k] = {"res": res, "orth": orth, "passes": L.gpu_last_passes(),
                               "shifted": L.gpu_last_variant() == 2, "device_check_res": cres,
                               "device_check_orth": corth, "fp64_fallback": L.gpu_last_fallback()}
        del A1
    del bufs
    # cost of the on-device check: the same steps with the check off
    prev_check = L.gpu_set_check(0)
    try:
        nb = fresh(nk, 0)
        torch.cuda.synchronize()
        c0 = torch.cuda.Event(enable_timing=True)
        c1 = torch.cuda.Event(enable_timing=True)
        c0.record(stream)
        for b in nb:
            mixed(b)
        c1.record(stream)
        torch.cuda.synchronize()
        ms_nocheck = c0.elapsed_time(c1) / nk
        del nb
    finally:
        L.gpu_set_check(prev_check)
    # the same steps with the check on and the per-launch event trace off
    nb = fresh(nk, 0)
    torch.cuda.synchronize()
    c0 = torch.cuda.Event(enable_timing=True)
    c1 = torch.cuda.Event(enable_timing=True)
    c0.record(stream)
    for b in nb:
        mixed(b)
    c1.record(stream)
    torch.cuda.synchronize()
    ms_untraced = c0.elapsed_time(c1) / nk
    del nb
    check_cost = {"ms_per_step_without_check": ms_nocheck, "ms_per_step_untraced": ms_untraced,
                  "ms_per_step_with_check": sum(sum(v) for v in per_kappa_ms.values()) / args.steps,
                  "what": "level 1: orthogonality from the last pass's Gram (n x n), residual over 8192 "
                          "sampled rows; a failure re-solves in FP64 (TSQR)"}

    # ---- plain FP64 drop-in (reference-structured lila_dgeqrf_w03_mt_hr)
    plain_res = None
    if not args.no_plain:
        psteps = max(1, min(args.steps, args.plain_steps))
        pb = fresh(1 + psteps, 0)
        plain(pb[0])
        torch.cuda.synchronize()
        p0 = torch.cuda.Event(enable_timing=True)
        p1 = torch.cuda.Event(enable_timing=True)
        p0.record(stream)
        for s in range(psteps):
            plain(pb[1 + s])
        p1.record(stream)
        torch.cuda.synchronize()
        pms = p0.elapsed_time(p1) / psteps
        # Q holds the last plain step's factor; that step factored pb[psteps]
        last = psteps % nk
        res, orth = _accuracy(torch, pb[psteps], Q, bases[last], n)
        acc_plain = {"%g" % kappas[last]: {"res": res, "orth": orth}}
        del pb
        plain_res = {"value": credited_flops(m, n) / (pms * 1e-3) / 1e9, "unit": "GFLOP/s", "ms_per_step": pms,
                     "steps": psteps, "accuracy_last_step": acc_plain,
                     "path": "lila_dgeqrf_w03_mt_hr (FP64 CUDA cores, reference algorithm)"}

    # ---- FP64 TSQR leaf: row-block Householder QRs and a reduction tree of
    # R factors (the reference's tree QR, tsqr/main_test_tsqr.c:234-395),
    # then the Householder reconstruction; the row-block size and the tree
    # arity come from lila_gpu_tsqr_autotune on this shape (untimed)
    tsqr_res = None
    if not args.no_plain:
        tsteps = max(1, min(args.steps, args.plain_steps))
        lw_ts = max(L.query_dgeqrf_w03_tsqr(b_, a_, m, n, 0, mt) for b_ in (128, 256) for a_ in (2, 4))
        W_ts = torch.empty(lw_ts, dtype=torch.float64, device="cuda")
        tb = fresh(1, 0)
        code = L.gpu_tsqr_autotune(m, n, tb[0], m, T, mt, Q, m, W_ts, lw_ts)
        t_mb, t_ar = code // 100, code % 100
        tb = fresh(1 + tsteps, 0)

        def tsqr(A):
            rc = L.dgeqrf_w03_tsqr(t_mb, t_ar, m, n, 0, mt, A, m, T, mt, Q, m, W_ts, lw_ts)
            assert rc == 0, rc

        tsqr(tb[0])
        torch.cuda.synchronize()
        t0 = torch.cuda.Event(enable_timing=True)
        t1 = torch.cuda.Event(enable_timing=True)
        t0.record(stream)
        for s in range(tsteps):
            tsqr(tb[1 + s])
        t1.record(stream)
        torch.cuda.synchronize()
        tms = t0.elapsed_time(t1) / tsteps
        last = tsteps % nk
        res, orth = _accuracy(torch, tb[tsteps], Q, bases[last], n)
        del tb, W_ts
        tsqr_res = {"value": credited_flops(m, n) / (tms * 1e-3) / 1e9, "unit": "GFLOP/s", "ms_per_step": tms,
                    "steps": tsteps, "mb": t_mb, "arity": t_ar,
                    "accuracy_last_step": {"%g" % kappas[last]: {"res": res, "orth": orth}},
                    "path": "lila_dgeqrf_w03_tsqr (FP64 tree QR + reconstruction, mb / arity autotuned)"}

    # ---- e2e: host buffers, copies inside the timed region.  A stream of
    # matrices, the condition numbers cycled: step i's input copy (pinned
    # host -> device) and its two output copies (V/R and Q, device -> pinned
    # host) run on three copy streams while other steps factor, over four
    # device slots, so that an input copy rarely waits for the slot's
    # previous outputs to leave; input copies are enqueued three steps ahead
    # (the leaf blocks the host once, when it reads its check values).  The
    # timed region runs from before the first input copy to after the last
    # output copy.
    e2e = None
    out_of_core = None
    if not args.no_e2e:
        e2e_steps = max(32, args.steps)
        nslot = 4
        hA = []
        for k in range(nk):
            h = torch.empty((n, m), dtype=torch.float64, pin_memory=True).t()
            h.copy_(bases[k].cpu())
            hA.append(h)
        hA_out = [torch.empty((n, m), dtype=torch.float64, pin_memory=True).t() for _ in range(2)]
        hQ_out = [torch.empty((n, m), dtype=torch.float64, pin_memory=True).t() for _ in range(2)]
        dAs = [torch.empty((n, m), dtype=torch.float64, device="cuda").t() for _ in range(nslot)]
        Qs = [Q] + [L.colmajor(m, n, fill=0.0) for _ in range(nslot - 1)]

        def mixed_q(A, Qb):
            rc = L.dgeqrf_w03_mt_hr_mixed(m, n, 0, mt, A, m, T, mt, Qb, m, W, lw_mixed)
            assert rc == 0, rc

        # copy rates of this host link, each direction alone
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        for _ in range(2):
            e0.record(stream)
            dAs[0].copy_(hA[0], non_blocking=True)
            e1.record(stream)
            torch.cuda.synchronize()
        h2d_gbs = 8.0 * m * n / (e0.elapsed_time(e1) * 1e-3) / 1e9
        for _ in range(2):
            e0.record(stream)
            hA_out[0].copy_(dAs[0], non_blocking=True)
            hQ_out[0].copy_(dAs[0], non_blocking=True)
            e1.record(stream)
            torch.cuda.synchronize()
        d2h_gbs = 16.0 * m * n / (e0.elapsed_time(e1) * 1e-3) / 1e9
        mixed_q(dAs[0], Qs[0])
        torch.cuda.synchronize()
        s_h2d, s_d2h, s_d2h_q = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
        ahead = nslot - 1
        # one step's copies all at once (an input copy in, V/R and Q out, on
        # the pipeline's three copy streams): the floor of a pipeline whose
        # copies always overlap
        both_ms = []
        for _ in range(2):
            torch.cuda.synchronize()
            e0.record(stream)
            for cs in (s_h2d, s_d2h, s_d2h_q):
                cs.wait_event(e0)
            with torch.cuda.stream(s_h2d):
                dAs[1].copy_(hA[1 % nk], non_blocking=True)
            with torch.cuda.stream(s_d2h):
                hA_out[1].copy_(dAs[2], non_blocking=True)
            with torch.cuda.stream(s_d2h_q):
                hQ_out[1].copy_(dAs[3], non_blocking=True)
            for cs in (s_h2d, s_d2h, s_d2h_q):
                ev = torch.cuda.Event()
                ev.record(cs)
                stream.wait_event(ev)
            e1.record(stream)
            torch.cuda.synchronize()
            both_ms.append(e0.elapsed_time(e1))
        both_ms = min(both_ms)

        gaps = []

        def pipeline(steps):
            """steps matrices through the copy / factor pipeline; returns the
            device time from before the first input copy to after the last
            output copy, in ms."""
            ev_h2d = [torch.cuda.Event() for _ in range(steps)]
            ev_done = [torch.cuda.Event() for _ in range(steps)]
            ev_out = [torch.cuda.Event() for _ in range(steps)]
            ev_out_q = [torch.cuda.Event(enable_timing=True) for _ in range(steps)]

            def h2d(i):
                if i >= nslot:
                    # the slot's previous outputs have left
                    s_h2d.wait_event(ev_out[i - nslot])
                    s_h2d.wait_event(ev_out_q[i - nslot])
                with torch.cuda.stream(s_h2d):
                    dAs[i % nslot].copy_(hA[i % nk], non_blocking=True)
                    ev_h2d[i].record(s_h2d)

            torch.cuda.synchronize()
            e0.record(stream)
            s_h2d.wait_event(e0)
            for i in range(min(ahead, steps)):
                h2d(i)
            for i in range(steps):
                if i + ahead < steps:
                    h2d(i + ahead)
                stream.wait_event(ev_h2d[i])
                mixed_q(dAs[i % nslot], Qs[i % nslot])
                ev_done[i].record(stream)
                s_d2h.wait_event(ev_done[i])
                s_d2h_q.wait_event(ev_done[i])
                with torch.cuda.stream(s_d2h):
                    hA_out[i % 2].copy_(dAs[i % nslot], non_blocking=True)
                    ev_out[i].record(s_d2h)
                with torch.cuda.stream(s_d2h_q):
                    hQ_out[i % 2].copy_(Qs[i % nslot], non_blocking=True)
                    ev_out_q[i].record(s_d2h_q)
            stream.wait_event(ev_out[steps - 1])
            stream.wait_event(ev_out_q[steps - 1])
            e1.record(stream)
            torch.cuda.synchronize()
            # when each matrix's last output copy completed, from the start
            gaps.clear()
            prev = 0.0
            for i in range(steps):
                t = e0.elapsed_time(ev_out_q[i])
                gaps.append(t - prev)
                prev = t
            return e0.elapsed_time(e1)

        # warm-up pass over every host buffer and slot (the first copies that
        # touch a page-locked buffer run slower), then the timed pass
        pipeline(max(nk, nslot))
        # no Python garbage collection inside the timed pipeline: a collection
        # delays the host's next copy enqueue while the link idles
        # three runs of e2e_steps matrices; the median run is reported (a
        # host stall of tens of ms in one run shows in its gaps)
        runs = []
        for _ in range(3):
            gc.collect()
            gc.disable()
            try:
                t_run = pipeline(e2e_steps) / e2e_steps
            finally:
                gc.enable()
            runs.append((t_run, list(gaps)))
        runs.sort(key=lambda x: x[0])
        e2e_ms, gaps_med = runs[1]
        gaps[:] = gaps_med
        if world > 1:
            import torch.distributed as dist

            t = torch.tensor([e2e_ms], dtype=torch.float64, device="cuda")
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            e2e_ms = float(t.item())
        floor_ms = max(8.0 * m * n / h2d_gbs, 16.0 * m * n / d2h_gbs) / 1e6
        floor_ms = max(floor_ms, both_ms)
        e2e = {"value": world * credited_flops(m, n) / (e2e_ms * 1e-3) / 1e9, "unit": "GFLOP/s",
               "ms_per_step": e2e_ms, "steps": e2e_steps, "kappas": list(kappas),
               "h2d_bytes_per_step": 8 * m * n, "d2h_bytes_per_step": 16 * m * n,
               "link_h2d_GBs": h2d_gbs, "link_d2h_GBs": d2h_gbs, "copy_floor_ms_per_step": floor_ms,
               "copies_of_one_step_concurrently_ms": both_ms,
               "ms_between_outputs": {"first": gaps[0], "median": sorted(gaps[1:])[len(gaps[1:]) // 2] if len(gaps) > 1
                                      else gaps[0], "max": max(gaps[1:] or gaps)},
               "ms_per_step_of_runs": [r[0] for r in runs], "reported": "the median of three runs",
               "copy_floor": "the larger of each direction alone at its measured rate and one step's three copies "
                             "run at once",
               "pipeline": "four device slots; input copies three steps ahead on one copy stream, V/R and Q "
                           "copies on two more, overlapping the factorization of other steps"}
        # the library's own out-of-core call on the same host matrix: A and Q
        # stay in page-locked host memory and stream through the device in
        # chunks (every pass reads A over the host link; the last one also
        # writes V and Q back)
        hA_w = torch.empty((n, m), dtype=torch.float64, pin_memory=True).t()
        lw_o = L.lib().lila_gpu_query_dgeqrf_tall_host(m, n, 0)
        W_o = torch.empty(lw_o, dtype=torch.float64, device="cuda")
        T_o = L.colmajor(mt, n, fill=0.0)
        o_ms = []
        for _ in range(3):
            hA_w.copy_(hA[0])
            torch.cuda.synchronize()
            e0.record(stream)
            rc = L.gpu_dgeqrf_tall_host(m, n, mt, hA_w, m, T_o, mt, hQ_out[0], m, 0, W_o, lw_o)
            e1.record(stream)
            torch.cuda.synchronize()
            assert rc == 0, rc
            o_ms.append(e0.elapsed_time(e1))
        o_ms = sorted(o_ms[1:])[0]
        o_passes = L.gpu_last_passes()
        out_of_core = {"value": credited_flops(m, n) / (o_ms * 1e-3) / 1e9, "unit": "GFLOP/s",
                       "ms_per_matrix": o_ms, "kappa": kappas[0], "passes": o_passes,
                       "rows_per_chunk": min(1048576, (m + 127) // 128 * 128),
                       "host_bytes_read": (o_passes + 1) * 8 * m * n, "host_bytes_written": 16 * m * n,
                       "device_bytes": int(lw_o) * 8,
                       "call": "lila_gpu_dgeqrf_tall_host (A, Q in page-locked host memory; best of 2 after 1 warm-up)"}
        del hA, hA_out, hQ_out, dAs, Qs, hA_w, W_o, T_o
        torch.cuda.empty_cache()

    flops = credited_flops(m, n)
    gflops = world * flops / (ms * 1e-3) / 1e9
    peaks, peak_src = load_peaks()
    total_traced = sum(v[1] for v in trace.values()) or 1.0
    # dominant kernel and its algorithmic bytes per launch (m x n FP64 panel)
    alg_bytes = {"ozaki_map": 16.0 * m * n, "ozaki_gram": 8.0 * m * n, "ozaki_colmax": 8.0 * m * n}
    # The leaf enqueues a fixed number of passes and the device decides how
    # many run: the Gram, factor and map launches of the passes after the
    # last one return at once.  The launches that did work per step follow
    # from the pass count of each step's condition number (P passes: P Grams
    # and factors, P - 1 maps between passes, two final maps); the traced
    # time of a kernel (which includes its few-microsecond skipped launches)
    # is divided by those.
    passes = [acc_mixed["%g" % kappas[s % nk]]["passes"] for s in range(args.steps)]
    working = {"ozaki_map": sum(p + 1 for p in passes), "ozaki_gram": sum(passes),
               "ozaki_gram_reduce": sum(passes), "factor_pass": sum(passes), "factor_rk_r": sum(passes)}
    dname, (dcnt, dms) = max(trace.items(), key=lambda kv: kv[1][1]) if trace else ("none", (1, 1.0))
    dcnt = working.get(dname, dcnt)
    bpl = alg_bytes.get(dname)
    achieved = bpl / (dms / dcnt * 1e-3) / 1e9 if bpl else None
    kernels = {k: {"launches_per_step": working.get(k, v[0]) / args.steps, "ms_per_step": v[1] / args.steps,
                   "share": v[1] / total_traced, "enqueued_per_step": v[0] / args.steps}
               for k, v in sorted(trace.items(), key=lambda kv: -kv[1][1])}
    result = {
        "metric": METRIC,
        "value": gflops,
        "unit": "GFLOP/s",
        "mats_per_s": world * 1e3 / ms,
        "n_gpus": world,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": ms,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f64",
        "data": "synthetic: A = U diag(sigma) V^T, U = Q of seeded N(0,1) m x n (seed 201), V Haar "
                "(seed 202), sigma log-spaced 1 -> 1/kappa, kappa cycled over %s" % list(kappas),
        "config": {"workload": "tall-skinny QR (V, R, T tiles and explicit Q) by split-precision Cholesky QR 2 "
                               "/ shifted + Householder reconstruction (lila_dgeqrf_w03_mt_hr_mixed)",
                   "m": m, "n": n, "mt": mt, "kappas": list(kappas), "variant": "mixed (BF16 tcgen05, "
                   "FP64-grade)", "l2": "inputs larger than L2 (fresh 2.1 GB copy of A per step, no flush needed)",
                   "parallelism": "replicas" if world > 1 else "single-gpu"},
        "per_kappa_ms": {k: sum(v) / len(v) for k, v in per_kappa_ms.items()},
        "accuracy": {"tol": 50 * n * 2.0 ** -53, "mixed": acc_mixed, "status": status_mixed,
                     "device_check": check_cost},
        "plain_fp64": plain_res,
        "tsqr_fp64": tsqr_res,
        "mixed_over_plain": (gflops / world / plain_res["value"]) if plain_res else None,
        "roofline": {
            "bound": "hbm",
            "kernel": dname,
            "achieved": achieved,
            "peak": peaks.get("hbm_gbs"),
            "unit": "GB/s",
            "frac": (achieved / peaks["hbm_gbs"]) if achieved else None,
            "traffic": MAP_DRAM_BYTES_PER_ROW * m if dname == "ozaki_map" else None,
            "traffic_source": ("dram__bytes_read.sum + dram__bytes_write.sum of one ncu capture of a "
                               "1,048,576 x 64 launch, scaled to m rows" if dname == "ozaki_map" else None),
            "peak_source": peak_src,
            "algorithmic_bytes_per_launch": bpl,
            "kernel_share_of_traced_time": dms / total_traced,
            "kernel_ms_per_launch": dms / dcnt,
        },
        "kernels": kernels,
        "e2e": e2e,
        "out_of_core": out_of_core,
        "gpu_launches": int(launches),
        "clocks": clk,
    }
    return result


# ---------------------------------------------------------------------------
# further workloads, reported under "workloads" of the same line
# ---------------------------------------------------------------------------
def _event_ms(torch, fn, reps, prep=None):
    """CUDA-event milliseconds of each fn() on the current stream; prep()
    (restoring inputs) runs before each, outside the timed region."""
    stream = torch.cuda.current_stream()
    out = []
    for _ in range(reps):
        if prep is not None:
            prep()
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        fn()
        e1.record(stream)
        torch.cuda.synchronize()
        out.append(e0.elapsed_time(e1))
    return out


def _probe_fro(torch, apply, ncols, probes=16, seed=7):
    """Stochastic Frobenius-norm estimate of a linear map X -> apply(X) from
    Gaussian probes: E ||M g||^2 = ||M||_F^2."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    G = torch.randn((ncols, probes), generator=g, dtype=torch.float64, device="cuda")
    Y = apply(G)
    return float(torch.sqrt((Y * Y).sum() / probes))


def run_recursive(L, torch, steps=3, warmup=1, mt=64, nx=64, autotune=True):
    """Recursive QR + explicit Q of a 4000 x 1000 Gaussian, then
    Q^T applied to a 4000 x 64 block (lila_dgeqrf_w03_recursive, lila_dormqrf_z03).
    With autotune, the panel width mt and the recursion cutoff nx come from
    lila_gpu_recursive_autotune on this matrix (untimed)."""
    import numpy as np

    m, n, k = 4000, 1000, 64
    A = np.asfortranarray(np.random.default_rng(101).standard_normal((m, n)))
    C = np.asfortranarray(np.random.default_rng(102).standard_normal((m, k)))
    dA0, dC0 = L.to_device_colmajor(A), L.to_device_colmajor(C)
    dA, dC = L.colmajor(m, n), L.colmajor(m, k)
    tuned = None
    if autotune:
        lw_t = max(L.query_dgeqrf_w03_recursive([0, 1, 1, x], m, n, 0, t, None, m, None, t, None, m, None, -1)
                   for t in (32, 64, 128, 256) for x in (32, 64, 128, 256, 512))
        W_t = torch.empty(lw_t, dtype=torch.float64, device="cuda")
        T_t, Q_t = L.colmajor(256, n, fill=0.0), L.colmajor(m, n, fill=0.0)
        rc, t_mt, t_nx = L.recursive_autotune([0, 1, 1, nx], m, n, dA0, m, dA, T_t, 256, Q_t, m, W_t, lw_t)
        if rc > 0:
            tuned = {"mt": t_mt, "nx": t_nx, "best_us": rc, "untuned": {"mt": mt, "nx": nx},
                     "candidates": "mt in {32, 64, 128, 256} x nx in {32, 64, 128, 256, 512}"}
            mt, nx = t_mt, t_nx
        del W_t, T_t, Q_t
    dT, dQ = L.colmajor(mt, n, fill=0.0), L.colmajor(m, n, fill=0.0)
    lp = [0, 1, 1, nx]
    lw = max(L.query_dgeqrf_w03_recursive(lp, m, n, 0, mt, None, m, None, mt, None, m, None, -1),
             L.query_dormqrf_w03(m, k, n, 0, 0, mt, None, m, None, mt, None, -1))
    W = torch.empty(lw, dtype=torch.float64, device="cuda")

    def prep():
        dA.copy_(dA0)
        dC.copy_(dC0)

    def step():
        assert L.dgeqrf_w03_recursive(lp, m, n, 0, mt, dA, m, dT, mt, dQ, m, W, lw) == 0
        assert L.dormqrf_z03(m, k, n, 0, 0, mt, dA, m, dT, mt, dC, m, W, lw) == 0

    _event_ms(torch, step, warmup, prep)
    l0 = L.launch_count()
    L.trace(True)
    ts = _event_ms(torch, step, steps, prep)
    trace = L.trace_summary()
    L.trace(False)
    launches = (L.launch_count() - l0) / steps
    ts = _event_ms(torch, step, steps, prep)  # untraced timing
    ms_direct = sorted(ts)[len(ts) // 2]
    tot = sum(v[1] for v in trace.values()) or 1.0
    kernels = {kk: {"launches_per_step": v[0] / steps, "ms_per_step": v[1] / steps, "share": v[1] / tot}
               for kk, v in sorted(trace.items(), key=lambda kv: -kv[1][1])[:12]}
    # graph mode: the first call of each argument set is captured, later ones replay
    prev = L.gpu_graph_mode(1)
    t_first = _event_ms(torch, step, 1, prep)[0]
    tg = _event_ms(torch, step, steps, prep)
    L.gpu_graph_mode(prev)
    L.gpu_graph_cache_clear()
    ms = sorted(tg)[len(tg) // 2]
    flops = 4.0 * m * n * n - 4.0 / 3.0 * n ** 3 + 4.0 * m * n * k - 2.0 * n * n * k
    R = torch.triu(dA[:n, :n])
    res = _fro(torch, dQ @ R - dA0) / _fro(torch, dA0)
    orth = _fro(torch, torch.eye(n, dtype=torch.float64, device="cuda") - dQ.t() @ dQ)
    qtc = dQ.t() @ dC0
    qtc_err = float((dC[:n] - qtc).abs().max() / qtc.abs().max())
    return {"workload": "recursive Householder QR + explicit Q of a 4000 x 1000 N(0,1) matrix (seed 101), "
                        "then Q^T applied to a 4000 x 64 N(0,1) block (seed 102)",
            "calls": "lila_dgeqrf_w03_recursive (leaf 1, panel 1, nx %d, mt %d) + lila_dormqrf_z03" % (nx, mt),
            "value": flops / (ms * 1e-3) / 1e9, "unit": "GFLOP/s", "ms_per_step": ms, "steps": steps,
            "mode": "graph replay (lila_gpu_graph_mode(1); the first call of the argument set captured)",
            "direct": {"ms_per_step": ms_direct, "gflops": flops / (ms_direct * 1e-3) / 1e9},
            "graph_first_call_ms": t_first, "kernels_direct_traced": kernels,
            "flops_per_step": flops, "dtype": "f64", "gpu_launches_per_step": launches, "autotune": tuned,
            "accuracy": {"res": res, "orth": orth, "qtc_vs_explicit_q": qtc_err, "tol": 50 * n * 2.0 ** -53}}


def run_square(L, torch, nsq=16384, steps=1, warmup=1, mt=128, nx=128, precision=0):
    """Square recursive QR (FP64 or split precision), columns graded by 10^(-6j/n)."""
    n = nsq
    g = torch.Generator(device="cuda")
    g.manual_seed(301)
    A0 = torch.randn((n, n), generator=g, dtype=torch.float64, device="cuda")  # rows = columns of A
    A0 *= torch.pow(10.0, -6.0 * torch.arange(n, dtype=torch.float64, device="cuda") / n)[:, None]
    dA0 = A0.t()  # column-major view
    dA = L.colmajor(n, n)
    dT, dQ = L.colmajor(mt, n, fill=0.0), L.colmajor(n, n, fill=0.0)
    lp = [0, 1, 1, nx]
    lw = L.query_dgeqrf_w03_recursive(lp, n, n, 0, mt, None, n, None, mt, None, n, None, -1)
    W = torch.empty(lw, dtype=torch.float64, device="cuda")

    def prep():
        dA.copy_(dA0)

    def step():
        assert L.dgeqrf_w03_recursive(lp, n, n, 0, mt, dA, n, dT, mt, dQ, n, W, lw) == 0

    prev = L.gpu_set_precision(precision)
    _event_ms(torch, step, warmup, prep)
    L.trace(True)
    ts = _event_ms(torch, step, steps, prep)
    trace = L.trace_summary()
    L.trace(False)
    L.gpu_set_precision(prev)
    ms = sorted(ts)[len(ts) // 2]
    flops_qr = 4.0 / 3.0 * n ** 3
    flops_all = 4.0 * n ** 3 - 4.0 / 3.0 * n ** 3  # geqrf + explicit Q
    R = torch.triu(dA[:n, :n])
    res = _probe_fro(torch, lambda G: dQ @ (R @ G) - dA0 @ G, n) / _fro(torch, dA0)
    orth = _probe_fro(torch, lambda G: G - dQ.t() @ (dQ @ G), n)
    d = torch.diagonal(R).abs()
    tot = sum(v[1] for v in trace.values()) or 1.0
    top = sorted(trace.items(), key=lambda kv: -kv[1][1])[:6]
    return {"workload": "square recursive Householder QR (V, R, T and explicit Q), n = %d, A N(0,1) (seed 301) "
                        "with column j scaled by 10^(-6j/n)" % n,
            "calls": "lila_dgeqrf_w03_recursive (leaf 1, panel 1, nx %d, mt %d)" % (nx, mt),
            "precision": "split (FP64-grade products on BF16 tcgen05)" if precision else "fp64",
            "value": flops_all / (ms * 1e-3) / 1e9, "unit": "GFLOP/s (QR + explicit Q, 8/3 n^3)",
            "geqrf_credit_gflops": flops_qr / (ms * 1e-3) / 1e9, "ms_per_step": ms, "steps": steps,
            "dtype": "f64",
            "accuracy": {"res_probe16": res, "orth_probe16": orth, "tol": 50 * n * 2.0 ** -53,
                         "r_diag_abs_min": float(d.min()), "r_diag_abs_max": float(d.max()),
                         "r_diag_abs_first_last": [float(d[0]), float(d[-1])]},
            "kernels": {k: {"ms_per_step": v[1] / steps, "share": v[1] / tot} for k, v in top}}


def run_update(L, torch, m=16384, n=8192, k=128, mt=128, steps=5, warmup=2, precision=0):
    """The trailing update that dominates the square QR: H^T of k reflectors
    applied to an m x n block (lila_dormqrf_w03), 4mnk + nk^2 flops."""
    g = torch.Generator(device="cuda")
    g.manual_seed(303)
    A0 = torch.randn((k + n, m), generator=g, dtype=torch.float64, device="cuda").t()  # column-major m x (k+n)
    dA = L.colmajor(m, k + n)
    dA.copy_(A0)
    dT, dQ = L.colmajor(mt, k, fill=0.0), L.colmajor(m, k, fill=0.0)
    lp = [0, 1, 1, min(k, 64)]
    lw = max(L.query_dgeqrf_w03_recursive(lp, m, k, 0, mt, None, m, None, mt, None, m, None, -1),
             L.query_dormqrf_w03(m, n, k, 0, k, mt, None, m, None, mt, None, -1))
    W = torch.empty(lw, dtype=torch.float64, device="cuda")
    assert L.dgeqrf_w03_recursive(lp, m, k, 0, mt, dA, m, dT, mt, dQ, m, W, lw) == 0
    C0 = dA[:, k:].clone()

    def prep():
        dA[:, k:].copy_(C0)

    def step():
        assert L.dormqrf_w03(m, n, k, 0, k, mt, dA, m, dT, mt, W, lw) == 0

    prev = L.gpu_set_precision(precision)
    _event_ms(torch, step, warmup, prep)
    L.trace(True)
    ts = _event_ms(torch, step, steps, prep)
    trace = L.trace_summary()
    L.trace(False)
    L.gpu_set_precision(prev)
    ms = sorted(ts)[len(ts) // 2]
    flops = 4.0 * m * n * k + n * k * k
    tot = sum(v[1] for v in trace.values()) or 1.0
    return {"workload": "H^T of %d reflectors applied to a %d x %d block (lila_dormqrf_w03, mt %d)" % (k, m, n, mt),
            "precision": "split" if precision else "fp64",
            "value": flops / (ms * 1e-3) / 1e9, "unit": "GFLOP/s", "ms_per_step": ms, "steps": steps,
            "dtype": "f64",
            "kernels": {kk: {"launches_per_step": v[0] / steps, "ms_per_step": v[1] / steps, "share": v[1] / tot}
                        for kk, v in sorted(trace.items(), key=lambda kv: -kv[1][1])}}


def _selector_params(L, torch, log):
    from lila_gb300 import selector_train as ST

    try:
        return ST.load_params(), "trained (lila_gb300/data/selector_params.f32)"
    except (OSError, RuntimeError) as e:
        log("selector parameters unavailable (%s): training on 50,000 instances" % e)
        p, rep = ST.train(50000, batch_instances=10000, epochs=12, log=log)
        return p, "trained in this run on 50,000 instances (holdout accuracy %.3f)" % rep["holdout_accuracy"]


def _ls_summary(batch, skip_rankdef=True):
    """Accuracy of a solved batch.  b = A x* + 1e-10 N(0,1), so the least
    residual is the noise's component outside range(A), about
    1e-10 sqrt((m - n) nrhs); a backward-stable solve lands on it.  The
    forward error against x* mostly measures the problem's sensitivity
    (kappa 1e-10 and kappa^2 u terms), reported for completeness."""
    import numpy as np

    fwd, res, rabs = batch.errors()
    ok = ~np.asarray(batch.rankdef) if skip_rankdef else np.ones(batch.count, dtype=bool)
    m = np.asarray(batch.m, dtype=np.float64)
    n = np.asarray(batch.n, dtype=np.float64)
    floor = 1e-10 * np.sqrt((m - n) * batch.nrhs)
    ratio = rabs / floor
    return {"residual_over_noise_floor_median": float(np.median(ratio)),
            "residual_over_noise_floor_max": float(ratio.max()),
            "residual_rel_median": float(np.median(res)), "residual_rel_max": float(res.max()),
            "fwd_err_vs_xstar_median": float(np.median(fwd[ok])), "fwd_err_vs_xstar_max": float(fwd[ok].max()),
            "nonfinite": int(np.sum(~np.isfinite(fwd)))}


def run_batched(L, torch, count=10000, steps=3, warmup=1, klo=1.0, khi=12.0, p_rankdef=0.0, seed=400000,
                params=None, log=print, stream_batches=1):
    """Batched uneven least squares (4 right-hand sides): 10,000 instances, m ~ U{64..4096},
    n ~ U{8..128}, kappa log-uniform, optionally a stream of such batches with rank-deficient ones."""
    import time as _time

    import numpy as np

    from lila_gb300 import workload as W

    out = {"count": count, "nrhs": 4, "kappa_log10": [klo, khi], "rank_deficient_fraction": p_rankdef}
    t0 = _time.time()
    batches = [W.make_ls_batch(count, seed + 1000 * s, klo=klo, khi=khi, p_rankdef=p_rankdef)
               for s in range(stream_batches)]
    out["generation_seconds"] = _time.time() - t0
    flops = sum(b.flops() for b in batches) / len(batches)
    out["flops_per_batch"] = flops
    b0 = batches[0]
    # ---- plain FP64: the batched Householder solver, up to three launches in a CUDA graph
    wbytes = L.lib().lila_query_dgels_batched(count)
    work = torch.empty(wbytes, dtype=torch.uint8, device="cuda")
    info = torch.zeros(count, dtype=torch.int32, device="cuda")
    plain_ms = []
    for b in batches:
        assert L.dgels_batched_prepare(count, b.m, b.n, 4, b.A_ptr, b.lda, b.B_ptr, b.lda, work, wbytes) == 0
        graph = L.lib().lila_dgels_batched_graph(count, 4, ctypes_ptr(work), ctypes_ptr(info))
        assert graph
        launch = lambda: L.gpu_graph_launch(graph)  # noqa: E731
        _event_ms(torch, launch, warmup, b.restore)
        plain_ms += _event_ms(torch, launch, steps, b.restore)
        L.gpu_graph_destroy(graph)
    plain_acc = _ls_summary(batches[-1], skip_rankdef=True)
    pm = float(np.median(plain_ms))
    out["plain_fp64"] = {"path": "lila_dgels_batched (FP64 Householder, CUDA graph)",
                         "ms_per_batch_median": pm, "mats_per_s": count / (pm * 1e-3),
                         "gflops": flops / (pm * 1e-3) / 1e9, "accuracy": plain_acc}

    # ---- routed variants with the on-device check and FP64 fallback
    def routed(policy, flags=0):
        lat, fails, mixed_n, fp64_n, routes = [], 0, 0, 0, np.zeros(3, dtype=np.int64)
        shifted_n = 0
        acc = None
        for b in batches:
            h = L.GelsMixed(b.m, b.n, 4, b.A_ptr, b.lda, b.B_ptr, b.lda)
            elig = [(b.n[t] <= 128) for t in range(count)]
            state = {}

            def solve():
                if policy == "learned":
                    rc, inf, orth, route = h.solve(params, flags)
                else:
                    route = [policy if elig[t] else 2 for t in range(count)]
                    rc, inf, orth = h.run(route, flags)
                state["rc"], state["route"], state["info"], state["orth"] = rc, route, inf, orth

            _event_ms(torch, solve, warmup, b.restore)
            for _ in range(steps):
                lat += _event_ms(torch, solve, 1, b.restore)
                assert state["rc"] >= 0, state["rc"]
                fails += state["rc"]
                r = np.asarray(state["route"])
                mixed_n += int(np.sum(r != 2))
                routes += np.bincount(r, minlength=3)
                # instances that ended in the FP64 solver: routed there, or a
                # failed check whose retry (if any) failed too
                inf, orth = np.asarray(state["info"]), np.asarray(state["orth"])
                lim = 50.0 * np.asarray(b.n, dtype=np.float64) * 2.0 ** -53
                fp64_n += int(np.sum((r == 2) | ((inf == 1) & ~((orth >= 0) & (orth <= lim)))))
                shifted_n += sum(h.shifted())
            acc = _ls_summary(b, skip_rankdef=True)
            # one more solve with the per-launch trace on (outside the timed
            # batches): where the batch's device time goes
            b.restore()
            torch.cuda.synchronize()
            L.trace(True)
            solve()
            torch.cuda.synchronize()
            tr = L.trace_summary()
            L.trace(False)
            h.close()
        lat = np.asarray(lat)
        tot = sum(v[1] for v in tr.values()) or 1.0
        kernels = {kk: {"launches": v[0], "ms": round(v[1], 2), "share": round(v[1] / tot, 3)}
                   for kk, v in sorted(tr.items(), key=lambda kv: -kv[1][1])[:6]}
        return {"ms_per_batch_median": float(np.median(lat)), "ms_per_batch_p99": float(np.percentile(lat, 99)),
                "mats_per_s": count / (float(np.mean(lat)) * 1e-3),
                "gflops_credited": flops / (float(np.mean(lat)) * 1e-3) / 1e9,
                "check_failure_rate_of_routed_to_mixed": fails / max(1, mixed_n),
                "fallback_rate_of_routed_to_mixed": fails / max(1, mixed_n),
                "fallback_rate_of_all": fails / (count * len(lat)),
                "fp64_solved_fraction": fp64_n / (count * len(lat)),
                "route_fractions": (routes / routes.sum()).tolist(),
                "trial_shifted_fraction": shifted_n / (count * len(lat)), "accuracy_last_batch": acc,
                "batches_timed": int(len(lat)), "kernels_traced_one_batch": kernels}

    out["always_shifted_cholqr3"] = routed(1)
    # variant 0 routing without the trial: Cholesky QR 2, instances whose
    # check fails retried by shifted Cholesky QR 3, FP64 Householder last
    out["always_cholqr2"] = routed(0, L.GELS_NO_TRIAL)
    out["always_cholqr2"]["policy"] = "Cholesky QR 2; failed checks retried by shifted Cholesky QR 3, then FP64"
    # variant 0 with its trial factor: the shift where the trial's condition
    # estimate asks for it, the same retry and fallback
    out["cholqr2_trial"] = routed(0)
    out["cholqr2_trial"]["policy"] = ("Cholesky QR 2 whose trial Cholesky of the FP64-grade Gram (1-norm condition "
                                      "above 1e8 or breakdown) switches to shifted Cholesky QR 3; retry and FP64 "
                                      "as above")
    fixed = ("always_shifted_cholqr3", "always_cholqr2", "cholqr2_trial")
    best_fixed = min(out[k]["ms_per_batch_median"] for k in fixed)
    out["best_mixed_over_plain"] = pm / best_fixed
    if params is not None:
        out["learned"] = routed("learned")
    if params is not None:
        lm = out["learned"]["ms_per_batch_median"]
        out["learned_over_plain"] = pm / lm
        out["learned_over_best_fixed_variant"] = best_fixed / lm
    for b in batches:
        del b
    return out


def fp64_peak_probe(L, torch):
    """The FP64 denominators of the plain kernels, measured here: independent
    DFMA chains and DMMA (mma.sync m8n8k4) over 8 CTAs per SM, GFLOP/s from
    CUDA events, with the SM clocks sampled while the probes run."""
    import datetime as _dt

    sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    out = torch.empty(sms * 8 * 256, dtype=torch.float64, device="cuda")
    clocks = ClockSampler(int(os.environ.get("LOCAL_RANK", "0")))
    clocks.start()
    w0 = _dt.datetime.now()
    dfma = max(L.lib().lila_prim_fp64_probe(0, out.data_ptr(), sms * 8, 256, 20000) for _ in range(2))
    dmma = max(L.lib().lila_prim_fp64_probe(1, out.data_ptr(), sms * 8, 256, 5000) for _ in range(2))
    w1 = _dt.datetime.now()
    clk = clocks.stop((w0, w1))
    return {"dfma_gflops": dfma, "dmma_gflops": dmma, "peak_gflops": max(dfma, dmma), "clocks": clk,
            "how": "lila_prim_fp64_probe: 8 independent FMA chains per thread (DFMA) and mma.sync m8n8k4 (DMMA), "
                   "%d CTAs x 256 threads, best of 2, CUDA events" % (sms * 8)}


def run_extra(args, which):
    import torch

    import lila_gb300 as L

    torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", "0")))
    L.lib()
    log = lambda msg: print(msg, file=sys.stderr)  # noqa: E731
    steps = args.extra_steps
    if which == "recursive":
        r = run_recursive(L, torch, steps=steps)
    elif which == "update":
        r = {"fp64": run_update(L, torch), "split": run_update(L, torch, precision=1)}
        r["split_over_fp64"] = r["split"]["value"] / r["fp64"]["value"]
        r["fp64_peak_probe"] = fp64_peak_probe(L, torch)
        r["fp64_frac_of_probe_peak"] = r["fp64"]["value"] / r["fp64_peak_probe"]["peak_gflops"]
    elif which == "square":
        kw = dict(nsq=args.square_n, steps=1, warmup=1, mt=args.square_mt, nx=args.square_nx)
        r = {"plain": run_square(L, torch, precision=0, **kw), "mixed": run_square(L, torch, precision=1, **kw)}
        r["mixed_over_plain"] = r["mixed"]["value"] / r["plain"]["value"]
        r["fp64_peak_probe"] = fp64_peak_probe(L, torch)
        r["plain_frac_of_probe_peak"] = r["plain"]["value"] / r["fp64_peak_probe"]["peak_gflops"]
    elif which == "batched":
        params, src = _selector_params(L, torch, log)
        r = run_batched(L, torch, count=args.batch_count, steps=steps, params=params)
        r["workload"] = ("batched uneven least squares: %d instances, m ~ U{64..4096}, n ~ U{8..128}, m >= 2n, "
                         "kappa log-uniform [1e1, 1e12], 4 right-hand sides" % args.batch_count)
        r["selector"] = src
    else:
        params, src = _selector_params(L, torch, log)
        r = run_batched(L, torch, count=args.batch_count, steps=steps, klo=1.0, khi=15.0, p_rankdef=0.05,
                        seed=500000, params=params, stream_batches=args.stream_batches)
        r["workload"] = ("stream of %d batches of %d instances as the batched workload with kappa log-uniform "
                         "[1e1, 1e15] and 5%% exactly rank-deficient instances; learned selector with on-device "
                         "check and FP64 Householder fallback" % (args.stream_batches, args.batch_count))
        r["selector"] = src
    torch.cuda.empty_cache()
    return r


def ctypes_ptr(t):
    import ctypes

    return ctypes.c_void_p(t.data_ptr())


def run_reference(args, rank, world):
    """CPU reference arm: the reference's FP64 Householder QR (leaf 1, panel 1,
    mt 200, nx 20) restated in C on OpenBLAS with every host core, one
    factorization of a full-size matrix per step, the condition numbers
    cycled as in the GPU arm; the Cholesky QR + reconstruction leaf is timed
    once per condition number beside it.  A run of more than 30 steps in all
    factors a row sample per step so that it ends within minutes."""
    import numpy as np

    lib, how = _cpu_lib()
    kappas = KAPPAS if args.kappa is None else (args.kappa,)
    total = args.warmup + args.steps
    m_step = args.m if total <= 30 else max(args.n * 64, int(args.m * 30 / total))
    bases = [make_tall_input_numpy(m_step, args.n, k) for k in kappas]
    t_steps = []
    acc = {}
    for s in range(total):
        k = s % len(kappas)
        t, A, Q = _cpu_factor(lib, bases[k], CPU_HH)
        if s >= args.warmup:
            t_steps.append(t)
        key = "%g" % kappas[k]
        if key not in acc:
            res, orth = _cpu_accuracy(bases[k], A, Q)
            acc[key] = {"res": res, "orth": orth}
        del A, Q
    t = sum(t_steps) / len(t_steps)
    value = credited_flops(m_step, args.n) / t / 1e9
    tol = 50 * args.n * 2.0 ** -53
    hr = {}
    for k, A0 in zip(kappas, bases):
        th, Ah, Qh = _cpu_factor(lib, A0, CPU_HR)
        rh, oh = _cpu_accuracy(A0, Ah, Qh)
        hr["%g" % k] = {"gflops": credited_flops(m_step, args.n) / th / 1e9, "res": rh, "orth": oh}
        del Ah, Qh
    cores = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else os.cpu_count()
    sample = ("the reference's FP64 Householder QR (lila_dgeqrf_w03_recursive, leaf 1, panel 1, mt 200, nx 20) "
              "restated in C %s; one %d x %d matrix per step, kappa cycled over %s; OPENBLAS threads %s"
              % (how, m_step, args.n, list(kappas), os.environ.get("OPENBLAS_NUM_THREADS", cores)))
    return {
        "metric": METRIC,
        "impl": "reference",
        "value": value,
        "unit": "GFLOP/s",
        "mats_per_s": 1.0 / (t * args.m / m_step),
        "n_gpus": world,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": t * 1e3,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f64",
        "data": "synthetic: A = U diag(sigma) V^T as in the GPU arm (seeds 201 / 202)",
        "config": {"workload": "tall-skinny QR (V, R, T tiles and explicit Q) by the reference's FP64 Householder "
                               "QR on the host cores",
                   "m": args.m, "n": args.n, "m_per_step": m_step, "kappas": list(kappas),
                   "family": CPU_HH, "variant": "plain-fp64 (CPU)"},
        "cpu_baseline": {"value": value, "unit": "GFLOP/s", "cores": cores, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": "GFLOP/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "cholqr_hr_leaf": hr,
        "accuracy": {"tol": tol, "householder": acc,
                     "note": "the gate 50 n 2^-53 does not grow with m; FP64 Householder's rounding grows with "
                             "the row count"},
    }


# What the result line keeps of the measurements beside the headline; stderr has
# all of them.
BRIEF = ("value", "ms_per_step", "ms_per_matrix", "ms_per_batch_median", "mats_per_s", "gflops", "gflops_credited",
         "fallback_rate_of_all", "mixed_over_plain", "best_mixed_over_plain", "learned_over_plain",
         "learned_over_best_fixed_variant", "passes", "res", "orth", "tol", "error")


def _brief(x):
    if isinstance(x, dict):
        kept = {k: _brief(v) for k, v in x.items() if k in BRIEF or (isinstance(v, dict) and "kernels" not in k)}
        return {k: v for k, v in kept.items() if v != {}}
    return float("%.5g" % x) if isinstance(x, float) else x


def result_line(out):
    """The one-line result: the headline whole, of everything else the values (a
    reader of the line may take a few KB only)."""
    line = {k: v for k, v in out.items() if k != "kernels"}
    for key in ("plain_fp64", "tsqr_fp64", "out_of_core", "workloads", "accuracy"):
        if key in line:
            line[key] = _brief(line[key])
    if "e2e" in line:
        line["e2e"] = {k: v for k, v in line["e2e"].items()
                       if k in ("value", "unit", "ms_per_step", "steps", "h2d_bytes_per_step", "d2h_bytes_per_step",
                                "copies_of_one_step_concurrently_ms")}
    if "cpu_baseline" in line:
        line["cpu_baseline"] = {k: v for k, v in line["cpu_baseline"].items()
                                if k in ("value", "unit", "cores", "kind", "sample")}
    if "roofline" in line:
        line["roofline"] = {k: v for k, v in line["roofline"].items() if k != "traffic_source"}
    # the per-condition-number times and accuracy close the line, so that
    # a record that keeps only the line's tail still shows them
    for key in ("per_kappa_ms", "accuracy"):
        if key in line:
            line[key] = line.pop(key)
    return line


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=16)
    ap.add_argument("--warmup", type=int, default=4)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--m", type=int, default=4194304)
    ap.add_argument("--n", type=int, default=64)
    ap.add_argument("--mt", type=int, default=32)
    ap.add_argument("--kappa", type=float, default=None, help="one kappa instead of the four of the workload")
    ap.add_argument("--plain-steps", type=int, default=4)
    ap.add_argument("--no-plain", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--workload", default="all",
                    choices=["all", "tall", "recursive", "square", "update", "batched", "learned"],
                    help="all: the tall-skinny headline plus the other workloads under 'workloads'")
    ap.add_argument("--square-n", type=int, default=16384)
    ap.add_argument("--square-mt", type=int, default=128)
    ap.add_argument("--square-nx", type=int, default=128)
    ap.add_argument("--batch-count", type=int, default=10000)
    ap.add_argument("--stream-batches", type=int, default=3)
    ap.add_argument("--extra-steps", type=int, default=3)
    ap.add_argument("--map-path", type=int, default=0, choices=[0, 1, 2, 3],
                    help="kernels of the tall Gram and row map (lila_prim_ozaki_map_path): 0 default, 1 register-fed, "
                         "2 / 3 TMA-fed transposed-tile row map")
    args = ap.parse_args()

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if args.impl == "reference":
        if rank != 0:
            return 0
        print(json.dumps(run_reference(args, rank, world)))
        return 0
    if world > 1:
        import torch.distributed as dist

        dist.init_process_group("nccl")
    if args.workload not in ("all", "tall"):
        if rank == 0:
            print(json.dumps(run_extra(args, args.workload)))
        return 0
    out = run_ours(args, rank, world)
    if rank == 0:
        if world == 1 and not args.no_cpu_baseline:
            out["cpu_baseline"] = cpu_baseline(args.m, args.n, 1e2)
        if args.workload == "all" and world == 1:
            out["workloads"] = {}
            for w in ("recursive", "square", "batched", "learned"):
                try:
                    out["workloads"][w] = run_extra(args, w)
                except Exception as e:  # reported, never hidden: the headline line still prints
                    out["workloads"][w] = {"error": "%s: %s" % (type(e).__name__, e)}
        print("detail: " + json.dumps(out), file=sys.stderr)
        print(json.dumps(result_line(out)))
    if world > 1:
        import torch.distributed as dist

        dist.barrier()
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
