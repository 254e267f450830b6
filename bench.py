"""Benchmark of the B200 Q2-P1disc Stokes operator (pTatin3D hot path).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--workload c2|c1|c0] [--no-cpu-baseline]

One step = one FP64 A11 apply (MatMult_MFStokes_A11: Dirichlet columns zeroed,
rows copied) over the whole 128^3 Q2 box of the precision workload (257^3
nodes, 50.9M velocity dofs; nodes perturbed +-0.05h; three viscosity layers
1e3/1/1e-1 plus 64 inclusions 1e-3..1e3; free-slip box BCs).  Inputs are
resident in HBM and larger than L2 (u, y 407 MB each; eta 453 MB), so no L2
flush is needed between steps.

value     = 3N / t_apply in GDoF/s, the device-timed apply (CUDA events on the
            op's stream), whole job over all ranks (replicas: each rank runs
            the same problem; the operator is single-GPU by design).
e2e       = the same metric through the public host-pointer API
            (pt_matmult_a11_h): pinned host x -> device, apply, device -> host y.
roofline  = algorithmic bytes of one apply / its device time against the
            measured HBM copy bandwidth (MEASURED_PEAKS.json).
cpu_baseline = the reference's own AVX A11 (oracle/_ref, compiled from the
            reference sources) on the same 128^3 box and inputs, on all host
            cores; the same leg runs the reference's diag, B, B^T and whole
            Stokes operator once and checks every device output of the line
            against them (parity: max-norm relative error).
extra     = FP32 A11, diag, B, B^T and whole-operator rates, and the rest of
            the metric: the precision-form solve (FP64- vs FP32-smoothed
            flexible CG to rtol 1e-8 on this box, true residual from the
            reference's A11 on the host), the batched form (256 boxes) and a
            served stream (p50/p99, solves/s against serial plain solves).
--impl reference times that reference CPU path only and prints its line.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(REPO, "ptatin-gene_b200"))

METRIC = "Q2 A11 GDoF/s FP64 vs FP32 @128³; batched solves/s & p99 @rtol 1e-8"

WORKLOAD_TEXT = {
    "c2": "perturbed +-0.05h, layered eta + 64 inclusions (1e6 contrast)",
    "c1": "undeformed, sinker eta (16 spheres r 0.08, 1e4)",
    "c0": "perturbed +-0.1h, log-uniform Gauss-point eta [1e-2, 1e2]",
    "box": "perturbed +-0.1h, log-uniform Gauss-point eta [1e-2, 1e2]",
    "sinker": "perturbed +-0.05h, sinker eta",
    "layered": "perturbed +-0.05h, layered eta + inclusions",
}
# DRAM bytes per element of one FP64 streaming apply (K 1.94 KB + u/y tiles),
# measured with ncu on a 128x128x32 box (rows of 128 elements): 2 colour
# launches averaged 0.3194 GB read + 0.0180 GB written for 128*128*32/4 elements.
TRAFFIC_PER_ELEMENT_F64 = 4 * (0.3194e9 + 0.0180e9) / (128 * 128 * 32)
UNIT = "GDoF/s"


def algorithmic_bytes(m, s=8):
    """u + coords + y (3N each) + eta (27 nel), s bytes per value."""
    return (9 * m.nnodes + 27 * m.nel) * s


def load_peaks():
    p = os.path.join(REPO, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index=0):
        self.index = index
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self._t = threading.Thread(target=self._read, daemon=True)
            self._t.start()
            # the timed region starts once samples flow
            t_end = time.time() + 3.0
            while not self.lines and time.time() < t_end:
                time.sleep(0.01)
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *exc):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def dist_setup(args):
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    pg = None
    if ws > 1:
        import datetime

        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local))
        pg = dist
    return ws, rank, local, pg


def max_over_ranks(x, pg, device):
    if pg is None:
        return x
    import torch
    t = torch.tensor([x], dtype=torch.float64, device=device)
    pg.all_reduce(t, op=pg.ReduceOp.MAX)
    return float(t.item())


def barrier(pg, device):
    import torch
    if pg is not None:
        t = torch.zeros(1, device=device)
        pg.all_reduce(t)
    if torch.cuda.is_available():
        torch.cuda.synchronize()


def reference_problem(workload):
    """The workload the reference CPU path runs: the same box, viscosity and
    BCs as the device leg (the whole problem, every size)."""
    from pt_b200 import mesh as M
    m, eta, mask = M.problem(workload, seed=0)
    return m, eta, mask, f"the whole {m.mx}x{m.my}x{m.mz} problem"


def cpu_model():
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                if line.startswith("model name"):
                    return line.split(":", 1)[1].strip()
    except OSError:
        pass
    return None


def _relerr(a, b):
    a = np.asarray(a, dtype=np.float64)
    b = np.asarray(b, dtype=np.float64)
    return float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))


def cpu_reference_leg(m, eta, mask, x, p, seconds=12.0, kind="avx", device_out=None):
    """The reference's own A11 (oracle/_ref, all host cores) on the device leg's
    box and inputs: best of the applies that fit in `seconds` (at least two),
    one apply on one thread, and one run of its diag, B, B^T and whole Stokes
    operator.  With device_out = {name: host array} each device result is
    checked against the reference's (MatShell-level BC rules of
    src/stokes_operators.c); returns (cpu_baseline dict, parity dict)."""
    import oracle
    if not oracle.RefCPU.available():
        oracle.build()
    r = oracle.RefCPU()

    def best_of(fn, budget):
        out = fn()  # warm-up (and the output to check)
        times, t_end = [], time.perf_counter() + budget
        while time.perf_counter() < t_end or len(times) < 2:
            t0 = time.perf_counter()
            fn()
            times.append(time.perf_counter() - t0)
        return min(times), len(times), out

    def once(fn):
        t0 = time.perf_counter()
        out = fn()
        return time.perf_counter() - t0, out

    nthreads = r.set_threads(os.cpu_count())
    best, nrep, y_ref = best_of(lambda: r.matmult_a11(m.dims, m.coords, eta, mask, x, kind), seconds)
    # one thread as well: the reference's element loop scatters under `omp critical`
    r.set_threads(1)
    t1, _ = once(lambda: r.matmult_a11(m.dims, m.coords, eta, mask, x, kind))
    r.set_threads(nthreads)
    t_diag, d_ref = once(lambda: r.getdiag_a11(m.dims, m.coords, eta, mask))
    t_a21, bu_ref = once(lambda: r.matmult_a21(m.dims, m.coords, mask, x))
    t_a12, btp_ref = once(lambda: r.matmult_a12(m.dims, m.coords, mask, p, kind))
    t_a, (au_ref, ap_ref) = once(lambda: r.matmult_a(m.dims, m.coords, eta, mask, x, p, kind))
    secs = {"diag": t_diag, "a21": t_a21, "a12": t_a12, "stokes_a": t_a}
    what = f"the whole {m.mx}x{m.my}x{m.mz} problem"
    cpu = {
        "value": m.nvel / best / 1e9,
        "unit": UNIT,
        "cores": nthreads,
        "kind": "reference",
        "sample": f"reference {kind} A11 (MatMult_MFStokes_A11 over MFStokesWrapper_A11_AVX, OpenMP {nthreads} "
                  f"threads) on {what}, same inputs as the device leg, best of {nrep} applies",
        "seconds_per_apply": best,
        "one_thread": {"value": m.nvel / t1 / 1e9, "seconds_per_apply": t1, "applies": 1},
        "cpu_model": cpu_model(),
        "ops_seconds": secs,
        "ops_gdofs": {k: (m.nvel + (m.npres if k == "stokes_a" else 0)) / v / 1e9 for k, v in secs.items()},
    }
    parity = None
    if device_out is not None:
        refs = {"a11": y_ref, "a11_e2e": y_ref, "diag": d_ref, "a21": bu_ref, "a12": btp_ref, "stokes_a_u": au_ref,
                "stokes_a_p": ap_ref}
        parity = {k: _relerr(device_out[k], v) for k, v in refs.items() if k in device_out}
        parity["max"] = max(parity.values()) if parity else None
        parity["against"] = (f"the reference's own CPU operators (oracle/_ref, {kind}) on {what}, "
                             "MatShell-level BC rules, max-norm relative error")
    return cpu, parity


def reference_residual(m, eta, mask, f, xsol, kind="avx"):
    """True FP64 relative residual ||f - A11 x|| / ||f|| of a device solution,
    with the reference's own A11 on the host (all cores); None where its
    library is not built and cannot be."""
    import oracle
    if not oracle.RefCPU.available():
        oracle.build()
    if not oracle.RefCPU.available():
        return None
    r = oracle.RefCPU()
    r.set_threads(os.cpu_count())
    res = f - r.matmult_a11(m.dims, m.coords, eta, mask, xsol, kind)
    return float(np.linalg.norm(res) / np.linalg.norm(f))


def run_reference(args):
    ws, rank, local, pg = int(os.environ.get("WORLD_SIZE", "1")), int(os.environ.get("RANK", "0")), 0, None
    if rank != 0:
        return 0
    try:
        import oracle
        if not oracle.RefCPU.available():
            oracle.build()
        oracle.RefCPU()
    except Exception as e:  # pragma: no cover
        print(json.dumps({"impl": "reference", "unavailable": f"reference CPU build missing: {e}"}))
        return 0
    from pt_b200 import mesh as M
    r = oracle.RefCPU()
    nthreads = r.set_threads(os.cpu_count())
    m, eta, mask, what = reference_problem(args.workload)
    x = M.uniform_vec(m.nvel, 7)
    # MatMult_MFStokes_A11 on the same inputs as the device leg (Dirichlet
    # columns zeroed, rows copied) through the reference's AVX element loop
    for _ in range(args.warmup):
        r.matmult_a11(m.dims, m.coords, eta, mask, x, "avx")
    t0 = time.perf_counter()
    for _ in range(args.steps):
        r.matmult_a11(m.dims, m.coords, eta, mask, x, "avx")
    dt = (time.perf_counter() - t0) / args.steps
    v = m.nvel / dt / 1e9
    line = {
        "impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": dt * 1e3, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": f"A11 FP64 MatMult, {m.mx}x{m.my}x{m.mz} Q2 box ({m.nvel} velocity dofs), "
                               f"{WORKLOAD_TEXT.get(args.workload.split(':')[0], args.workload)}, free-slip BCs",
                   "global_batch": 1, "seq_len": 0, "parallelism": "cpu-openmp",
                   "impl_detail": "reference CPU (oracle/_ref: MFStokesWrapper_A11_AVX compiled from the "
                                  "reference sources)"},
        "cpu_baseline": {"value": v, "unit": UNIT, "cores": nthreads, "kind": "reference",
                         "sample": f"{what}, every step one MatMult_MFStokes_A11 through the reference's AVX "
                                   "element loop compiled from its sources"},
        "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))
    return 0


def run_ours(args):
    import torch

    from pt_b200 import MatStokesMF
    from pt_b200 import mesh as M

    ws, rank, local, pg = dist_setup(args)
    dev = torch.device("cuda", local)
    torch.cuda.set_device(dev)

    m, eta, mask = M.problem(args.workload, seed=0)
    stream = torch.cuda.Stream(device=dev)
    op = MatStokesMF(*m.dims, a11_op=args.a11_op, stream=stream)
    op.SetUp(m.coords, eta, mask)
    x = torch.from_numpy(M.uniform_vec(m.nvel, 7)).to(dev)
    y = torch.empty_like(x)
    x32, y32 = x.float(), torch.empty(m.nvel, dtype=torch.float32, device=dev)
    p = torch.from_numpy(M.uniform_vec(m.npres, 8)).to(dev)
    yp = torch.empty(m.npres, dtype=torch.float64, device=dev)
    torch.cuda.synchronize()

    def timed(fn, k):
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with torch.cuda.stream(stream):
            ev0.record(stream)
            for _ in range(k):
                fn()
            ev1.record(stream)
        ev1.synchronize()
        return ev0.elapsed_time(ev1) / 1e3

    # ---- tile schedule by the autotuner (untimed), then the headline --------
    tiling = {"lz": op.tiling, "autotune": None}
    if not args.no_autotune and op.a11_op == "b200_stream":
        best, table = op.autotune_tiling(x)
        tiling = {"lz": best, "autotune_ms": {str(k): round(v, 4) for k, v in table.items()}}
    # ---- headline: FP64 A11 (MatShell level), device resident ----------------
    for _ in range(max(args.warmup, 3)):
        op.MatMult_MFStokes_A11(x, y)
    barrier(pg, dev)
    op.reset_launch_count()
    with ClockSampler(local) as clk:
        t = timed(lambda: op.MatMult_MFStokes_A11(x, y), args.steps)
    launches = op.launch_count()
    t = max_over_ranks(t, pg, dev)
    t_apply = t / args.steps
    value = ws * m.nvel / t_apply / 1e9

    # the timed apply's own output, checked against the reference below
    stream.synchronize()
    y_timed = y.cpu().numpy() if rank == 0 and ws == 1 else None
    a11_op = op.a11_op

    # ---- roofline of the A11 apply ---------------------------------------------
    peak, peak_kind = load_peaks()
    bytes_alg = algorithmic_bytes(m)
    achieved = bytes_alg / t_apply / 1e9

    # ---- other operators and FP32 (device resident) ------------------------------
    extra = {}
    if not args.quick:
        def rate(fn, n):
            for _ in range(2):
                fn()
            dt = timed(fn, max(2, args.steps // 2)) / max(2, args.steps // 2)
            return n / dt / 1e9, dt * 1e3
        extra["a11_fp32_gdofs"], extra["a11_fp32_ms"] = rate(lambda: op.MatMult_MFStokes_A11(x32, y32), m.nvel)
        # the SpMVOp-level apply (no Dirichlet columns or rows)
        extra["a11_spmvop_gdofs"], extra["a11_spmvop_ms"] = rate(lambda: op.MFStokesWrapper_A11(x, y), m.nvel)
        extra["diag_gdofs"], extra["diag_ms"] = rate(lambda: op.MatGetDiagonal_MFStokes_A11(y), m.nvel)
        extra["a21_gdofs"], extra["a21_ms"] = rate(lambda: op.MatMult_MFStokes_A21(x, yp), m.nvel)
        extra["a12_gdofs"], extra["a12_ms"] = rate(lambda: op.MatMult_MFStokes_A12(p, y), m.nvel)
        # the whole Stokes operator (A11 u + A12 p, A21 u), rate over velocity + pressure dofs
        extra["stokes_a_gdofs"], extra["stokes_a_ms"] = rate(lambda: op.MatMult_MFStokes_A(x, p, y, yp),
                                                             m.nvel + m.npres)
        extra["a11_flops_per_element_ref_count"] = 17253

    # ---- e2e through the host-pointer API (pinned buffers) ----------------------------
    xh = torch.empty(m.nvel, dtype=torch.float64, pin_memory=True)
    xh.copy_(x.cpu())
    yh = torch.empty(m.nvel, dtype=torch.float64, pin_memory=True)
    xn, yn = xh.numpy(), yh.numpy()
    # the host-pointer apply overlaps its copies with the compute group by group
    # of z-chunks; shorter chunks make a finer pipeline, so its chunk depth is
    # tuned (untimed) like the device apply's: the device choice or 2 layers
    lz_dev = op.tiling
    e2e_tune = {}
    if op.a11_op == "b200_stream" and not args.no_autotune:
        for lz in dict.fromkeys((lz_dev, 2)):
            op.set_tiling(lz)
            op.MatMult_MFStokes_A11(xn, yn)
            t0 = time.perf_counter()
            for _ in range(2):
                op.MatMult_MFStokes_A11(xn, yn)
            e2e_tune[op.tiling] = (time.perf_counter() - t0) / 2
        op.set_tiling(min(e2e_tune, key=e2e_tune.get))
    op.MatMult_MFStokes_A11(xn, yn)
    k_e2e = max(2, min(args.steps, 5))
    barrier(pg, dev)
    t0 = time.perf_counter()
    for _ in range(k_e2e):
        op.MatMult_MFStokes_A11(xn, yn)
    t_e2e = max_over_ranks((time.perf_counter() - t0) / k_e2e, pg, dev)
    e2e = {"value": ws * m.nvel / t_e2e / 1e9, "unit": UNIT, "h2d_bytes_per_step": 8 * m.nvel,
           "d2h_bytes_per_step": 8 * m.nvel, "ms_per_step": t_e2e * 1e3,
           "path": "pt_matmult_a11_h (MatMult_MFStokes_A11 on pinned numpy arrays)",
           "lz": op.tiling, "lz_tune_ms": {str(k): round(v * 1e3, 3) for k, v in e2e_tune.items()}}
    y_e2e = yn.copy() if rank == 0 and ws == 1 else None
    op.set_tiling(lz_dev)

    cpu, parity = None, None
    if rank == 0 and ws == 1 and not args.no_cpu_baseline:
        # device outputs of every operator on the bench inputs (host copies)
        dout = {"a11": y_timed, "a11_e2e": y_e2e}
        if not args.quick:
            # the op runs on its own stream: wait for it before each copy
            def host(t):
                stream.synchronize()
                return t.cpu().numpy()
            dout["diag"] = host(op.MatGetDiagonal_MFStokes_A11(y))
            dout["a21"] = host(op.MatMult_MFStokes_A21(x, yp))
            dout["a12"] = host(op.MatMult_MFStokes_A12(p, y))
            au, ap = op.MatMult_MFStokes_A(x, p, y, yp)
            dout["stokes_a_u"], dout["stokes_a_p"] = host(au), host(ap)
        try:
            cpu, parity = cpu_reference_leg(m, eta, mask, x.cpu().numpy(), p.cpu().numpy(),
                                            seconds=args.cpu_seconds, device_out=dout)
        except Exception as e:  # pragma: no cover
            cpu = {"value": None, "unit": UNIT, "cores": os.cpu_count(), "kind": "reference",
                   "sample": f"unavailable: {e}"}
        del dout

    # ---- the rest of the metric: precision-form solve, batched, served ------------
    if rank == 0 and ws == 1 and not args.quick and not args.no_legs:
        extra["solve"] = solve_leg(op, m, eta, mask, args, check=not args.no_cpu_baseline)
    op.Destroy()
    del x, y, x32, y32, p, yp
    torch.cuda.empty_cache()
    if rank == 0 and ws == 1 and not args.quick and not args.no_legs:
        extra["batched"] = batched_leg(args.nbatch, args.steps)
        torch.cuda.empty_cache()
        extra["serve"] = serve_leg(args, nreq=args.leg_nreq, ncal=args.leg_ncal, nserial=args.leg_nserial)

    if rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
            "warmup": max(args.warmup, 3), "ms_per_step": t_apply * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": f"A11 FP64 MatMult, {m.mx}x{m.my}x{m.mz} Q2 box ({m.nvel} velocity dofs), "
                                   f"{WORKLOAD_TEXT.get(args.workload.split(':')[0], args.workload)}, free-slip BCs",
                       "global_batch": 1, "seq_len": 0, "parallelism": f"replicas{ws}",
                       "a11_op": a11_op, "tiling": tiling, "l2": "inputs larger than L2 (no flush)"},
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": TRAFFIC_PER_ELEMENT_F64 * m.nel,
                         "traffic_source": "ncu dram__bytes_read+write per element of colour launches on a "
                                           "128x128x32 box (rows of 128 elements), times the element count",
                         "peak_kind": peak_kind, "algorithmic_bytes_per_apply": bytes_alg},
            "cpu_baseline": cpu,
            "parity_relerr": parity["max"] if parity else None,
            "parity": parity,
            "e2e": e2e,
            "gpu_launches": launches,
            "clocks": clk.summary(),
            "extra": extra,
        }
        print(json.dumps(line))
    if pg is not None:
        pg.destroy_process_group()
    return 0


def solve_leg(op, m, eta, mask, args, check=True):
    """Precision form on the op's box: A11 u = f (f uniform [-1, 1] on free
    dofs), FP64 outer Krylov (args.ksp) to rtol args.rtol, preconditioned by the
    geometric V-cycle with Chebyshev-Jacobi smoothing (args.pc) in FP64 and in
    FP32.  Each solver is set up first (levels, eigenvalue estimates, the
    V-cycle graph: one PCApply, timed apart), then one solve is timed.  With
    check=True the true residual of each solution comes from the reference's
    own A11 on the host, and the FP32-smoothed solution's error is stated
    against the FP64-smoothed one."""
    import torch

    from pt_b200 import mesh as M
    from pt_b200.solver import KSPSolveA11
    f = M.uniform_vec(m.nvel, 11)
    f[mask.astype(bool)] = 0.0
    fd = torch.from_numpy(f).to(torch.device("cuda", torch.cuda.current_device()))
    emin, emax = (float(v) for v in args.cheby_window.split(","))
    out = {"workload": f"{m.mx}x{m.my}x{m.mz} box of the apply leg", "nvel": m.nvel, "ksp": args.ksp,
           "pc": args.pc, "cheby_degree": args.cheby_degree, "cheby_window": [emin, emax], "rtol": args.rtol,
           "tiling_lz": op.tiling}
    sols = {}
    modes = [(n, f) for n, f in (("fp64", 0), ("fp32_smoothed", 1)) if n in args.solve_modes.split(",")]
    if args.fine_degree:
        out["fine_degree"] = args.fine_degree
    for name, fp32 in modes:
        x = torch.zeros_like(fd)
        with KSPSolveA11(op, ksp=args.ksp, pc=args.pc, cheby_degree=args.cheby_degree, cheby_fp32=fp32,
                         rtol=args.rtol, max_it=args.max_it, restart=args.restart,
                         mg_fine_degree=args.fine_degree, cheby_emin=emin, cheby_emax=emax) as k:
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            k.apply_pc(fd, x)   # PCSetUp + one V-cycle
            torch.cuda.synchronize()
            t_setup = time.perf_counter() - t0
            x.zero_()
            st = k.solve(fd, x)
        st["setup_seconds"] = t_setup
        sols[name] = x.cpu().numpy()
        del x
        out[name] = st
    if len(sols) == 2:
        out["solution_relerr_fp32_vs_fp64"] = _relerr(sols["fp32_smoothed"], sols["fp64"])
        out["time_to_solution_speedup"] = out["fp64"]["seconds"] / out["fp32_smoothed"]["seconds"]
    if check:
        for name in sols:
            out[name]["true_relres_reference_a11"] = reference_residual(m, eta, mask, f, sols[name])
    return out


def run_solve(args):
    """--mode solve: the precision-form leg alone on args.workload; prints one
    JSON line."""
    import torch

    from pt_b200 import MatStokesMF
    from pt_b200 import mesh as M
    torch.cuda.set_device(0)
    m, eta, mask = M.problem(args.workload, seed=0)
    op = MatStokesMF(*m.dims)
    op.SetUp(m.coords, eta, mask)
    if not args.no_autotune:
        op.autotune_tiling(torch.from_numpy(M.uniform_vec(m.nvel, 7)).cuda())
    out = {"mode": "solve", "workload": args.workload}
    out.update(solve_leg(op, m, eta, mask, args, check=not args.no_cpu_baseline))
    print(json.dumps(out))
    op.Destroy()
    return 0


def batched_problems(n=256, seed=0):
    """The batched workload: n boxes with axes drawn from {8,12,16,24,32},
    per-element log-uniform eta with contrast drawn from {1e2,1e4,1e6},
    nodes perturbed +-0.05h, free-slip box BCs."""
    from pt_b200 import mesh as M
    rng = np.random.default_rng(seed)
    axes = np.array([8, 12, 16, 24, 32])
    out = []
    for i in range(n):
        mx, my, mz = (int(v) for v in rng.choice(axes, size=3))
        c = float(rng.choice([1e2, 1e4, 1e6]))
        m = M.make_mesh(mx, my, mz, perturb=0.05, seed=seed * 100003 + i)
        eta = M.eta_per_element(m, contrast=c, seed=seed * 100003 + i)
        out.append((m, eta, M.bc_mask_freeslip(mx, my, mz)))
    return out


def batched_leg(nbatch, steps):
    """Batched form: one batched A11 apply over all problems (work-list
    launches) vs the same problems applied one after another, FP64 and FP32."""
    import torch

    from pt_b200 import MatStokesMF
    from pt_b200.batch import BatchA11, autotune_lz
    probs = batched_problems(nbatch, seed=0)
    ops, us64 = [], []
    for i, (m, eta, mask) in enumerate(probs):
        op = MatStokesMF(*m.dims)
        op.SetUp(m.coords, eta, mask)
        ops.append(op)
        us64.append(torch.from_numpy(M_uniform(m.nvel, 1000 + i)).cuda())
    ndof = sum(m.nvel for m, _, _ in probs)
    out = {"mode": "batched", "problems": len(probs), "velocity_dofs": ndof,
           "elements": int(sum(m.nel for m, _, _ in probs))}

    def timed(fn, k):
        for _ in range(2):
            fn()
        torch.cuda.synchronize()
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev0.record()
        for _ in range(k):
            fn()
        ev1.record()
        ev1.synchronize()
        return ev0.elapsed_time(ev1) / k

    for prec, us in (("fp64", us64), ("fp32", [u.float() for u in us64])):
        ys = [torch.empty_like(u) for u in us]
        best, table = autotune_lz(ops, us, ys)
        with BatchA11(ops, lz=best if best else None) as b:
            t_b = timed(lambda: b.apply(us, ys, masked=True), steps)
            launches = b.launches_per_apply
        # sequential baselines: each box's own default apply ("b200": stored element
        # matrices up to 32^3, else streaming), and the streaming kernel the batch runs
        t_s = timed(lambda: [op.MatMult_MFStokes_A11(u, y) for op, u, y in zip(ops, us, ys)], max(2, steps // 4))
        for op in ops:
            op.set_a11_op("b200_stream")
        t_ss = timed(lambda: [op.MatMult_MFStokes_A11(u, y) for op, u, y in zip(ops, us, ys)], max(2, steps // 4))
        for op in ops:
            op.set_a11_op("b200")
        out[prec] = {"batched_ms": t_b, "sequential_ms": t_s, "batched_gdofs": ndof / t_b / 1e6,
                     "sequential_gdofs": ndof / t_s / 1e6, "speedup": t_s / t_b,
                     "sequential_stream_ms": t_ss, "speedup_vs_sequential_stream": t_ss / t_b,
                     "launches_per_apply": launches, "autotune_lz": best, "autotune_ms": table}
    for op in ops:
        op.Destroy()
    return out


def run_batched(args):
    """--mode batched: the batched leg alone; prints one JSON line."""
    import torch
    torch.cuda.set_device(0)
    print(json.dumps(batched_leg(args.nbatch, args.steps)))
    return 0


class RequestStream:
    """The served stream: cubic boxes m^3, m uniform over sizes; nodes
    perturbed +-0.05h; viscosity 1 with 8 seeded inclusions (radius 0.1), four
    at c^(1/2) and four at c^(-1/2), c log-uniform in [1e2, 1e6]; free-slip box
    BCs; f uniform [-1, 1] on free dofs.  Request i is (mesh, eta, mask, f, c),
    built on demand from its seeds (the size and contrast draws are made up
    front, in order); start(ahead) builds requests in a background thread up to
    `ahead` beyond the last one taken, so a long stream never holds more than a
    window of requests in host memory."""

    def __init__(self, n, seed=0, sizes=(8, 48)):
        rng = np.random.default_rng(seed)
        self.n, self.seed, self.draws = n, seed, []
        for _ in range(n):
            m = int(rng.integers(sizes[0], sizes[1] + 1))
            self.draws.append((m, 10.0 ** rng.uniform(2.0, 6.0)))
        self._ready, self._next, self._taken = {}, 0, 0
        self._cv = threading.Condition()
        self._thread = None
        self.build_seconds = 0.0

    def __len__(self):
        return self.n

    def make(self, i):
        from pt_b200 import mesh as M
        m, c = self.draws[i]
        seed = self.seed
        mesh = M.make_mesh(m, m, m, perturb=0.05, seed=seed * 1000003 + i)
        r = np.random.default_rng(seed * 7919 + i + 1)
        centres = r.uniform(0.0, 1.0, size=(8, 3))
        vals = [c ** 0.5] * 4 + [c ** -0.5] * 4
        eta = M.eta_spheres(mesh, centres, [0.1] * 8, vals)
        mask = M.bc_mask_freeslip(m, m, m)
        f = M_uniform(mesh.nvel, seed * 31 + i)
        f[mask.astype(bool)] = 0.0
        return mesh, eta, mask, f, c

    def start(self, ahead=48):
        def run():
            while True:
                with self._cv:
                    while self._next < self.n and self._next >= self._taken + ahead:
                        self._cv.wait()
                    if self._next >= self.n:
                        return
                    i = self._next
                    self._next += 1
                t0 = time.perf_counter()
                req = self.make(i)
                with self._cv:
                    self.build_seconds += time.perf_counter() - t0
                    self._ready[i] = req
                    self._cv.notify_all()
        self._thread = threading.Thread(target=run, daemon=True)
        self._thread.start()
        return self

    def take(self, i):
        """Request i, in order; blocks until the producer has built it."""
        if self._thread is None:
            return self.make(i)
        with self._cv:
            while i not in self._ready:
                self._cv.wait()
            req = self._ready.pop(i)
            self._taken = i + 1
            self._cv.notify_all()
        return req


def serve_requests(n, seed=0, sizes=(8, 48)):
    """All n requests of the stream, built at once (short streams)."""
    st = RequestStream(n, seed, sizes)
    return [st.make(i) for i in range(n)]


def serve_run(reqs, arrivals, iters, keep_x=None, **opts):
    """Serve reqs (a list or a started RequestStream) arriving at the given
    times (seconds on the server clock, relative to the first arrival).
    Returns (results by id, stats); solutions are kept for the ids in keep_x
    (all when None)."""
    from pt_b200.serve import Server
    res, max_active, max_bytes = {}, 0, 0
    take = reqs.take if isinstance(reqs, RequestStream) else (lambda i: reqs[i])
    n = len(reqs)
    with Server(**opts) as s:
        t0 = s.time()
        nxt = 0
        while len(res) < n:
            now = s.time() - t0
            while nxt < n and arrivals[nxt] <= now:
                m, eta, mask, f, _ = take(nxt)
                s.submit(nxt, m.dims, m.coords, eta, mask, f)
                nxt += 1
            act, queued = s.step(iters)
            max_active = max(max_active, act)
            max_bytes = max(max_bytes, s.stats()["bytes_in_use"])
            for d in s.done():
                d["t_done"] -= t0
                d["t_submit"] -= t0
                d["t_admit"] -= t0
                if keep_x is not None and d["id"] not in keep_x:
                    d.pop("x")
                res[d["id"]] = d
            if act == 0 and queued == 0 and nxt < n:
                time.sleep(max(0.0, min(0.01, arrivals[nxt] - (s.time() - t0))))
        st = s.stats()
    st.update(max_active=max_active, max_bytes_in_use=max_bytes)
    return res, st


def serve_leg(args, nreq, ncal, nserial):
    """Serving form: Poisson arrivals at ~80% of the measured capacity, solves
    of A11 u = f to rtol 1e-8 by FP32 Chebyshev(3)-Jacobi-preconditioned FP64
    CG, continuously batched; p50/p99 latency and solves/s against serial
    plain FP64 solves of the same requests.  The true FP64 residual of a sample
    of served results comes from the reference's own A11 on the host."""
    import torch

    from pt_b200 import MatStokesMF
    from pt_b200.solver import KSPSolveA11
    t_gen = time.time()
    cal = serve_requests(ncal, seed=1)
    reqs = RequestStream(nreq, seed=0)
    t_gen = time.time() - t_gen
    # tile schedule (tile width, z-chunk depth) by the autotuner, on the
    # calibration requests' FP32 applies
    from pt_b200.batch import autotune
    ops = []
    for m, eta, mask, _, _ in cal:
        op = MatStokesMF(*m.dims)
        op.SetUp(m.coords, eta, mask)
        ops.append(op)
    us = [torch.ones(op.nvel, dtype=torch.float32, device="cuda") for op in ops]
    ys = [torch.empty_like(u) for u in us]
    (lz, tile_x), table = autotune(ops, us, ys, lz_candidates=(1, 2, 0), tile_candidates=(0, 64, 128))
    for op in ops:
        op.Destroy()
    emin, emax = (float(v) for v in args.cheby_window.split(","))
    opts = dict(rtol=args.rtol, max_it=args.max_it, cheby_fp32=1, cheby_degree=args.cheby_degree,
                cheby_emin=emin, cheby_emax=emax, memory_budget_bytes=120 << 30, max_active=256, lz=lz,
                tile_x=tile_x)
    # capacity: a saturated queue (everything arrives at once)
    res_cal, _ = serve_run(cal, [0.0] * len(cal), args.serve_iters, **opts)
    capacity = len(cal) / max(d["t_done"] for d in res_cal.values())
    rate = 0.8 * capacity
    rng = np.random.default_rng(12345)
    arrivals = np.cumsum(rng.exponential(1.0 / rate, size=len(reqs)))
    arrivals -= arrivals[0]
    sample = list(range(0, len(reqs), max(1, len(reqs) // 8)))
    reqs.start()
    res, st = serve_run(reqs, arrivals, args.serve_iters, keep_x=set(sample), **opts)
    lat = np.array([res[i]["t_done"] - arrivals[i] for i in range(len(reqs))])
    wall = max(d["t_done"] for d in res.values())
    its = np.array([res[i]["its"] for i in range(len(reqs))])
    conv = all(res[i]["converged"] for i in range(len(reqs)))
    # true FP64 residual of a sample of served results
    relres = []
    for i in sample:
        m, eta, mask, f, _ = reqs.make(i)
        relres.append(reference_residual(m, eta, mask, f, res[i]["x"]))
    relres = [r for r in relres if r is not None]
    # serial plain FP64 solves (one request at a time, set-up included)
    serial = []
    for i in np.linspace(0, len(reqs) - 1, min(nserial, len(reqs))).astype(int):
        m, eta, mask, f, _ = reqs.make(int(i))
        torch.cuda.synchronize()
        t = time.time()
        with MatStokesMF(*m.dims) as op:
            op.SetUp(m.coords, eta, mask)
            fd = torch.from_numpy(f).cuda()
            x = torch.zeros_like(fd)
            with KSPSolveA11(op, ksp="fcg", pc="cheby_jacobi", cheby_fp32=0, cheby_degree=args.cheby_degree,
                             cheby_emin=emin, cheby_emax=emax, rtol=args.rtol, max_it=args.max_it) as k:
                sst = k.solve(fd, x)
            x.cpu()
        serial.append({"seconds": time.time() - t, "its": sst["its"], "converged": sst["converged"],
                       "elements": m.nel, "served_its": res[int(i)]["its"]})
    serial_rate = len(serial) / sum(d["seconds"] for d in serial)
    out = {"mode": "serve", "requests": len(reqs), "sizes": "m^3, m uniform 8..48",
           "contrast": "log-uniform [1e2, 1e6]", "rtol": args.rtol, "cheby_window": [emin, emax],
           "iterations_per_step": args.serve_iters,
           "capacity_solves_per_s": capacity, "arrival_rate_per_s": rate, "calibration_requests": len(cal),
           "solves_per_s": len(reqs) / wall, "p50_latency_s": float(np.percentile(lat, 50)),
           "p99_latency_s": float(np.percentile(lat, 99)), "mean_its": float(its.mean()),
           "max_its": int(its.max()), "all_converged": conv, "true_relres_sample_max": max(relres, default=None),
           "serial_fp64_solves_per_s": serial_rate, "serial_sample": len(serial),
           "serial_mean_its": float(np.mean([d["its"] for d in serial])),
           "serial_mean_served_its_same_requests": float(np.mean([d["served_its"] for d in serial])),
           "speedup_solves_per_s": (len(reqs) / wall) / serial_rate, "server": st,
           "autotune": {"lz": lz, "tile_x": tile_x, "ms": {f"lz{a}_tx{b}": v for (a, b), v in table.items()}},
           "host_generation_s": t_gen + reqs.build_seconds,
           "latency_percentiles_s": {str(q): float(np.percentile(lat, q)) for q in (10, 25, 50, 75, 90, 95, 99, 99.9)},
           "contrast_its": {f"1e{k}-1e{k + 1}": float(np.mean([res[i]["its"] for i in range(len(reqs))
                                                              if 10 ** k <= reqs.draws[i][1] < 10 ** (k + 1)]))
                            for k in (2, 3, 4, 5)}}
    return out


def run_serve(args):
    """--mode serve: the served stream alone (args.nreq requests); prints one
    JSON line."""
    import torch
    torch.cuda.set_device(0)
    print(json.dumps(serve_leg(args, args.nreq, args.ncal, args.nserial)))
    return 0


def run_markers(args):
    """Coefficient producer: Gauss-point (eta, rho) from material points by the
    reference's Q1 projection, device-resident markers (CUDA events) and the
    host path, against the reference's own CPU projection on the same markers."""
    import torch

    from pt_b200 import MatStokesMF
    from pt_b200 import mesh as M
    torch.cuda.set_device(0)
    m, _, _ = M.problem(args.workload, seed=0)
    wil, xi, _, eta, rho = M.markers(m, args.markers_per_element, seed=3)
    n = len(wil)
    op = MatStokesMF(*m.dims)
    op.set_coords(m.coords)
    dw, dx = torch.from_numpy(wil).cuda(), torch.from_numpy(xi).cuda()
    de, dr = torch.from_numpy(eta).cuda(), torch.from_numpy(rho).cuda()
    for _ in range(max(args.warmup, 3)):
        op.ProjectMarkers(dw, dx, de, dr, install=False)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        op.ProjectMarkers(dw, dx, de, dr, install=False)
    torch.cuda.synchronize()
    t_dev = (time.perf_counter() - t0) / args.steps
    t0 = time.perf_counter()
    for _ in range(max(1, args.steps // 4)):
        eq, rq = op.ProjectMarkers(wil, xi, eta, rho, install=False)
    t_host = (time.perf_counter() - t0) / max(1, args.steps // 4)
    out = {"mode": "markers", "workload": args.workload, "elements": m.nel, "markers": n,
           "gpu_ms": t_dev * 1e3, "gpu_markers_per_s": n / t_dev, "e2e_ms": t_host * 1e3}
    if not args.no_cpu_baseline:
        import oracle
        if not oracle.RefCPU.available():
            oracle.build()
        r = oracle.RefCPU()
        t0 = time.perf_counter()
        req, rrq = r.marker_project(m.dims, wil, xi, eta, rho)
        t_cpu = time.perf_counter() - t0
        rel = float(np.abs(eq - req).max() / np.abs(req).max())
        out.update(cpu_ms=t_cpu * 1e3, cpu_kind="reference (material_point_utils.c, one thread: its loops are serial)",
                   speedup=t_cpu / t_dev, relerr_vs_reference=rel)
    op.Destroy()
    print(json.dumps(out))
    return 0


def M_uniform(n, seed):
    return np.random.default_rng(seed).uniform(-1.0, 1.0, size=n)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="c2")
    ap.add_argument("--a11-op", default="b200")
    ap.add_argument("--quick", action="store_true", help="headline A11 only")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-autotune", action="store_true", help="apply: keep the default tile schedule")
    ap.add_argument("--cpu-seconds", type=float, default=12.0)
    ap.add_argument("--mode", default="apply", choices=["apply", "solve", "batched", "serve", "markers"])
    ap.add_argument("--markers-per-element", type=int, default=8)
    ap.add_argument("--nreq", type=int, default=200, help="serve: requests in the measured stream")
    ap.add_argument("--ncal", type=int, default=48, help="serve: requests of the capacity calibration")
    ap.add_argument("--nserial", type=int, default=12, help="serve: requests solved one at a time")
    ap.add_argument("--serve-iters", type=int, default=8, help="serve: iterations per server step")
    ap.add_argument("--nbatch", type=int, default=256)
    ap.add_argument("--no-legs", action="store_true",
                    help="apply mode: skip the solve / batched / served legs of the default line")
    ap.add_argument("--leg-nreq", type=int, default=100, help="served leg of the default line: requests")
    ap.add_argument("--leg-ncal", type=int, default=32, help="served leg: capacity calibration requests")
    ap.add_argument("--leg-nserial", type=int, default=100,
                    help="served leg: requests solved one at a time (all of the leg's requests by default)")
    ap.add_argument("--ksp", default="fcg")
    ap.add_argument("--rtol", type=float, default=1e-8)
    ap.add_argument("--max-it", type=int, default=20000)
    ap.add_argument("--restart", type=int, default=30)
    ap.add_argument("--pc", default="mg", choices=["mg", "cheby_jacobi", "jacobi", "none"])
    ap.add_argument("--cheby-degree", type=int, default=3)
    ap.add_argument("--fine-degree", type=int, default=0, help="solve: Chebyshev degree on the finest level (0 = same)")
    ap.add_argument("--cheby-window", default="0.03,1.1",
                    help="solve and serve: Chebyshev window as fractions of lambda_max (the reference's esteig "
                         "window is 0.2,1.1; 0.03,1.1 measured 23%% faster to rtol 1e-8 on the 128^3 workload "
                         "and 17%% faster on served-request boxes)")
    ap.add_argument("--solve-modes", default="fp64,fp32_smoothed", help="solve: which smoother precisions to run")
    args = ap.parse_args()
    if args.mode == "solve":
        return run_solve(args)
    if args.mode == "batched":
        return run_batched(args)
    if args.mode == "serve":
        return run_serve(args)
    if args.mode == "markers":
        return run_markers(args)
    if args.impl == "reference":
        return run_reference(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
