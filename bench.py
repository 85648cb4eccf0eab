"""Benchmark of the elastic solve path on GB300.

Workload: the polycrystal configuration the headline metric is quoted on -- 3D nodal linear
elasticity, 256^3-cell coarse level plus a refined (ratio 2) patch over the central 1/8 of the
volume (two AMR levels of 257^3 nodes each), cubic C11/C12/C44 = 1.68/1.21/0.75 on 64 seeded
Voronoi grains with Haar-uniform rotations, u = 0 on z = 0, u_z = 0.01 on z = 1, traction-free
lateral faces, V-cycle with 2 pre/2 post damped-Jacobi sweeps and a CG bottom solve, to a 1e-8
relative residual.  One step = one full solve from u = 0 on inputs resident in HBM.

  value        mixed-precision solves/s (FP32 cycle inside FP64 refinement), device-timed
  fp64         plain FP64 solves/s (same solver, FP64 throughout)
  e2e          mixed solves/s through ae_solve with pinned HOST buffers (H2D + D2H in the region)
  roofline     the FP32 fused Jacobi sweep on the finest coarse level (the dominant kernel)
  cpu_baseline the FP64 oracle (a C++ restatement of the reference's CPU path) on a bounded
               sample of the same workload, extrapolated to one solve
  batch        batched periodic RVEs: 512 polycrystal cells, edges uniform in {16,24,32,48,64}
               (seed 4), 8-32 grains each (seed 5 + cell), exx = 1e-3, to 1e-8; all cells in one
               graph-replayed batch (mixed precision, and FP64) against the same solves run one
               cell at a time in FP64; the FP64 oracle on a sample of cells as the CPU baseline
  serve        served homogenisation: Poisson request streams (seed 6) of cells with edges
               uniform in {32, 40, ..., 128}, 8-64 grains and the six unit strains (1e-3) as
               load cases, into the continuous-batching server; p50/p99 latency and solves/s per
               arrival rate, mixed against FP64

python bench.py --gpus N --steps K --warmup W [--impl reference]
"""
import argparse
import ctypes as C
import functools
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "mixed vs FP64 elastic solves/s @1e-8 resid; p50/p99 latency; Fapply HBM GB/s"
UNIT = "solves/s"
L2_BYTES = 129 * 2 ** 20
# FP32 fused Jacobi sweep, cubic 21-coefficient stiffness: x in 12 + b 12 + diag 12 + C 84 + x out 12
JACOBI32_BYTES_PER_NODE = 132
FAPPLY64_BYTES_PER_NODE = 216
FAPPLY32_BYTES_PER_NODE = 108
# the same kernels on a grain map: stiffness 2 B per node (uint16 grain id) instead of 84 / 168
JACOBI32_BYTES_PER_NODE_GRAINS = 12 + 12 + 12 + 2 + 12
FAPPLY64_BYTES_PER_NODE_GRAINS = 24 + 2 + 24
FAPPLY32_BYTES_PER_NODE_GRAINS = 12 + 2 + 12
# measured DRAM bytes per node of the FP32 Jacobi sweep (ncu dram__bytes_read.sum +
# dram__bytes_write.sum at 193^3, larger than L2), keyed by grain map on/off.  Grain map: the
# split sweep's tiled kernel over the interior box (x 12, b 12, 1/D 12, id + direction mask 4,
# out 12 = 52 algorithmic bytes), per node of that box; per node: the one-pass kernel.
JACOBI32_TRAFFIC_PER_NODE = {True: 52.1, False: 131.1}
# FP64 operations per node (FMA counted as 2) of the FP64 Fapply on a grain map: the interior row's 99
# operations, 60 of them FMAs; the 6 % of the nodes with a grad C column add to it
FAPPLY64_FLOPS_PER_NODE_GRAINS = 159.0
# FP64 composite iterations the config needs (measured by this benchmark's FP64 solve, which
# matches the oracle iteration for iteration); used to extrapolate the CPU oracle's per-iteration
# time to a full solve in the reference arm, which cannot afford a full CPU solve.
FP64_ITERS_OVERRIDE = int(os.environ.get("AE_FP64_ITERS", "0"))


def workload_label(n):
    """The workload both arms report in config.workload."""
    return ("polycrystal 2-level AMR: %d^3 cells + ratio-2 patch over the central 1/8 (2 x %d^3 nodes), "
            "cubic 1.68/1.21/0.75, 64 Voronoi grains" % (n, n + 1))


def workload(n=256, nseeds=64, seed_points=1, seed_rot=2):
    """Levels, stiffness and right-hand sides of the two-level polycrystal (host arrays)."""
    from anisotropicfracture_gb300 import microstructure, models
    from anisotropicfracture_gb300.elastic import BCElastic
    levels = [dict(cells=n, lo=0, hi=n, ng=0),
              dict(cells=2 * n, lo=n // 2, hi=3 * n // 2, ng=2)]
    seeds = microstructure.voronoi_seeds(nseeds, seed_points)
    rot = models.random_rotations(nseeds, np.random.default_rng(seed_rot))
    table = models.cubic(1.68, 1.21, 0.75, rot)
    bc = BCElastic()
    for f in ["XLO", "XHI", "YLO", "YHI", "XLO_YLO", "XLO_YHI", "XHI_YLO", "XHI_YHI"]:
        for d in range(3):
            bc.Set(f, d, bc.Traction, 0.0)
    from anisotropicfracture_gb300.elastic import FACES
    for f in FACES:
        if "ZHI" in f:
            bc.Set(f, 2, bc.Displacement, 0.01)
    out = []
    for L in levels:
        dx = 1.0 / L["cells"]
        lo = [L["lo"] - L["ng"]] * 3
        hi = [L["hi"] + L["ng"]] * 3
        gid = microstructure.voronoi_grain_ids(lo, hi, (dx, dx, dx), seeds)
        Cf = np.ascontiguousarray(np.moveaxis(table[gid].astype(np.float64), -1, 0))
        out.append(dict(L, dx=dx, store_lo=lo, store_hi=hi, C=Cf, gid=np.ascontiguousarray(gid[None].astype(np.int32)),
                        table=table))
    return out, bc


def level_shape(level):
    return tuple(level["store_hi"][d] - level["store_lo"][d] + 1 for d in (2, 1, 0))


def valid_part(level, arr):
    """The valid nodes of a level array (storage minus the ghost layers of a refined patch): the
    composite solution the residual norm constrains.  Ghost values depend on the iteration
    history (they receive interpolated corrections), so errors are measured without them."""
    g = level["ng"]
    if g == 0:
        return arr
    return arr[:, g:-g, g:-g, g:-g]


def rel_err(levels, xs, ref):
    """max |x - ref| / max |ref| over the valid nodes of every level"""
    scale = max(float(np.abs(valid_part(L, r)).max()) for L, r in zip(levels, ref))
    return max(float(np.abs(valid_part(L, a) - valid_part(L, b)).max()) for L, a, b in zip(levels, xs, ref)) / scale


def oracle_level(level):
    from oracle import pyoracle as po
    return po.level(level["cells"], lo=(level["lo"],) * 3, hi=(level["hi"],) * 3, ng=level["ng"])


def oracle_rhs(level, bc):
    """BC values on domain-boundary nodes (BC::Operator::Elastic::Init), zero elsewhere; CPU."""
    from oracle import pyoracle as po
    return po.bc_init(oracle_level(level), bc.type, bc.val, np.zeros((3,) + level_shape(level)))


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms during the timed region."""
    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), "--query-gpu=" + self.Q,
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 8:
                continue
            try:
                sm.append(float(f[0]))
                mx.append(float(f[1]))
            except ValueError:
                continue
            for nm, v in zip(names, f[4:8]):
                if v.lower().startswith("active"):
                    reasons.add(nm)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def fp64_peak_tflops(n=4096, reps=3):
    """The FP64 rate the GPU sustains on a cuBLAS DGEMM (torch.matmul of two n x n float64
    matrices), best of reps, CUDA events: the denominator of the FP64 kernels' FLOP fraction."""
    import torch
    a = torch.randn(n, n, dtype=torch.float64, device="cuda")
    b = torch.randn(n, n, dtype=torch.float64, device="cuda")
    torch.matmul(a, b)
    torch.cuda.synchronize()
    best = float("inf")
    for _ in range(reps):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        torch.matmul(a, b)
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    del a, b
    torch.cuda.empty_cache()
    return 2.0 * n ** 3 / (best * 1e-3) / 1e12


def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


def cpu_oracle_sample(levels, bc, n_iters_solve, sample_iters=1, threads=None, rhs=None):
    """Time the FP64 oracle on the full workload: set-up plus `sample_iters` composite
    iterations; extrapolate to a solve of `n_iters_solve` iterations."""
    from oracle import pyoracle as po
    if threads:
        po.set_threads(threads)
    Ls, Cs, us, bs = [], [], [], []
    for a, L in enumerate(levels):
        Ls.append(oracle_level(L))
        Cs.append(L["C"])
        bs.append(rhs[a] if rhs is not None else oracle_rhs(L, bc))
        us.append(np.zeros_like(bs[-1]))
    t0 = time.perf_counter()
    po.solve_amr(Ls, po.ORC_MAJORMINOR, Cs, bc.type, us, bs, 1e-30, 0.0, max_iter=0)
    t_setup = time.perf_counter() - t0
    t0 = time.perf_counter()
    po.solve_amr(Ls, po.ORC_MAJORMINOR, Cs, bc.type, us, bs, 1e-30, 0.0, max_iter=sample_iters)
    t_iters = time.perf_counter() - t0 - t_setup
    t_iter = max(t_iters, 1e-9) / sample_iters
    t_solve = t_setup + n_iters_solve * t_iter
    return dict(value=1.0 / t_solve, unit=UNIT, cores=po.lib().orc_num_threads(), kind="port",
                sample="FP64 oracle on the full two-level 257^3 workload: set-up %.1f s + %d composite "
                       "iteration(s) at %.2f s each, extrapolated to the %d iterations a solve needs"
                       % (t_setup, sample_iters, t_iter, n_iters_solve))


def cpu_single_thread(levels, bc, cpu):
    """The same solve on one host thread (the reference's per-rank Fapply/Fsmooth are
    single-threaded), estimated from the oracle's Fapply on the coarse level timed at one thread
    and at all threads: one solve at one thread ~ the all-thread solve x that ratio."""
    from oracle import pyoracle as po
    L = levels[0]
    Lo = oracle_level(L)
    u = np.random.default_rng(0).standard_normal((3,) + level_shape(L))
    nthreads = po.lib().orc_num_threads()

    def t_apply(threads):
        po.set_threads(threads)
        po.fapply(Lo, po.ORC_MAJORMINOR, L["C"], bc.type, u)  # warm
        t0 = time.perf_counter()
        po.fapply(Lo, po.ORC_MAJORMINOR, L["C"], bc.type, u)
        return time.perf_counter() - t0

    t1 = t_apply(1)
    tn = t_apply(nthreads)
    po.set_threads(nthreads)
    ratio = t1 / tn
    return {"value": cpu["value"] / ratio, "unit": UNIT, "cores": 1,
            "sample": "all-thread oracle solve time x the Fapply time ratio 1 thread / %d threads on the "
                      "%d^3-node coarse level (%.2f s / %.3f s = %.1f)" % (nthreads, L["cells"] + 1, t1, tn, ratio)}


def config1_solve_iters():
    """(iterations of the two-level workload's FP64 solve, where that count comes from): the
    oracle's own full solve (tests/golden/config1_oracle.npz, made by
    tests/golden/make_config1_oracle.py) when its record is present."""
    path = os.path.join(ROOT, "tests", "golden", "config1_oracle.npz")
    if FP64_ITERS_OVERRIDE:
        return FP64_ITERS_OVERRIDE, "AE_FP64_ITERS"
    if os.path.exists(path):
        z = np.load(path)
        return int(z["iters"]), "the oracle's full FP64 solve of this workload (%.0f s on %d host threads)" % (
            float(z["seconds"]), int(z["threads"]))
    return 167, "the GPU FP64 solve of this workload"


def config_of(n):
    """The config both arms print (identical dicts; the precision each arm computes in is a
    top-level key)."""
    return {"workload": workload_label(n), "cycle": "V-cycle, 2 pre + 2 post damped-Jacobi sweeps, CG bottom",
            "tol_rel": 1e-8, "nodes": 2 * (n + 1) ** 3}


def run_reference(args, rank):
    """Reference arm: the reference's CPU path (its C++ restatement in oracle/, pinned bit for bit
    to the reference's own compiled per-node code; the reference as a whole needs AMReX, Eigen and
    MPI, absent here) on the host cores.  The set-up (stiffness restricted to every multigrid
    level, diagonals) is timed once; each step then runs set-up plus --ref-sample-iters composite
    iterations, and the solve time is extrapolated to the iteration count of a full solve."""
    if rank != 0:
        return
    from oracle import pyoracle as po
    po.set_threads(os.cpu_count())
    levels, bc = workload(args.cells)
    iters, src = config1_solve_iters()
    Ls = [oracle_level(L) for L in levels]
    Cs = [L["C"] for L in levels]
    bs = [oracle_rhs(L, bc) for L in levels]
    us = [np.zeros_like(b) for b in bs]
    kw = dict(max_fmg_iter=0, bottom=0, nu1=1, nu2=1)
    t0 = time.perf_counter()
    po.solve_amr(Ls, po.ORC_MAJORMINOR, Cs, bc.type, us, bs, 1e-30, 0.0, max_iter=0, **kw)
    t_setup = time.perf_counter() - t0
    m = max(1, args.ref_sample_iters)
    steps = []
    for k in range(args.warmup + args.steps):
        it = 1 if k < args.warmup else m
        t0 = time.perf_counter()
        po.solve_amr(Ls, po.ORC_MAJORMINOR, Cs, bc.type, us, bs, 1e-30, 0.0, max_iter=it, **kw)
        if k >= args.warmup:
            steps.append(time.perf_counter() - t0)
    t_step = float(np.mean(steps))
    t_iter = max(t_step - t_setup, 1e-9) / m
    t_solve = t_setup + iters * t_iter
    v = 1.0 / t_solve
    cores = po.lib().orc_num_threads()
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": t_step * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "precision": "fp64", "data": "synthetic",
            "config": config_of(args.cells),
            "solve_seconds_extrapolated": t_solve,
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
                             "sample": "FP64 oracle on the full two-level 257^3 workload, %d threads: each step = "
                                       "set-up + %d composite iterations (%.1f s); set-up %.1f s, %.2f s per "
                                       "iteration; one solve = set-up + %d iterations (from %s) = %.0f s"
                                       % (cores, m, t_step, t_setup, t_iter, iters, src, t_solve)},
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def pull_z_bc(uz):
    """u = 0 on z = 0, u_z = uz (u_x = u_y = 0) on z = 1, traction-free lateral faces; edges and
    corners touching z = 0 / z = 1 take the z-face type."""
    from anisotropicfracture_gb300.elastic import BCElastic, FACES
    bc = BCElastic()
    for f in FACES:
        for d in range(3):
            bc.Set(f, d, bc.Displacement, 0.0)
    for f in ["XLO", "XHI", "YLO", "YHI", "XLO_YLO", "XLO_YHI", "XHI_YLO", "XHI_YHI"]:
        for d in range(3):
            bc.Set(f, d, bc.Traction, 0.0)
    for f in FACES:
        if "ZHI" in f:
            bc.Set(f, 2, bc.Displacement, uz)
    return bc


def pernode_err(a, ref, floor=1e-3):
    """max over nodes of |a - ref| / max(|ref_node|, floor * max|ref|)"""
    s = float(np.abs(ref).max())
    return float((np.abs(a - ref) / np.maximum(np.abs(ref), floor * (s if s > 0 else 1.0))).max())


def normwise(a, ref):
    s = float(np.abs(ref).max())
    return float(np.abs(a - ref).max() / (s if s > 0 else 1.0))


# ---------------------------------------------------------------- the 64^3 single-level workload
def bench_config0(args):
    """64^3 cells (65^3 nodes), isotropic sphere inclusion (E 10 / 1, nu 0.3, 2-cell diffuse
    interface), pulled along z, V(2,2) + CG to 1e-8: GPU FP64 and mixed solves/s (device time over
    several solves, and end to end through host buffers), against the oracle's full FP64 solve on
    the host cores, timed in full: its iterations, the displacement error of each GPU solution
    against it, and the oracle's residual of each GPU solution."""
    import torch
    from anisotropicfracture_gb300 import microstructure, models
    from anisotropicfracture_gb300.elastic import Elastic, Field, Linear, level_desc
    from oracle import pyoracle as po
    n = 64
    Cf = microstructure.sphere_inclusion_iso((0, 0, 0), (n, n, n), (1.0 / n,) * 3)
    bc = pull_z_bc(0.01)
    L = po.level(n)
    b = po.bc_init(L, bc.type, bc.val, np.zeros((3,) + L.shape))
    op = Elastic([level_desc(n)], models.ISOTROPIC)
    op.SetModel(0, Field(Cf))
    op.SetBC(bc)
    op.SetUniform(False)
    op.prepareForSolve()
    stream = torch.cuda.Stream()
    op.set_stream(stream.cuda_stream)
    s = Linear(op)
    s.setMaxFmgIter(0)
    s.setBottomSolver("cg")
    s.setPreSmooth(1)
    s.setPostSmooth(1)
    s.opts.max_iter = 400
    bd = torch.from_numpy(b).cuda()
    xd = torch.zeros_like(bd)
    bh = torch.from_numpy(b).pin_memory()
    xh = torch.zeros_like(bh).pin_memory()
    reps = max(1, args.config0_reps)
    out = {"workload": "64^3 cells (65^3 nodes), isotropic sphere inclusion r 0.25 (E 10 / 1, nu 0.3, 2-cell diffuse "
                       "interface), u_z = 0.01 on z = 1, traction-free sides, V(2,2) Jacobi + CG, tol_rel 1e-8",
           "unit": UNIT, "l2": "resident in L2 (17.6 MB per FP64 apply): reported in solves/s, not as HBM fraction"}
    xs = {}
    for prec, inner in (("fp64", 1), ("mixed", args.config0_inner)):
        s.setPrecision(prec)
        s.opts.inner_cycles = inner

        def one():
            with torch.cuda.stream(stream):
                xd.zero_()
            s.solve(Field(xd), Field(bd), 1e-8, 0.0)

        for _ in range(2):
            one()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(reps):
            one()
        e1.record(stream)
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / reps
        xs[prec] = xd.cpu().numpy()
        st = s.stats
        rec = {"value": 1000.0 / ms, "ms_per_solve": ms, "iters": st.iters, "cycles": st.cycles,
               "inner_cycles": inner, "converged": bool(st.converged), "resfinal": st.resfinal, "target": st.target}
        t0 = time.perf_counter()
        for _ in range(reps):
            xh.zero_()
            s.solve(Field(xh.numpy()), Field(bh.numpy()), 1e-8, 0.0)
        e2e = (time.perf_counter() - t0) / reps
        rec["e2e"] = {"value": 1.0 / e2e, "unit": UNIT, "h2d_bytes_per_step": 2 * b.nbytes,
                      "d2h_bytes_per_step": b.nbytes}
        out[prec] = rec
    out["mixed_over_fp64"] = out["mixed"]["value"] / out["fp64"]["value"]
    op.close()
    if not args.no_cpu:
        po.set_threads(os.cpu_count())
        t0 = time.perf_counter()
        ref, st, rc = po.solve(L, po.ORC_ISOTROPIC, Cf, bc.type, np.zeros_like(b), b, 1e-8, 0.0, max_fmg_iter=0,
                               bottom=0, nu1=1, nu2=1, max_iter=400)
        t_cpu = time.perf_counter() - t0
        bn = float(np.abs(b).max())
        out["oracle"] = {"iters": st.iters, "converged": bool(rc == 0 and st.converged), "seconds": t_cpu,
                         "threads": po.lib().orc_num_threads()}
        for prec in ("fp64", "mixed"):
            _, rn = po.residual(L, po.ORC_ISOTROPIC, Cf, bc.type, xs[prec], b)
            out[prec]["displacement_err_vs_oracle"] = normwise(xs[prec], ref)
            out[prec]["oracle_rel_residual"] = rn / bn
        out["cpu_baseline"] = {"value": 1.0 / t_cpu, "unit": UNIT, "cores": po.lib().orc_num_threads(),
                               "kind": "port", "sample": "the oracle's full FP64 solve (%d V-cycles), timed in full"
                                                         % st.iters}
    return out


def oracle_check(levels, bc, rhs, sols):
    """The oracle on the GPU's final solutions of the two-level workload: its composite residual
    ||b - A x||_inf / ||b||_inf (MLMG's computeMLResidual restated), and, when the committed record
    of the oracle's own full solve (tests/golden/config1_oracle.npz) is present, the displacement
    error at its subsampled nodes, relative to the max-norm of the oracle's solution there."""
    from oracle import pyoracle as po
    Ls = [oracle_level(L) for L in levels]
    Cs = [L["C"] for L in levels]
    bn = max(float(np.abs(valid_part(L, b)).max()) for L, b in zip(levels, rhs))
    out = {"residual": "oracle composite ||b - A x||_inf / ||b||_inf of each GPU solution (solve target 1e-8)"}
    for name, xs in sols.items():
        t0 = time.perf_counter()
        rn = po.residual_amr(Ls, po.ORC_MAJORMINOR, Cs, bc.type, xs, rhs)
        out[name] = {"oracle_rel_residual": rn / bn, "seconds": time.perf_counter() - t0}
    path = os.path.join(ROOT, "tests", "golden", "config1_oracle.npz")
    if os.path.exists(path):
        z = np.load(path)
        k = int(z["stride"])
        subs = [z["sub%d" % a] for a in range(len(levels))]
        scale = max(float(np.abs(v).max()) for v in subs)
        out["cpu_oracle_solve"] = {"iters": int(z["iters"]), "seconds": float(z["seconds"]),
                                   "threads": int(z["threads"]), "resfinal": float(z["resfinal"]),
                                   "compared": "every %d-th node of each level's valid box (%d nodes)"
                                               % (k, sum(v[0].size for v in subs))}
        for name, xs in sols.items():
            err = max(float(np.abs(valid_part(L, x)[:, ::k, ::k, ::k] - v).max())
                      for L, x, v in zip(levels, xs, subs))
            out[name]["displacement_err_vs_cpu_oracle_solve"] = err / scale
    return out


def parity_at_size(op, levels, bc, device):
    """One FP64 Fapply, residual and Fsmooth (two sweeps) of the GPU on each full-size level,
    against the oracle on the same seeded inputs: normwise error and the worst per-node relative
    error (floor 1e-3 of the field's max-norm)."""
    import torch
    from anisotropicfracture_gb300.elastic import Field
    from oracle import pyoracle as po
    rng = np.random.default_rng(11)
    out = {"tolerance": "1e-12 normwise and per node (floor 1e-3 of the max-norm)"}
    for a, L in enumerate(levels):
        Lo = oracle_level(L)
        lo = tuple(L["store_lo"])
        shape = (3,) + level_shape(L)
        u = rng.standard_normal(shape)
        b = rng.standard_normal(shape)
        ud, bd = torch.from_numpy(u).to(device), torch.from_numpy(b).to(device)
        f, r, xd = torch.zeros_like(ud), torch.zeros_like(ud), ud.clone()
        torch.cuda.synchronize()  # the operator runs on a stream of the caller's, not on the default one
        op.Fapply(a, 0, Field(f, lo), Field(ud, lo))
        op.Residual(a, 0, Field(r, lo), Field(ud, lo), Field(bd, lo))
        op.Fsmooth(a, 0, Field(xd, lo), Field(bd, lo), 2, 2.0 / 3.0)
        torch.cuda.synchronize()
        got = {"fapply": f.cpu().numpy(), "residual": r.cpu().numpy(), "fsmooth": xd.cpu().numpy()}
        del ud, bd, f, r, xd
        t0 = time.perf_counter()
        ref = {"fapply": po.fapply(Lo, po.ORC_MAJORMINOR, L["C"], bc.type, u),
               "residual": po.residual(Lo, po.ORC_MAJORMINOR, L["C"], bc.type, u, b)[0]}
        D = po.diagonal(Lo, po.ORC_MAJORMINOR, L["C"], bc.type)
        ref["fsmooth"] = po.fsmooth(Lo, po.ORC_MAJORMINOR, L["C"], bc.type, D, u, b, 2, 2.0 / 3.0)
        rec = {"nodes": int(np.prod(shape[1:])), "oracle_seconds": time.perf_counter() - t0}
        for k in got:
            g, e = valid_part(L, got[k]), valid_part(L, ref[k])
            rec[k] = {"normwise": normwise(g, e), "per_node": pernode_err(g, e)}
        out["level%d" % a] = rec
    return out


# ---------------------------------------------------------------- damaged polycrystal, 193^3 nodes
def bench_damaged_polycrystal(args):
    """Phase-field-degraded cubic polycrystal, single level, mixed vs FP64 and the displacement error.
    The stiffness floor of g(c) = (1-c)^2 + floor is args.damage_floor (see the returned note)."""
    import torch
    from anisotropicfracture_gb300 import microstructure, models
    from anisotropicfracture_gb300.elastic import BCElastic, Elastic, FACES, Field, Linear, level_desc
    n = args.damaged_cells
    dx = (1.0 / n,) * 3
    C, _, _ = microstructure.cubic_polycrystal((0, 0, 0), (n, n, n), dx, nseeds=64, seed_points=1, seed_rot=2)
    c = microstructure.penny_crack_damage((0, 0, 0), (n, n, n), dx, ncracks=8, seed=3, width_cells=3.0,
                                          cell=1.0 / n)
    C *= ((1.0 - c) ** 2 + args.damage_floor)[None]
    bc = BCElastic()
    for f in FACES:
        for d in range(3):
            bc.Set(f, d, bc.Displacement, 0.0)
    for f in ["XLO", "XHI", "YLO", "YHI", "XLO_YLO", "XLO_YHI", "XHI_YLO", "XHI_YHI"]:
        for d in range(3):
            bc.Set(f, d, bc.Traction, 0.0)
    for f in FACES:
        if "ZHI" in f:
            bc.Set(f, 2, bc.Displacement, 0.005)
    C = np.ascontiguousarray(C)
    op = Elastic([level_desc(n)], models.MAJORMINOR)
    op.SetModel(0, Field(C))
    op.SetBC(bc)
    op.SetUniform(False)
    op.prepareForSolve()
    dev = torch.device("cuda", 0)
    b = torch.zeros((3, n + 1, n + 1, n + 1), dtype=torch.float64, device=dev)
    op.BCInit(0, Field(b))
    s = Linear(op)
    s.setMaxFmgIter(0)
    s.setBottomSolver("cg")
    s.setPreSmooth(2)
    s.setPostSmooth(2)
    s.opts.max_iter = 400
    s.opts.inner_cycles = args.inner
    out = {"workload": "%d^3 cells, cubic 64-grain polycrystal x g(c), 8 penny cracks (seed 3, width 3 cells), "
                       "u_z = 0.005 on z = 1, V(2,2) + CG, tol_rel 1e-8" % n,
           "damage_floor": args.damage_floor,
           "note": "with the specified floor 1e-6 the reference's operator and smoother diverge (the oracle "
                   "and this library both report it); floors 0.03, 0.01 and 1e-3 diverge too, 0.1 converges",
           "unit": UNIT}
    xs = {}
    for prec in ("fp64", "mixed"):
        s.setPrecision(prec)
        x = torch.zeros_like(b)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        s.solve([Field(x)], [Field(b)], 1e-8, 0.0)
        torch.cuda.synchronize()
        secs = time.perf_counter() - t0
        out[prec] = {"value": 1.0 / secs, "seconds": secs, "iters": s.stats.iters, "converged": bool(s.stats.converged)}
        xs[prec] = x.cpu().numpy()
    out["mixed_over_fp64"] = out["mixed"]["value"] / out["fp64"]["value"]
    out["displacement_err_mixed_vs_fp64"] = float(np.abs(xs["mixed"] - xs["fp64"]).max() / np.abs(xs["fp64"]).max())
    op.close()
    if not args.no_cpu:
        # the FP64 oracle on the host cores: set-up plus one V-cycle, extrapolated to the
        # iterations of the GPU FP64 solve (the same algorithm)
        try:
            from oracle import pyoracle as po
            L = po.level(n)
            bh = po.bc_init(L, bc.type, bc.val, np.zeros((3,) + L.shape))
            kw = dict(max_fmg_iter=0, bottom=0, nu1=2, nu2=2)
            t0 = time.perf_counter()
            po.solve(L, po.ORC_MAJORMINOR, C, bc.type, np.zeros_like(bh), bh, 1e-30, 0.0, max_iter=0, **kw)
            t_setup = time.perf_counter() - t0
            t0 = time.perf_counter()
            po.solve(L, po.ORC_MAJORMINOR, C, bc.type, np.zeros_like(bh), bh, 1e-30, 0.0, max_iter=1, **kw)
            t_iter = max(time.perf_counter() - t0 - t_setup, 1e-9)
            iters = out["fp64"]["iters"]
            out["cpu_baseline"] = {"value": 1.0 / (t_setup + iters * t_iter), "unit": UNIT,
                                   "cores": po.lib().orc_num_threads(), "kind": "port",
                                   "sample": "FP64 oracle, set-up %.1f s + 1 V-cycle at %.2f s, extrapolated to the "
                                             "%d cycles of the FP64 solve" % (t_setup, t_iter, iters)}
            if not args.no_parity:  # the oracle's residual of each GPU solution
                bn = float(np.abs(bh).max())
                for prec in ("fp64", "mixed"):
                    _, rn = po.residual(L, po.ORC_MAJORMINOR, C, bc.type, xs[prec], bh)
                    out[prec]["oracle_rel_residual"] = rn / bn
        except Exception as e:  # pragma: no cover
            out["cpu_baseline"] = {"value": None, "sample": "failed: %s" % e}
    del C
    return out


# ---------------------------------------------------------------- batched and served cells
BATCH_EDGES = (16, 24, 32, 48, 64)
SERVE_EDGES = tuple(range(32, 129, 8))
CELL_SOLVER = dict(max_fmg_iter=0, nu1=2, nu2=2, sweeps=2, bottom=1, bottom_max_iter=200, bottom_reltol=1e-4,
                   nuf=8, max_iter=200)


def batch_workload(ncells=512, seed=4):
    """Cells of the batched workload: edge, grain count, seeds and per-grain stiffness tables."""
    from anisotropicfracture_gb300 import cells
    rng = np.random.default_rng(seed)
    edges = rng.choice(BATCH_EDGES, size=ncells)
    out = []
    for c in range(ncells):
        g = np.random.default_rng(5 + c)
        ngr = int(g.integers(8, 33))
        seeds, table = cells.rve_grains(int(edges[c]), ngr, int(g.integers(1 << 30)))
        out.append({"n": int(edges[c]), "ngrains": ngr, "seeds": seeds, "table": table})
    return out


def serve_workload(nreq, seed=6):
    from anisotropicfracture_gb300 import cells
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(nreq):
        n = int(rng.choice(SERVE_EDGES))
        ngr = int(rng.integers(8, 65))
        seeds, table = cells.rve_grains(n, ngr, int(rng.integers(1 << 30)))
        out.append({"n": n, "ngrains": ngr, "seeds": seeds, "table": table})
    return out


def _exx():
    E = np.zeros((3, 3))
    E[0, 0] = 1e-3
    return E


def make_cell_batch(work, nrhs_loads=None):
    from anisotropicfracture_gb300 import cells, models
    loads = [_exx()] if nrhs_loads is None else nrhs_loads
    B = cells.CellBatch([(w["n"], len(loads)) for w in work], models.MAJORMINOR)
    s = 0
    for c, w in enumerate(work):
        B.set_grains(c, w["seeds"], w["table"])
        for E in loads:
            B.set_load(s, E)
            s += 1
    B.prepare()
    return B


def cpu_cells_sample(work, nsample, threads=None):
    """FP64 oracle cell solves of a sample of cells (stiffness built outside the timed region);
    returns (seconds, nodes) of the sample."""
    from anisotropicfracture_gb300 import cells, models
    from oracle import pyoracle as po
    if threads:
        po.set_threads(threads)
    secs, nodes = 0.0, 0
    for w in work[:nsample]:
        n = w["n"]
        Cf = cells.rve_stiffness(n, w["seeds"], w["table"])
        t0 = time.perf_counter()
        po.rve_solve(po.rve_level(n), models.MAJORMINOR, Cf, _exx(), **CELL_SOLVER)
        secs += time.perf_counter() - t0
        nodes += n ** 3
    return secs, nodes


def _max_over_ranks(x, world):
    """Max of a host float over the ranks (the slowest rank bounds a weak-scaling step)."""
    if world <= 1:
        return x
    import torch
    import torch.distributed as dist
    t = torch.tensor([x], dtype=torch.float64, device="cuda")
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def _barrier(world):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


def _nvtx_push(name):
    import torch
    torch.cuda.nvtx.range_push(name)


def _nvtx_pop():
    import torch
    torch.cuda.nvtx.range_pop()


def bench_batch(args, lib, rank=0, world=1):
    """Batched cells: mixed and FP64 in one batch, FP64 one cell at a time, CPU oracle sample.
    With N ranks each takes its largest-first share of the cells (no collective on the data path)
    and times are the max over ranks; solves/s count all ranks' cells (weak scaling)."""
    from anisotropicfracture_gb300 import cells as _cells
    work_all = batch_workload(args.batch_cells)
    if world > 1:
        share = _cells.partition_cells([_cells.plan_bytes(w["n"]) for w in work_all], world)[rank]
        work = [work_all[c] for c in share]
    else:
        work = work_all
    total = len(work_all)
    nodes = sum(w["n"] ** 3 for w in work_all)
    t0 = time.perf_counter()
    B = make_cell_batch(work)
    setup_s = time.perf_counter() - t0
    out = {"workload": "%d periodic polycrystal RVEs, edges uniform in %s cells (seed 4), 8-32 grains each, "
                       "cubic 1.68/1.21/0.75, exx = 1e-3, tol_rel 1e-8" % (total, list(BATCH_EDGES)),
           "cells": total, "nodes": nodes, "device_bytes": B.device_bytes(), "setup_s": setup_s,
           "cycle": "V-cycle, 2 pre + 2 post smoother calls of 2 damped-Jacobi sweeps, BiCGStab bottom",
           "inner_cycles": args.batch_inner, "unit": UNIT,
           "ranks": world, "scaling": "weak" if world > 1 else None}
    res = {}
    sols = {}
    for prec, name in ((1, "mixed"), (0, "fp64_batched")):
        st, rc = B.solve(precision=prec, inner_cycles=args.batch_inner, check=False, **CELL_SOLVER)  # warm/tune
        l0 = lib.ae_kernel_launches()
        _barrier(world)
        t0 = time.perf_counter()
        reps = max(1, args.batch_steps)
        _nvtx_push("batch_" + name)  # ncu --nvtx --nvtx-include "batch_mixed/" lists the timed launches
        for _ in range(reps):
            st, rc = B.solve(precision=prec, inner_cycles=args.batch_inner, check=False, **CELL_SOLVER)
        _nvtx_pop()
        secs = _max_over_ranks((time.perf_counter() - t0) / reps, world)
        launches = (lib.ae_kernel_launches() - l0) // reps
        res[name] = {"value": total / secs, "s_per_batch": secs, "converged": rc == 0,
                     "max_iters": max(s["iters"] for s in st), "mean_iters": float(np.mean([s["iters"] for s in st])),
                     "gpu_launches": int(launches)}
        sols[name] = [B.solution(s) for s in range(len(work))]
    shapes = [B.get_shape(m) for m in range(6)]
    B.close()
    # the same solves one cell at a time in FP64 (set-up outside the timed region)
    lim = len(work) if args.batch_single_limit <= 0 else min(len(work), args.batch_single_limit)
    singles = [make_cell_batch([w]) for w in work[:lim]]
    for Bs in singles[:2]:
        Bs.solve(precision=0, check=False, **CELL_SOLVER)
    _barrier(world)
    t0 = time.perf_counter()
    ok = True
    for Bs in singles:
        st, rc = Bs.solve(precision=0, check=False, **CELL_SOLVER)
        ok = ok and rc == 0
    secs = _max_over_ranks(time.perf_counter() - t0, world)
    w64 = [Bs.solution(0) for Bs in singles]
    for Bs in singles:
        Bs.close()
    timed = lim * world if args.batch_single_limit > 0 else total
    res["fp64_one_at_a_time"] = {"value": timed / secs, "cells_timed": timed, "seconds": secs, "converged": ok}
    err = 0.0
    for a, b in zip(sols["mixed"][:lim], w64):
        err = max(err, float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)))
    err_b = max(float(np.abs(a - b).max() / max(np.abs(b).max(), 1e-300))
                for a, b in zip(sols["fp64_batched"][:lim], w64))
    out.update(res)
    out["mixed_over_fp64_one_at_a_time"] = res["mixed"]["value"] / res["fp64_one_at_a_time"]["value"]
    out["mixed_over_fp64_batched"] = res["mixed"]["value"] / res["fp64_batched"]["value"]
    out["displacement_err_mixed_vs_fp64"] = err
    out["fp64_batched_vs_one_at_a_time"] = err_b
    out["shapes"] = shapes
    if not args.no_cpu and rank == 0:
        try:
            ns = max(1, args.batch_cpu_sample)
            secs, nn = cpu_cells_sample(work, ns, threads=os.cpu_count())
            per_node = secs / nn
            out["cpu_baseline"] = {"value": 1.0 / (per_node * nodes / total), "unit": UNIT,
                                   "cores": os.cpu_count(), "kind": "port",
                                   "sample": "FP64 oracle cell solves of the first %d cells (%d nodes, %.1f s), "
                                             "scaled per node to the mean cell" % (ns, nn, secs)}
        except Exception as e:  # pragma: no cover
            out["cpu_baseline"] = {"value": None, "sample": "failed: %s" % e}
        if not args.no_parity:
            out["oracle_check"] = cells_oracle_check(work, sols, max(1, args.batch_cpu_sample))
    return out


def cells_oracle_check(work, sols, nsample):
    """The oracle's mean-free residual ||b - A w - c||_inf / ||b||_inf of the GPU's batched
    solutions (mixed and FP64) for the first `nsample` cells."""
    from anisotropicfracture_gb300 import cells, models
    from oracle import pyoracle as po
    out = {"cells": nsample, "what": "oracle mean-free residual / ||b||_inf of the batched GPU solutions"}
    worst = {k: 0.0 for k in sols}
    for c, w in enumerate(work[:nsample]):
        n = w["n"]
        L = po.rve_level(n)
        Cf = cells.rve_stiffness(n, w["seeds"], w["table"])
        b = po.rve_rhs(L, models.MAJORMINOR, Cf, _exx())
        bn = float(np.abs(b).max())
        for k, ws in sols.items():
            _, _, rn = po.rve_residual(L, models.MAJORMINOR, Cf, np.ascontiguousarray(ws[c]), b)
            worst[k] = max(worst[k], rn / bn)
    for k in sols:
        out[k + "_worst_rel_residual"] = worst[k]
    return out


def serve_run(work, rate, precision, inner, seed=7, rank=0, world=1):
    """Poisson arrivals at `rate` requests/s into a fresh server.  With world > 1 this rank's server
    takes the requests i = rank (mod world) of the stream, at their times in the whole stream."""
    from anisotropicfracture_gb300 import cells, models
    S = cells.CellServer(models.MAJORMINOR, precision=precision, inner_cycles=inner, **CELL_SOLVER)
    loads = cells.unit_strains()
    times = np.cumsum(np.random.default_rng(seed).exponential(1.0 / rate, size=len(work)))
    mine = list(range(rank, len(work), world))
    work = [work[i] for i in mine]
    offsets = [float(times[i]) for i in mine]
    tickets = []

    def producer():
        t0 = time.perf_counter()
        for w, t in zip(work, offsets):
            dt = t0 + t - time.perf_counter()
            if dt > 0:
                time.sleep(dt)
            tickets.append(S.submit(w["n"], loads, w["seeds"], w["table"]))

    th = threading.Thread(target=producer)
    th.start()
    th.join()
    res = [S.wait(t, 3600.0) for t in tickets]
    st = S.stats()
    S.close()
    lat = np.array([r["latency"] for r in res])
    queue = np.array([r["t_admit"] - r["t_submit"] for r in res])
    service = np.array([r["t_done"] - r["t_admit"] for r in res])
    good = [r for r in res if r["status"] == 0]
    first = min(r["t_submit"] for r in res)
    last = max(r["t_done"] for r in res)
    nsolves = sum(len(r["stats"]) for r in good)
    # requests resident on the device (admitted, not yet done) over time: time-weighted mean, max
    ev = sorted([(r["t_admit"], 1) for r in res] + [(r["t_done"], -1) for r in res])
    live, peak, area, t_prev = 0, 0, 0.0, ev[0][0]
    for t, d in ev:
        area += live * (t - t_prev)
        live += d
        peak = max(peak, live)
        t_prev = t
    span = max(ev[-1][0] - ev[0][0], 1e-9)

    def pct(a, q):
        return float(np.percentile(a, q))

    return {"rate": rate, "requests": len(work), "ok": len(good) == len(res), "lat": lat.tolist(),
            "queue": queue.tolist(), "service": service.tolist(), "solves": nsolves,
            "offered_solves_per_s": rate * len(cells.unit_strains()),
            "p50_s": pct(lat, 50), "p99_s": pct(lat, 99),
            "queue_p50_s": pct(queue, 50), "queue_p99_s": pct(queue, 99),
            "service_p50_s": pct(service, 50), "service_p99_s": pct(service, 99),
            "resident_mean": area / span, "resident_max": peak,
            "solves_per_s": nsolves / (last - first), "iterations": st["iterations"], "busy_s": st["busy_seconds"]}


def _serve_over_ranks(work, rate, precision, inner, rank, world):
    """One arrival rate: every rank serves its share of the stream; rank 0 merges the records
    (latency percentiles over all requests, solves/s summed over the concurrently serving ranks)."""
    _barrier(world)
    r = serve_run(work, rate, precision, inner, rank=rank, world=world)
    if world > 1:
        import torch.distributed as dist
        parts = [None] * world
        dist.all_gather_object(parts, r)
    else:
        parts = [r]
    lat = np.concatenate([p["lat"] for p in parts])
    queue = np.concatenate([p["queue"] for p in parts])
    service = np.concatenate([p["service"] for p in parts])

    def pct(a, q):
        return float(np.percentile(a, q))

    out = {"rate": rate, "requests": int(lat.size), "ok": all(p["ok"] for p in parts),
           "offered_solves_per_s": parts[0]["offered_solves_per_s"],
           "p50_s": pct(lat, 50), "p99_s": pct(lat, 99), "queue_p50_s": pct(queue, 50), "queue_p99_s": pct(queue, 99),
           "service_p50_s": pct(service, 50), "service_p99_s": pct(service, 99),
           "resident_mean": float(sum(p["resident_mean"] for p in parts)),
           "resident_max": int(sum(p["resident_max"] for p in parts)),
           "solves_per_s": float(sum(p["solves_per_s"] for p in parts)),
           "iterations": int(max(p["iterations"] for p in parts)), "busy_s": float(max(p["busy_s"] for p in parts))}
    if world > 1:
        out["ranks"] = world
    return out


def bench_serve(args, rank=0, world=1):
    """Served cells: for each arrival rate a fresh server takes a Poisson stream of requests.
    Latency (submission to result) is split into queueing delay (submission to admission) and
    service time (admission to result); `resident_*` counts requests on the device at once.
    The sub-capacity rates show overlap below saturation; above capacity the queue grows and
    latency measures the backlog.  With N ranks each GPU serves every N-th request of the stream
    (no exchange between the servers) and solves/s adds up over the ranks."""
    rates = [float(r) for r in args.serve_rates.split(",") if r]
    rates64 = [float(r) for r in args.serve_fp64_rates.split(",") if r]
    work = serve_workload(max(args.serve_requests, args.serve_fp64_requests))
    out = {"workload": "Poisson streams (seed 6) of periodic polycrystal cells, edges uniform in {32..128 step 8}, "
                       "8-64 grains, 6 unit strains (1e-3) per request, tol_rel 1e-8",
           "requests_per_rate": {"mixed": args.serve_requests, "fp64": args.serve_fp64_requests},
           "mean_nodes": float(np.mean([w["n"] ** 3 for w in work[:args.serve_requests]])),
           "inner_cycles": args.batch_inner, "unit": UNIT, "ranks": world}
    # warm-up: one small request (library load, first graph capture)
    serve_run(work[:1], 1000.0, 1, args.batch_inner)
    out["mixed"] = [_serve_over_ranks(work[:args.serve_requests], r, 1, args.batch_inner, rank, world) for r in rates]
    out["fp64"] = [_serve_over_ranks(work[:args.serve_fp64_requests], r, 0, args.batch_inner, rank, world)
                   for r in rates64]
    cap_m = max(r["solves_per_s"] for r in out["mixed"])
    cap_f = max(r["solves_per_s"] for r in out["fp64"])
    out["capacity_solves_per_s"] = {"mixed": cap_m, "fp64": cap_f,
                                    "how": "highest delivered solves/s over the arrival rates"}
    for name, cap in (("mixed", cap_m), ("fp64", cap_f)):
        for r in out[name]:
            r["load"] = r["offered_solves_per_s"] / cap
    out["mixed_over_fp64"] = cap_m / cap_f
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--cells", type=int, default=256)
    ap.add_argument("--fp64-steps", type=int, default=1)
    ap.add_argument("--oracle-tol", type=float, default=1e-9,
                    help="residual of the FP64 oracle solution the displacement errors are measured against (0: off)")
    ap.add_argument("--path-check", action="store_true",
                    help="also solve in FP64 with F-cycles and report its distance to the oracle solution")
    ap.add_argument("--mixed-tight-tol", type=float, default=0.0,
                    help="also time the mixed solve to this residual and report its error (0: off)")
    ap.add_argument("--e2e-steps", type=int, default=2)
    ap.add_argument("--bicgstab-steps", type=int, default=1,
                    help="timed mixed solves with the BiCGStab bottom solver (0: off)")
    ap.add_argument("--ref-sample-iters", type=int, default=3,
                    help="composite oracle iterations per step of the reference arm")
    ap.add_argument("--cpu-sample-iters", type=int, default=1)
    ap.add_argument("--no-config0", action="store_true", help="skip the 64^3 single-level workload")
    ap.add_argument("--config0-reps", type=int, default=5)
    ap.add_argument("--config0-inner", type=int, default=4, help="FP32 cycles per FP64 residual, 64^3 workload")
    ap.add_argument("--no-parity", action="store_true",
                    help="skip the full-size operator comparison and the oracle residuals of the GPU solutions")
    ap.add_argument("--no-cpu", action="store_true")
    # 12: an FP64 composite residual costs about one FP32 V-cycle here, and a solve overshoots its
    # cycle count by (inner - 1) / 2 cycles on average; 8 / 12 / 16 gave 0.413 / 0.430 / 0.419
    # solves/s on the polycrystal (168, 168 and 176 cycles)
    ap.add_argument("--inner", type=int, default=int(os.environ.get("AE_INNER_CYCLES", "12")),
                    help="FP32 cycles per FP64 residual in mixed precision")
    ap.add_argument("--per-node-model", action="store_true",
                    help="give the single-box stiffness per node (ae_op_set_model) instead of as grain ids + table")
    ap.add_argument("--no-damaged", action="store_true", help="skip the damaged-polycrystal workload")
    ap.add_argument("--damaged-cells", type=int, default=192)
    ap.add_argument("--damage-floor", type=float, default=0.1,
                    help="stiffness floor of g(c) in the damaged workload (the specified 1e-6 diverges)")
    ap.add_argument("--no-batch", action="store_true", help="skip the batched-cell workload")
    ap.add_argument("--no-neohookean", action="store_true", help="skip the NeoHookean Newton workload")
    ap.add_argument("--neo-cells", type=int, default=96)
    ap.add_argument("--neo-nriters", type=int, default=4)
    ap.add_argument("--no-serve", action="store_true", help="skip the served-cell workload")
    ap.add_argument("--no-builders", action="store_true",
                    help="skip timing the device-side model builders (mixture, degradation)")
    ap.add_argument("--only-cells", action="store_true", help="run only the batched/served cell workloads")
    ap.add_argument("--batch-cells", type=int, default=512)
    ap.add_argument("--batch-steps", type=int, default=2)
    ap.add_argument("--batch-inner", type=int, default=4,
                    help="FP32 cycles per FP64 residual for the batched and served cells")
    ap.add_argument("--batch-single-limit", type=int, default=0, help="cells timed one at a time (0: all)")
    ap.add_argument("--batch-cpu-sample", type=int, default=4)
    ap.add_argument("--serve-requests", type=int, default=200, help="requests per arrival rate, mixed precision")
    ap.add_argument("--serve-rates", default="4,50,100,200,500,1000,2000",
                    help="arrival rates (requests/s), mixed precision")
    ap.add_argument("--serve-fp64-requests", type=int, default=40, help="requests per arrival rate, FP64")
    ap.add_argument("--serve-fp64-rates", default="1,50", help="arrival rates (requests/s), FP64")
    args = ap.parse_args()

    if args.gpus > 1 and "WORLD_SIZE" not in os.environ:
        # --gpus N outside a launcher: start N ranks, one per GPU, as torchrun would
        import socket
        sk = socket.socket()
        sk.bind(("127.0.0.1", 0))
        port = sk.getsockname()[1]
        sk.close()
        os.execvp(sys.executable, [sys.executable, "-m", "torch.distributed.run", "--nnodes=1",
                                   "--nproc-per-node", str(args.gpus), "--master-addr", "127.0.0.1",
                                   "--master-port", str(port), os.path.abspath(__file__)] + sys.argv[1:])
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank)
        return
    if args.only_cells:
        main_cells_only(args)
        return

    import torch
    import torch.distributed as dist
    from anisotropicfracture_gb300 import _lib, build as libbuild, models
    from anisotropicfracture_gb300.elastic import Elastic, Field, Linear, level_desc

    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl")
    libbuild.build()
    lib = _lib.load()

    levels, bc = workload(args.cells)
    descs = [level_desc(L["cells"], lo=(L["lo"],) * 3, hi=(L["hi"],) * 3) for L in levels]
    op = Elastic(descs, models.MAJORMINOR)
    for a, L in enumerate(levels):
        if args.per_node_model:
            op.SetModel(a, Field(L["C"], tuple(L["store_lo"])))
        else:  # the Voronoi map itself: grain ids + per-grain table (same values, 2 B per node)
            op.SetModelGrains(a, Field(L["gid"], tuple(L["store_lo"])), L["table"])
    op.SetBC(bc)
    op.SetUniform(False)
    op.prepareForSolve()
    stream = torch.cuda.Stream()
    op.set_stream(stream.cuda_stream)
    dev = torch.device("cuda", local)
    rhs_d = [torch.zeros((3,) + level_shape(L), dtype=torch.float64, device=dev) for L in levels]
    torch.cuda.synchronize()  # the operator runs on `stream`, the fill above on the default one
    for a, L in enumerate(levels):  # BC::Operator::Elastic::Init through the library
        op.BCInit(a, Field(rhs_d[a], tuple(L["store_lo"])))
    torch.cuda.synchronize()
    rhs_h = [b.cpu().numpy() for b in rhs_d]
    sol_d = [torch.zeros_like(b) for b in rhs_d]
    nodes = sum(int(np.prod(b.shape[1:])) for b in rhs_h)

    solver = Linear(op)
    solver.setMaxFmgIter(0)
    solver.setBottomSolver("cg")
    solver.setPreSmooth(1)
    solver.setPostSmooth(1)
    solver.opts.max_iter = 400
    solver.opts.inner_cycles = args.inner

    def fields(xs, rs):
        return ([Field(x, tuple(L["store_lo"])) for x, L in zip(xs, levels)],
                [Field(r, tuple(L["store_lo"])) for r, L in zip(rs, levels)])

    def solve_device(prec):
        solver.setPrecision(prec)
        with torch.cuda.stream(stream):
            for x in sol_d:
                x.zero_()
        xs, rs = fields(sol_d, rhs_d)
        solver.solve(xs, rs, 1e-8, 0.0)
        return solver.stats

    def barrier():
        if world > 1:
            dist.barrier()

    def timed(prec, steps):
        barrier()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        st = None
        # NVTX range "timed_<prec>": ncu --nvtx --nvtx-include "timed_mixed/" lists exactly the
        # launches of the timed solves
        torch.cuda.nvtx.range_push("timed_" + prec)
        for _ in range(steps):
            st = solve_device(prec)
        torch.cuda.nvtx.range_pop()
        e1.record(stream)
        torch.cuda.synchronize()
        barrier()
        ms = e0.elapsed_time(e1) / steps
        if world > 1:
            t = torch.tensor([ms], device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms, st

    # warm-up (mixed is the headline; one FP64 warm-up as well)
    for _ in range(args.warmup):
        solve_device("mixed")
    iters_mixed = solver.stats.iters
    clocks = ClockSampler(torch.cuda.current_device())
    clocks.start()
    l0 = lib.ae_kernel_launches()
    ms_mixed, st_mixed = timed("mixed", args.steps)
    launches = lib.ae_kernel_launches() - l0
    clk = clocks.stop()
    res_mixed = (st_mixed.iters, st_mixed.resfinal, st_mixed.target, st_mixed.converged)
    x_mixed = [x.cpu().numpy() for x in sol_d]

    # FP64 reference solve of the same problem (also the displacement-error yardstick)
    ms_fp64, fp64_iters, disp_err = None, None, None
    if args.fp64_steps > 0:
        solve_device("fp64")
        ms_fp64, st64 = timed("fp64", args.fp64_steps)
        fp64_iters = st64.iters
        x64 = [x.cpu().numpy() for x in sol_d]
        disp_err = rel_err(levels, x_mixed, x64)

    # FP64 oracle solution: the FP64 solve continued from its 1e-8 solution down to a much tighter
    # residual (--oracle-tol); the yardstick for the displacement error of every 1e-8 solve.  Two
    # solutions that both meet a 1e-8 residual differ by up to cond(A) x 1e-8, so the error of
    # each is measured against this one rather than against the other.
    oracle = None
    if args.fp64_steps > 0 and args.oracle_tol > 0:
        solver.setPrecision("fp64")
        xs, rs = fields(sol_d, rhs_d)  # sol_d holds the FP64 1e-8 solution: the initial guess
        # (1e-9 sits a decade above the FP64 floor of this residual: b is 0.01 on one face, while
        # A x sums about 50 terms of order C u / dx^2 ~ 1e3, so its rounding is ~1e-12 = 1e-10 |b|)
        solver.solve(xs, rs, args.oracle_tol, 0.0)
        st_or = solver.stats
        x_or = [x.cpu().numpy() for x in sol_d]

        def err_vs_oracle(xs_):
            return rel_err(levels, xs_, x_or)

        # with the refined patch's ghost layers included, for reference (they are not part of the
        # composite solution and follow the iteration history)
        scale_all = max(float(np.abs(x).max()) for x in x_or)
        ghost_err = max(float(np.abs(a - b).max()) for a, b in zip(x_mixed, x_or)) / scale_all
        def where(xs_):
            # per level: relative error on valid nodes and the (comp, i, j, k) of its maximum
            out = []
            scale = max(float(np.abs(valid_part(L, r)).max()) for L, r in zip(levels, x_or))
            for L, a, b in zip(levels, xs_, x_or):
                d = np.abs(valid_part(L, a) - valid_part(L, b))
                c, k, j, i = np.unravel_index(int(np.argmax(d)), d.shape)
                out.append({"err": float(d.max()) / scale, "at": [int(c), int(i) + L["lo"], int(j) + L["lo"],
                                                                  int(k) + L["lo"]]})
            return out

        def away(xs_, margin=4):
            # relative error on valid nodes at least `margin` coarse cells (2 margin fine cells)
            # from the refined patch's boundary, where the coarse/fine interface rows sit
            scale = max(float(np.abs(valid_part(L, r)).max()) for L, r in zip(levels, x_or))
            lo_c, hi_c = levels[1]["lo"] // 2, levels[1]["hi"] // 2
            out = 0.0
            for lev, (L, a, b) in enumerate(zip(levels, xs_, x_or)):
                d = np.abs(valid_part(L, a) - valid_part(L, b)).max(axis=0)
                idx = [np.arange(n) + L["lo"] for n in d.shape]
                k, j, i = np.meshgrid(*idx, indexing="ij", sparse=True)
                lo, hi, m = (lo_c, hi_c, margin) if lev == 0 else (2 * lo_c, 2 * hi_c, 2 * margin)
                inside = functools.reduce(np.minimum, [np.minimum(c - lo, hi - c) for c in (i, j, k)])
                outside = functools.reduce(np.maximum, [np.maximum(np.maximum(lo - c, c - hi), 0) for c in (i, j, k)])
                dist = np.where(inside >= 0, inside, outside)
                sel = d[dist >= m]
                if sel.size:
                    out = max(out, float(sel.max()) / scale)
            return out

        oracle = {"tol_rel": args.oracle_tol, "iters_from_fp64": st_or.iters, "converged": bool(st_or.converged),
                  "displacement_err_mixed_away_from_interface": away(x_mixed),
                  "displacement_err_fp64_away_from_interface": away(x64),
                  "displacement_err_fp64": err_vs_oracle(x64), "displacement_err_mixed": err_vs_oracle(x_mixed),
                  "per_level_mixed": where(x_mixed),
                  "displacement_err_mixed_incl_ghosts": ghost_err,
                  "measured_on": "valid nodes of both levels (the composite solution)"}
        # another FP64 iteration path (F-cycles) to the same 1e-8 residual: how far two FP64 paths
        # land apart measures the non-uniqueness of the composite solution on its own
        if args.path_check:
            solver.setPrecision("fp64")
            solver.setMaxFmgIter(1 << 30)
            with torch.cuda.stream(stream):
                for x in sol_d:
                    x.zero_()
            xs3, rs3 = fields(sol_d, rhs_d)
            solver.solve(xs3, rs3, 1e-8, 0.0)
            solver.setMaxFmgIter(0)
            x_f = [x.cpu().numpy() for x in sol_d]
            oracle["fp64_fcycle"] = {"iters": solver.stats.iters, "displacement_err": err_vs_oracle(x_f),
                                     "displacement_err_away_from_interface": away(x_f)}
        # the mixed solve to a tighter residual, timed the same way, with its error
        if args.mixed_tight_tol > 0:
            def solve_tight():
                solver.setPrecision("mixed")
                with torch.cuda.stream(stream):
                    for x in sol_d:
                        x.zero_()
                xs2, rs2 = fields(sol_d, rhs_d)
                solver.solve(xs2, rs2, args.mixed_tight_tol, 0.0)
                return solver.stats
            solve_tight()
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            st_t = solve_tight()
            e1.record(stream)
            torch.cuda.synchronize()
            ms_t = e0.elapsed_time(e1)
            oracle["mixed_tight"] = {"tol_rel": args.mixed_tight_tol, "value": world * 1000.0 / ms_t, "unit": UNIT,
                                     "ms_per_solve": ms_t, "iters": st_t.iters, "converged": bool(st_t.converged),
                                     "displacement_err": err_vs_oracle([x.cpu().numpy() for x in sol_d])}

    # the same mixed solve with the reference's default bottom solver (BiCGStab, Linear.H:25): CG
    # fails on the non-symmetric coarsest operator every call and falls back to smoothing
    bicg = None
    if args.bicgstab_steps > 0:
        solver.setBottomSolver("bicgstab")
        solve_device("mixed")
        ms_b, st_b = timed("mixed", args.bicgstab_steps)
        bicg = {"value": world * 1000.0 / ms_b, "unit": UNIT, "ms_per_solve": ms_b, "iters": st_b.iters,
                "bottom_failures": st_b.bottom_fail, "converged": bool(st_b.converged),
                "cycle": "V-cycle, 2 pre + 2 post damped-Jacobi sweeps, BiCGStab bottom"}
        solver.setBottomSolver("cg")
    bottom_fail_cg = st_mixed.bottom_fail

    # end to end through the C ABI with pinned host buffers
    solver.setPrecision("mixed")
    rhs_p = [torch.from_numpy(b).pin_memory() for b in rhs_h]
    sol_p = [torch.zeros_like(b).pin_memory() for b in rhs_p]
    t0 = time.perf_counter()
    e2e_steps = max(1, args.e2e_steps)
    for _ in range(e2e_steps):
        for x in sol_p:
            x.zero_()
        xs, rs = fields([x.numpy() for x in sol_p], [r.numpy() for r in rhs_p])
        solver.solve(xs, rs, 1e-8, 0.0)
    e2e_s = (time.perf_counter() - t0) / e2e_steps
    h2d = sum(b.numel() * 8 for b in rhs_p) * 2  # rhs and initial guess
    d2h = sum(b.numel() * 8 for b in sol_p)

    # the oracle on the GPU's solutions, and the FP64 operators at full size against the oracle
    checks, parity = None, None
    if rank == 0 and not args.no_cpu and not args.no_parity:
        sols = {"mixed": x_mixed}
        if args.fp64_steps > 0:
            sols["fp64"] = x64
        checks = oracle_check(levels, bc, rhs_h, sols)
        parity = parity_at_size(op, levels, bc, dev)

    # roofline of the dominant kernel: FP32 fused Jacobi sweep on the finest coarse level
    ms_jac = C.c_double(0.0)
    _lib.check(lib.ae_profile_kernel(op.handle, 1, 0, 0, 1, 20, C.byref(ms_jac)))
    ms_f64 = C.c_double(0.0)
    _lib.check(lib.ae_profile_kernel(op.handle, 0, 0, 0, 0, 5, C.byref(ms_f64)))
    ms_f32 = C.c_double(0.0)
    _lib.check(lib.ae_profile_kernel(op.handle, 0, 0, 0, 1, 20, C.byref(ms_f32)))
    n0 = int(np.prod(rhs_h[0].shape[1:]))
    peak, peak_kind = measured_peaks()
    f64_peak = fp64_peak_tflops() if rank == 0 else None
    # achieved = canonical algorithmic bytes (per-node stiffness) / time; the bytes the kernels
    # actually have to move on a grain map (2-byte id per node; the per-grain table stays in
    # L1/L2) are reported beside them
    grains = not args.per_node_model
    a_jac = JACOBI32_BYTES_PER_NODE_GRAINS if grains else JACOBI32_BYTES_PER_NODE
    a_f64 = FAPPLY64_BYTES_PER_NODE_GRAINS if grains else FAPPLY64_BYTES_PER_NODE
    a_f32 = FAPPLY32_BYTES_PER_NODE_GRAINS if grains else FAPPLY32_BYTES_PER_NODE
    jac_gbs = JACOBI32_BYTES_PER_NODE * n0 / (ms_jac.value * 1e-3) / 1e9
    fapply64_gbs = FAPPLY64_BYTES_PER_NODE * n0 / (ms_f64.value * 1e-3) / 1e9
    fapply32_gbs = FAPPLY32_BYTES_PER_NODE * n0 / (ms_f32.value * 1e-3) / 1e9

    cpu = None
    if rank == 0 and not args.no_cpu:
        try:
            cpu = cpu_oracle_sample(levels, bc, config1_solve_iters()[0], sample_iters=args.cpu_sample_iters,
                                    rhs=rhs_h)
            cpu["single_thread"] = cpu_single_thread(levels, bc, cpu)
        except Exception as e:  # pragma: no cover
            cpu = {"value": None, "unit": UNIT, "cores": None, "kind": "port", "sample": "failed: %s" % e}

    value = world * 1000.0 / ms_mixed
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_mixed, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32+f64", "data": "synthetic",
        "precision": "mixed: FP32 cycle in FP64 refinement",
        "config": config_of(args.cells),
        "run": {"inner_cycles": args.inner,
                "stiffness": ("per-node coefficients (ae_op_set_model)" if args.per_node_model else
                              "Voronoi grain ids + per-grain table (ae_op_set_model_grains)"),
                "parallelism": "replicas" if world > 1 else "single GPU",
                "l2": "inputs larger than L2 (stiffness %.1f GB)" % (sum(L["C"].nbytes for L in levels) / 1e9)},
        "iters_mixed": res_mixed[0], "resfinal_mixed": res_mixed[1], "target": res_mixed[2],
        "converged": bool(res_mixed[3]),
        "fp64": {"value": (world * 1000.0 / ms_fp64) if ms_fp64 else None, "unit": UNIT,
                 "ms_per_solve": ms_fp64, "iters": fp64_iters},
        "mixed_over_fp64": (ms_fp64 / ms_mixed) if ms_fp64 else None,
        "displacement_err_mixed_vs_fp64": disp_err,
        "fp64_oracle": oracle,
        "bottom_failures_cg": bottom_fail_cg,
        "mixed_bicgstab_bottom": bicg,
        "oracle_check": checks,
        "parity_at_size": parity,
        "e2e": {"value": world / e2e_s, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h},
        "roofline": {"bound": "hbm",
                     "kernel": ("FP32 damped-Jacobi sweep of the grain-map level (split: TMA-staged tile kernel "
                                "over the interior + per-node list over the boundary shell), level 0, 257^3 nodes"
                                if grains else "FP32 fused Jacobi sweep (per-node cubic stiffness), level 0, 257^3"),
                     "achieved": a_jac * n0 / (ms_jac.value * 1e-3) / 1e9, "peak": peak, "unit": "GB/s",
                     "frac": a_jac * n0 / (ms_jac.value * 1e-3) / 1e9 / peak,
                     "peak_kind": peak_kind, "traffic": JACOBI32_TRAFFIC_PER_NODE.get(grains, 0) * n0 or None,
                     "traffic_source": ("ncu dram bytes of the tile kernel per interior-box node at 193^3, times the "
                                        "level's nodes (the list kernel, 2 % of the nodes, not captured)" if grains
                                        else "ncu dram bytes of the same kernel per node at 193^3, times the nodes"),
                     "bytes_per_node": a_jac, "ms_per_launch": ms_jac.value,
                     "stiffness": "grain ids + table" if grains else "per node",
                     "canonical_bytes_per_node": JACOBI32_BYTES_PER_NODE,
                     "canonical_gbs": jac_gbs, "canonical_frac": jac_gbs / peak,
                     "canonical": "the same sweep's bytes with a per-node 21-coefficient stiffness (132 B/node)"},
        "fapply": {"fp64_gbs": fapply64_gbs, "fp64_ms": ms_f64.value, "fp32_gbs": fapply32_gbs,
                   "fp64_tflops": (FAPPLY64_FLOPS_PER_NODE_GRAINS * n0 / (ms_f64.value * 1e-3) / 1e12
                                   if grains else None),
                   "fp64_flops_per_node": FAPPLY64_FLOPS_PER_NODE_GRAINS if grains else None,
                   "fp64_peak_tflops_dgemm": f64_peak,
                   "fp64_frac_of_dgemm": (FAPPLY64_FLOPS_PER_NODE_GRAINS * n0 / (ms_f64.value * 1e-3) / 1e12 / f64_peak
                                          if grains and f64_peak else None),
                   "fp32_ms": ms_f32.value, "bytes_per_node_fp64": FAPPLY64_BYTES_PER_NODE,
                   "bytes_per_node_fp32": FAPPLY32_BYTES_PER_NODE,
                   "actual_bytes_per_node_fp64": a_f64, "actual_bytes_per_node_fp32": a_f32},
        "clocks": clk,
        "gpu_launches": int(launches),
        "cpu_baseline": cpu,
    }
    op.close()
    if rank == 0 and not args.no_config0:
        try:
            line["config0"] = bench_config0(args)
        except Exception as e:  # pragma: no cover
            line["config0"] = {"error": str(e)}
    add_cell_workloads(args, lib, line, rank, world)
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def add_cell_workloads(args, lib, line, rank, world):
    """The damaged-polycrystal, batched and served cell workloads.  The batch and the served stream
    shard over ranks (cells / requests, no data-path exchange); the single-box damaged solve and
    the model builders run on a 1-GPU job."""
    if not args.no_batch:
        try:
            line["batch"] = bench_batch(args, lib, rank, world)
        except Exception as e:  # pragma: no cover
            line["batch"] = {"error": str(e)}
    if not args.no_serve:
        try:
            sv = bench_serve(args, rank, world)
            if rank == 0:
                line["serve"] = sv
        except Exception as e:  # pragma: no cover
            line["serve"] = {"error": str(e)}
    if world > 1 or rank != 0:
        return
    if not args.no_damaged:
        try:
            line["damaged_polycrystal"] = bench_damaged_polycrystal(args)
        except Exception as e:  # pragma: no cover
            line["damaged_polycrystal"] = {"error": str(e)}
    if not args.no_builders:
        try:
            line["model_builders"] = bench_model_builders(args)
        except Exception as e:  # pragma: no cover
            line["model_builders"] = {"error": str(e)}
    if not args.no_neohookean:
        try:
            line["neohookean"] = bench_neohookean(args)
        except Exception as e:  # pragma: no cover
            line["neohookean"] = {"error": str(e)}


def bench_neohookean(args):
    """Newton<NeoHookean> (finite kinematics, the 45-slot Sym::Major tangent) on a box of
    (cells)^3 cells: mu 1, kappa 2.5, symmetry rollers on the low faces, x = 1 pulled by 5 %, a
    smooth body force; nriters Newton iterations from u = 0, each one ae_newton_neohookean (the
    tangent DDW(I + grad u) and rhs = b - N(u)) and one Linear solve of the correction to 1e-10.
    Device time per Newton solve in FP64 and mixed precision, the end-to-end time through host
    buffers, the Newton residual max|b - N(u)| / max|b| left after the last iteration, and the
    FP32 tangent Jacobi sweep (228 algorithmic B per node: 45 slots + x, b, 1/D, out) timed alone."""
    import ctypes as C
    import torch
    from anisotropicfracture_gb300 import _lib, models
    from anisotropicfracture_gb300.elastic import FACES, BCElastic, Elastic, Field, Newton, level_desc
    from oracle import pyoracle as po
    n = args.neo_cells
    neo = models.NeoHookean(1.0, 2.5)
    bc = BCElastic()
    for f, name in enumerate(FACES):
        for p, ax in enumerate("XYZ"):
            bc.type[f, p] = bc.Traction
            if ax + "LO" in name:
                bc.type[f, p] = bc.Displacement
            elif ax == "X" and "XHI" in name:
                bc.type[f, p], bc.val[f, p] = bc.Displacement, 0.05
    L = po.level(n)
    X, Y, Z = po.node_coords(L)
    force = np.zeros((3,) + L.shape)
    force[1] = 0.05 * np.sin(np.pi * X) * np.sin(np.pi * Z)
    b = po.bc_init(L, bc.type, bc.val, force)
    op = Elastic([level_desc(n)], models.MAJOR)
    op.SetBC(bc)
    op.SetUniform(False)  # the operator's own stream, ordered with the legacy default stream
    s = Newton(op)
    s.setNRIters(args.neo_nriters)
    s.setMaxFmgIter(0)
    s.setBottomSolver("bicgstab")
    s.setPreSmooth(2)
    s.setPostSmooth(2)
    s.opts.max_iter = 400
    bd = torch.from_numpy(b).cuda()
    out = {"workload": "%d^3 cells NeoHookean (mu 1, kappa 2.5), x = 1 pulled 5 %%, rollers on the low faces, "
                       "body force 0.05 sin(pi x) sin(pi z) e_y, %d Newton iterations, V(2,2) + BiCGStab, "
                       "corrections to tol_rel 1e-10" % (n, args.neo_nriters), "unit": "newton solves/s"}
    for prec, inner in (("fp64", 1), ("mixed", 4)):
        s.setPrecision(prec)
        s.opts.inner_cycles = inner
        ud = torch.zeros_like(bd)

        def one():
            ud.zero_()
            s.solve(Field(ud), Field(bd), model=neo, tol_rel=1e-10, tol_abs=0.0)

        one()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        one()
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        rec = {"value": 1000.0 / ms, "ms_per_newton_solve": ms, "mg_iters_last": s.stats.iters,
               "inner_cycles": inner}
        rd = bd.clone()
        op.NewtonNeoHookean(0, Field(rd), Field(ud), Field(bd), neo)
        torch.cuda.synchronize()
        rec["newton_residual"] = float(rd.abs().max()) / float(bd.abs().max())
        uh = np.zeros_like(b)
        t0 = time.perf_counter()
        s.solve(Field(uh), Field(b), model=neo, tol_rel=1e-10, tol_abs=0.0)
        e2e = time.perf_counter() - t0
        rec["e2e"] = {"value": 1.0 / e2e, "unit": "newton solves/s", "h2d_bytes_per_step": 2 * b.nbytes,
                      "d2h_bytes_per_step": b.nbytes}
        rec["e2e_vs_device_max_abs_diff"] = float(np.abs(uh - ud.cpu().numpy()).max())
        out[prec] = rec
    ms = C.c_double(0.0)
    lib = _lib.load()
    _lib.check(lib.ae_profile_kernel(op.handle, 1, 0, 0, 1, 20, C.byref(ms)))
    nodes = (n + 1) ** 3
    gbs = 228.0 * nodes / (ms.value * 1e-3) / 1e9
    peak, kind = measured_peaks()
    out["tangent_jacobi_fp32"] = {"ms": ms.value, "bytes_per_node": 228, "GB/s": gbs, "frac": gbs / peak,
                                  "peak": kind}
    op.close()
    return out


def bench_model_builders(args, reps=5):
    """The per-node stiffness built on the device from cell-centred order parameters over the
    (cells+1)^3 nodes of the single-box workload: the phase-field mixture of two cubic phases with
    eigenstrains (ae_op_set_model_mixture) and the isotropic degradation (ae_op_set_model_degraded).
    Inputs and outputs resident on the device; host clock around the call, which synchronises.
    Algorithmic bytes per node: mixture 21 slots + 9 eigenstrain written + one cell per phase read
    = 8 (21 + 9 + 2) = 256; degradation 2 slots written + one cell read = 24."""
    import torch
    from anisotropicfracture_gb300 import models
    from anisotropicfracture_gb300.elastic import Elastic, Field, level_desc
    n = args.cells
    nodes = (n + 1) ** 3
    rng = np.random.default_rng(7)
    torch.manual_seed(7)
    out = {"nodes": nodes, "timing": "host clock around %d synchronous calls, after one warm-up call" % reps}

    def timed(fn):
        fn()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(reps):
            fn()
        torch.cuda.synchronize()
        return (time.perf_counter() - t0) * 1e3 / reps

    eta = 0.05 + torch.rand((2, n + 1, n + 2, n + 2), dtype=torch.float64, device="cuda")
    table = models.cubic(1.68, 1.21, 0.75, models.random_rotations(2, rng))
    F0table = 0.01 * rng.standard_normal((2, 9))
    F0 = torch.zeros((9, n + 1, n + 1, n + 1), dtype=torch.float64, device="cuda")
    op = Elastic([level_desc(n)], models.MAJORMINOR)
    try:
        ms = timed(lambda: op.SetModelMixture(0, Field(eta, (-1, -1, 0)), table, F0table, Field(F0)))
    finally:
        op.close()
    del eta, F0
    out["mixture"] = {"ms": ms, "bytes_per_node": 256, "GB/s": 256.0 * nodes / (ms * 1e-3) / 1e9}

    damage = 0.9 * torch.rand((1, n + 2, n + 2, n + 2), dtype=torch.float64, device="cuda")
    op = Elastic([level_desc(n)], models.ISOTROPIC)
    try:
        ms = timed(lambda: op.SetModelDegraded(0, Field(damage, (-1, -1, -1)), 2.0, 1.0))
    finally:
        op.close()
    del damage
    torch.cuda.empty_cache()
    out["degraded"] = {"ms": ms, "bytes_per_node": 24, "GB/s": 24.0 * nodes / (ms * 1e-3) / 1e9}
    return out


def main_cells_only(args):
    """--only-cells: the batched and served workloads without the single-box configuration."""
    import torch
    from anisotropicfracture_gb300 import _lib, build as libbuild
    torch.cuda.set_device(0)
    libbuild.build()
    lib = _lib.load()
    line = {"metric": METRIC, "unit": UNIT, "n_gpus": 1, "data": "synthetic", "impl": "ours-cells"}
    add_cell_workloads(args, lib, line, 0, 1)
    print(json.dumps(line), flush=True)


if __name__ == "__main__":
    main()
