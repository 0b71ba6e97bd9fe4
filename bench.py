"""Benchmark of the MLFMA solve on GB300: FP64 MLFMA matvecs/s and time-to-RCS.

Workload (default): PEC sphere of radius 6 lambda at lambda = 1 m, icosphere
subdivided 6 times (81920 triangles, 122880 RWG unknowns), octree leaves
criterio_ladomax = 0.25 lambda (7 levels, L 51/31/20/13/9), plain FP64
MLFMA matvec as in the reference.  Synthetic mesh, seeded random
complex-Gaussian input vectors.  A step is one matvec over one right-hand
side; the working set (1.27 GB of radiation patterns, 0.58 GB of fields,
0.15 GB of near field) is far larger than L2, so no flush is needed.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

--impl reference times the CPU restatement of the reference's algorithm
(the reference itself is Fortran with no compiler here) on the host cores
with all threads, on the same workload, and prints the same JSON line.
Under torchrun each rank runs an independent replica (the solve does not
shard); value = matvecs of all ranks / max time over ranks.
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

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "time-to-RCS & MLFMA matvec/s at 123k RWG, rel.res 1e-4, ≤0.1 dB vs FP64 plain"
TRANSLATE6_DRAM_BYTES = 246.6e6 + 178.9e6   # read, written by the translation launch
WORKLOADS = {
    "sphere6": dict(level=6, radius=6.0, lam=1.0, ladomax=0.25,
                    name="PEC sphere r=6 lambda, icosphere-6 (81920 tri, 122880 RWG), leaf 0.25 lambda, FP64"),
    "sphere5": dict(level=5, radius=3.0, lam=1.0, ladomax=0.25,
                    name="PEC sphere r=3 lambda, icosphere-5 (20480 tri, 30720 RWG), leaf 0.25 lambda, FP64"),
}


def _jsonable(o):
    """numpy scalars and arrays in the JSON line"""
    if hasattr(o, "tolist"):
        return o.tolist()
    return str(o)


def _dist():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    lrank = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, lrank


class ClockSampler:
    """nvidia-smi clocks/throttle reasons sampled every 200 ms during the timed region."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index=0):
        self.index = index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for l in self.lines:
            f = [x.strip() for x in l.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                smax.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def fp64_peak_tflops(torch):
    """Measured FP64 rate of this GPU: cuBLAS DGEMM 4096^3, best of 5 (library roof, like the
    copy and bf16 GEMM roofs of the measured-peaks file)."""
    n = 4096
    a = torch.randn(n, n, dtype=torch.float64, device="cuda")
    b = torch.randn(n, n, dtype=torch.float64, device="cuda")
    for _ in range(2):
        a @ b
    torch.cuda.synchronize()
    best = 1e9
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        a @ b
        e1.record()
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1) / 1e3)
    return 2.0 * n ** 3 / best / 1e12


def replica_rate(steps: int, t_local: float, ws: int, device="cpu"):
    """Replicas only: every rank times its own `steps` matvecs; the job rate is
    all ranks' matvecs over the slowest rank's time (max over ranks)."""
    t = float(t_local)
    if ws > 1:
        import torch
        import torch.distributed as dist
        tt = torch.tensor([t], dtype=torch.float64, device=device)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        t = float(tt.item())
    return ws * steps / t, t


def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as fh:
            d = json.load(fh)
        return d.get("hbm_gbs", 6800.0), "measured"
    return 6800.0, "fallback"


def build_problem(wl):
    from lywell_gb300 import meshes
    return meshes.icosphere(wl["level"], wl["radius"])


def run_reference(args, wl):
    """CPU restatement of the reference (oracle/), all host threads, bounded sample."""
    ws, rank, _ = _dist()
    if rank != 0:
        return
    subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "oracle")], check=True)
    from oracle import core
    from oracle.rwg import RWG as ORWG
    ncores = os.cpu_count() or 1
    core.set_threads(ncores)
    tris = build_problem(wl)
    t0 = time.time()
    o = core.OracleMLFMA(ORWG(tris), lam=wl["lam"], ladomax=wl["ladomax"])
    setup = time.time() - t0
    rng = np.random.default_rng(0)
    x = rng.standard_normal(o.N) + 1j * rng.standard_normal(o.N)
    warm = max(3, args.warmup)
    t0 = time.time()
    for _ in range(warm):
        o.matvec(x)
    per = (time.time() - t0) / warm
    # the K steps asked for, unless they would take over two minutes of host time
    steps = max(1, min(args.steps, int(120.0 / max(per, 1e-3))))
    t0 = time.time()
    for _ in range(steps):
        o.matvec(x)
    dt = (time.time() - t0) / steps
    v = 1.0 / dt
    capped = "" if steps == args.steps else f" (capped from {args.steps} to two minutes)"
    line = {"impl": "reference", "metric": METRIC, "value": v, "unit": "matvec/s", "n_gpus": args.gpus,
            "steps": steps, "warmup": warm, "ms_per_step": dt * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "c128", "data": "synthetic",
            "config": {"workload": wl["name"], "N": o.N, "levels": o.nlev},
            "cpu_baseline": {"value": v, "unit": "matvec/s", "cores": core.get_threads(), "kind": "port",
                             "sample": f"{steps} FP64 MLFMA matvecs after {warm} warm-up ones and a "
                                       f"{setup:.1f}s set-up{capped}"},
            "e2e": {"value": v, "unit": "matvec/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line, default=_jsonable), flush=True)


def cpu_baseline_sample(wl, budget_s=10.0):
    from oracle import core
    from oracle.rwg import RWG as ORWG
    subprocess.run(["make", "-s", "-C", os.path.join(ROOT, "oracle")], check=True)
    core.set_threads(os.cpu_count() or 1)
    tris = build_problem(wl)
    t0 = time.time()
    o = core.OracleMLFMA(ORWG(tris), lam=wl["lam"], ladomax=wl["ladomax"])
    setup = time.time() - t0
    rng = np.random.default_rng(0)
    x = rng.standard_normal(o.N) + 1j * rng.standard_normal(o.N)
    o.matvec(x)
    # about budget_s seconds of matvecs (at least two)
    n, t0 = 0, time.time()
    while n < 2 or time.time() - t0 < budget_s:
        o.matvec(x)
        n += 1
    dt = (time.time() - t0) / n
    return {"value": 1.0 / dt, "unit": "matvec/s", "cores": core.get_threads(), "kind": "port",
            "sample": f"{n} FP64 MLFMA matvecs of the same workload ({n * dt:.1f} s) after one untimed "
                      f"and a {setup:.1f}s set-up"}


SPHEROID = dict(level=6, axes=(3.0, 0.75, 0.75), noise=0.01, seed=1234, lam=1.0, ladomax=0.25,
                name="PEC prolate spheroid 3 x 0.75 x 0.75 lambda from icosphere-6 (122880 RWG), seeded 2-ring-smoothed "
                     "radial noise 0.01 lambda, monostatic phi = 0..180 deg step 0.5 deg x {VV, HH} = 722 RHS")


def project_sequential(t_sample, iters, nang=722):
    """The reference's warm-started sequential sweep over nang angles, from a
    sample of its first angles: every iteration costs one FP64 operator
    application, so time is split over the sampled angles by iteration count;
    the first angle starts cold, every later one warm."""
    it = np.asarray(iters, dtype=float)
    return t_sample / it.sum() * (it[0] + (nang - 1) * it[1:].mean())


def batched_rcs_722(seq_angles=3, block=0, maxit=4000):
    """The 722-RHS monostatic sweep on the spheroid, measured end to end:
    phi = 0..180 deg in 0.5 deg steps (361 angles) x {VV, HH}, theta = 90 deg,
    solved as mixed-precision GMRES-IR (FP32 operator, FP64 residual to 1e-4)
    in blocks of right-hand sides (autotuned block size and engine), each
    block column sweeping a run of angles with extrapolated warm starts
    (mlf_monostatic mode 4).  Time to RCS = geometry and operator set-up +
    preconditioner set-up (27-box neighbourhood inverse, blocked FP32 LU) + autotuning + the two
    sweeps, which include the backscatter RCS of every angle.  The plain FP64
    GPU path -- the reference's sequential warm-started CGS sweep
    (gen_rcs_monostatica, main.f90:967-1089) on the FP64 operator, same
    preconditioner -- is run on the first `seq_angles` angles of each
    polarisation, which also give the per-angle RCS check, and projected to
    the 722 angles (its full run would take over an hour)."""
    import torch
    from lywell_gb300 import MLFMA, RWG, meshes

    t0 = time.time()
    tris = meshes.spheroid(SPHEROID["level"], SPHEROID["axes"], noise=SPHEROID["noise"], seed=SPHEROID["seed"])
    m = MLFMA(RWG(tris), lam=SPHEROID["lam"], ladomax=SPHEROID["ladomax"])
    torch.cuda.synchronize()
    t_tree = time.time() - t0
    t0 = time.time()
    bad = m.nearinv()
    torch.cuda.synchronize()
    t_pre = time.time() - t0
    t0 = time.time()
    # blocks of at most a quarter of the 361 angles of a sweep, so that every
    # column sweeps a run of at least four angles from extrapolated warm starts
    tune = (m.autotune_block(candidates=(8, 16, 32, 64)) if block <= 0
            else dict(block=block, tile_cols=0, per_rhs_ms={}))
    t_tune = time.time() - t0
    B = int(tune["block"])
    nang = 361
    phis = np.arange(nang) * np.deg2rad(0.5)
    sweeps = {}
    t0 = time.time()
    for pol in ("VV", "HH"):
        sweeps[pol] = m.monostatic(nang, phis=phis, pol=pol, errmax=1e-4, maxit=maxit, precond="nearinv", mode=4,
                                   block=B)
    t_sweep = time.time() - t0
    nrun = -(-nang // B)
    blocks = {pol: [int(max(sweeps[pol]["iters"][q * nrun + k] for q in range(B) if q * nrun + k < nang))
                    for k in range(nrun)] for pol in sweeps}
    t0 = time.time()
    seq, t_seq = {}, {}
    for pol in ("VV", "HH"):
        t1 = time.time()
        seq[pol] = m.monostatic(seq_angles, phis=phis[:seq_angles], pol=pol, errmax=1e-4, maxit=maxit,
                                precond="nearinv", mode=0)
        t_seq[pol] = time.time() - t1
    # column 0 of every block sweeps the first angles, as the sequential sample
    db = np.concatenate([np.abs(sweeps[pol]["sigma_db"][:seq_angles] - seq[pol]["sigma_db"]) for pol in seq])
    proj_seq = sum(project_sequential(t_seq[pol], seq[pol]["iters"], nang) for pol in seq)
    status = sorted({s for pol in sweeps for s in sweeps[pol]["status"]})
    ttr = t_tree + t_pre + t_tune + t_sweep
    out = {"workload": SPHEROID["name"], "N": m.N, "near_nnz": m.nnz, "setup_s": t_tree, "precond_setup_s": t_pre,
           "precond": "27-box neighbourhood inverse (blocked FP32 LU per leaf box)", "nearinv_bad_box": bad,
           "autotune": tune, "autotune_s": t_tune,
           "block": B,
           "measured_722": {"mode": 4, "angles": 2 * nang, "sweep_s": t_sweep, "time_to_rcs_s": ttr,
                            "status": status, "iters_per_block": blocks,
                            "iters_per_angle": {pol: [int(v) for v in sweeps[pol]["iters"]] for pol in sweeps}},
           "fp64_sequential_sample": {"angles_per_pol": seq_angles, "seconds": t_seq,
                                      "iters": {pol: [int(v) for v in seq[pol]["iters"]] for pol in seq},
                                      "status": sorted({s for pol in seq for s in seq[pol]["status"]}),
                                      "projected_722_s": t_tree + t_pre + proj_seq,
                                      "note": "projected: the sampled angles' time split by iteration count, "
                                              "the cold first angle of each polarisation once, every later "
                                              "angle as the sampled warm ones"},
           "rcs_db_vs_fp64_per_angle": [float(v) for v in db],
           "rcs_db_maxdiff_vs_fp64": float(db.max()),
           "speedup_vs_fp64_projected": (t_tree + t_pre + proj_seq) / ttr}
    m.close()
    return out


def learned_sample(steps=3000, seed=0):
    """Learned preconditioner: trained on three seeded superellipsoids
    (exponent U[2, 6], semi-axes (2, 1, 1) lambda x U[0.85, 1.15], 7680 RWG)
    with the library's MLP kernels, evaluated on the held-out superellipsoid
    (exponent 4, 2 x 1 x 1 lambda): CGS to 1e-4, x-polarised wave from -z,
    against no preconditioner, ILU0 and the exact neighbourhood inverse it
    corrects; time to RCS = preconditioner set-up + solve + two bistatic cuts."""
    import torch
    from lywell_gb300 import MLFMA, RWG, meshes
    from lywell_gb300.learned import solve_with_fallback, train

    rng = np.random.default_rng(7)
    d = np.array([0.0, 0.0, 1.0])
    p = np.array([1.0, 0.0, 0.0], dtype=complex)
    th = np.deg2rad(np.arange(0, 181, 1.0))
    t0 = time.time()
    ctxs, bs = [], []
    for _ in range(3):
        e = rng.uniform(2, 6)
        ax = np.array([2.0, 1.0, 1.0]) * rng.uniform(0.85, 1.15, 3)
        mt = MLFMA(RWG(meshes.superellipsoid(4, tuple(ax), e)), lam=1.0, ladomax=0.25)
        mt.nearinv()
        ctxs.append(mt)
        bs.append(mt.excitation(d, p))
    lp = train(ctxs, bs, steps=steps, batch=8192, lr=1e-3, seed=seed)
    t_train = time.time() - t0
    for mt in ctxs:
        mt.close()
    m = MLFMA(RWG(meshes.superellipsoid(4, (2.0, 1.0, 1.0), 4.0)), lam=1.0, ladomax=0.25)
    b = m.excitation(d, p)
    res = {}
    ref_db = None

    def finish(label, t_setup, out):
        torch.cuda.synchronize()
        t1 = time.time()
        s0 = m.rcs(out["x"], p, th, 0 * th)
        s9 = m.rcs(out["x"], p, th, 0 * th + np.pi / 2)
        t_rcs = time.time() - t1
        db = 10 * np.log10(np.concatenate([s0, s9]))
        rel = float(np.linalg.norm(m.matvec(out["x"]) - b) / np.linalg.norm(b))
        res[label] = {"iters": int(out["iters"]), "status": out["status"], "setup_s": t_setup,
                      "solve_s": out["_t"], "time_to_rcs_s": t_setup + out["_t"] + t_rcs, "true_relres": rel,
                      "_db": db}

    def timed(fn):
        t1 = time.time()
        out = fn()
        out["_t"] = time.time() - t1
        return out

    finish("none", 0.0, timed(lambda: m.cgs(b, errmax=1e-4, maxit=3000)))
    plain = res["none"]["iters"] if res["none"]["status"] == "converged" else 3000
    t1 = time.time(); ierr = m.ilu0(); t_ilu = time.time() - t1
    finish("ilu0", t_ilu, timed(lambda: m.cgs(b, errmax=1e-4, maxit=300, precond="ilu0")))   # capped: it stalls
    t1 = time.time(); m.nearinv(); t_nb = time.time() - t1
    finish("exact_neighbourhood_inverse", t_nb, timed(lambda: m.cgs(b, errmax=1e-4, maxit=3000, precond="nearinv")))
    t1 = time.time(); lp.apply_to(m); t_inst = time.time() - t1
    out = timed(lambda: solve_with_fallback(m, b, lp, plain_iters=plain, install_first=False))
    finish("learned", t_nb + t_inst, out)
    res["learned"]["used"] = out["used"]
    ref = res["exact_neighbourhood_inverse"]["_db"]
    for k in res:
        db = res[k].pop("_db")
        res[k]["rcs_db_maxdiff_vs_exact"] = float(np.abs(db - ref).max()) if res[k]["status"] == "converged" else None
    m.close()
    return {"workload": "superellipsoid exponent 4, 2 x 1 x 1 lambda, icosphere-4 (7680 RWG); trained on 3 seeded "
                        "superellipsoids of the same mesh density", "train_s": t_train, "gamma": lp.gamma,
            "trace": {str(k): v for k, v in lp.trace.items()}, "ilu0_ierr": ierr, "results": res}


def learned_heldout_123k(steps=3000, seed=0):
    """The learned preconditioner on the task's held-out body: superellipsoid of
    exponent 4, semi-axes 4 x 2 x 2 lambda, icosphere-6 (122 880 RWG, about
    60 bases per 0.25 lambda leaf box, neighbourhoods of ~1000-2500
    unknowns).  Trained on three seeded superellipsoids of 30 720 RWG
    (icosphere-5), exponent U[2, 6], semi-axes (a, a/2, a/2) x U[0.85, 1.15]
    with a = U[1.5, 2.5] lambda -- the low end of the 1.5-5 lambda range,
    where 30 720 RWG has the held-out body's mesh density -- with 2-ring
    targets from the blocked FP32 LU.
    x-polarised wave from -z, solves to 1e-4, time to RCS = preconditioner
    set-up + solve + two bistatic cuts; compared with ILU0 (the reference's
    preconditioner, CGS capped at 300 iterations), no preconditioner (capped
    at 3000) and the exact neighbourhood inverse M1 the network corrects.
    The learned preconditioner is run with mixed GMRES-IR and with FP64 CGS,
    the latter falling back to ILU0 (capped at 300 iterations) if it has not
    converged within the unpreconditioned iteration count."""
    import torch
    from lywell_gb300 import MLFMA, RWG, meshes
    from lywell_gb300.learned import solve_with_fallback, train

    rng = np.random.default_rng(23)
    d = np.array([0.0, 0.0, 1.0])
    p = np.array([1.0, 0.0, 0.0], dtype=complex)
    th = np.deg2rad(np.arange(0, 181, 1.0))
    t0 = time.time()
    ctxs, bs, bodies = [], [], []
    for _ in range(3):
        e = float(rng.uniform(2, 6))
        a = float(rng.uniform(1.5, 2.5))
        ax = np.array([a, a / 2, a / 2]) * rng.uniform(0.85, 1.15, 3)
        mt = MLFMA(RWG(meshes.superellipsoid(5, tuple(ax), e)), lam=1.0, ladomax=0.25)
        assert mt.nearinv() == 0
        ctxs.append(mt)
        bs.append(mt.excitation(d, p))
        bodies.append({"exponent": e, "semi_axes": [float(v) for v in ax], "N": mt.N})
    lp = train(ctxs, bs, steps=steps, batch=8192, lr=1e-3, seed=seed)
    torch.cuda.synchronize()
    t_train = time.time() - t0
    for mt in ctxs:
        mt.close()
    m = MLFMA(RWG(meshes.superellipsoid(6, (4.0, 2.0, 2.0), 4.0)), lam=1.0, ladomax=0.25)
    b = m.excitation(d, p)
    res, ref = {}, {}

    def finish(label, t_setup, out, t_solve):
        torch.cuda.synchronize()
        t1 = time.time()
        db = 10 * np.log10(np.concatenate([m.rcs(out["x"], p, th, 0 * th), m.rcs(out["x"], p, th, 0 * th + np.pi / 2)]))
        t_rcs = time.time() - t1
        rel = float(np.linalg.norm(m.matvec(out["x"]) - b) / np.linalg.norm(b))
        res[label] = {"iters": int(out["iters"]), "status": out["status"], "setup_s": t_setup, "solve_s": t_solve,
                      "time_to_rcs_s": t_setup + t_solve + t_rcs, "true_relres": rel}
        ref[label] = db

    def timed(fn):
        torch.cuda.synchronize()
        t1 = time.time()
        out = fn()
        torch.cuda.synchronize()
        return out, time.time() - t1

    out, ts = timed(lambda: m.cgs(b, errmax=1e-4, maxit=3000))
    finish("none", 0.0, out, ts)
    plain = res["none"]["iters"] if res["none"]["status"] == "converged" else 3000
    (ierr, t_ilu) = timed(lambda: m.ilu0())
    if ierr == 0:
        out, ts = timed(lambda: m.cgs(b, errmax=1e-4, maxit=300, precond="ilu0"))   # capped: it stalls
        finish("ilu0_reference", t_ilu, out, ts)
    else:
        res["ilu0_reference"] = {"status": f"zero pivot at row {ierr}", "setup_s": t_ilu}
    (_, t_m1) = timed(lambda: m.nearinv())
    out, ts = timed(lambda: m.cgs(b, errmax=1e-4, maxit=3000, precond="nearinv"))
    finish("fp64_cgs_exact_M1", t_m1, out, ts)
    out, ts = timed(lambda: m.solve(b, errmax=1e-4, maxit=3000, precond="nearinv", mixed=True))
    finish("mixed_exact_M1", t_m1, out, ts)
    (_, t_inst) = timed(lambda: lp.apply_to(m))
    out, ts = timed(lambda: m.solve(b, errmax=1e-4, maxit=3000, precond="nearinv", mixed=True))
    finish("mixed_learned", t_m1 + t_inst, out, ts)
    # FP64 CGS with the ILU0 fallback; the fallback solve is capped like the ILU0 run above
    out, ts = timed(lambda: solve_with_fallback(m, b, lp, plain_iters=plain, install_first=False, maxit=300))
    used = out["used"]
    finish("fp64_cgs_learned_with_fallback", t_m1 + t_inst, out, ts)
    res["fp64_cgs_learned_with_fallback"]["used"] = used
    base = ref["fp64_cgs_exact_M1"]
    for k in res:
        res[k]["rcs_db_maxdiff_vs_exact_M1"] = (float(np.abs(ref[k] - base).max())
                                              if res[k]["status"] == "converged" and k in ref else None)
    nnz = m.nnz
    m.close()
    return {"workload": "superellipsoid exponent 4, 4 x 2 x 2 lambda, icosphere-6 (122880 RWG), leaf 0.25 lambda; "
                        "trained on 3 seeded superellipsoids of 30720 RWG at the same mesh density",
            "N": 122880, "near_nnz": nnz, "training_bodies": bodies, "train_s": t_train, "gamma": lp.gamma,
            "trace": {str(k): v for k, v in lp.trace.items()}, "ilu0_ierr": ierr, "results": res}


def learned_at_scale(steps=3000, seed=0):
    """Learned preconditioner on the bench's 122 880-RWG sphere: trained on three
    seeded superellipsoids at the sphere's mesh density (icosphere-5, 30 720 RWG,
    exponent U[2, 6], semi-axes 3 lambda x U[0.8, 1.2]), then the sphere
    (held out) is solved to 1e-4 with the exact neighbourhood inverse and with
    the learned correction, by FP64 CGS and by mixed GMRES-IR; ILU0 (the
    reference's preconditioner) is run capped at 300 CGS iterations.  Time to
    RCS = preconditioner set-up + solve + two bistatic cuts."""
    import torch
    from lywell_gb300 import MLFMA, RWG, meshes
    from lywell_gb300.learned import train

    rng = np.random.default_rng(11)
    d = np.array([0.0, 0.0, 1.0])
    p = np.array([1.0, 0.0, 0.0], dtype=complex)
    th = np.deg2rad(np.arange(0, 181, 1.0))
    t0 = time.time()
    ctxs, bs = [], []
    for _ in range(3):
        e = rng.uniform(2, 6)
        ax = 3.0 * rng.uniform(0.8, 1.2, 3)
        mt = MLFMA(RWG(meshes.superellipsoid(5, tuple(ax), e)), lam=1.0, ladomax=0.25)
        mt.nearinv()
        ctxs.append(mt)
        bs.append(mt.excitation(d, p))
    lp = train(ctxs, bs, steps=steps, batch=8192, lr=1e-3, seed=seed)
    t_train = time.time() - t0
    for mt in ctxs:
        mt.close()
    wl = WORKLOADS["sphere6"]
    m = MLFMA(RWG(meshes.icosphere(wl["level"], wl["radius"])), lam=wl["lam"], ladomax=wl["ladomax"])
    b = m.excitation(d, p)
    out = {}
    ref_db = None

    def run(label, setup, mixed, precond, maxit=4000):
        nonlocal ref_db
        torch.cuda.synchronize()
        t1 = time.time()
        setup()
        t_setup = time.time() - t1
        t1 = time.time()
        o = m.solve(b, errmax=1e-4, maxit=maxit, precond=precond, mixed=mixed)
        t_solve = time.time() - t1
        t1 = time.time()
        s0 = m.rcs(o["x"], p, th, 0 * th)
        s9 = m.rcs(o["x"], p, th, 0 * th + np.pi / 2)
        t_rcs = time.time() - t1
        db = 10 * np.log10(np.concatenate([s0, s9]))
        ent = {"iters": int(o["iters"]), "status": o["status"], "setup_s": t_setup, "solve_s": t_solve,
               "time_to_rcs_s": t_setup + t_solve + t_rcs, "outer": int(o.get("outer", 0))}
        if o["status"] == "converged":
            if ref_db is None:
                ref_db = db
            ent["rcs_db_maxdiff_vs_fp64_exact"] = float(np.abs(db - ref_db).max())
        out[label] = ent

    def learned_setup():
        m.nearinv()
        lp.apply_to(m)

    run("fp64_cgs_exact_neighbourhood", m.nearinv, False, "nearinv")
    run("fp64_cgs_learned", learned_setup, False, "nearinv")
    run("mixed_exact_neighbourhood", m.nearinv, True, "nearinv")
    run("mixed_learned", learned_setup, True, "nearinv")
    run("fp64_cgs_ilu0_reference", lambda: m.ilu0(), False, "ilu0", maxit=300)
    # the three additions together: the 722-RHS monostatic sweep on the sphere (phi = 0..180 deg
    # step 0.5 deg x {VV, HH}), mixed + batched (autotuned block) + learned, measured over all
    # 722 angles; the plain FP64 path (the reference's warm-started sequential CGS, exact
    # neighbourhood inverse) on the first 3 angles of each polarisation, projected
    nang = 361
    phis = np.arange(nang) * np.deg2rad(0.5)
    t1 = time.time()
    m.nearinv()
    t_exact = time.time() - t1
    seq, t_seq = {}, {}
    for pol in ("VV", "HH"):
        torch.cuda.synchronize()
        t1 = time.time()
        seq[pol] = m.monostatic(3, phis=phis[:3], pol=pol, errmax=1e-4, maxit=4000, precond="nearinv", mode=0)
        t_seq[pol] = time.time() - t1
    t1 = time.time()
    lp.apply_to(m)
    t_inst = time.time() - t1
    t1 = time.time()
    tune = m.autotune_block(candidates=(8, 16, 32, 64))   # runs of at least four angles per column
    t_tune = time.time() - t1
    B = int(tune["block"])
    torch.cuda.synchronize()
    bat = {}
    t1 = time.time()
    for pol in ("VV", "HH"):
        bat[pol] = m.monostatic(nang, phis=phis, pol=pol, errmax=1e-4, maxit=4000, precond="nearinv", mode=4,
                                block=B)
    t_bat = time.time() - t1
    m.close()
    nrun = -(-nang // B)
    p_seq = t_exact + sum(project_sequential(t_seq[pol], seq[pol]["iters"], nang) for pol in seq)
    ttr = t_exact + t_inst + t_tune + t_bat
    db = np.concatenate([np.abs(bat[pol]["sigma_db"][:3] - seq[pol]["sigma_db"]) for pol in seq])
    sweep = {"fp64_sequential_exact": {"angles_per_pol": 3, "seconds": t_seq,
                                       "iters": {pol: [int(v) for v in seq[pol]["iters"]] for pol in seq},
                                       "projected_722_s": p_seq,
                                       "note": "projected: the cold first angle of each polarisation once, every "
                                               "later angle as the sampled warm ones, time split by iteration "
                                               "count; + the exact neighbourhood inverse set-up"},
             "mixed_batched_learned": {"mode": 4, "angles": 2 * nang, "block": B, "autotune": tune,
                                       "sweep_s": t_bat, "time_to_rcs_s": ttr,
                                       "setup_s": {"exact_inverse": t_exact, "learned_install": t_inst,
                                                   "autotune": t_tune},
                                       "status": sorted({v for pol in bat for v in bat[pol]["status"]}),
                                       "iters_per_block": {pol: [int(max(bat[pol]["iters"][q * nrun + k]
                                                                         for q in range(B) if q * nrun + k < nang))
                                                                 for k in range(nrun)] for pol in bat}},
             "rcs_db_vs_fp64_per_angle": [float(v) for v in db],
             "rcs_db_maxdiff": float(db.max())}
    sweep["speedup_vs_fp64_projected"] = p_seq / ttr
    base = out["fp64_cgs_exact_neighbourhood"]["time_to_rcs_s"]
    return {"workload": WORKLOADS["sphere6"]["name"] + "; trained on 3 seeded superellipsoids (30720 RWG, same "
                                                       "mesh density)",
            "train_s": t_train, "gamma": lp.gamma, "trace": {str(k): v for k, v in lp.trace.items()},
            "results": out,
            "speedup_vs_fp64_exact": {k: base / v["time_to_rcs_s"] for k, v in out.items()
                                      if v["status"] == "converged"},
            "sweep_722": sweep}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="sphere6", choices=list(WORKLOADS))
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-time-to-rcs", action="store_true")
    ap.add_argument("--rcs-maxit", type=int, default=4000)
    ap.add_argument("--no-batched", action="store_true", help="skip the 722-RHS spheroid sweep")
    ap.add_argument("--learned", action="store_true", help="add the learned-preconditioner samples (about 6 min)")
    ap.add_argument("--seq-angles", type=int, default=3)
    ap.add_argument("--block", type=int, default=0, help="RHS per block of the batched sweep (0: autotuned)")
    args = ap.parse_args()
    wl = WORKLOADS[args.workload]
    if args.impl == "reference":
        run_reference(args, wl)
        return

    import torch
    ws, rank, lrank = _dist()
    torch.cuda.set_device(lrank)
    if ws > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl", device_id=torch.device("cuda", lrank))
    from lywell_gb300 import MLFMA, RWG, ajustar_polariz, direction

    tris = build_problem(wl)
    torch.cuda.synchronize()
    t0 = time.time()
    rwg = RWG(tris)
    m = MLFMA(rwg, lam=wl["lam"], ladomax=wl["ladomax"])
    torch.cuda.synchronize()
    setup_s = time.time() - t0
    N = m.N
    rng = np.random.default_rng(rank)
    xh = rng.standard_normal(N) + 1j * rng.standard_normal(N)
    x = torch.from_numpy(xh).to("cuda")
    y = torch.empty_like(x)
    stream = torch.cuda.current_stream().cuda_stream

    def step():
        m.matvec_device(x.data_ptr(), y.data_ptr(), 1, stream)

    for _ in range(max(3, args.warmup)):
        step()
    torch.cuda.synchronize()
    cnt = m.algorithmic_counts()
    clocks = ClockSampler(lrank)
    clocks.start()
    time.sleep(0.3)
    m.set_profiling(True)
    stage = np.zeros(5)
    if ws > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(args.steps):
        step()
        stage += m.stage_times()
    e1.record()
    torch.cuda.synchronize()
    if ws > 1:
        torch.distributed.barrier()
    m.set_profiling(False)
    clk = clocks.stop()
    value, t = replica_rate(args.steps, e0.elapsed_time(e1) / 1e3, ws, "cuda")
    stage_ms = stage / args.steps

    # end to end through the public host API: pinned host x -> device -> host y
    xp = torch.from_numpy(xh).pin_memory()
    yp = torch.empty_like(xp).pin_memory()
    import ctypes
    from lywell_gb300 import _capi
    lib = _capi.load()
    for _ in range(2):
        lib.mlf_matvec(m.handle, ctypes.c_void_p(xp.data_ptr()), ctypes.c_void_p(yp.data_ptr()), 1, N)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        rc = lib.mlf_matvec(m.handle, ctypes.c_void_p(xp.data_ptr()), ctypes.c_void_p(yp.data_ptr()), 1, N)
        assert rc == 0
    t_e2e = time.perf_counter() - t0
    e2e = ws * args.steps / t_e2e if ws == 1 else args.steps / t_e2e * ws

    # roofline of the dominant stage (translation) against the FP64 roof, HBM beside it
    fp64 = fp64_peak_tflops(torch)
    hbm, hbm_kind = measured_peaks()
    tr_s = stage_ms[2] / 1e3
    tr_flops = cnt["flops"]["translation"]
    achieved = tr_flops / tr_s / 1e12
    total_tflops = cnt["flops_total"] / (t / args.steps * ws) / 1e12
    roof = {"bound": "fp64", "kernel": "k_translate (all levels, 1 launch/matvec)", "achieved": achieved, "peak": fp64,
            "unit": "TFLOP/s", "frac": achieved / fp64,
            "traffic": (TRANSLATE6_DRAM_BYTES if wl is WORKLOADS["sphere6"] else None),
            "traffic_unit": "bytes per matvec",
            "traffic_source": ("ncu dram__bytes_read.sum + dram__bytes_write.sum of the stage's launch in one "
                               "matvec of this workload, from a separate capture of this kernel (not "
                               "measured in this run)" if wl is WORKLOADS["sphere6"] else None),
            "peak_source": "measured here: cuBLAS DGEMM 4096^3 (GB300 FP64 pipe)",
            "algorithmic_flops_per_matvec": tr_flops,
            "hbm": {"achieved_gbs": cnt["translation_bytes"] / tr_s / 1e9, "peak_gbs": hbm,
                    "peak_source": hbm_kind,
                    "frac": cnt["translation_bytes"] / tr_s / 1e9 / hbm},
            "matvec": {"flops": cnt["flops_total"], "bytes": cnt["bytes_total"],
                       "achieved_tflops": total_tflops, "frac_fp64": total_tflops / fp64,
                       "achieved_gbs": cnt["bytes_total"] / (t / args.steps * ws) / 1e9,
                       "frac_hbm": cnt["bytes_total"] / (t / args.steps * ws) / 1e9 / hbm},
            "stage_ms": {"aggregation": stage_ms[0], "interpolation": stage_ms[1], "translation": stage_ms[2],
                         "anterpolation": stage_ms[3], "receive_near": stage_ms[4]}}

    # time to RCS: set-up (octree, tables, patterns, near field, preconditioner) + solve to
    # 1e-4 + two bistatic cuts (phi = 0, 90 deg; theta = 0..180 deg step 1)
    ttr = None
    if not args.no_time_to_rcs:
        d = np.array([0.0, 0.0, 1.0])      # x-polarised wave incident from -z (propagating along +z)
        pol = np.array([1.0, 0, 0], dtype=np.complex128)
        th = np.deg2rad(np.arange(0, 181, 1.0))
        ttr = {}
        rcs_ref = None
        for label, mixed in (("fp64_cgs_nearinv", False), ("mixed_gmres_ir_nearinv", True)):
            torch.cuda.synchronize()
            t0 = time.time()
            m2 = MLFMA(RWG(tris), lam=wl["lam"], ladomax=wl["ladomax"])
            bad = m2.nearinv()
            t_setup = time.time() - t0
            t1 = time.time()
            b = m2.excitation(d, pol)
            out = m2.solve(b, errmax=1e-4, maxit=args.rcs_maxit, precond="nearinv", mixed=mixed)
            t_solve = time.time() - t1
            t2 = time.time()
            s0 = m2.rcs(out["x"], pol, th, np.zeros_like(th))
            s9 = m2.rcs(out["x"], pol, th, np.full_like(th, np.pi / 2))
            t_rcs = time.time() - t2
            true_res = float(np.linalg.norm(m2.matvec(out["x"]) - b) / np.linalg.norm(b))
            db = 10 * np.log10(np.concatenate([s0, s9]))
            ent = {"seconds": t_setup + t_solve + t_rcs, "setup_s": t_setup, "solve_s": t_solve, "rcs_s": t_rcs,
                   "iters": out["iters"], "outer": out.get("outer", 0), "status": out["status"],
                   "relres_fp64": true_res, "nearinv_bad_box": bad, "rcs_angles": int(db.size)}
            if rcs_ref is None:
                rcs_ref = db
            else:
                ent["rcs_db_maxdiff_vs_fp64"] = float(np.abs(db - rcs_ref).max())
            ttr[label] = ent
            m2.close()
        ttr["speedup_mixed_vs_fp64"] = ttr["fp64_cgs_nearinv"]["seconds"] / ttr["mixed_gmres_ir_nearinv"]["seconds"]

    batched = None
    if not args.no_batched and rank == 0:
        batched = batched_rcs_722(args.seq_angles, args.block, args.rcs_maxit)

    learned = None
    if args.learned and rank == 0:
        learned = {"held_out_superellipsoid_7680": learned_sample(),
                   "held_out_superellipsoid_122880": learned_heldout_123k(),
                   "sphere_122880": learned_at_scale()}

    launches_per_matvec = 1 + (m.nlev - 3) + 1 + (m.nlev - 3) + 1   # translation: all levels in one
    line = {"metric": METRIC, "value": value, "unit": "matvec/s", "n_gpus": ws, "steps": args.steps,
            "warmup": max(3, args.warmup), "ms_per_step": t / args.steps * 1e3, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "c128", "data": "synthetic",
            "config": {"workload": wl["name"], "N": N, "levels": m.nlev,
                       "samples_per_level": [m.levels[l]["K"] for l in range(3, m.nlev + 1)],
                       "near_nnz": m.nnz, "parallelism": f"replicas x{ws}",
                       "l2": "inputs larger than L2 (patterns 1.27 GB streamed per matvec)"},
            "e2e": {"value": e2e, "unit": "matvec/s", "h2d_bytes_per_step": N * 16, "d2h_bytes_per_step": N * 16},
            "roofline": roof, "clocks": clk, "gpu_launches": launches_per_matvec * args.steps,
            "setup_s": setup_s, "time_to_rcs": ttr, "batched_rcs": batched}
    if learned is not None:
        line["learned_preconditioner"] = learned
    if rank == 0 and ws == 1 and not args.no_cpu_baseline:
        line["cpu_baseline"] = cpu_baseline_sample(wl)
    if rank == 0:
        print(json.dumps(line, default=_jsonable), flush=True)
    m.close()
    if ws > 1:
        torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
