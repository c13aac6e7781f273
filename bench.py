#!/usr/bin/env python
"""Benchmark of the B200 3x3-block CG drop-in (FrontISTR hecmw_solve, METHOD=CG).

Workload (default): the 100x100x100 HEX8 linear-elastic cantilever cube --
1,030,301 nodes, 3,090,903 DOF, 27,270,901 3x3 FP64 blocks (~2 GB of values) --
E=210000, nu=0.3, 2x2x2 Gauss, face z=0 clamped, -1.0 y-load on every node of
face z=100, assembled on the host like fistr1 (synthetic input; there is no
public dataset).  One step = one solve to relative residual 1e-8 with CG + SSOR
(PRECOND=1, iterPREmax=1, ncolor_in=10, sigma_diag=1), X0 = 0.

  value        seconds per solve with B, X and the matrix resident in HBM
               (device events around the one-graph CG solve), max over ranks
  e2e          seconds per solve through the drop-in C-ABI call with host buffers (pinned)
               (hecmw33_gpu_solve: matrix values + B + X uploaded, numeric
               preconditioner rebuild, solve, X downloaded), wall clock
  roofline     the dominant kernel of the headline solve, one SSOR application (the
               forward + backward colour sweeps; for the learned variants the two-grid
               cycle's smoother, the same SSOR in first-fit colour order), against
               measured HBM bandwidth; roofline_spmv the plain FP64 SpMV (spmv_kernel)
  cpu_baseline the CPU oracle (C restatement of the reference's CG + SSOR,
               OpenMP over all host cores) solving the same system to the same
               tolerance, measured (setup reported separately)
  parity       the GPU solves against that oracle solve: iterations, solution,
               colour schedule

The path does not shard (one GPU domain): with --gpus N, N independent replicas
run, one per GPU (torch.distributed only for the barrier and the max).
`--impl reference` times the CPU oracle alone, full solves to tolerance (the
reference's own CPU path is Fortran and cannot be built on this image).
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "s to rel-res 1e-8, 3M-DOF HEX8 elasticity: learned+mixed vs FP64 CG on 1 B200"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--mesh", default="100,100,100", help="nx,ny,nz HEX8 elements")
    ap.add_argument("--precond", type=int, default=1)
    ap.add_argument("--tol", type=float, default=1e-8)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-mixed", action="store_true", help="skip the mixed-precision variant")
    ap.add_argument("--no-learned", action="store_true", help="skip the learned-preconditioner variants")
    ap.add_argument("--train-steps", type=int, default=40)
    ap.add_argument("--train-lr", type=float, default=5e-3)
    ap.add_argument("--no-multi", action="store_true", help="skip the 16-load-case multi-RHS measurement")
    ap.add_argument("--no-batched", action="store_true", help="skip the 256-system batched measurement")
    ap.add_argument("--no-assembly", action="store_true", help="skip the HEX8 assembly measurement")
    ap.add_argument("--no-domains", action="store_true", help="skip the decomposed-mesh measurement")
    ap.add_argument("--no-config3", action="store_true",
                    help="skip the mixed-precision measurement on the jittered heterogeneous 80^3 system")
    ap.add_argument("--no-ilu0", action="store_true", help="skip the CG + ILU(0) measurement")
    ap.add_argument("--no-newton", action="store_true",
                    help="skip the learned preconditioner's Neo-Hookean Newton sequence (--learned-newton alone)")
    ap.add_argument("--batch-systems", type=int, default=256)
    ap.add_argument("--batch-edges", default="8,40", help="element range per box edge of the batch")
    ap.add_argument("--spmv-only", type=int, default=0,
                    help="only build the system and run this many SpMV launches (profiling)")
    ap.add_argument("--learned-newton", action="store_true",
                    help="the learned preconditioner in a Neo-Hookean Newton sequence (prints its own JSON line)")
    ap.add_argument("--newton-mesh", default="64,64,64")
    ap.add_argument("--profile-solve", action="store_true",
                    help="one solve capped at 5 CG iterations, nothing printed (profiling)")
    ap.add_argument("--profile-mode", type=int, default=0,
                    help="precision mode (Iarray(42)) of the --profile-solve solve")
    ap.add_argument("--profile-coarse", type=int, default=-1,
                    help="with --profile-solve or --profile-multi: the two-level preconditioner with these "
                         "smoothing weights (Iarray(44): 1 none, 2 one half; no training needed)")
    ap.add_argument("--profile-e2e", action="store_true",
                    help="one drop-in call with host buffers and a forced numeric rebuild (learned + mode 1, "
                         "network trained for 2 steps on 1 recorded solve), the last of 3 inside "
                         "cudaProfilerStart/Stop (for ncu --profile-from-start off)")
    ap.add_argument("--profile-multi", action="store_true",
                    help="one 16-load-case solve capped at 3 CG iterations, nothing printed (profiling)")
    ap.add_argument("--profile-batch", action="store_true",
                    help="one batched solve of --batch-systems boxes, nothing printed (profiling)")
    return ap.parse_args()


def pin_local_gpu():
    """One process per GPU: expose only this rank's GPU before CUDA initialises."""
    lr = os.environ.get("LOCAL_RANK")
    if lr is None:
        return
    vis = os.environ.get("CUDA_VISIBLE_DEVICES")
    ids = vis.split(",") if vis else None
    os.environ["CUDA_VISIBLE_DEVICES"] = ids[int(lr)] if ids else lr


class Clocks:
    """Samples nvidia-smi every 200 ms while the timed region runs."""

    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, uuid):
        self.uuid, self.proc, self.lines = uuid, None, []

    def start(self):
        try:
            cmd = ["nvidia-smi", "--query-gpu=" + self.Q, "--format=csv,noheader,nounits", "-lms", "200"]
            if self.uuid:
                cmd += ["-i", self.uuid]
            self.proc = subprocess.Popen(cmd, stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, smax, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 7:
                continue
            try:
                sm.append(float(f[0]))
                smax = max(smax, float(f[1]))
            except ValueError:
                continue
            for n, v in zip(names, f[3:7]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": smax, "reasons": sorted(reasons),
                "samples": len(sm)}


def max_over_ranks(values, dist, device):
    """Every rank's timings -> the maximum over ranks (the job is as slow as its
    slowest replica); identity without a process group."""
    import torch
    vals = torch.tensor([float(v) for v in values], dtype=torch.float64, device=device)
    if dist is not None:
        dist.all_reduce(vals, op=dist.ReduceOp.MAX)
    return [float(v) for v in vals]


def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    return 6650.0, "fallback"


def traffic_from_profile(name, key="dram_bytes_per_launch_full"):
    """Per-launch (or per-application) DRAM bytes from a committed ncu summary, if present."""
    p = os.path.join(ROOT, "profiles", name)
    if not os.path.exists(p):
        return None
    for line in open(p):
        if line.startswith(key + ":"):
            return float(line.split(":")[1])
    return None


def build_system(nx, ny, nz):
    from frontistr_b200.mesh import box_system
    m = box_system(nx, ny, nz)
    return m


def solver_flags(m, precond, tol, maxit=20000):
    m.set_precond(precond)
    m.set_iter(maxit)
    m.set_resid(tol)
    return m


def _oracle():
    sys.path.insert(0, os.path.join(ROOT, "tests"))
    import oracle_ctypes
    oracle_ctypes.build()
    return oracle_ctypes


def oracle_full_solve(m, precond, tol, maxit=40000, reps=1, colouring=False):
    """The CPU oracle (test infrastructure; the C restatement of hecmw_solve_CG with
    the reference's SSOR / ILU(0) and serial dots, OpenMP over all host cores) solving
    the same system to the same tolerance: preconditioner setup timed on its own, then
    `reps` complete CG solves from X0 = 0, each timed; the last one's solution, its
    iteration count and its true residual ||b - Ax|| / ||b||."""
    oc = _oracle()
    orc = oc.Oracle(m)
    t0 = time.perf_counter()
    pc = orc.precond(precond, 10, 1.0, 1)
    t_setup = time.perf_counter() - t0
    times, out = [], None
    for _ in range(reps):
        t = time.perf_counter()
        out = pc.cg(m.B, maxit=maxit, tol=tol)
        times.append(time.perf_counter() - t)
    res = {"X": out["X"], "iter": int(out["iter"]), "error": int(out["error"]), "solve_s": times,
           "setup_s": t_setup, "cores": int(oc.lib().o33_max_threads()),
           "true_resid": float(orc.rel_resid(out["X"], m.B))}
    if colouring and precond == 1:
        ci, perm, _ = pc.ordering()
        res["colouring"] = (ci, perm)
    return res


def cpu_baseline_from(ref, what, tol):
    """The cpu_baseline object of a measured oracle solve."""
    return {"value": statistics.median(ref["solve_s"]), "unit": "s", "cores": ref["cores"], "kind": "port",
            "iterations": ref["iter"], "true_resid": ref["true_resid"], "setup_s": ref["setup_s"],
            "runs": len(ref["solve_s"]),
            "sample": "measured to tolerance: %d complete %s solve(s) of the C oracle to rel. residual %g "
                      "(median), %d iterations, true residual %.3g; OpenMP over %d host threads, serial dots "
                      "as the reference; preconditioner setup %.2f s reported separately"
                      % (len(ref["solve_s"]), what, tol, ref["iter"], ref["true_resid"], ref["cores"],
                         ref["setup_s"])}


def parity_block(ref, gpu_iters, sols, colouring=None):
    """GPU results against the oracle's solve of the same system: iteration difference,
    ||X - X_oracle|| / ||X_oracle|| per variant, colour schedule identity."""
    import numpy as np
    xo = ref["X"]
    nx = float(np.linalg.norm(xo))
    out = {"oracle_iterations": ref["iter"], "gpu_iterations": gpu_iters,
           "iter_diff": abs(int(gpu_iters) - ref["iter"]),
           "x_rel_err_vs_oracle": {k: float(np.linalg.norm(v[:len(xo)] - xo) / nx) for k, v in sols.items()},
           "oracle_true_resid": ref["true_resid"], "bars": {"iterations": 2, "x_rel": 1e-8}}
    if colouring is not None and "colouring" in ref:
        ci, perm = colouring
        ci_o, perm_o = ref["colouring"]
        out["colour_schedule_equal"] = bool(np.array_equal(ci, ci_o) and np.array_equal(perm, perm_o))
        out["ncolors"] = int(len(ci) - 1)
    first = next(iter(sols))
    out["ok"] = bool(out["iter_diff"] <= 2 and out["x_rel_err_vs_oracle"][first] <= 1e-8 and
                     out.get("colour_schedule_equal", True))
    return out


def run_reference(args, rank, world):
    """The reference arm: the CPU oracle (the reference's CG + SSOR restated in C; the
    Fortran original cannot be built here) on the bench's system, each step one complete
    solve to tolerance.  A solve takes tens of seconds on the host, so at most three
    timed solves run (after `warmup` untimed solves capped at 20 iterations), and the
    value is their median."""
    if rank != 0:
        return
    nx, ny, nz = (int(v) for v in args.mesh.split(","))
    m = solver_flags(build_system(nx, ny, nz), args.precond, args.tol)
    reps = max(1, min(args.steps, 3))
    oc = _oracle()
    orc = oc.Oracle(m)
    warm = orc.precond(args.precond, 10, 1.0, 1)
    for _ in range(args.warmup):
        warm.cg(m.B, maxit=20, tol=args.tol)  # warm-up: threads and pages, not timed
    del warm
    ref = oracle_full_solve(m, args.precond, args.tol, reps=reps)
    value = statistics.median(ref["solve_s"])
    what = {1: "CG+SSOR", 3: "CG+DIAG", 10: "CG+ILU(0)"}.get(args.precond, "CG")
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "s", "n_gpus": world,
        "steps": reps, "steps_requested": args.steps, "warmup": args.warmup, "ms_per_step": value * 1e3,
        "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic", "config": config_dict(nx, ny, nz, m, args),
        "iterations": ref["iter"], "true_resid": ref["true_resid"], "error": ref["error"],
        "cpu_baseline": cpu_baseline_from(ref, what, args.tol),
        "e2e": {"value": value, "unit": "s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


def face_load_cases(m, k, seed):
    """k load cases: random unit-norm tractions on every node of the loaded face."""
    import numpy as np
    rng = np.random.default_rng(seed)
    top = np.unique(np.nonzero(m.B)[0] // 3)
    out = np.zeros((k, 3 * m.N))
    for j in range(k):
        t = rng.standard_normal(3)
        t /= np.linalg.norm(t)
        for c in range(3):
            out[j, 3 * top + c] = t[c]
    return out


def bench_multi(solver, m, nrhs=16, learned=False):
    """16 load cases on the resident matrix: one multi-RHS solve (SpMM + 16-vector
    sweeps) against the same 16 cases solved one after another (device times).
    learned: the same with the learned two-level preconditioner (Iarray(43) = 1, the
    network trained above; FP64), against 16 learned solves one after another."""
    import numpy as np
    B = face_load_cases(m, nrhs, seed=11)
    ia, ra = m.Iarray.copy(), m.Rarray.copy()
    ia[96] = ia[97] = 0
    X = np.zeros_like(B)
    solver.solve_multi(B, X, ia.copy(), ra.copy())  # warm (buffers, graph)
    X = np.zeros_like(B)
    rec = solver.solve_multi(B, X, ia.copy(), ra.copy())
    t_multi = rec["t_solve"]
    kernels = solver.last_solve_info()["kernels"]
    t_seq, it_seq = 0.0, []
    for k in range(nrhs):
        x = np.zeros(3 * m.N)
        r1 = solver.solve_resident(B[k].copy(), x, ia.copy(), ra.copy())
        t_seq += r1["t_solve"]
        it_seq.append(int(r1["iter"]))
    out = {"load_cases": nrhs, "s": t_multi, "rhs_per_s": nrhs / t_multi, "sequential_s": t_seq,
           "sequential_rhs_per_s": nrhs / t_seq, "speedup_vs_sequential": t_seq / t_multi,
           "iterations": [int(v) for v in rec["iter"]], "sequential_iterations": it_seq,
           "max_true_resid": float(np.max(rec["true_resid"])),
           "errors": sorted(set(int(v) for v in rec["errors"])), "gpu_launches": kernels,
           "workload": "%d random unit-norm tractions on the loaded face of the same matrix, CG+SSOR to 1e-8"
                       % nrhs}
    if learned:
        il = ia.copy()
        il[42] = 1
        X = np.zeros_like(B)
        solver.solve_multi(B, X, il.copy(), ra.copy())  # warm
        X = np.zeros_like(B)
        rl = solver.solve_multi(B, X, il.copy(), ra.copy())
        t_l = rl["t_solve"]
        t_lseq, it_lseq = 0.0, []
        for k in range(nrhs):
            x = np.zeros(3 * m.N)
            r1 = solver.solve_resident(B[k].copy(), x, il.copy(), ra.copy())
            t_lseq += r1["t_solve"]
            it_lseq.append(int(r1["iter"]))
        out["learned"] = {"s": t_l, "rhs_per_s": nrhs / t_l, "speedup_vs_cg_ssor_multi": t_multi / t_l,
                          "sequential_learned_s": t_lseq, "speedup_vs_sequential_learned": t_lseq / t_l,
                          "iterations": [int(v) for v in rl["iter"]], "sequential_iterations": it_lseq,
                          "max_true_resid": float(np.max(rl["true_resid"])),
                          "errors": sorted(set(int(v) for v in rl["errors"])),
                          "workload": "the same 16 cases, Iarray(43) = 1: flexible CG with the learned two-level "
                                      "preconditioner (trained network, FP64 smoother), to 1e-8"}
    return out


def bench_config3(tol=1e-10):
    """Mixed precision on the harder system: 80x80x80 HEX8, interior nodes jittered by
    +-0.2h, log-normal E (median 210000, sigma 1.0), nu uniform in [0.25, 0.40]
    (seeded), same supports and load; FP64 CG+SSOR and the three mixed modes to 1e-10
    (mode 1 runs mode 0's one FP64 launch), each with its error against the FP64 solution."""
    import numpy as np
    from frontistr_b200.mesh import box_system
    from frontistr_b200.solver import GpuSolver
    m = box_system(80, 80, 80, jitter=0.2, sigma_E=1.0, nu_range=(0.25, 0.40), seed=3)
    out = {"workload": "80x80x80 HEX8, jitter 0.2h, log-normal E (sigma 1), nu U[0.25, 0.40], seed 3; "
                       "CG+SSOR to %g" % tol, "dof": 3 * m.N, "modes": {}}
    ref = None
    sols = {}
    colouring = None
    with GpuSolver() as s:
        for name, mode in (("fp64", 0), ("bf16_precond", 1), ("fp32_restart", 2), ("fp32_reliable", 3)):
            recs = []
            for _ in range(2):  # warm + timed
                g = m.copy()
                g.set_iter(40000)
                g.set_resid(tol)
                g.Iarray[41] = mode
                rec = s.solve(g)
                recs.append(rec)
            info = s.last_solve_info()
            if mode == 0:
                ref = g.X.copy()
                colouring = s.colouring()
            sols[name] = g.X.copy()
            out["modes"][name] = {"s": recs[-1]["t_solve"], "iterations": int(recs[-1]["iter"]),
                                  "outer": info["outer"], "error": int(recs[-1]["error"]),
                                  "true_resid": info["true_resid"],
                                  "rel_err_vs_fp64": float(np.linalg.norm(g.X - ref) / np.linalg.norm(ref))}
    # for the oracle comparison made after the GPU work (bench main)
    m.set_iter(40000)
    m.set_resid(tol)
    out.update(_sols=sols, _system=m, _colouring=colouring)
    return out


def bench_domains(m, solver, ndom=2):
    """The cube as `ndom` domains of a decomposed mesh (slabs of node ids,
    domain.partition): each a GpuSolver handle driven by its own thread on this GPU,
    exchanging halos and sums through the host (LocalExchange), FP64 CG + SSOR of every
    domain's internal block to 1e-8.  Wall time of the concurrent solves; iterations
    against the one-domain solve's (the local SSOR changes them, as in the reference);
    the true residual of the gathered solution on the whole matrix."""
    import threading
    import numpy as np
    from frontistr_b200.domain import LocalExchange, gather_solution, partition
    from frontistr_b200.matrix import default_iarray_rarray
    from frontistr_b200.solver import GpuSolver
    t0 = time.perf_counter()
    doms = partition(m, ndom)
    t_part = time.perf_counter() - t0
    ex = LocalExchange(doms, timeout=600.0)
    mats, solvers = [], []
    for k, d in enumerate(doms):
        lm = d.matrix.copy()
        lm.Iarray, lm.Rarray = default_iarray_rarray()
        lm.set_iter(20000)
        lm.set_resid(1e-8)
        s = GpuSolver()
        s.set_matrix(lm)
        s.set_domain(d.comm, ex.endpoint(k))
        mats.append(lm)
        solvers.append(s)
    out, errs = [None] * ndom, []

    def run(k):
        try:
            out[k] = solvers[k].solve_resident(mats[k].B, mats[k].X, mats[k].Iarray, mats[k].Rarray)
        except BaseException as e:  # noqa: BLE001 -- re-raised below
            errs.append(e)
            ex.barrier.abort()

    threads = [threading.Thread(target=run, args=(k,)) for k in range(ndom)]
    t0 = time.perf_counter()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    wall = time.perf_counter() - t0
    for s in solvers:
        s.close()
    if errs:
        raise errs[0]
    X = gather_solution(doms, [lm.X for lm in mats], m.N)
    r = m.B[:3 * m.N] - solver.matvec(X)[:3 * m.N]
    return {"workload": "the same cube as %d slab domains (N internal of NP nodes each), one GPU handle and "
                        "host thread per domain on this GPU, halo exchange and sums through the host" % ndom,
            "domains": ndom, "nodes": [[d.N, d.NP] for d in doms], "partition_s": t_part, "wall_s": wall,
            "errors": [o["error"] for o in out], "iterations": [o["iter"] for o in out],
            "device_solve_s": [o["t_solve"] for o in out],
            "true_resid": float(np.linalg.norm(r) / np.linalg.norm(m.B[:3 * m.N]))}


def bench_assembly(n=64, seed=3):
    """HEX8 linear-elastic assembly of an n^3 box (interior nodes jittered by +-0.2h,
    log-normal E, nu in [0.25, 0.40], clamped base, loaded top) on the device
    (hecmw33_gpu_assemble_hex8: profile and per-block lists on the host once, element
    blocks and element-order sums on the device, constraints) against the host
    restatement it is bitwise equal to (fistr_mesh_assemble + fistr_mat_ass_bc, one
    thread).  Times: the first call (symbolic + numeric), a re-assembly of new values
    on the same mesh (a Newton iteration), and the host call."""
    import numpy as np
    from frontistr_b200.mesh import mesh_system
    from frontistr_b200.solver import GpuSolver
    rng = np.random.default_rng(seed)
    n1 = n + 1
    g = np.arange(n1, dtype=np.float64)
    X = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).transpose(2, 1, 0, 3).reshape(-1, 3).copy()
    inner = np.all((X > 0) & (X < n), axis=1)
    X[inner] += rng.uniform(-0.2, 0.2, size=(int(inner.sum()), 3))
    e = np.arange(n)
    ex, ey, ez = (a.reshape(-1) for a in np.meshgrid(e, e, e, indexing="ij"))
    order = np.lexsort((ex, ey, ez))
    ex, ey, ez = ex[order], ey[order], ez[order]
    nid = lambda x, y, z: x + n1 * (y + n1 * z)
    el = np.stack([nid(ex, ey, ez), nid(ex + 1, ey, ez), nid(ex + 1, ey + 1, ez), nid(ex, ey + 1, ez),
                   nid(ex, ey, ez + 1), nid(ex + 1, ey, ez + 1), nid(ex + 1, ey + 1, ez + 1),
                   nid(ex, ey + 1, ez + 1)], 1).astype(np.int32)
    E = 2.1e5 * np.exp(rng.standard_normal(len(el)))
    nu = rng.uniform(0.25, 0.40, len(el))
    F = np.zeros(3 * len(X))
    top = np.nonzero(X[:, 2] == n)[0]
    F[3 * top + 1] = -1.0
    base = np.nonzero(X[:, 2] == 0)[0]
    fixed = [(int(b), d, 0.0) for b in base for d in (1, 2, 3)]
    with GpuSolver() as s:
        t0 = time.perf_counter()
        s.assemble_hex8(X, el, E, nu, F=F, fixed=fixed)
        t1 = time.perf_counter()
        s.assemble_hex8(X, el, 1.1 * E, nu, F=F, fixed=fixed, symbolic=False)
        t2 = time.perf_counter()
        g2 = s.get_matrix()
    t3 = time.perf_counter()
    cload = [(int(i) // 3, int(i) % 3 + 1, float(F[i])) for i in np.nonzero(F)[0]]
    ref = mesh_system(X, el, 361, 1.1 * E, nu, fixed=fixed, cload=cload)
    t4 = time.perf_counter()
    same = bool(np.array_equal(g2.D, ref.D) and np.array_equal(g2.AL[:9 * ref.NPL], ref.AL[:9 * ref.NPL])
                and np.array_equal(g2.AU[:9 * ref.NPU], ref.AU[:9 * ref.NPU]) and np.array_equal(g2.B, ref.B))
    out = {"workload": "%d^3 HEX8 box, jitter 0.2h, log-normal E, nu U[0.25, 0.40], clamped base" % n,
           "elements": int(len(el)), "nodes": int(len(X)), "gpu_first_call_s": t1 - t0,
           "gpu_reassembly_s": t2 - t1, "host_s": t4 - t3, "host_kind": "fistr_mesh_assemble, 1 thread",
           "bitwise_equal_to_host": same, "speedup_reassembly_vs_host": (t4 - t3) / (t2 - t1)}
    # Neo-Hookean tangent + residual of the Newton workload's block (64^3, h = 1) at a
    # displacement field, against the host's OpenMP assembly (fistr_box_neohooke)
    from frontistr_b200.newton import NeoHookeBox
    box = NeoHookeBox(n, n, n, h=1.0, C10=1.0, D1=0.01)
    Xg = X.copy()
    Xg[:] = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).transpose(2, 1, 0, 3).reshape(-1, 3)
    U = np.zeros(3 * box.N)
    U[2::3] = -0.02 * Xg[:, 2]
    with GpuSolver() as s:
        s.assemble_hex8_neohooke(Xg, el, 1.0, 0.01, U)
        t5 = time.perf_counter()
        s.assemble_hex8_neohooke(Xg, el, 1.0, 0.01, U, symbolic=False)
        t6 = time.perf_counter()
    t7 = time.perf_counter()
    box.tangent(U)
    t8 = time.perf_counter()
    out["neohooke"] = {"gpu_reassembly_s": t6 - t5, "host_s": t8 - t7,
                       "host_kind": "fistr_box_neohooke, OpenMP over %d threads" % (os.cpu_count() or 1),
                       "speedup_vs_host": (t8 - t7) / (t6 - t5)}
    return out


def bench_learned_newton(args):
    """The learned preconditioner where the network is meant to live: a Newton
    sequence.  64x64x64 compressible Neo-Hookean block (C10 = 1.0, D1 = 0.01, h = 1),
    clamped at z = 0, top face held in x, y and moved down by 10 % of the height over
    12 equal increments.  Increments 1-4 are solved with plain FP64 CG + SSOR while
    (r, e) pairs are recorded; the network is trained on them on the GPU; every
    tangent system of increments 5-12 is solved both ways (plain, and flexible CG
    with the network), and the learned solution advances the sequence."""
    import numpy as np
    from frontistr_b200.newton import NeoHookeBox, newton_sequence
    from frontistr_b200.solver import GpuSolver
    nx, ny, nz = (int(v) for v in args.newton_mesh.split(","))
    box = NeoHookeBox(nx, ny, nz, h=1.0, C10=1.0, D1=0.01)
    top_uz = -0.1 * nz
    rows = []
    train = {}
    t_asm = [0.0]
    s = GpuSolver()
    s.learn_record(1, max_pairs=32)

    first = [True]

    def solve(inc, it, m):
        m.set_iter(40000)
        m.set_resid(args.tol)
        if not first[0]:
            m.Iarray[97] = 0  # same structure: keep the orderings and layouts
            m.Iarray[96] = 2  # new tangent values: rebuild the preconditioner numerically
        first[0] = False
        if inc == 5 and it == 1 and not train:
            n = s.learn_record(0)
            t0 = time.perf_counter()
            l0, l1 = s.learn_train(steps=args.train_steps, lr=args.train_lr)
            train.update(pairs=n, steps=args.train_steps, loss_before=l0, loss_after=l1,
                         train_s=time.perf_counter() - t0)
        rec = {"increment": inc, "newton": it}
        if inc >= 5:
            g = m.copy()
            r = s.solve(g)
            rec["plain"] = {"iter": int(r["iter"]), "s": float(r["t_solve"]), "error": int(r["error"]),
                            "true_resid": s.last_solve_info()["true_resid"]}
            g = m.copy()
            g.Iarray[42] = 1
            r = s.solve(g)
            info = s.last_solve_info()
            rec["learned"] = {"iter": int(r["iter"]), "s": float(r["t_solve"]), "error": int(r["error"]),
                              "true_resid": info["true_resid"], "fallback_iter": info["fallback"]}
        else:
            g = m.copy()
            r = s.solve(g)
            rec["plain"] = {"iter": int(r["iter"]), "s": float(r["t_solve"]), "error": int(r["error"]),
                            "true_resid": s.last_solve_info()["true_resid"]}
        rows.append(rec)
        return g.X.copy()

    t0 = time.perf_counter()
    steps = list(newton_sequence(box, solve, top_uz=top_uz, n_incr=12, max_newton=6, tol=1e-6))
    wall = time.perf_counter() - t0
    s.close()
    late = [r for r in rows if "learned" in r]
    sum_plain = sum(r["plain"]["s"] for r in late)
    sum_learned = sum(r["learned"]["s"] for r in late)
    return {"impl": "ours", "workload": "%dx%dx%d Neo-Hookean HEX8 (C10 1.0, D1 0.01), top z displaced by %g "
                                        "in 12 increments; CG+SSOR to %g" % (nx, ny, nz, top_uz, args.tol),
            "dof": 3 * box.N, "newton_systems": len(rows), "training": train,
            "increments_5_12": {"systems": len(late), "plain_s": sum_plain, "learned_s": sum_learned,
                                "plain_iterations": sum(r["plain"]["iter"] for r in late),
                                "learned_iterations": sum(r["learned"]["iter"] for r in late),
                                "speedup": sum_plain / sum_learned if sum_learned else None,
                                "max_true_resid_learned": max(r["learned"]["true_resid"] for r in late)},
            "newton": [{"increment": x["increment"], "newton": x["newton"], "residual": x["residual"]}
                       for x in steps], "systems": rows, "wall_s": wall}


def iteration_bytes(n, nz, fused=False):
    """Algorithmic bytes of one FP64 CG+SSOR iteration on a one-domain system of n block
    rows and nz blocks: the reference's SpMV model (hecmw_solver_Iterative.f90:211-217),
    one SSOR application (off-diagonal blocks with their columns, the diagonal LU read
    by both sweeps, row pointers, vectors) and the minimum fused vector traffic.
    fused: the iteration without a product (h33_persist.cuh): each off-diagonal block and
    column once, the diagonal LU twice, the vector passes of its two sweeps and its update."""
    off = nz - n
    if fused:
        return 76 * off + 2 * 72 * n + (4 + 11 + 9) * 24 * n
    spmv = 72 * nz + 4 * off + 8 * (n + 1) + 24 * n + 24 * n
    ssor = 76 * off + 2 * 72 * n + 2 * 8 * (n + 1) + 4 * 24 * n
    vec = 10 * 24 * n
    return spmv + ssor + vec


def bench_batched(args):
    """Independent boxes (edges uniform in [8, 40] elements, E log-uniform in
    [1e3, 1e6], nu in [0.2, 0.45], random traction on the top face; seeded) solved
    in one persistent launch with the autotuned schedule, against the same systems
    solved one after another on one handle (device times, set-up excluded)."""
    import numpy as np
    from frontistr_b200.batch import BatchSolver, stack_systems
    from frontistr_b200.mesh import random_box_batch
    from frontistr_b200.solver import GpuSolver
    lo, hi = (int(v) for v in args.batch_edges.split(","))
    t0 = time.perf_counter()
    systems = random_box_batch(args.batch_systems, edge_range=(lo, hi), seed=2024)
    big, sys_ptr = stack_systems(systems)
    t_asm = time.perf_counter() - t0
    ia, ra = big.Iarray.copy(), big.Rarray.copy()
    ia[0] = 20000
    ra[0] = args.tol
    out = {"systems": len(systems), "nodes": int(big.N), "dof": 3 * int(big.N), "blocks": int(big.NZ),
           "dof_range": [3 * min(m.N for m in systems), 3 * max(m.N for m in systems)], "assemble_s": t_asm}
    with BatchSolver() as bs:
        t = time.perf_counter()
        bs.set_matrix(big, sys_ptr, ia, ra)
        out["setup_s"] = time.perf_counter() - t
        t = time.perf_counter()
        bs.autotune(big.B, np.zeros(3 * big.N), ia.copy(), ra.copy())
        out["autotune_s"] = time.perf_counter() - t
        X = np.zeros(3 * big.N)
        bs.solve(big.B, X, ia.copy(), ra.copy())  # warm
        times = []
        for _ in range(2):
            X = np.zeros(3 * big.N)
            rec = bs.solve(big.B, X, ia.copy(), ra.copy())
            times.append(rec["t_solve"])
        info = bs.info()
    t_b = min(times)
    out.update({"s": t_b, "systems_per_s": len(systems) / t_b,
                "schedule": {k: info[k] for k in ("lanes", "cluster", "big", "small", "grid", "big_frac")},
                "total_iterations": int(np.sum(rec["iter"])), "max_iterations": int(np.max(rec["iter"])),
                "max_true_resid": float(np.max(rec["true_resid"])),
                "errors": sorted(set(int(v) for v in rec["errors"])), "gpu_launches": info["kernels_per_solve"]})
    t_seq = 0.0
    with GpuSolver() as s:
        for m in systems:
            g = m.copy()
            g.set_iter(20000)
            g.set_resid(args.tol)
            s.solve(g)  # set-up (not timed)
            g.X[:] = 0.0
            g.Iarray[96] = g.Iarray[97] = 0
            r1 = s.solve_resident(g.B, g.X, g.Iarray, g.Rarray)
            t_seq += r1["t_solve"]
    # algorithmic bytes of the batch: every system's CG+SSOR iterations times the
    # per-iteration bytes of the kernel that ran (fused with four lanes per row or more)
    its = np.asarray(rec["iter"], dtype=np.float64)
    nbytes = float(sum(it * iteration_bytes(mk.N, mk.NZ, info["lanes"] >= 4) for it, mk in zip(its, systems)))
    peak, peak_kind = measured_peaks()
    out["roofline"] = {"bound": "hbm", "kernel": "batch_cg_kernel (the whole batched solve, one launch)",
                       "algorithmic_bytes": nbytes, "achieved": nbytes / t_b / 1e9, "peak": peak,
                       "frac": nbytes / t_b / 1e9 / peak, "unit": "GB/s", "peak_kind": peak_kind}
    out.update({"sequential_s": t_seq, "sequential_systems_per_s": len(systems) / t_seq,
                "speedup_vs_sequential": t_seq / t_b,
                "workload": "%d HEX8 boxes, edges uniform in [%d, %d] elements, E log-uniform [1e3, 1e6], "
                            "nu [0.2, 0.45], random unit traction on z = nz; CG+SSOR to %g" %
                            (len(systems), lo, hi, args.tol)})
    return out


def roofline_sweeps(sweeps, head, peak, peak_kind, tag):
    """The roofline object for one SSOR application (forward + backward colour
    sweeps), in the storage of the headline variant; the learned variants apply the
    two-grid cycle's smoother (the same SSOR on its own layouts, first-fit colours)."""
    store = "bf16" if head.endswith("mixed") else "fp64"
    smoother = head.startswith("learned") and ("smoother_" + store) in sweeps
    key = ("smoother_" if smoother else "") + store
    if key not in sweeps:
        key = "fp64"
        store = "fp64"
    sw = sweeps[key]
    what = "BF16-stored values, FP32 diagonal LU" if store == "bf16" else "FP64"
    if smoother:
        kernel = ("sweep_fwd_uni_kernel + sweep_bwd_uni_kernel: one application of the learned preconditioner's "
                  "SSOR smoother (first-fit colour order), all colours, %s" % what)
        prof = "ssor_smoother_sweeps_%s.txt" % tag
    else:
        kernel = "sweep_fwd_uni_kernel + sweep_bwd_uni_kernel: one SSOR application, all colours, %s" % what
        prof = "ssor_sweeps_%s.txt" % tag
    return {"bound": "hbm", "kernel": kernel,
            "achieved": sw["achieved"], "peak": peak, "unit": "GB/s", "frac": sw["frac"], "peak_kind": peak_kind,
            "traffic": traffic_from_profile(prof, "dram_bytes_per_apply_%s" % store),
            "algorithmic_bytes": sw["algorithmic_bytes"], "ms_per_apply": sw["ms_per_apply"]}


def bench_ilu0(m, args, peak):
    """CG + block ILU(0) (PRECOND = 10: natural order, hecmw_precond_BILU_33.f90:90-362)
    on the same system, on its own handle: FP64 and BF16-stored factors, device time of
    the solve, one preconditioner application timed live, the level count."""
    import numpy as np
    from frontistr_b200.solver import GpuSolver
    out = {"workload": "same system, CG + block ILU(0) (PRECOND=10, natural order, level-scheduled sweeps) "
                       "to %g" % args.tol}
    sols = {}
    with GpuSolver() as s:
        g = m.copy()
        g.set_precond(10)
        rec = s.solve(g)
        if rec["error"] != 0:
            return {"failed": rec}
        out["setup_s_first_call"] = rec["t_setup"]
        ia, ra = g.Iarray.copy(), g.Rarray.copy()
        for name, mode in (("fp64", 0), ("bf16_factors", 1)):
            recs = []
            for _ in range(3):  # warm + 2 timed
                X = np.zeros(3 * m.N)
                iam = ia.copy()
                iam[41] = mode
                recs.append(s.solve_resident(m.B, X, iam, ra.copy()))
            info = s.last_solve_info()
            sols[name] = X
            out[name] = {"s": statistics.mean(r["t_solve"] for r in recs[1:]), "iterations": int(recs[-1]["iter"]),
                         "error": int(recs[-1]["error"]), "true_resid": info["true_resid"],
                         "levels_fwd_plus_bwd": info["sweep_groups"], "kernels": info["kernels"]}
        for key, lp in (("fp64", 0), ("bf16_factors", 1)):
            ms, nbytes = s.time_precond(5, lp)
            out[key]["precond_apply"] = {"ms_per_apply": ms, "algorithmic_bytes": nbytes,
                                         "achieved": nbytes / (ms * 1e-3) / 1e9,
                                         "frac": nbytes / (ms * 1e-3) / 1e9 / peak}
    out["_sols"] = sols
    return out


def config_dict(nx, ny, nz, m, args):
    return {"workload": "HEX8 cantilever %dx%dx%d elements (%d nodes, %d DOF, %d blocks), CG+%s to %g"
                        % (nx, ny, nz, m.N, 3 * m.N, m.NZ, {1: "SSOR", 3: "DIAG", 10: "ILU(0)"}.get(args.precond),
                           args.tol),
            "nodes": m.N, "dof": 3 * m.N, "blocks": m.NZ, "precond": args.precond, "tol": args.tol,
            "solver": "plain FP64 CG (drop-in)", "l2": "inputs larger than L2 (matrix ~2 GB)",
            "parallelism": "replicas"}


def main():
    args = parse()
    pin_local_gpu()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    if args.impl == "reference":
        return run_reference(args, rank, world)
    if args.learned_newton:
        if rank == 0:
            print(json.dumps(bench_learned_newton(args)))
        return

    import numpy as np
    import torch
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(0)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
    from frontistr_b200.solver import GpuSolver

    nx, ny, nz = (int(v) for v in args.mesh.split(","))
    m = solver_flags(build_system(nx, ny, nz), args.precond, args.tol)
    solver = GpuSolver()
    if args.spmv_only:
        solver.set_matrix(m)
        solver.time_spmv(args.spmv_only)
        torch.cuda.synchronize()
        return
    if args.profile_multi:
        import numpy as np
        solver.set_matrix(m)
        B = face_load_cases(m, 16, seed=11)
        ia, ra = m.Iarray.copy(), m.Rarray.copy()
        ia[0] = 3
        if args.profile_coarse >= 1:
            ia[42] = 1
            ia[43] = args.profile_coarse
        solver.solve_multi(B, np.zeros_like(B), ia, ra)
        return
    if args.profile_batch:
        import numpy as np
        from frontistr_b200.batch import BatchSolver, stack_systems
        from frontistr_b200.mesh import random_box_batch
        lo, hi = (int(v) for v in args.batch_edges.split(","))
        big, sys_ptr = stack_systems(random_box_batch(args.batch_systems, edge_range=(lo, hi), seed=2024))
        ia, ra = big.Iarray.copy(), big.Rarray.copy()
        ia[0] = 20000
        with BatchSolver() as bs:
            bs.set_matrix(big, sys_ptr, ia, ra)
            bs.solve(big.B, np.zeros(3 * big.N), ia, ra)
        return
    if args.profile_e2e:
        solver.learn_record(1, max_pairs=4)
        rec = solver.solve(m.copy())
        solver.learn_record(0)
        solver.learn_train(steps=2, lr=5e-3)
        for i in range(3):
            mm = m.copy()
            mm.Iarray[97] = 0
            mm.Iarray[96] = 2  # numeric rebuild, as at a new Newton increment
            mm.Iarray[41] = 1
            mm.Iarray[42] = 1
            torch.cuda.synchronize()
            if i == 2:
                torch.cuda.profiler.start()
            rec = solver.solve(mm)
            torch.cuda.synchronize()
            if i == 2:
                torch.cuda.profiler.stop()
            if rec["error"] != 0:
                raise SystemExit("solve failed: %r" % rec)
        return
    if args.profile_solve:
        mm = m.copy()
        mm.set_iter(5)
        mm.Iarray[41] = args.profile_mode
        if args.profile_coarse >= 1:
            mm.Iarray[42] = 1
            mm.Iarray[43] = args.profile_coarse
        rec = solver.solve(mm)
        if rec["error"] not in (0, 3001):
            raise SystemExit("solve failed: %r" % rec)
        return

    # first drop-in call: symbolic setup, preconditioner, graph
    first = m.copy()
    info0 = solver.solve(first)
    if info0["error"] != 0:
        raise SystemExit("solve failed: %r" % info0)
    ia, ra = first.Iarray.copy(), first.Rarray.copy()  # flags 97/98 now 0: reuse
    dev = torch.device("cuda", 0)
    dB = torch.from_numpy(m.B).to(dev)
    dX = torch.zeros_like(dB)
    uuid = None
    try:
        uuid = "GPU-" + str(torch.cuda.get_device_properties(0).uuid)
    except Exception:
        pass

    def barrier():
        torch.cuda.synchronize()
        if dist is not None:
            dist.barrier()

    train = None
    if not args.no_learned:
        # training data: FP64 SSOR-CG solves of other load cases (random unit top-face
        # tractions), as earlier load increments would provide them; not timed
        rng = np.random.default_rng(7)
        top = np.unique(np.nonzero(m.B)[0] // 3)
        t0 = time.perf_counter()
        solver.learn_record(1, max_pairs=16)
        for _ in range(4):
            t = rng.standard_normal(3)
            t /= np.linalg.norm(t)
            mm = m.copy()
            mm.B = np.zeros_like(m.B)
            for node in top:
                mm.B[3 * node:3 * node + 3] = t
            mm.Iarray[97] = 0
            mm.Iarray[96] = 0
            # on the resident matrix: values uploaded again without a rebuild would keep
            # the plain solves below off the one-launch CG
            rec = solver.solve_resident(mm.B, mm.X, mm.Iarray, mm.Rarray)
            assert rec["error"] == 0
        npairs = solver.learn_record(0)
        t1 = time.perf_counter()
        loss0, loss1 = solver.learn_train(steps=args.train_steps, lr=args.train_lr)
        torch.cuda.synchronize()
        t2 = time.perf_counter()
        train = {"pairs": npairs, "record_s": t1 - t0, "train_s": t2 - t1, "steps": args.train_steps,
                 "loss_before": loss0, "loss_after": loss1}

    class VariantFailed(Exception):
        pass

    def step(mode, learned=0, coarse=0):
        dX.zero_()
        torch.cuda.synchronize()
        iam = ia.copy()
        iam[41] = mode
        iam[42] = learned
        iam[43] = coarse
        rec = solver.solve_resident_device(dB.data_ptr(), dX.data_ptr(), iam, ra.copy())
        if rec["error"] != 0:
            if mode == 0 and learned == 0:
                raise SystemExit("solve failed: %r" % rec)
            raise VariantFailed(rec)
        return rec

    variants = {}
    modes = [("fp64", 0, 0, 0)] + ([] if args.no_mixed else [("mixed", 1, 0, 0)])
    if train is not None:
        modes += [("learned_fp64", 0, 1, 0), ("learned_mixed", 1, 1, 0)]
    if not args.no_learned and not args.no_mixed:
        # ablations of the learned two-level preconditioner (not headline candidates):
        # the same coarse space without the network's smoothing weights, and with the
        # untrained network's weights (1/2 everywhere)
        modes += [("twolevel_unsmoothed_mixed", 1, 1, 1), ("twolevel_uniform_mixed", 1, 1, 2)]
    clocks = Clocks(uuid)
    sols = {}
    failed = {}
    clocks.start()  # sampled over every variant's solves, the headline's among them
    for name, mode, learned, coarse in modes:
        # every rank runs the same steps; a variant that fails (non-FP64 only) is
        # reported and left out of the headline
        try:
            for _ in range(args.warmup):
                step(mode, learned, coarse)
            barrier()
            t0 = time.perf_counter()
            recs = [step(mode, learned, coarse) for _ in range(args.steps)]
        except VariantFailed as exc:
            barrier()
            r = exc.args[0]
            failed[name] = {"error": int(r["error"]), "iter": int(r["iter"]), "resid": float(r["resid"])}
            continue
        barrier()
        wall = (time.perf_counter() - t0) / args.steps
        info = solver.last_solve_info()
        sols[name] = dX.cpu().numpy().copy()
        variants[name] = {"s": statistics.mean(r["t_solve"] for r in recs), "wall_s": wall,
                          "iterations": recs[-1]["iter"], "outer": info["outer"],
                          "true_resid": info["true_resid"], "kernels": info["kernels"],
                          "fallback_iter": info["fallback"]}
    clk = clocks.stop()
    for name in sols:
        variants[name]["rel_err_vs_fp64"] = float(np.linalg.norm(sols[name] - sols["fp64"]) /
                                                  np.linalg.norm(sols["fp64"]))
    # headline: the fastest variant whose FP64 true residual meets the tolerance
    ok = [k for k, v in variants.items() if v["true_resid"] <= args.tol and not k.startswith("twolevel_")]
    head = min(ok, key=lambda k: variants[k]["s"]) if ok else "fp64"
    variants.update({k: {"failed": v} for k, v in failed.items()})
    dev_s = variants[head]["s"]
    wall = variants[head]["wall_s"]
    iters = variants["fp64"]["iterations"]
    step(0)  # leave the FP64 solve as the last one for the bookkeeping below
    info = solver.last_solve_info()
    iter_s = variants["fp64"]["s"] / max(iters, 1)

    # SpMV roofline, live: device events over back-to-back launches on the solver's stream
    spmv_ms = solver.time_spmv(20)
    peak, peak_kind = measured_peaks()
    achieved = info["spmv_bytes"] / (spmv_ms * 1e-3) / 1e9
    gpu_colouring = solver.colouring() if args.precond == 1 else None

    # the dominant kernels of an iteration: one preconditioner application (SSOR: the
    # forward + backward colour sweeps), FP64 and BF16-stored, timed live the same way
    sweeps = {}
    for key, lp, sm in (("fp64", 0, False), ("bf16", 1, False), ("smoother_fp64", 0, True),
                        ("smoother_bf16", 1, True)):
        if (lp and args.no_mixed) or (sm and train is None):
            continue
        ms, nbytes = solver.time_precond(20, lp, smoother=sm)
        sweeps[key] = {"ms_per_apply": ms, "algorithmic_bytes": nbytes, "achieved": nbytes / (ms * 1e-3) / 1e9,
                       "frac": nbytes / (ms * 1e-3) / 1e9 / peak}

    # end-to-end through the drop-in call with host buffers: the caller's matrix
    # values, B and X sit in pinned host memory (page-locked, as a GPU-aware caller
    # allocates them); the call copies them in, rebuilds the numeric preconditioner,
    # solves and copies X back
    e2e = None
    if not args.no_e2e:
        def pinned(a):
            t_ = torch.empty(a.size, dtype=torch.float64, pin_memory=True)
            out = t_.numpy()
            out[:] = a
            return out
        pin = {k: pinned(getattr(m, k)) for k in ("D", "AL", "AU", "B", "X")}
        e2e_t = []
        for i in range(max(1, min(args.steps, 3)) + 1):
            mm = m.copy()
            for k, v in pin.items():
                v[:] = getattr(m, k)
                setattr(mm, k, v)
            mm.Iarray[97] = 0  # structure unchanged (flag 98)
            mm.Iarray[96] = 2  # numerical preconditioner rebuild forced (flag 97), as a new Newton increment
            mm.Iarray[41] = 1 if head.endswith("mixed") else 0
            mm.Iarray[42] = 1 if head.startswith("learned") else 0
            torch.cuda.synchronize()
            t = time.perf_counter()
            rec = solver.solve(mm)
            e2e_t.append(time.perf_counter() - t)
            assert rec["error"] == 0
        e2e_t = e2e_t[1:]
        h2d = 8 * 9 * m.NZ + 2 * 8 * 3 * m.N
        d2h = 8 * 3 * m.N
        e2e = {"value": statistics.mean(e2e_t), "unit": "s", "h2d_bytes_per_step": h2d,
               "d2h_bytes_per_step": d2h, "solver": head, "host_buffers": "pinned"}

    dev_s, wall, e2e_v = max_over_ranks([dev_s, wall, e2e["value"] if e2e else 0.0], dist, dev)
    if e2e:
        e2e["value"] = e2e_v

    if world > 1:
        # the 16-load-case, batched and config-3 figures are single-GPU measurements
        # reported at N = 1; replicas only repeat the headline
        args.no_multi = args.no_batched = args.no_config3 = args.no_assembly = args.no_domains = True
    multi = None if args.no_multi else bench_multi(solver, m, learned=train is not None)
    config3 = None if args.no_config3 else bench_config3()
    assembly = None if args.no_assembly else bench_assembly()
    batched = None if args.no_batched else bench_batched(args)
    domains = None if args.no_domains else bench_domains(m, solver)
    newton = None
    if not (args.no_newton or args.no_learned or world > 1):
        # the learned preconditioner in the Newton sequence of the 64^3 Neo-Hookean block
        newton = bench_learned_newton(args)
        newton.pop("systems", None)
        newton.pop("impl", None)

    ilu0 = None if (args.no_ilu0 or world > 1) else bench_ilu0(m, args, peak)

    cpu = parity = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        ref = oracle_full_solve(m, args.precond, args.tol, colouring=True)
        what = {1: "CG+SSOR", 3: "CG+DIAG", 10: "CG+ILU(0)"}.get(args.precond, "CG")
        cpu = cpu_baseline_from(ref, what, args.tol)
        parity = parity_block(ref, variants["fp64"]["iterations"], sols, gpu_colouring)
        if ilu0 is not None:
            ref0 = oracle_full_solve(m, 10, args.tol)
            ilu0["cpu_baseline"] = cpu_baseline_from(ref0, "CG+ILU(0)", args.tol)
            ilu0["parity"] = parity_block(ref0, ilu0["fp64"]["iterations"], ilu0.pop("_sols"))
        if config3 is not None:
            sols3 = config3.pop("_sols")
            m3 = config3.pop("_system")
            ref3 = oracle_full_solve(m3, 1, 1e-10, colouring=True)
            config3["cpu_baseline"] = cpu_baseline_from(ref3, "CG+SSOR", 1e-10)
            config3["parity"] = parity_block(ref3, config3["modes"]["fp64"]["iterations"], sols3,
                                             config3.pop("_colouring"))
    for d in (ilu0, config3):
        if d is not None:
            for k in ("_sols", "_system", "_colouring"):
                d.pop(k, None)

    if rank == 0:
        tag = "%dcube" % nx if nx == ny == nz else "%dx%dx%d" % (nx, ny, nz)
        cfg = config_dict(nx, ny, nz, m, args)
        cfg["solver"] = {"fp64": "plain FP64 CG + SSOR (drop-in)",
                         "mixed": "FP64 CG + SSOR called with Iarray(42)=1: the one FP64 launch, as without",
                         "learned_fp64": "flexible CG, learned two-level preconditioner (SSOR two-grid cycle with "
                                         "the coarse space the network shapes), FP64 (Iarray(43)=1)",
                         "learned_mixed": "flexible CG, learned two-level preconditioner with BF16-stored SSOR and "
                                          "FP32 inner residuals, FP64 iterations (Iarray(42)=1, Iarray(43)=1)"}[head]
        line = {
            "metric": METRIC, "value": dev_s, "unit": "s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": dev_s * 1e3, "higher_is_better": False,
            "scaling": "weak", "vs_baseline": None,
            "dtype": "f64+bf16" if head.startswith(("learned_mixed", "twolevel")) else "f64",
            "data": "synthetic", "config": cfg,
            "variants": variants,
            "training": train,
            "speedup_vs_fp64": variants["fp64"]["s"] / dev_s,
            "iterations": variants[head]["iterations"], "wall_s_per_step": wall,
            "fp64_ms_per_iteration": iter_s * 1e3,
            "fp64_iteration_GBps": info["iter_bytes"] / iter_s / 1e9,
            "setup_s_first_call": info0["t_setup"],
            "roofline": roofline_sweeps(sweeps, head, peak, peak_kind, tag),
            "roofline_spmv": {"bound": "hbm", "kernel": "spmv_kernel (plain FP64 SpMV, y = A x)",
                              "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                              "peak_kind": peak_kind,
                              "traffic": traffic_from_profile("spmv_kernel_%s.txt" % tag),
                              "algorithmic_bytes": info["spmv_bytes"], "ms_per_launch": spmv_ms},
            "precond_apply": sweeps,
            "cpu_baseline": cpu,
            "parity": parity,
            "ilu0": ilu0,
            "e2e": e2e,
            "gpu_launches": variants[head]["kernels"] * args.steps,
            "clocks": clk,
            "multi_rhs": multi,
            "mixed_config3": config3,
            "assembly": assembly,
            "batched": batched,
            "domains": domains,
            "learned_newton": newton,
        }
        print(json.dumps(line))
    solver.close()
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
