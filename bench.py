"""Benchmark: harmonic BEM assemble+solve throughput (solves/s) on the
time-harmonic elastodynamic quad8 cube, 8x8 elements per face (384 elements,
1154 nodes, 3462 complex DOF), E=1, nu=0.25, rho=1, xi=0.05, 20 frequencies
a0 = 0.1..2.0, bottom face clamped, uniform harmonic t_z=-1 on the top face.

One step = one full frequency sweep on the device = 20 solves, mixed precision:
double-float assembly of the 20 systems (binary64 results), complex64 LU with
binary16-split tensor-core trailing updates, FP64 iterative refinement to a 1e-12
backward error (solutions within 1e-8 of the FP64 oracle's). value: device time
(CUDA events inside the library) with the mesh resident in HBM; inputs (20 x
192 MB systems) exceed L2. e2e: the same sweep through the public C-ABI from
host buffers: mesh upload (H2D) + sweep + solution download (D2H) every step.

Beside the headline: the plain FP64 GPU path on the same sweep
(plain_fp64_gpu), the 14883-DOF surface patch with mixed vs plain FP64
(precision_form), the learned quadrature on the thin slab (learned_quadrature),
48 uneven problems in one batched call (batching_form), the static cube
(870 DOF), the thin slab (5190 DOF) and a half-space footing with their CPU
arms (configs_form), the roofline of the dominant kernel and the CPU oracle
timed on the host cores.

--impl reference times the reference-equivalent CPU path (the oracle: OpenMP
assembly on all host cores + OpenBLAS getrf/getrs) on one frequency per step.
Under torchrun (N > 1) the sweep is sharded: 20 frequencies per rank of a
20*N-frequency sweep (weak scaling), no device collective.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "harmonic BEM assemble+solve solves/sec vs plain FP64 GPU at rel-err ≤1e-8"
WORKLOAD = "harela cube 8x8 quad8 per face, 3462 complex DOF, 20 frequencies a0=0.1..2.0"
WORKLOAD_P = "harela surface patch 40x40 quad8 (20x20), 14883 complex DOF, a0=0.5"

# Algorithmic work of the regular-pair assembly kernel (the dominant kernel):
# bytes = the complex system A (n^2) and b (n) written once per frequency;
# flops = FLOPS_PER_REGULAR_POINT real flops per regular quadrature point of the
# time-harmonic kernel, counted on the binary64 formulation with the radial
# functions from the call's table: distance, 1/r and interval 16, five complex
# Horner sums of degree 7 with their singular parts 160, dr, dr/dn and the
# products with it 12, u*/t* components 108, 120 complex accumulations 480.
FLOPS_PER_REGULAR_POINT = 776
# GB300 FP64 rate (nominal; not in the measured peaks): the binary64
# formulation of the same kernel (the plain path's) could at best run at this rate
FP64_NOMINAL_TFLOPS = 1.25
# DRAM bytes per frequency of that kernel from ncu (dram__bytes_read.sum +
# dram__bytes_write.sum of one launch of the 2-frequency profile case, 449.6 +
# 394.1 MB, divided by 2; profiles/k_mixed_cube8x2freq.md): A written once
# and read once (the pair sums are added to the zeroed system at the L2). Traffic grows in
# proportion to the frequencies (one system per frequency).
REG_TRAFFIC_PER_FREQ = 421.9e6
# Pipe utilisation of the same launch (ncu, same small case and
# file): the kernel is bound by instruction issue on the FP32 pipe
# (double-float arithmetic), not by HBM.
REG_NCU_PIPES = {"issue_slots_busy_pct": 53.2, "fp32_fma_pipe_pct": 28.0, "fp64_pipe_pct": 34.9,
                 "source": "profiles/k_mixed_cube8x2freq.md"}


def _dist():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    return ws, rank


class Clocks:
    """nvidia-smi sampling during the timed region."""

    def __init__(self):
        self.samples = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", os.environ.get("LOCAL_RANK", "0"),
                 "--query-gpu=clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
                 "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
                 "clocks_event_reasons.sw_power_cap", "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.samples.append([x.strip() for x in line.split(",")])

    def stop(self):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
        sm = [float(s[0]) for s in self.samples if len(s) >= 7 and s[0].replace(".", "").isdigit()]
        mx = [float(s[1]) for s in self.samples if len(s) >= 7 and s[1].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[i] for s in self.samples if len(s) >= 7 for i in range(4) if s[3 + i] == "Active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(sm)}


def cpu_baseline_sample(deck, mat, omega, threads=None):
    """Oracle (reference-equivalent CPU path) assemble + getrf/getrs for one
    frequency on all host cores. Returns (seconds, cores, solution)."""
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    cores = threads or os.cpu_count()
    os.environ.setdefault("OMP_NUM_THREADS", str(cores))
    P = O.Problem(deck)
    t0 = time.perf_counter()
    A, b = P.assemble_harela(mat, omega, nthreads=cores)
    x = O.lu_solve(A, b, overwrite=True)
    return time.perf_counter() - t0, cores, x


def cpu_sweep_rate(deck, mat, om, samples):
    """The CPU path's solves/s on a bounded sample of a sweep: one untimed
    frequency (threads, pages), then `samples` frequencies spread over the
    sweep, each assembled and solved. The same sampling serves the reference
    arm and the GPU line's cpu_baseline. Returns (solves/s, cores, seconds)."""
    cpu_baseline_sample(deck, mat, om[0])
    idx = [int(round(i * (len(om) - 1) / max(1, samples - 1))) for i in range(samples)] if samples > 1 else [0]
    ts = []
    cores = os.cpu_count()
    for i in idx:
        t, cores, _ = cpu_baseline_sample(deck, mat, om[i])
        ts.append(t)
    return len(ts) / sum(ts), cores, sum(ts)


def bench_config(n, nf):
    """config dict of the headline workload, identical in both arms."""
    return {"workload": WORKLOAD, "n_dof": n, "frequencies": nf,
            "l2": "inputs larger than L2 (20 x 192 MB systems per step)"}


def run_reference(args):
    ws, rank = _dist()
    if rank != 0:
        return 0
    from multifebe_gb300 import meshgen as M
    deck, mat, om = M.workload(2)
    # untimed warm-up frequencies (threads, pages); each a full assemble + solve
    for i in range(max(1, min(args.warmup, 2))):
        cpu_baseline_sample(deck, mat, om[i % len(om)])
    ts = []
    cores = os.cpu_count()
    for i in range(args.steps):
        t, cores, _ = cpu_baseline_sample(deck, mat, om[i % len(om)])
        ts.append(t)
    tot = sum(ts)
    value = len(ts) / tot
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * tot / len(ts), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "complex128", "data": "synthetic",
            "config": bench_config(deck.n_dof, len(om)),
            "cpu_baseline": {"value": value, "unit": "solves/s", "cores": cores, "kind": "port",
                             "sample": "each step assembles and solves (getrf/getrs) one frequency of the sweep, "
                                       "frequencies taken in turn, after untimed warm-up frequencies (oracle "
                                       "restatement of the Fortran path, OpenMP + OpenBLAS)"},
            "e2e": {"value": value, "unit": "solves/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def run_gpu(args):
    ws, rank = _dist()
    if ws > 1:
        # one GPU per rank, selected before the library initialises CUDA
        os.environ.setdefault("CUDA_VISIBLE_DEVICES", os.environ.get("LOCAL_RANK", str(rank)))
        import torch.distributed as dist
        dist.init_process_group("gloo")
    from multifebe_gb300 import meshgen as M, BemRegion, _abi, shard
    from multifebe_gb300.bem import _p
    deck, mat, om = M.workload(2)
    if ws > 1:
        # weak scaling: a 20*N-frequency sweep over a0 in [0.1, 2.0], 20 per rank
        om_all = M.omega_from_a0(shard.weak_scaled_frequencies(0.1, 2.0, len(om), ws), mat)
        om = om_all[shard.frequency_shard(len(om_all), rank, ws)]
    nf = len(om)
    R = BemRegion(deck)
    n = R.n
    # warm-up (also loads every kernel)
    for _ in range(args.warmup):
        R.sweep_harela(mat, om, precision="mixed")
    if ws > 1:
        dist.barrier()
    clocks = Clocks()
    clocks.start()
    dev_ms = []
    launches = 0
    t0 = time.perf_counter()
    for _ in range(args.steps):
        R.sweep_harela(mat, om, precision="mixed")
        s = R.last_stats
        dev_ms.append(s["ms_assemble"] + s["ms_factor"] + s["ms_solve"])
        launches += s.get("kernel_launches", 0)
    wall = time.perf_counter() - t0
    clk = clocks.stop()
    if ws > 1:
        dist.barrier()
    st = R.last_stats
    per_step_ms = statistics.mean(dev_ms)
    if ws > 1:
        import torch
        tt = torch.tensor([per_step_ms, wall], dtype=torch.float64)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        per_step_ms, wall = float(tt[0]), float(tt[1])
    value = ws * nf / (per_step_ms / 1e3)

    # e2e: public C-ABI from host buffers, mesh upload + sweep + download per step
    L = _abi.load()
    desc = R.desc
    lam = np.array([complex(mat["lambda"]).real, complex(mat["lambda"]).imag])
    mu = np.array([complex(mat["mu"]).real, complex(mat["mu"]).imag])
    nu = np.array([complex(mat["nu"]).real, complex(mat["nu"]).imag])
    omv = np.ascontiguousarray(om)
    X = np.zeros((nf, n), dtype=np.complex128)
    h2d = _desc_bytes(desc.contents, deck)
    d2h = X.nbytes
    e2e_t = []
    for it in range(args.warmup + args.steps):
        t1 = time.perf_counter()
        h = ctypes.c_void_p()
        _abi.check(L.mfbem_mesh_upload(desc, ctypes.byref(h)))
        stt = _abi.Stats()
        _abi.check(L.mfbem_sweep_harela(h, _p(lam), _p(mu), float(mat["rho"]), _p(nu), nf, _p(omv), 1, 1e-12, _p(X), 0,
                                        ctypes.byref(stt)))
        L.mfbem_mesh_release(h)
        if it >= args.warmup:
            e2e_t.append(time.perf_counter() - t1)
    e2e_step = statistics.mean(e2e_t)
    if ws > 1:
        tt = torch.tensor([e2e_step], dtype=torch.float64)
        dist.all_reduce(tt, op=dist.ReduceOp.MAX)
        e2e_step = float(tt[0])

    if rank != 0:
        return 0
    # the plain FP64 GPU path on the same sweep (FP64 assembly + FP64 LU), and
    # the accuracy of the timed path against it (the plain path is itself
    # pinned to the oracle in the tests)
    Xm = R.sweep_harela(mat, om, precision="mixed")
    Xp = R.sweep_harela(mat, om, precision="plain")
    plain_ms = []
    for _ in range(max(1, args.steps // 2)):
        Xp = R.sweep_harela(mat, om, precision="plain")
        sp = R.last_stats
        plain_ms.append(sp["ms_assemble"] + sp["ms_factor"] + sp["ms_solve"])
    plain_step = statistics.mean(plain_ms)
    relerr = max(np.abs(Xm[i] - Xp[i]).max() / np.abs(Xp[i]).max() for i in range(nf))
    # the plain path with binary64 arithmetic in its trailing updates too
    # (SIMT FMA on the FP64 pipe instead of the Ozaki-scheme tensor-core GEMM)
    native = _plain_native(R, mat, om)
    line = {"metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": ws, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": per_step_ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None,
            "dtype": "double-float assembly (binary64 x - x_i) into binary64 systems / complex64 LU with binary16 hi/lo "
                     "tensor-core updates + FP64 refinement",
            "data": "synthetic",
            "config": bench_config(n, nf),
            "detail": {"precision": "mixed", "rel_err_vs_fp64_gpu": relerr,
                       "max_backward_error": st["max_backward_error"],
                       "ms_assemble": st["ms_assemble"], "ms_factor": st["ms_factor"], "ms_solve": st["ms_solve"],
                       "ms_regular": st["ms_regular"], "ms_singular": st["ms_singular"],
                       "ms_adaptive": st["ms_adaptive"], "ms_free": st["ms_free"],
                       "parallelism": f"replicas x{ws}"},
            "e2e": {"value": ws * nf / e2e_step, "unit": "solves/s", "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h},
            "gpu_launches": launches, "clocks": clk,
            "plain_fp64_gpu": {"value": nf / (plain_step / 1e3), "unit": "solves/s", "ms_per_step": plain_step,
                               "ms_factor": sp["ms_factor"], "ms_assemble": sp["ms_assemble"],
                               "ms_solve": sp["ms_solve"],
                               "speedup_of_mixed": (nf / (per_step_ms / 1e3)) / (nf / (plain_step / 1e3)),
                               "trailing_updates": "FP64-accurate Ozaki scheme on the bf16 tensor cores"},
            "plain_fp64_gpu_native": dict(native, speedup_of_mixed=native["ms_per_step"] / per_step_ms)}
    line["roofline"] = roofline(st, n, nf)
    if args.precision_form:
        line["precision_form"] = precision_form()
    if args.learned:
        line["learned_quadrature"] = learned_quadrature()
    if args.batching:
        line["batching_form"] = batching_form()
    if args.configs:
        line["configs_form"] = configs_form()
    # cpu baseline: the reference arm's sampling on a bounded sample of the sweep
    try:
        v, cores, secs = cpu_sweep_rate(deck, mat, om, 5)
        line["cpu_baseline"] = {"value": v, "unit": "solves/s", "cores": cores, "kind": "port",
                                "sample": "5 of the sweep's 20 frequencies spread over a0 0.1..2.0, each "
                                          "assembled and solved by the oracle restatement (OpenMP + OpenBLAS "
                                          "getrf/getrs) after one untimed frequency, %.1f s" % secs}
        line["plain_fp64_gpu"]["speedup_over_cpu"] = line["plain_fp64_gpu"]["value"] / v
    except Exception as ex:  # the oracle must build on the host; report why not
        line["cpu_baseline"] = {"value": None, "unit": "solves/s", "cores": os.cpu_count(), "kind": "port",
                                "sample": f"unavailable: {ex}"}
    print(json.dumps(line), flush=True)
    return 0


def _plain_native(R, mat, om, steps=1):
    """The plain sweep with MFBEM_FP64_GEMM=dfma: binary64 FMA throughout (the
    LU's trailing updates on the FP64 pipe). One untimed and `steps` timed sweeps."""
    old = os.environ.get("MFBEM_FP64_GEMM")
    os.environ["MFBEM_FP64_GEMM"] = "dfma"
    try:
        R.sweep_harela(mat, om, precision="plain")
        ts = []
        for _ in range(steps):
            R.sweep_harela(mat, om, precision="plain")
            st = R.last_stats
            ts.append(st["ms_assemble"] + st["ms_factor"] + st["ms_solve"])
    finally:
        if old is None:
            del os.environ["MFBEM_FP64_GEMM"]
        else:
            os.environ["MFBEM_FP64_GEMM"] = old
    t = statistics.mean(ts)
    return {"value": len(om) / (t / 1e3), "unit": "solves/s", "ms_per_step": t, "ms_factor": st["ms_factor"],
            "trailing_updates": "binary64 SIMT FMA (own kernel)"}


def _peaks():
    try:
        return json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json"))), "measured"
    except Exception:
        return {"hbm_gbs": 6800.0, "bf16_tflops": 1900.0}, "fallback"


def roofline(st, n, nf):
    """Roofline of the dominant kernel (regular-pair assembly, one launch for
    all nf frequencies), timed by CUDA events on the library's stream."""
    pk, src = _peaks()
    t = st["ms_regular"] / 1e3
    alg_bytes = nf * (n * n + n) * 16
    achieved = alg_bytes / t / 1e9
    pts = st["points_regular"] * nf
    tfl = pts * FLOPS_PER_REGULAR_POINT / t / 1e12
    return {"kernel": "k_mixed<MIX_REG> (regular pairs, double-float, all frequencies in one launch)",
            "bound": "hbm", "achieved": achieved,
            "peak": pk["hbm_gbs"], "unit": "GB/s", "frac": achieved / pk["hbm_gbs"], "peak_source": src,
            "traffic": (REG_TRAFFIC_PER_FREQ * nf) if REG_TRAFFIC_PER_FREQ else None,
            "algorithmic_bytes": alg_bytes, "ms": st["ms_regular"],
            "compute": {"points": pts, "flops_per_point": FLOPS_PER_REGULAR_POINT, "achieved_tflops": tfl,
                        "fp64_nominal_peak_tflops": FP64_NOMINAL_TFLOPS,
                        "frac_of_fp64_nominal": tfl / FP64_NOMINAL_TFLOPS,
                        "ncu_pipes_of_active_cycles": REG_NCU_PIPES,
                        "note": "SIMT-issue bound (double-float on the FP32 pipe, binary64 for x - x_i and the "
                                "pair sums' last addition): FP64-equivalent flops of the tabulated formulation; "
                                "HBM and tensor pipes are not the limit of this kernel"}}


def batching_form():
    """48 uneven problems: the cube at n x n elements per face, n in
    {4,5,6,7,8,10} (870 .. 5406 DOF), 8 frequencies a0 = 0.2..1.6 each, mixed
    precision. One call for all meshes (concurrent sweeps) against the same
    sweeps one after another (wall clock, host API), and every problem's
    difference to the plain FP64 GPU solution (itself pinned to the oracle)."""
    import time as _t
    from multifebe_gb300 import meshgen as M, BemRegion, sweep_harela_batch
    work = M.batch_workload()
    regions = [BemRegion(d) for d, _, _ in work]
    mats = [m for _, m, _ in work]
    oms = [o for _, _, o in work]
    nsol = sum(len(o) for o in oms)
    for _ in range(2):  # warm-up: kernels, autotuner classes
        sweep_harela_batch(regions, mats, oms, precision="mixed")
    t0 = _t.perf_counter()
    Xb, _ = sweep_harela_batch(regions, mats, oms, precision="mixed")
    t_batch = _t.perf_counter() - t0
    t0 = _t.perf_counter()
    dev_ms = 0.0
    for r, m, o in zip(regions, mats, oms):
        r.sweep_harela(m, o, precision="mixed")
        st = r.last_stats
        dev_ms += st["ms_assemble"] + st["ms_factor"] + st["ms_solve"]
    t_seq = _t.perf_counter() - t0
    errs = []
    for r, m, o, x in zip(regions, mats, oms, Xb):
        xp = r.sweep_harela(m, o, precision="plain")
        errs += [float(np.abs(x[i] - xp[i]).max() / np.abs(xp[i]).max()) for i in range(len(o))]
    for r in regions:
        r.close()
    return {"workload": "harela cubes n x n quad8 per face, n in {4,5,6,7,8,10} (870..5406 DOF), 8 frequencies "
                        "a0=0.2..1.6 each: 48 problems", "problems": nsol,
            "batched": {"value": nsol / t_batch, "unit": "solves/s", "wall_s": t_batch},
            "one_after_another": {"value": nsol / t_seq, "unit": "solves/s", "wall_s": t_seq,
                                  "device_s": dev_ms / 1e3,
                                  "note": "device_s: the six sweeps' own CUDA-event time (assembly, factorisation, "
                                          "refinement) summed; the batched wall time against it shows how much "
                                          "of the GPU the concurrent sweeps leave idle"},
            "max_rel_err_vs_fp64": max(errs), "n_dof": [r_.n for r_ in regions]}


def _pair_stats(err, cost, sel):
    """Quadrature points and log10 relative errors (against the converged
    integral) of the selected pairs."""
    e, c = err[sel], cost[sel]
    return {"pairs": int(sel.sum()), "points": int(c.sum()),
            "frac_within_1e-7": float((e <= -7.0).mean()) if e.size else None,
            "log10_err_p50": float(np.median(e)) if e.size else None,
            "log10_err_p95": float(np.percentile(e, 95)) if e.size else None,
            "log10_err_max": float(e.max()) if e.size else None}


def learned_quadrature():
    """The thin slab (16x16 + 16x1 quad8 per face, 5190 DOF, a0 0.2 and 1.0).
    The network is trained on 8000 seeded random harmonic pairs (|k| x size in
    0..0.5, the slab's material) labelled on the GPU. At equal tolerance 1e-7:
    the reference adaptive rule at qsi_relative_error 1e-7 against the learned
    rule at log10 tolerance -7 (falling back to that reference rule). Reported:
    over the slab's own quasi-singular pairs, labelled against their converged
    integrals (graded depth-9 rule, g = 30), the points and the error
    distribution -- over all pairs and over the pairs the network changes --;
    in the device sweep, the adaptive-pair points and kernel time, the
    assembly error against the converged assembly (qsi_relative_error 1e-10)
    and the sweep's solves/s."""
    import time as _t
    from multifebe_gb300 import meshgen as M, BemRegion, qlearn as Q
    t0 = _t.perf_counter()
    e, p, k, kc = Q.random_pairs(8000, seed=21, kernel=1)
    F, Y, C, V = Q.label_pairs(e, p, k, kc)
    t1 = _t.perf_counter()
    w = Q.init_weights(2)
    hist = Q.train(w, F, Y, V, steps=3000, batch=2048, lr=2e-3, seed=6)
    t2 = _t.perf_counter()
    deck, mat, om = M.workload(5)
    # |k2| x element size at the highest frequency (largest slab element size 1/16)
    k2 = float(om[-1]) / abs(np.sqrt(complex(mat["mu"]) / mat["rho"]))
    kcl = k2 * (1.0 / 16.0)
    out = {"workload": "harela slab 1x1x0.02, 16x16 + 16x1 quad8 per face, 5190 complex DOF, a0 0.2 and 1.0",
           "training": {"pairs": 8000, "kernel": "harmonic", "valid": int(V.sum()), "label_s": t1 - t0,
                        "train_s": t2 - t1, "steps": 3000, "loss_first": float(hist[:10].mean()),
                        "loss_last": float(hist[-100:].mean())}}
    tol = 1e-7
    ref_c = Q.reference_candidate(tol)
    R = BemRegion(deck, qsi_relative_error=tol)
    # the slab's own quasi-singular pairs against their converged integrals
    el, pts, _ = Q.mesh_adaptive_pairs(R)
    Fm, Ym, Cm, Vm = Q.label_pairs(el, pts, 1, np.full(len(pts), kcl))
    pred = Q.forward(w, Fm)
    ch = Q.choose(pred, Cm, np.log10(tol), fallback=ref_c)
    idx = np.arange(len(ch))
    valid = Vm.astype(bool)
    err_ref, cost_ref = Ym[:, ref_c], Cm[:, ref_c]
    err_l, cost_l = Ym[idx, ch], Cm[idx, ch]
    changed = valid & (ch != ref_c)
    # the learned rule at equal accuracy: the loosest learned tolerance whose
    # error distribution over the slab's pairs is no worse than the reference
    # rule's at 1e-7 (fraction within 1e-7 and 95th percentile)
    ref_st = _pair_stats(err_ref, cost_ref, valid)
    eq = None
    for lt in np.arange(-7.0, -10.01, -0.25):
        c2 = Q.choose(pred, Cm, lt, fallback=ref_c)
        st2 = _pair_stats(Ym[idx, c2], Cm[idx, c2], valid)
        if st2["frac_within_1e-7"] >= ref_st["frac_within_1e-7"] and st2["log10_err_p95"] <= ref_st["log10_err_p95"]:
            eq = dict(st2, log10_tol=float(lt), points_vs_reference=st2["points"] / ref_st["points"])
            break
    # accuracy / cost curves over the slab's pairs: the reference rule at
    # qsi_relative_error 1e-6 .. 1e-9 and the learned rule at log10 tolerance
    # -7 .. -10; then, for each reference setting, the cheapest learned
    # tolerance whose worst pair error and 95th percentile are no larger
    ref_curve = []
    for c in range(Q.REF_DEFAULT, min(Q.REF_DEFAULT + 4, Cm.shape[1])):
        st_c = _pair_stats(Ym[:, c], Cm[:, c], valid)
        ref_curve.append(dict(st_c, qsi_relative_error=10.0 ** -(3 + c)))
    learned_curve = []
    for lt in np.arange(-7.0, -10.01, -0.25):
        c2 = Q.choose(pred, Cm, lt, fallback=ref_c)
        learned_curve.append(dict(_pair_stats(Ym[idx, c2], Cm[idx, c2], valid), log10_tol=float(lt)))
    # the same selection with the true labels instead of the network's
    # predictions: the cheapest candidate per pair whose converged-integral
    # error meets the tolerance -- the best any predictor of this candidate
    # set can do
    label_curve = []
    for lt in np.arange(-6.0, -9.01, -0.25):
        c3 = Q.choose(Ym, Cm, lt, fallback=ref_c)
        label_curve.append(dict(_pair_stats(Ym[idx, c3], Cm[idx, c3], valid), log10_tol=float(lt)))
    at_equal = []
    for rc_ in ref_curve:
        best = None
        for lc in learned_curve:
            if lc["log10_err_max"] <= rc_["log10_err_max"] and lc["log10_err_p95"] <= rc_["log10_err_p95"]:
                if best is None or lc["points"] < best["points"]:
                    best = lc
        bl = None
        for lc in label_curve:
            if lc["log10_err_max"] <= rc_["log10_err_max"] and (bl is None or lc["points"] < bl["points"]):
                bl = lc
        at_equal.append({"reference_qsi": rc_["qsi_relative_error"], "reference_points": rc_["points"],
                         "true_label_choice_points": bl["points"] if bl else None,
                         "reference_log10_err_max": rc_["log10_err_max"],
                         "learned_log10_tol": best["log10_tol"] if best else None,
                         "learned_points": best["points"] if best else None,
                         "learned_log10_err_max": best["log10_err_max"] if best else None,
                         "points_vs_reference": (best["points"] / rc_["points"]) if best else None})
    out["mesh_pairs"] = {
        "adaptive_pairs": int(len(ch)), "labelled_valid": int(valid.sum()),
        "learned_at_equal_accuracy": eq,
        "reference_curve": ref_curve, "learned_curve": learned_curve, "true_label_curve": label_curve,
        "learned_vs_reference_at_equal_worst_error": at_equal,
        "reference_1e-7": _pair_stats(err_ref, cost_ref, valid),
        "learned_1e-7": _pair_stats(err_l, cost_l, valid),
        "changed_pairs": {"reference_1e-7": _pair_stats(err_ref, cost_ref, changed),
                          "learned_1e-7": _pair_stats(err_l, cost_l, changed)},
        "reference_1e-6": _pair_stats(Ym[:, Q.REF_DEFAULT], Cm[:, Q.REF_DEFAULT], valid)}
    Rc = BemRegion(deck, qsi_relative_error=1e-10)
    Ac, _ = Rc.build_lse_harela(mat, float(om[-1]))
    Rc.close()
    scale = float(np.abs(Ac).max())
    runs = [("reference_1e-7", None, np.log10(tol)), ("learned_1e-7", w, np.log10(tol))]
    if eq is not None:
        runs.append(("learned_equal_accuracy", w, eq["log10_tol"]))
    for name, wt, lt in runs:
        nl = R.set_learned_quadrature(wt, log10_tol=lt, kernel=1, kcl=kcl)
        A, _ = R.build_lse_harela(mat, float(om[-1]))
        err = float(np.abs(A - Ac).max() / scale)
        R.sweep_harela(mat, om, precision="mixed")
        R.sweep_harela(mat, om, precision="mixed")
        st = R.last_stats
        out[name] = {"pairs_learned": nl, "points_adaptive": st["points_adaptive"],
                     "ms_adaptive_sweep": st["ms_adaptive"], "assembly_rel_err_vs_converged": err,
                     "sweep_solves_per_s": len(om) / ((st["ms_assemble"] + st["ms_factor"] + st["ms_solve"]) / 1e3)}
    R.close()
    return out


def _sweep_e2e(R, deck, mat, om, precision, reps):
    """The public C-ABI from host buffers: mesh upload (H2D) + sweep +
    solution download (D2H) per repetition. Returns (mean seconds, h2d, d2h)."""
    from multifebe_gb300 import _abi
    from multifebe_gb300.bem import _p, PRECISION
    L = _abi.load()
    lam = np.array([complex(mat["lambda"]).real, complex(mat["lambda"]).imag])
    mu = np.array([complex(mat["mu"]).real, complex(mat["mu"]).imag])
    nu = np.array([complex(mat["nu"]).real, complex(mat["nu"]).imag])
    omv = np.ascontiguousarray(om, dtype=np.float64)
    X = np.zeros((len(om), R.n), dtype=np.complex128)
    ts = []
    for _ in range(reps):
        t1 = time.perf_counter()
        h = ctypes.c_void_p()
        _abi.check(L.mfbem_mesh_upload(R.desc, ctypes.byref(h)))
        stt = _abi.Stats()
        _abi.check(L.mfbem_sweep_harela(h, _p(lam), _p(mu), float(mat["rho"]), _p(nu), len(om), _p(omv),
                                        PRECISION[precision], 1e-12, _p(X), 0, ctypes.byref(stt)))
        L.mfbem_mesh_release(h)
        ts.append(time.perf_counter() - t1)
    return statistics.mean(ts), _desc_bytes(R.desc.contents, deck), X.nbytes


def precision_form(steps=3, warmup=1):
    """The 14883-DOF surface patch at a0=0.5 (one solve per step).
    mixed: `steps` device-timed solves after `warmup` untimed ones, and the
    same through the C-ABI from host buffers (e2e); plain FP64 GPU: one timed
    solve after an untimed one; CPU: the oracle's assemble + getrf/getrs on
    all host cores, whose solution is also the FP64 reference of the u and t
    errors of both GPU paths."""
    from multifebe_gb300 import meshgen as M, BemRegion
    deck, mat, om = M.workload(3)
    R = BemRegion(deck)
    for _ in range(warmup):
        R.sweep_harela(mat, om, precision="mixed")
    tms, st = [], None
    for _ in range(steps):
        Xm = R.sweep_harela(mat, om, precision="mixed")
        st = dict(R.last_stats)
        tms.append(st["ms_assemble"] + st["ms_factor"] + st["ms_solve"])
    tm = statistics.mean(tms)
    e2e_s, h2d, d2h = _sweep_e2e(R, deck, mat, om, "mixed", steps)
    R.sweep_harela(mat, om, precision="plain")
    Xp = R.sweep_harela(mat, om, precision="plain")
    sp = dict(R.last_stats)
    tp = sp["ms_assemble"] + sp["ms_factor"] + sp["ms_solve"]
    nat = _plain_native(R, mat, om)
    out = {"workload": WORKLOAD_P, "n_dof": int(Xm.shape[1]), "steps": steps, "warmup": warmup,
           "mixed": {"value": 1e3 / tm, "unit": "solves/s", "ms_per_step": tm, "ms_assemble": st["ms_assemble"],
                     "ms_factor": st["ms_factor"], "ms_solve": st["ms_solve"],
                     "refinement_iterations": st["refinement_iterations"],
                     "max_backward_error": st["max_backward_error"],
                     "e2e": {"value": 1.0 / e2e_s, "unit": "solves/s", "h2d_bytes_per_step": h2d,
                             "d2h_bytes_per_step": d2h}},
           "plain_fp64_gpu": {"value": 1e3 / tp, "unit": "solves/s", "ms_assemble": sp["ms_assemble"],
                              "ms_factor": sp["ms_factor"], "ms_solve": sp["ms_solve"]},
           "plain_fp64_gpu_native": dict(nat, speedup_of_mixed=nat["ms_per_step"] / tm),
           "speedup_of_mixed": tp / tm,
           "rel_err_mixed_vs_fp64_gpu": float(np.abs(Xm - Xp).max() / np.abs(Xp).max())}
    try:
        t, cores, xo = cpu_baseline_sample(deck, mat, float(om[0]))
        uo, to = R.solution(xo)
        errs = {}
        for name, X in (("mixed", Xm[0]), ("plain_fp64_gpu", Xp[0])):
            u, tt = R.solution(X)
            errs[name] = {"u": float(np.abs(u - uo).max() / np.abs(uo).max()),
                          "t": float(np.abs(tt - to).max() / np.abs(to).max())}
        out["rel_err_vs_fp64_oracle"] = errs
        out["cpu_baseline"] = {"value": 1.0 / t, "unit": "solves/s", "cores": cores, "kind": "port",
                               "sample": "one assemble + getrf/getrs of the patch by the oracle restatement "
                                         "(OpenMP + OpenBLAS), %.1f s" % t}
        out["plain_fp64_gpu"]["speedup_over_cpu"] = out["plain_fp64_gpu"]["value"] * t
    except Exception as ex:
        out["cpu_baseline"] = {"value": None, "unit": "solves/s", "kind": "port", "sample": f"unavailable: {ex}"}
    R.close()
    return out


def _oracle():
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import oracle as O
    return O


def configs_form():
    """The other benchmark configurations, each with its CPU arm (the oracle
    on all host cores) and the error of the GPU solutions against the
    oracle's FP64 solution:
      cfg 1: staela cube 4x4 per face (870 real DOF), plain and mixed;
      cfg 5: harela thin slab (5190 complex DOF), both frequencies, plain and
             mixed sweeps;
      half-space footing: staela, 8x8 quad8 loaded square on the surface of a
             half-space (complementary kernel), plain, with Love's closed form;
      penny crack in a cube: staela, a crack-like boundary (dual BEM, six
             rows per crack node) inside a clamped cube, plain and mixed;
      Burton & Miller cube: the cube 8x8 of the headline with the
             'dual_bm_same' formulation (SBIE + i/c2 HBIE at the 3072 HBIE
             points), four frequencies, plain and mixed sweeps, the oracle on
             one of them."""
    from multifebe_gb300 import meshgen as M, BemRegion
    O = _oracle()
    cores = os.cpu_count()
    out = {}

    def rel(a, b):
        return float(np.abs(a - b).max() / np.abs(b).max())

    def static_case(deck, mat, hs, reps, crack=None):
        R = BemRegion(deck, crack=crack)
        if hs:
            R.set_halfspace(-3, 0.0, 1)
        res = {}
        xs = {}
        for prec in ("plain", "mixed"):
            R.solve_staela(mat["mu"], mat["nu"], precision=prec)  # warm-up
            ms = []
            for _ in range(reps):
                xs[prec] = R.solve_staela(mat["mu"], mat["nu"], precision=prec)
                st = R.last_stats
                ms.append(st["ms_assemble"] + st["ms_factor"] + st["ms_solve"])
            res[prec] = {"value": 1e3 / statistics.mean(ms), "unit": "solves/s", "ms_per_solve": statistics.mean(ms),
                         "ms_assemble": st["ms_assemble"], "ms_factor": st["ms_factor"], "ms_solve": st["ms_solve"]}
        P = O.Problem(deck)
        if hs:
            P.set_halfspace(-3, 0.0, 1)
        if crack is not None:
            P.set_crack(*crack)
        P.assemble_staela(mat["mu"], mat["nu"], nthreads=cores)  # warm-up
        ts = []
        for _ in range(3):
            t0 = time.perf_counter()
            A, b = P.assemble_staela(mat["mu"], mat["nu"], nthreads=cores)
            xo = O.lu_solve(A, b, overwrite=True)
            ts.append(time.perf_counter() - t0)
        res["cpu_baseline"] = {"value": 1.0 / statistics.mean(ts), "unit": "solves/s", "cores": cores, "kind": "port",
                               "sample": "3 assemble + getrf/getrs of the oracle after one untimed assembly"}
        for prec in ("plain", "mixed"):
            res[prec]["rel_err_vs_fp64_oracle"] = rel(xs[prec], xo)
            res[prec]["speedup_over_cpu"] = res[prec]["value"] / res["cpu_baseline"]["value"]
        R.close()
        return res, xs, P

    deck, mat, _ = M.workload(1)
    out["cfg1_staela_cube4"], _, _ = static_case(deck, mat, False, 20)
    out["cfg1_staela_cube4"]["n_dof"] = deck.n_dof

    deck = M.halfspace_footing(1.0, 8, 1.0)
    mat = M.elastic(1.0, 0.25)
    res, xs, P = static_case(deck, mat, True, 10)
    u, _ = P.solution(xs["plain"])
    c = int(np.argmin(np.linalg.norm(deck.nodes, axis=1)))
    w = M.love_square_centre(1.0, 1.0, 1.0, 0.25)
    res["love_centre_settlement"] = {"gpu": float(u[c, 2]), "closed_form": w, "rel_err": abs(u[c, 2] - w) / w}
    res["n_dof"] = deck.n_dof
    out["halfspace_footing_8x8"] = res

    # crack-like boundary (dual BEM): pressurised penny crack inside a clamped
    # cube 8 x 8 x 8 (crack 4 x 4 + 4 x (4 x 3) quad8, cube 4 x 4 per face)
    deck, crack = M.penny_crack_in_box(1.0, 4, 3, 4.0, 4)
    res, xs, P = static_case(deck, mat, False, 10, crack=crack)
    u1, _, u2, _ = P.solution_faces(xs["plain"])
    c = int(np.argmin(np.linalg.norm(deck.nodes, axis=1)))
    res["n_dof"] = P.n
    res["opening_at_centre"] = {"gpu": float(u2[c, 2] - u1[c, 2]),
                                "sneddon_full_space": float(M.sneddon_opening(0.0, 1.0, 1.0, 1.0, 0.25))}
    out["penny_crack_in_cube"] = res

    deck, mat, om = M.workload(5)
    R = BemRegion(deck)
    res = {"n_dof": deck.n_dof, "frequencies": len(om)}
    X = {}
    for prec in ("plain", "mixed"):
        R.sweep_harela(mat, om, precision=prec)  # warm-up
        ms = []
        for _ in range(3):
            X[prec] = R.sweep_harela(mat, om, precision=prec)
            st = R.last_stats
            ms.append(st["ms_assemble"] + st["ms_factor"] + st["ms_solve"])
        res[prec] = {"value": len(om) / (statistics.mean(ms) / 1e3), "unit": "solves/s",
                     "ms_per_sweep": statistics.mean(ms), "ms_assemble": st["ms_assemble"],
                     "ms_factor": st["ms_factor"], "ms_solve": st["ms_solve"]}
    R.close()
    P = O.Problem(deck)
    ts, errs = [], {"plain": 0.0, "mixed": 0.0}
    for i, wv in enumerate(om):
        t0 = time.perf_counter()
        A, b = P.assemble_harela(mat, float(wv), nthreads=cores)
        xo = O.lu_solve(A, b, overwrite=True)
        ts.append(time.perf_counter() - t0)
        del A
        for prec in errs:
            errs[prec] = max(errs[prec], rel(X[prec][i], xo))
    res["cpu_baseline"] = {"value": len(ts) / sum(ts), "unit": "solves/s", "cores": cores, "kind": "port",
                           "sample": "both frequencies assembled and solved by the oracle (first includes warm-up)"}
    for prec in errs:
        res[prec]["rel_err_vs_fp64_oracle"] = errs[prec]
        res[prec]["speedup_over_cpu"] = res[prec]["value"] / res["cpu_baseline"]["value"]
    res["note"] = ("the slab's systems are ill-conditioned (1/rcond ~1e7 at a0 = 0.2): both GPU paths differ "
                   "from the oracle by the conditioning times ~1e-12 assembly differences")
    out["cfg5_harela_slab16"] = res

    deck, mat, _ = M.workload(2)
    om = M.omega_from_a0(np.array([0.5, 1.0, 1.5, 2.0]), mat)
    R = BemRegion(deck, formulation="dual_bm")
    res = {"n_dof": deck.n_dof, "frequencies": len(om), "formulation": "dual_bm_same, alpha 1"}
    X = {}
    for prec in ("plain", "mixed"):
        R.sweep_harela(mat, om[:1], precision=prec)  # warm-up
        ms = []
        for _ in range(2):
            X[prec] = R.sweep_harela(mat, om, precision=prec)
            st = R.last_stats
            ms.append(st["ms_assemble"] + st["ms_factor"] + st["ms_solve"])
        res[prec] = {"value": len(om) / (statistics.mean(ms) / 1e3), "unit": "solves/s",
                     "ms_per_sweep": statistics.mean(ms), "ms_assemble": st["ms_assemble"],
                     "ms_regular": st["ms_regular"], "ms_adaptive": st["ms_adaptive"],
                     "ms_singular": st["ms_singular"], "ms_factor": st["ms_factor"], "ms_solve": st["ms_solve"]}
    R.close()
    P = O.Problem(deck)
    P.set_formulation("dual_bm")
    t0 = time.perf_counter()
    A, b = P.assemble_harela(mat, float(om[-1]), nthreads=cores)
    xo = O.lu_solve(A, b, overwrite=True)
    t = time.perf_counter() - t0
    del A
    res["cpu_baseline"] = {"value": 1.0 / t, "unit": "solves/s", "cores": cores, "kind": "port",
                           "sample": "one frequency (a0 = 2.0) assembled and solved by the oracle"}
    for prec in ("plain", "mixed"):
        res[prec]["rel_err_vs_fp64_oracle"] = rel(X[prec][-1], xo)
        res[prec]["speedup_over_cpu"] = res[prec]["value"] / res["cpu_baseline"]["value"]
    out["burton_miller_cube8"] = res
    return out


def _profiler(on):
    """cuProfilerStart / cuProfilerStop (driver API): with `ncu
    --profile-from-start off` only the launches between the two are captured."""
    lib = ctypes.CDLL("libcuda.so.1")
    return (lib.cuProfilerStart if on else lib.cuProfilerStop)()


def profile_case(nf, precision="mixed"):
    """Small fixed case for ncu captures: the benchmark mesh, nf frequencies,
    two sweeps of the given precision (the second one between
    cuProfilerStart / cuProfilerStop)."""
    from multifebe_gb300 import meshgen as M, BemRegion
    deck, mat, om = M.workload(2)
    R = BemRegion(deck)
    R.sweep_harela(mat, om[:nf], precision=precision)
    _profiler(True)
    R.sweep_harela(mat, om[:nf], precision=precision)
    _profiler(False)
    print(json.dumps(R.last_stats))
    return 0


def profile_patch(precision):
    """ncu case for the 14883-DOF surface patch: two sweeps at a0=0.5, the
    second between cuProfilerStart / cuProfilerStop."""
    from multifebe_gb300 import meshgen as M, BemRegion
    deck, mat, om = M.workload(3)
    R = BemRegion(deck)
    R.sweep_harela(mat, om, precision=precision)
    _profiler(True)
    R.sweep_harela(mat, om, precision=precision)
    _profiler(False)
    print(json.dumps(R.last_stats))
    return 0


def profile_static(precision):
    """ncu case for the static cube (870 DOF): three solves of the given
    precision (the first loads the kernels)."""
    from multifebe_gb300 import meshgen as M, BemRegion
    deck, mat, _ = M.workload(1)
    R = BemRegion(deck)
    for _ in range(3):
        R.solve_staela(mat["mu"], mat["nu"], precision=precision)
    print(json.dumps(R.last_stats))
    return 0


def _desc_bytes(d, deck):
    ne, nn = deck.n_elements, deck.n_nodes
    return int(ne * (24 + 1 + 4 + 24 + 24 + 16 + 24) * 8 + ne * (8 + 1 + 1) * 4 + nn * (3 + 6 + 3 + 1) * 4 + nn * 6 * 8)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--no-precision-form", dest="precision_form", action="store_false",
                    help="skip the 14883-DOF surface-patch mixed/plain comparison")
    ap.add_argument("--no-learned", dest="learned", action="store_false",
                    help="skip the learned-quadrature measurement on the thin slab")
    ap.add_argument("--no-batching", dest="batching", action="store_false",
                    help="skip the 48-problem batch of uneven meshes")
    ap.add_argument("--no-configs", dest="configs", action="store_false",
                    help="skip configurations 1 and 5 and the half-space footing")
    ap.add_argument("--profile-case", type=int, default=0,
                    help="profiling helper: run the benchmark mesh for this many frequencies twice, print stats, exit")
    ap.add_argument("--profile-precision", default="mixed", choices=["mixed", "plain"],
                    help="precision of the --profile-case sweeps")
    ap.add_argument("--profile-patch", default="", choices=["", "mixed", "plain"],
                    help="profiling helper: one sweep of the 14883-DOF surface patch, print stats, exit")
    ap.add_argument("--profile-static", default="", choices=["", "mixed", "plain"],
                    help="profiling helper: three static solves of the 870-DOF cube, print stats, exit")
    args = ap.parse_args()
    if args.profile_static:
        return profile_static(args.profile_static)
    if args.profile_case:
        return profile_case(args.profile_case, args.profile_precision)
    if args.profile_patch:
        return profile_patch(args.profile_patch)
    if args.impl == "reference":
        return run_reference(args)
    return run_gpu(args)


if __name__ == "__main__":
    sys.exit(main())
