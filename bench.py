#!/usr/bin/env python
"""Benchmark: Laplace G FMM matvec + adjoint on one B200 per rank.

Headline workload (one "step" = one forward and one backward pass of the
Laplace G FMM as a torch.autograd operator):
  1,048,576 points from 32 Gaussian clusters (sigma 0.02) in the unit cube,
  charges N(0,1), targets = sources (zero-distance pairs excluded), order
  p = 12 -- the lowest order whose potential meets rel. err <= 1e-6 against
  the FP64 direct sum on this point set -- mixed precision (FP32 near field,
  FP16x3 tensor-core M2L, FP64 expansions).  The backward gives the
  gradients of L = sum(w * pot) w.r.t. the charges (the transposed FMM) and
  the positions (the forward's field and the transposed FMM's field).
Metric: FMM matvec Mpts/s at rel err <= 1e-6 vs FP64 direct (points per
second of forward + backward on a built tree); the same step in the plain FP64
form is timed beside it (mixed_over_fp64, backward_over_forward).

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                  [--config adjoint1m|bem|uniform32k|batch64|batch64_matvec|helmholtz1m]

Under torchrun each rank runs its own independent problem (a different point
seed): one FMM does not shard here, so N GPUs run N independent problems (weak
scaling, no collective on the data path).  The reference arm (--impl
reference) times the reference's own CPU fmm() (built from its sources into
oracle/_ref) on the host cores.
"""
from __future__ import annotations

import argparse
import json
import multiprocessing as mp
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

# C2: Laplace Gnj double-layer matvec on an icosphere (--config bem, and a
# secondary key of the headline line)
P_ORDER = 10
SUBDIV = 6
LMAX = 5
METRIC = "FMM matvec Mpts/s (Laplace Gn double-layer BEM, 245,760 pts, p=10)"
# C3, the headline: Laplace G forward + backward on clustered points
C3_N = 1 << 20
C3_P = 12
C3_SEED = 13
C3_METRIC = "FMM matvec Mpts/s at rel err <=1e-6 vs FP64 direct; mixed+adjoint vs plain FP64"
# the reference arm's bounded sample: the C3 point set cut into 16 disjoint
# slices of 65,536 points, each one reference forward + adjoint at depth 4
# (the reference's fastest depth for this size, measured), one process per
# core; then single runs at 1/4 N (depth 5) and 1/2 N (depth 6) for the fit
C3_REF_SLICES = 16
C3_REF_LMAX = {C3_N // 16: 4, C3_N // 4: 5, C3_N // 2: 6}
L2_FLUSH_BYTES = 256 << 20  # > 126 MB L2
# DRAM bytes (read + write) per evaluate of the two dominant kernels, from
# single-pass ncu captures of the timed steps of each workload (the near field
# runs as two launches per evaluate; the M2L is translate_h16 + reduce_pairs)
NCU_TRAFFIC = {
    "adjoint1m": {"p2p_mixed": 2 * (31.84e6 + 0.07e6), "translate_tc": 118.2e6 + 1328.8e6 + 1497.1e6 + 5.3e6},
    "bem": {"p2p_mixed": 2 * 10.0e6, "translate_tc": 25.6e6 + 88.2e6 + 148.3e6 + 3.2e6},
}


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f), "measured"
    except Exception:
        return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0}, "fallback"


class ClockSampler:
    """Polls the SM clock and the clock-event (throttle) reasons of one GPU
    through NVML every `period` seconds while the timed region runs (the same
    counters nvidia-smi's clocks.sm / clocks_event_reasons.* report)."""

    REASONS = {0x8: "hw_slowdown", 0x40: "hw_thermal_slowdown", 0x20: "sw_thermal_slowdown", 0x4: "sw_power_cap"}

    def __init__(self, gpu_index, period=0.002):
        self.gpu, self.period = gpu_index, period
        self.sm, self.mask, self.smax = [], 0, None
        self._stop = threading.Event()

    def __enter__(self):
        try:
            import pynvml
            pynvml.nvmlInit()
            self.nv = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(self.gpu)
            self.smax = float(pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM))
            self.t = threading.Thread(target=self._poll, daemon=True)
            self.t.start()
        except Exception:
            self.nv = None
        return self

    def _poll(self):
        nv = self.nv
        get_reasons = getattr(nv, "nvmlDeviceGetCurrentClocksEventReasons", None) or \
            nv.nvmlDeviceGetCurrentClocksThrottleReasons
        while not self._stop.is_set():
            try:
                self.sm.append(float(nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM)))
                self.mask |= int(get_reasons(self.h))
            except Exception:
                pass
            time.sleep(self.period)

    def __exit__(self, *a):
        self._stop.set()
        if self.nv:
            self.t.join(timeout=2)
            try:
                self.nv.nvmlShutdown()
            except Exception:
                pass

    def summary(self):
        reasons = sorted(nm for bit, nm in self.REASONS.items() if self.mask & bit)
        return {"sm_mhz": statistics.median(self.sm) if self.sm else None, "sm_max_mhz": self.smax,
                "reasons": reasons, "samples": len(self.sm), "source": "NVML, 2 ms polling"}


def max_over_ranks(x, world):
    """The largest of the ranks' values of x: an all-reduce MAX over the
    process group (a device tensor with NCCL, a host tensor with gloo)."""
    if world <= 1:
        return float(x)
    import torch
    dev = "cuda" if torch.distributed.get_backend() == "nccl" else "cpu"
    t = torch.tensor([float(x)], dtype=torch.float64, device=dev)
    torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    return float(t.item())


def job_mpts_s(world, npts_per_rank, ms_step):
    """Whole-job throughput: every rank's points over the slowest rank's time."""
    return world * npts_per_rank / (ms_step * 1e-3) / 1e6


def workload(seed):
    from old_fmm_bem_b200 import geometry
    return geometry.bem_double_layer_problem(SUBDIV, seed=seed)


# ------------------------------------------------------------------ reference arm
def _ref_sample():
    """Bounded sample of the workload for the CPU reference: the same surface
    family at 4 subdivisions (5,120 triangles, 15,360 points), lmax 3."""
    from old_fmm_bem_b200 import geometry
    return geometry.bem_double_layer_problem(4, seed=1), 3


def _ref_worker(args):
    from oracle import pyoracle
    rep = args
    (x, n, q), lmax = _ref_sample()
    lo = x.min(axis=1)
    rd = float((x.max(axis=1) - lo).max() * (1 + 1e-5))
    t0 = time.perf_counter()
    for _ in range(rep):
        pyoracle.ref_fmm(x, x, q, neq=2, p=P_ORDER, lmax=lmax, sn=n, bbox=(lo[0], lo[1], lo[2], rd))
    return time.perf_counter() - t0, x.shape[1] * rep


def cpu_reference_time(workers, rep=1, pool=None):
    if pool is None:
        return _ref_worker(rep)
    res = pool.map(_ref_worker, [rep] * workers)
    return max(r[0] for r in res), sum(r[1] for r in res)


def run_reference_c2(args, rank, world):
    if rank != 0:
        return
    from oracle import pyoracle
    if not pyoracle.ref_available(P_ORDER):
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref reference library not built"}))
        return
    cores = os.cpu_count() or 1
    ctx = mp.get_context("spawn")
    with ctx.Pool(cores) as pool:
        for _ in range(args.warmup):
            cpu_reference_time(cores, 1, pool)
        t0 = time.perf_counter()
        pts = 0
        for _ in range(args.steps):
            dt, n = cpu_reference_time(cores, 1, pool)
            pts += n
        el = time.perf_counter() - t0
    value = pts / el / 1e6
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "Mpts/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * el / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": "Laplace Gnj double-layer matvec, icosphere r=1, p=10 (reference CPU fmm(), "
                                   "bounded sample: 4 subdivisions, 15,360 points, lmax 3, one process per core)",
                       "points_per_process": 15360, "processes": cores},
            "cpu_baseline": {"value": value, "unit": "Mpts/s", "cores": cores, "kind": "reference",
                             "sample": "reference fmm(ni,nj,2) at p=10 on a 15,360-point icosphere, one per core"},
            "e2e": {"value": value, "unit": "Mpts/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


def gaussian_clusters(n, seed, nclusters=32, sigma=0.02):
    """n points from nclusters Gaussian clusters (centres U[0.1, 0.9]^3, the
    given sigma) clipped to [0, 1]^3, and charges N(0, 1).  The first m points
    of a draw are a draw of m points of the same mixture (labels are iid)."""
    rng = np.random.default_rng(seed)
    c = rng.uniform(0.1, 0.9, (3, nclusters))
    lab = rng.integers(0, nclusters, n)
    x = np.clip(c[:, lab] + sigma * rng.standard_normal((3, n)), 0.0, 1.0).astype(np.float32)
    return x, rng.standard_normal(n).astype(np.float32)


def c3_problem(seed):
    """The headline point set, charges and backward weights w = dL/dpot."""
    x, q = gaussian_clusters(C3_N, seed)
    w = np.random.default_rng(seed + 1000).standard_normal(C3_N).astype(np.float32)
    return x, q, w


def _ref_c3_worker(job):
    """One reference forward + adjoint (fmm(ni,nj,0) with charges q, then with
    weights w; the position gradient w*grad(pot) + q*grad(psi) assembled in
    numpy) on points [a, b) of the C3 set.  Returns the seconds of the two
    fmm() calls without their tree builds (tfmm[0..13]) and the point count."""
    from oracle import pyoracle
    a, b, lmax = job
    x, q, w = c3_problem(C3_SEED)
    x, q, w = np.ascontiguousarray(x[:, a:b]), q[a:b].copy(), w[a:b].copy()
    el = 0.0
    for charges in (q, w):
        tm = np.zeros(100)
        t0 = time.perf_counter()
        v, g = pyoracle.ref_fmm(x, x, charges, neq=0, p=C3_P, lmax=lmax, bbox=(0, 0, 0, 1), timings=tm, perf=True)
        el += time.perf_counter() - t0 - float(tm[0:14].sum())
        if charges is q:
            field = g
    t0 = time.perf_counter()
    _dx = w * field + q * g
    el += time.perf_counter() - t0
    return el, b - a


def c3_reference_fit(pool):
    """One-core seconds of the reference forward + adjoint at 1/16, 1/4 and
    1/2 of the C3 points (run side by side, one process each), the linear fit
    t = a + b N through them and its value at the full N."""
    sizes = sorted(C3_REF_LMAX)
    res = pool.map(_ref_c3_worker, [(0, n, C3_REF_LMAX[n]) for n in sizes])
    secs = [r[0] for r in res]
    b, a = np.polyfit(np.asarray(sizes, float), np.asarray(secs), 1)
    t_full = a + b * C3_N
    return {"points": sizes, "lmax": [C3_REF_LMAX[n] for n in sizes], "one_core_s": secs,
            "fit": "t = a + b N (least squares)", "a_s": float(a), "b_s_per_point": float(b),
            "full_n_one_core_s": float(t_full), "full_n_one_core_mpts_s": C3_N / t_full / 1e6}


def run_reference(args, rank, world):
    """The reference's own CPU fmm() on the headline workload, all host cores
    (one process per core: the reference is serial).  A step runs every one of
    the 16 disjoint 65,536-point slices of the C3 point set through a
    reference forward + adjoint; after the timed steps, single runs at 1/4 and
    1/2 of the points give a linear fit to the full set."""
    if rank != 0:
        return
    from oracle import pyoracle
    if not pyoracle.ref_available(C3_P, perf=True):
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref reference library (p=12, perf) not built"}))
        return
    cores = os.cpu_count() or 1
    n_slice = C3_N // C3_REF_SLICES
    jobs = [(k * n_slice, (k + 1) * n_slice, C3_REF_LMAX[n_slice]) for k in range(C3_REF_SLICES)]
    ctx = mp.get_context("spawn")
    with ctx.Pool(min(cores, C3_REF_SLICES)) as pool:
        pool.map(_ref_c3_worker, [(0, 4096, 2)] * min(cores, C3_REF_SLICES))  # load the library in every worker
        for _ in range(args.warmup):
            pool.map(_ref_c3_worker, [(0, 4096, 2)] * min(cores, C3_REF_SLICES))
        walls, one_core = [], []
        for _ in range(args.steps):
            t0 = time.perf_counter()
            res = pool.map(_ref_c3_worker, jobs)
            walls.append(time.perf_counter() - t0)
            one_core.extend(r[0] for r in res)
        fit = c3_reference_fit(pool)
    ms_step = 1e3 * float(np.mean(walls))
    value = C3_N / (ms_step * 1e-3) / 1e6
    procs = min(cores, C3_REF_SLICES)
    line = {"impl": "reference", "metric": C3_METRIC, "value": value, "unit": "Mpts/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": "Laplace G forward + adjoint (charges and positions), 1,048,576 points from 32 "
                                   "Gaussian clusters (sigma 0.02) in [0,1]^3, q N(0,1), p=12: reference CPU fmm(), "
                                   "bounded sample = the point set cut into 16 disjoint slices of 65,536 points, one "
                                   "forward + adjoint each (depth 4), one process per core",
                       "points_per_step": C3_N, "slices": C3_REF_SLICES, "processes": procs,
                       "build": "reference sources, g++ -O3 -march=x86-64-v3 (oracle/Makefile perf)"},
            "one_core_s_per_slice": float(np.mean(one_core)),
            "full_n_fit": fit,
            "cpu_baseline": {"value": value, "unit": "Mpts/s", "cores": procs, "kind": "reference",
                             "sample": "reference fmm() forward + adjoint on 16 disjoint 65,536-point slices of the "
                                       "1,048,576-point C3 set per step, one process per core; full-N one-core time "
                                       "from the linear fit in full_n_fit"},
            "e2e": {"value": value, "unit": "Mpts/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line))


# ------------------------------------------------------------------ accuracy
def rel_err_vs_direct(ob, kernel, x_t, x_s, q, pot_fmm, grad_fmm=None, n_t=None, n_s=None, ntarget=1024, seed=7):
    """Relative 2-norm error of FMM potentials (and gradients) at `ntarget`
    random targets against the FP64 direct sum on the GPU (fmmb_direct_f64,
    itself checked against the oracle by the test suite), zero-distance pairs
    excluded and no softening, like the FMM plans measured here."""
    rng = np.random.default_rng(seed)
    sel = np.sort(rng.choice(x_t.shape[1], size=min(ntarget, x_t.shape[1]), replace=False))
    pd = ob.Plan(kernel=kernel, p=4, lmax=2, precision=ob.FP64, semantics=ob.SEM_ACCURATE, exclude_self=True)
    pd.set_geometry(np.ascontiguousarray(x_t[:, sel]), x_s,
                    np.ascontiguousarray(n_t[:, sel]) if n_t is not None else None, n_s)
    vd, gd = pd.direct(q)
    pd.close()
    out = {"pot": float(np.linalg.norm(pot_fmm[sel] - vd) / np.linalg.norm(vd)), "targets": int(len(sel))}
    if grad_fmm is not None and gd is not None:
        g = grad_fmm.reshape(3, -1)[:, sel]
        out["grad"] = float(np.linalg.norm(g - gd) / np.linalg.norm(gd))
    return out


def setup_line(plan, npts, ms_step):
    """Geometry setup of the plan (fmmb_get_setup_times): the octree build on
    the GPU against the HBM roofline of its algorithmic bytes -- per point,
    targets and sources alike: 12 B coordinates read + 4 B key written, 16 B
    (key + index, read and written) per 8-bit radix pass, 28 B gathered into
    sorted order -- and the whole fmmb_set_geometry (host-built tiles and work
    lists included); the matvec rate with one setup per matvec."""
    tree_ms, setup_ms = plan.setup_times()
    st = plan.stats()
    passes = (3 * st["lmax"] + 7) // 8
    nbytes = (st["ni"] + st["nj"]) * (16 + 16 * passes + 28)
    peaks, kind = measured_peaks()
    gbs = nbytes / (tree_ms * 1e-3) / 1e9
    return {"tree_build_ms": tree_ms, "set_geometry_ms": setup_ms, "tree_algorithmic_bytes": nbytes,
            "tree_gbs": gbs, "tree_frac_of_hbm": gbs / peaks.get("hbm_gbs", 6650.0),
            "mpts_s_with_setup_per_matvec": npts / ((ms_step + setup_ms) * 1e-3) / 1e6,
            "note": f"tree build = keys, radix sort, levels, lists (scratch from a stream-ordered pool, one host synchronisation for all level sizes); "
                    f"HBM peak {kind}"}


# ------------------------------------------------------------------ our arm
def phase_rooflines(plan, p, lmax, npts, phase, phase_alone, ms_step, mixed, traffic=None):
    """Rooflines of the two dominant kernels, from their CUDA-event durations
    in a step's launches run once more after an L2 flush (phase timers on the
    launching streams; phase_alone = with the near field run after the far
    field):
      * p2p_mixed: 20 flops per algorithmic pair (Laplace G: differences 3,
        r^2 6, rsqrt 1, r^-3 2, q r^-1 and q r^-3 2, potential 1, gradient 6;
        Gni/Gnj: the normal dot in place of the gradient); bound by the FP32
        pipes (peak 148 SMs x 128 lanes x 2 flops at the maximum SM clock);
      * M2L (translate_h16 / translate_tc + its pair-row reduction): 2 K^2
        algorithmic flops per box pair on the tensor cores; peak = the
        measured dense bf16 for the FP16 kernel (p <= 12: FP16 and BF16 run at
        the same rate), half of it (TF32) above; where the FP64 M2L runs (the
        FP64 form, p > 15, few box pairs) the flops of its two blocks and the
        nominal FP64 peak;
    and the whole matvec against the sum of its phases' roofline times
    (algorithmic work of each phase over the peak of the unit it runs on: P2P,
    P2M, L2P FP32; M2L FP16 or TF32; M2M, L2L FP64 at the nominal 37 TFLOP/s).
    traffic: DRAM bytes of one launch from an ncu capture, or None.
    Returns (dominant, other, matvec)."""
    st = plan.stats()
    peaks, peak_kind = measured_peaks()
    traffic = traffic or {}
    names = ["p2p", "p2m", "m2m", "m2l", "l2l", "l2p"]
    K = (p + 1) ** 2
    sm_max = float(peaks.get("sm_max_mhz", 1965.0))
    fp32_peak = 148 * 128 * 2 * sm_max * 1e6 / 1e12
    p2p_ach = 20.0 * st["p2p_pairs"] / (phase_alone[0] * 1e-3) / 1e12
    tc_peak = peaks["bf16_tflops"] if p <= 12 else peaks["bf16_tflops"] / 2  # FP16 / TF32 dense
    fp64_peak = 37.0
    # FP64 M2L: blocks of (p+1)(p+2)/2 and p(p+1)/2 rows; taken by the FP64 form, above p = 15 and, for K <= 169, by
    # geometries of few box pairs (few_pairs in csrc/api.cpp, whose limit this restates)
    par = not mixed or K > 256 or (K <= 169 and st["m2l_pairs"] * K * K <= 7e8)
    m2l_flops = 2.0 * (((p + 1) * (p + 2) // 2) ** 2 + (p * (p + 1) // 2) ** 2) if par else 2.0 * K * K
    if par:
        tc_peak = fp64_peak
    m2l_ach = m2l_flops * st["m2l_pairs"] / (phase_alone[3] * 1e-3) / 1e12
    roof_p2p = {"kernel": "p2p_mixed" if mixed else "p2p_f64", "bound": "fp32", "achieved": p2p_ach,
                "peak": fp32_peak, "unit": "TFLOP/s", "frac": p2p_ach / fp32_peak,
                "traffic": traffic.get("p2p_mixed"), "ms": float(phase_alone[0]),
                "ms_in_overlapped_step": float(phase[0]),
                "note": f"20 flops per algorithmic pair ({st['p2p_pairs']} pairs); ms = the kernel's own launches "
                        f"(near field not overlapped), summed per evaluate; peak = nominal FP32 at "
                        f"{sm_max:.0f} MHz (no FP32 figure in MEASURED_PEAKS.json); traffic per evaluate"}
    roof_m2l = {"kernel": "m2l_parity (M2L)" if par else
                "translate_h16+reduce_pairs (M2L)" if p <= 12 else "translate_tc+reduce_pairs (M2L)",
                "bound": "fp64 tensor" if par else "tensor",
                "achieved": m2l_ach, "peak": tc_peak, "unit": "TFLOP/s", "frac": m2l_ach / tc_peak,
                "traffic": traffic.get("translate_tc"), "ms": float(phase_alone[3]),
                "ms_in_overlapped_step": float(phase[3]),
                "note": f"{m2l_flops:.0f} flops of the even and odd blocks per box pair ({st['m2l_pairs']} pairs); "
                        f"peak = nominal FP64 of a B200" if par else
                        f"algorithmic 2*K^2 flops per box pair (K={K}, {st['m2l_pairs']} pairs); the tensor cores "
                        f"execute 3 FP16 MMAs per product (p <= 12; TF32 above) on operators padded to a multiple "
                        f"of 16 rows; peak = {peak_kind} dense bf16 (= FP16) for p <= 12, half of it (TF32) above; "
                        f"traffic per evaluate (translate + reduce_pairs)"}
    nb_i, nb_j = plan.tree(4), plan.tree(5)
    ideal = {"p2p": 20.0 * st["p2p_pairs"] / fp32_peak,
             "p2m": 2.0 * npts * K / fp32_peak,
             "m2m": 2.0 * K * K * float(nb_j[3:lmax + 1].sum()) / fp64_peak,
             "m2l": m2l_flops * st["m2l_pairs"] / tc_peak,
             "l2l": 2.0 * K * K * float(nb_i[3:lmax + 1].sum()) / fp64_peak,
             "l2p": 2.0 * npts * K / fp32_peak}
    ideal = {k: v / 1e9 for k, v in ideal.items()}  # flops / (TFLOP/s) -> ms
    matvec_roof = {"ideal_ms": ideal, "sum_ideal_ms": sum(ideal.values()), "step_ms": ms_step,
                   "frac_of_step": sum(ideal.values()) / ms_step,
                   "frac_per_phase_alone": {k: ideal[k] / float(phase_alone[i]) for i, k in enumerate(names)},
                   "note": "algorithmic flops per phase (P2P 20 per pair, P2M/L2P 2(p+1)^2 per point, M2L/M2M/L2L "
                           "2(p+1)^4 per box pair) over FP32 (nominal), FP16 (the measured bf16; TF32 = half of it "
                           "above p = 12) and FP64 (nominal 37) peaks"}
    dom = int(np.argmax(phase_alone[:6]))
    if names[dom] == "m2l":
        return roof_m2l, roof_p2p, matvec_roof
    return roof_p2p, roof_m2l, matvec_roof


def run_ours(args, rank, world, secondary=False):
    """The C2 workload (--config bem): Laplace Gnj double-layer matvec on the
    icosphere.  secondary: no CPU baseline, and a compact dict returned
    instead of the printed line (the headline line carries it)."""
    import torch
    import old_fmm_bem_b200 as ob

    dev = int(os.environ.get("LOCAL_RANK", 0))
    torch.cuda.set_device(dev)
    x, n, q = workload(seed=rank)
    npts = x.shape[1]
    stream = torch.cuda.Stream()
    plan = ob.Plan(kernel=ob.LAPLACE_GNJ, p=P_ORDER, lmax=LMAX, precision=ob.MIXED if args.precision == "mixed" else ob.FP64,
                   semantics=ob.SEM_ACCURATE, exclude_self=True)
    plan.set_stream(stream)
    xd, nd = torch.from_numpy(x).cuda(), torch.from_numpy(n).cuda()
    plan.set_geometry(xd, xd, source_normals=nd)
    qd = torch.from_numpy(q).cuda()
    pot = torch.zeros(npts, device="cuda")
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device="cuda")

    def step():
        plan.evaluate(qd, pot)

    with torch.cuda.stream(stream):
        for _ in range(args.warmup):
            step()
    torch.cuda.synchronize()
    if world > 1:
        torch.distributed.barrier()

    # device-resident timed region: per-step CUDA events on the plan's stream,
    # L2 flushed between steps (outside the events)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    phase = np.zeros(7)
    with ClockSampler(dev) as clk:
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for k in range(args.steps):
                flush.fill_(float(k))
                ev[k][0].record(stream)
                step()
                ev[k][1].record(stream)
                stream.synchronize()
                phase += np.array(list(_phases(plan, stream, flush).values()))
        torch.cuda.synchronize()
    ms = [a.elapsed_time(b) for a, b in ev]
    ms_step = float(np.mean(ms))
    phase /= args.steps
    launches = plan.stats()["launches"]
    # each kernel's own duration: the same steps with the near field run
    # after the far field instead of beside it (phase timers: CUDA events on the
    # launching stream around each phase of the step's launches run once more)
    plan.set_overlap(False)
    phase_alone = np.zeros(7)
    with torch.cuda.stream(stream):
        for _ in range(3):
            step()
        for k in range(args.steps):
            flush.fill_(float(k))
            step()
            stream.synchronize()
            phase_alone += np.array(list(_phases(plan, stream, flush).values()))
    phase_alone /= args.steps
    plan.set_overlap(True)
    ms_step = max_over_ranks(ms_step, world)

    # end to end through the public API with host (pinned) buffers: the copy of
    # the charges in and of the potentials out are inside the timed call
    qh = torch.from_numpy(q).pin_memory()
    ph = torch.zeros(npts).pin_memory()
    e2e = []
    for k in range(max(3, args.steps // 2)):
        flush.fill_(float(k))
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        plan.evaluate(qh.numpy(), ph.numpy())
        e2e.append(time.perf_counter() - t0)
    e2e_s = float(np.median(e2e))
    e2e_s = max_over_ranks(e2e_s, world)

    if rank != 0:
        plan.close()
        return
    pot64, _ = plan.evaluate(q, f64=True)
    err = rel_err_vs_direct(ob, ob.LAPLACE_GNJ, x, x, q, pot64, n_s=n)
    st = plan.stats()
    names = ["p2p", "p2m", "m2m", "m2l", "l2l", "l2p"]
    roof, roof2, matvec_roof = phase_rooflines(plan, P_ORDER, LMAX, npts, phase, phase_alone, ms_step,
                                               args.precision == "mixed", NCU_TRAFFIC["bem"])
    # CPU baseline: the reference's own fmm() on a bounded sample, one core
    cpu = None
    if not args.no_cpu and not secondary:
        try:
            from oracle import pyoracle
            if pyoracle.ref_available(P_ORDER):
                dt, npt = cpu_reference_time(1, rep=2)
                cpu = {"value": npt / dt / 1e6, "unit": "Mpts/s", "cores": 1, "kind": "reference",
                       "sample": "reference fmm(ni,nj,2) at p=10 on a 15,360-point icosphere (4 subdivisions, "
                                 "lmax 3), 2 runs, 1 core"}
        except Exception as e:  # the baseline is reported, not required
            cpu = {"error": str(e)}
    value = job_mpts_s(world, npts, ms_step)
    line = {
        "metric": METRIC, "value": value, "unit": "Mpts/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32+fp16x3+f64" if args.precision == "mixed" else "f64", "data": "synthetic",
        "config": {"workload": "Laplace Gnj double-layer BEM matvec, icosphere r=1, 81,920 triangles x 3 Gauss "
                               "points = 245,760 points, p=10, lmax=5, self pairs excluded",
                   "precision": args.precision, "points": npts, "p": P_ORDER, "lmax": LMAX,
                   "l2": "flushed between steps (256 MB write)", "parallelism": f"replicas x{world}"},
        "rel_err_vs_fp64_direct": err,
        "phase_ms": dict(zip(names + ["total"], [float(v) for v in phase])),
        "phase_ms_alone": dict(zip(names + ["total"], [float(v) for v in phase_alone])),
        "stats": st,
        "roofline": roof,
        "roofline_secondary": roof2,
        "matvec_roofline": matvec_roof,
        "cpu_baseline": cpu,
        "e2e": {"value": world * npts / e2e_s / 1e6, "unit": "Mpts/s", "h2d_bytes_per_step": 4 * npts,
                "d2h_bytes_per_step": 4 * npts},
        "gpu_launches": launches * args.steps,
        "setup": setup_line(plan, npts, ms_step),
        "clocks": clk.summary(),
    }
    plan.close()
    if secondary:
        return {k: line[k] for k in ("metric", "value", "unit", "ms_per_step", "dtype", "config",
                                     "rel_err_vs_fp64_direct", "phase_ms", "phase_ms_alone", "stats", "roofline",
                                     "roofline_secondary", "matvec_roofline", "e2e", "setup", "clocks")}
    print(json.dumps(line))


# ------------------------------------------------------------------ other configurations
def _timed(step, stream, steps, warmup, flush, out=None):
    """Mean CUDA-event time (ms) of `step` on `stream`, L2 flushed before each
    (the per-step times are appended to `out` when given)."""
    import torch
    with torch.cuda.stream(stream):
        for _ in range(warmup):
            step()
    torch.cuda.synchronize()
    ms = []
    with torch.cuda.stream(stream):
        for k in range(steps):
            flush.fill_(float(k))
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            step()
            b.record(stream)
            b.synchronize()
            ms.append(a.elapsed_time(b))
    if out is not None:
        out.extend(ms)
    return float(np.mean(ms))


def _phases(plan, stream, flush):
    """Phase times (ms) of the plan's last evaluate from a cold L2: timings()
    runs its launches once more on the plan's stream, here after a flush."""
    import torch
    with torch.cuda.stream(stream):
        flush.fill_(0.0)
    return plan.timings()


def uniform_cube(n, seed):
    rng = np.random.default_rng(seed)
    return rng.random((3, n), dtype=np.float32), rng.uniform(-1, 1, n).astype(np.float32)


def run_c1(args):
    """Plain Laplace G potential FMM in FP64: 32,768 points uniform in [0,1]^3,
    charges U[-1,1], p = 8, lmax 3 (64 points per leaf)."""
    import torch
    import old_fmm_bem_b200 as ob
    x, q = uniform_cube(32768, 11)
    stream = torch.cuda.Stream()
    plan = ob.Plan(kernel=ob.LAPLACE_G, p=8, lmax=3, precision=ob.FP64, semantics=ob.SEM_ACCURATE, exclude_self=True)
    plan.set_stream(stream)
    xd, qd = torch.from_numpy(x).cuda(), torch.from_numpy(q).cuda()
    plan.set_geometry(xd, xd, bbox=(0, 0, 0, 1))
    pot = torch.zeros(x.shape[1], device="cuda")
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device="cuda")
    with ClockSampler(int(os.environ.get("LOCAL_RANK", 0))) as clk:
        ms = _timed(lambda: plan.evaluate(qd, pot), stream, args.steps, max(3, args.warmup), flush)
    pot64, _ = plan.evaluate(q, f64=True)
    err = rel_err_vs_direct(ob, ob.LAPLACE_G, x, x, q, pot64)
    # the reference's own fmm() (oracle/_ref, p = 8, lmax = 3) on the same points, one core
    cpu = None
    if not args.no_cpu:
        from oracle import pyoracle
        if pyoracle.ref_available(8):
            t0 = time.perf_counter()
            pyoracle.ref_fmm(x, x, q, neq=0, p=8, lmax=3)
            dt = time.perf_counter() - t0
            cpu = {"value": x.shape[1] / dt / 1e6, "unit": "Mpts/s", "cores": 1, "kind": "reference",
                   "sample": "reference fmm(ni,nj,0) at p=8, lmax=3 on the same 32,768 points (reference semantics, "
                             "tree build included), one core"}
    print(json.dumps({"metric": "FMM matvec Mpts/s (Laplace G potential, 32,768 uniform points, p=8, FP64)",
                      "value": x.shape[1] / (ms * 1e-3) / 1e6, "unit": "Mpts/s", "n_gpus": 1, "steps": args.steps,
                      "ms_per_step": ms, "dtype": "f64", "data": "synthetic",
                      "config": {"workload": "Laplace G, 32,768 points U[0,1]^3, q U[-1,1], p=8, lmax=3, FP64, "
                                             "self pairs excluded"},
                      "rel_err_vs_fp64_direct": err, "phase_ms": _phases(plan, stream, flush), "cpu_baseline": cpu,
                      "clocks": clk.summary()}))
    plan.close()


def run_headline(args, rank, world):
    """The headline (C3): Laplace G as a torch.autograd operator on 1,048,576
    clustered points, p = 12; one step = forward + backward (gradients w.r.t.
    charges and positions of L = sum(w * pot)); mixed form timed over the
    driver's steps, the plain FP64 form beside it; octree depth of each form
    from fmmb_autotune_lmax.  Rank r runs its own point set (seed 13 + r)."""
    import torch
    import old_fmm_bem_b200 as ob
    from old_fmm_bem_b200.autograd import FMMOperator

    dev = int(os.environ.get("LOCAL_RANK", 0))
    torch.cuda.set_device(dev)
    x, q, w = c3_problem(C3_SEED + rank)
    n = x.shape[1]
    bbox = (0.0, 0.0, 0.0, 1.0)
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    xd = torch.from_numpy(x).cuda()
    qd = torch.from_numpy(q).cuda()
    wd = torch.from_numpy(w).cuda().to(torch.float64)
    kw = dict(kernel=ob.LAPLACE_G, p=C3_P, semantics=ob.SEM_ACCURATE, exclude_self=True, bbox=bbox)

    def make(prec):
        lmax, tune = ob.autotune_lmax(xd, xd, precision=prec, reps=2, **kw)
        X = xd.clone().requires_grad_(True)
        Q = qd.to(torch.float64).requires_grad_(True)
        op = FMMOperator(X, X, kernel=ob.LAPLACE_G, p=C3_P, lmax=lmax, precision=prec, bbox=bbox)
        box = {}

        def fwd():
            box["pot"] = op(Q)

        def fwd_bwd():
            X.grad = None
            Q.grad = None
            (op(Q) * wd).sum().backward()

        return op, X, Q, fwd, fwd_bwd, lmax, tune

    res = {}
    with ClockSampler(dev) as clk:
        # mixed form: the driver's steps
        op, X, Q, fwd, fwd_bwd, lmax, tune = make(ob.MIXED)
        t_f = _timed(fwd, stream, max(3, args.steps // 2), max(3, args.warmup), flush)
        per_step = []
        torch.cuda.nvtx.range_push("timed")  # the timed steps, for a profiler's launch list
        t_fb = _timed(fwd_bwd, stream, args.steps, max(3, args.warmup), flush, per_step)
        torch.cuda.nvtx.range_pop()
        ph = np.array(list(_phases(op.plan, stream, flush).values()))
        launches = op.plan.stats()["launches"]
    # each kernel's own duration: one evaluate with gradient, near field after
    # the far field (phase timers, CUDA events on the launching streams)
    op.plan.set_overlap(False)
    ph_alone = np.zeros(7)
    with torch.cuda.stream(stream):
        for _ in range(3):
            fwd()
        for k in range(max(3, args.steps // 2)):
            flush.fill_(float(k))
            fwd()
            stream.synchronize()
            ph_alone += np.array(list(_phases(op.plan, stream, flush).values()))
    ph_alone /= max(3, args.steps // 2)
    op.plan.set_overlap(True)
    t_fb_job = max_over_ranks(t_fb, world)

    # end to end through the C ABI with pinned host buffers: charges and
    # weights in, potential, charge gradient and position gradients out (the
    # forward's field stays on the device for the backward)
    plan = op.plan
    qh = torch.from_numpy(q).pin_memory()
    wh = torch.from_numpy(w).pin_memory()
    f64h = [torch.zeros(k * n, dtype=torch.float64).pin_memory() for k in (1, 1, 3, 3)]
    field_d = torch.empty(3 * n, dtype=torch.float64, device="cuda")
    e2e = []
    with torch.cuda.stream(stream):
        for k in range(max(3, args.steps // 2) + 2):
            flush.fill_(float(k))
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            plan.evaluate(qh.numpy(), f64h[0].numpy(), field_d, f64=True)
            plan.adjoint(qh.numpy(), wh.numpy(), field_d, f64h[1].numpy(), f64h[2].numpy(), f64h[3].numpy(),
                         want_dxs=True)
            e2e.append(time.perf_counter() - t0)
    e2e_s = max_over_ranks(float(np.median(e2e[2:])), world)

    # plain FP64 form, same step
    op64, X64, Q64, fwd64, fwd_bwd64, lmax64, tune64 = make(ob.FP64)
    t_f64 = _timed(fwd64, stream, min(args.steps, 5), 2, flush)
    t_fb64 = _timed(fwd_bwd64, stream, min(args.steps, 5), 2, flush)

    # C2 (the Gnj BEM matvec on the icosphere) as a secondary key
    c2 = run_ours(args, rank, world, secondary=True)

    if rank != 0:
        op.close()
        op64.close()
        return
    # accuracy on 1,024 random points against FP64 direct sums: potential,
    # field, charge gradient psi = A^T w and position gradient w grad(pot) +
    # q grad(psi), for both forms
    sel = np.sort(np.random.default_rng(7).choice(n, size=1024, replace=False))
    pd = ob.Plan(kernel=ob.LAPLACE_G, p=4, lmax=2, precision=ob.FP64, semantics=ob.SEM_ACCURATE, exclude_self=True)
    pd.set_geometry(np.ascontiguousarray(x[:, sel]), x)
    vd, gd = pd.direct(q)
    psid, gpsid = pd.direct(w)
    pd.close()
    dxd = w[sel] * gd + q[sel] * gpsid

    def rel(a, b):
        return float(np.linalg.norm(a - b) / np.linalg.norm(b))

    errs = {}
    for name, o in (("mixed", op), ("fp64", op64)):
        pot, field = o.plan.evaluate(q, f64=True)
        dq, dxt, dxs = o.plan.adjoint(q, w, field, want_dxs=True)
        dx = (dxt + dxs).reshape(3, -1)[:, sel]
        errs[name] = {"pot": rel(pot[sel], vd), "field": rel(field.reshape(3, -1)[:, sel], gd),
                      "dq": rel(dq[sel], psid), "dx": rel(dx, dxd), "targets": 1024}
    fd = c3_finite_differences(ob, x, q, w, lmax, ob.MIXED, args.fd)
    st = op.plan.stats()
    roof, roof2, matvec_roof = phase_rooflines(op.plan, C3_P, lmax, n, ph, ph_alone, t_f, True,
                                               NCU_TRAFFIC["adjoint1m"] if lmax == 6 else None)
    # CPU baseline: the reference's own forward + adjoint on one 65,536-point
    # slice of this point set, one core
    cpu = None
    if not args.no_cpu:
        try:
            from oracle import pyoracle
            if pyoracle.ref_available(C3_P, perf=True):
                el, npt = _ref_c3_worker((0, C3_N // C3_REF_SLICES, C3_REF_LMAX[C3_N // C3_REF_SLICES]))
                cpu = {"value": npt / el / 1e6, "unit": "Mpts/s", "cores": 1, "kind": "reference",
                       "sample": "reference fmm() forward + adjoint (two fmm(ni,nj,0) calls, tree builds excluded) "
                                 "at p=12, depth 4, on the first 65,536 points of this set, 1 core"}
        except Exception as e:  # the baseline is reported, not required
            cpu = {"error": str(e)}
    setup = setup_line(op.plan, n, t_f)
    op.close()
    op64.close()
    line = {
        "metric": C3_METRIC, "value": job_mpts_s(world, n, t_fb_job), "unit": "Mpts/s", "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": t_fb_job, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f32+fp16x3+f64", "data": "synthetic",
        "config": {"workload": "Laplace G FMM forward + backward (torch.autograd: gradients w.r.t. charges and "
                               "positions of sum(w*pot)), 1,048,576 points from 32 Gaussian clusters (sigma 0.02) in "
                               "[0,1]^3, q N(0,1), w N(0,1), p=12, mixed precision, self pairs excluded",
                   "points": n, "p": C3_P, "lmax": lmax, "lmax_fp64": lmax64, "precision": "mixed",
                   "l2": "flushed between steps (256 MB write)", "parallelism": f"replicas x{world}"},
        "rel_err_vs_fp64_direct": errs["mixed"],
        "rel_err_fp64_form": errs["fp64"],
        "finite_differences": fd,
        "forward_ms": t_f, "forward_backward_ms": t_fb, "backward_over_forward": (t_fb - t_f) / t_f,
        "ms_per_step_each": per_step,
        "fp64_form": {"lmax": lmax64, "forward_ms": t_f64, "forward_backward_ms": t_fb64,
                      "backward_over_forward": (t_fb64 - t_f64) / t_f64, "autotune_ms": tune64},
        "mixed_over_fp64": t_fb64 / t_fb,
        "autotune_ms": tune,
        "phase_ms": dict(zip(["p2p", "p2m", "m2m", "m2l", "l2l", "l2p", "total"], [float(v) for v in ph])),
        "phase_ms_alone": dict(zip(["p2p", "p2m", "m2m", "m2l", "l2l", "l2p", "total"],
                                   [float(v) for v in ph_alone])),
        "stats": st,
        "roofline": roof,
        "roofline_secondary": roof2,
        "matvec_roofline": matvec_roof,
        "cpu_baseline": cpu,
        "e2e": {"value": world * n / e2e_s / 1e6, "unit": "Mpts/s", "ms": 1e3 * e2e_s,
                "h2d_bytes_per_step": 16 * n, "d2h_bytes_per_step": 64 * n,
                "note": "fmmb_evaluate_f64 (q in; potential out, field kept on the device) + fmmb_adjoint_f64 "
                        "(q, w in; dq, dL/dx_t, dL/dx_s out), pinned host buffers"},
        "gpu_launches": (2 * launches + 2) * args.steps,
        "setup": setup,
        "c2_bem_gnj": c2,
        "clocks": clk.summary(),
    }
    print(json.dumps(line))


def c3_finite_differences(ob, x, q, w, lmax, prec, ncoord, h=1e-4):
    """Central differences of L = sum(w * pot) w.r.t. ncoord random
    coordinates (step h; each side a fresh tree on the moved point set)
    against the backward's position gradient, in the given form.  The
    coordinates are drawn among points with no neighbour closer than 30 h
    (the difference quotient's O(h^2 / r^2) truncation stays below 1e-3)."""
    if ncoord <= 0:
        return None
    rng = np.random.default_rng(11)
    x64 = x.astype(np.float64)
    pts, dims = [], []
    while len(pts) < ncoord:
        i = int(rng.integers(0, x.shape[1]))
        r2 = ((x64 - x64[:, i:i + 1]) ** 2).sum(0)
        r2[i] = np.inf
        if r2.min() >= (30 * h) ** 2 and i not in pts:
            pts.append(i)
            dims.append(int(rng.integers(0, 3)))
    pts, dims = np.array(pts), np.array(dims)
    plan = ob.Plan(kernel=ob.LAPLACE_G, p=C3_P, lmax=lmax, precision=prec, semantics=ob.SEM_ACCURATE,
                   exclude_self=True)
    bbox = (0.0, 0.0, 0.0, 1.0)
    plan.set_geometry(x, x, bbox=bbox)
    pot, field = plan.evaluate(q, f64=True)
    _, dxt, dxs = plan.adjoint(q, w, field, want_dxs=True)
    grad = (dxt + dxs).reshape(3, -1)
    t0 = time.perf_counter()
    fdv = np.zeros(ncoord)
    xm = x.copy()
    w64 = w.astype(np.float64)
    for k, (i, d) in enumerate(zip(pts, dims)):
        vals = []
        for sgn in (1.0, -1.0):
            xm[d, i] = np.float32(x[d, i] + sgn * h)
            plan.set_geometry(xm, xm, bbox=bbox)
            vals.append(float(w64 @ plan.evaluate(q, f64=True)[0]))
        hh = float(np.float32(x[d, i] + h)) - float(np.float32(x[d, i] - h))  # the float32 step taken
        xm[d, i] = x[d, i]
        fdv[k] = (vals[0] - vals[1]) / hh
    an = grad[dims, pts]
    plan.close()
    return {"coordinates": ncoord, "h": h, "rel_err": float(np.linalg.norm(fdv - an) / np.linalg.norm(an)),
            "max_abs_rel": float(np.max(np.abs(fdv - an) / np.maximum(np.abs(an), 1e-30))),
            "seconds": time.perf_counter() - t0,
            "note": "central differences of sum(w * pot) over fresh trees, against the backward's dL/dx; points "
                    "with no neighbour closer than 30 h"}


def run_c4(args):
    """Batched BEM: 64 independent unit-sphere problems with triangle counts
    log-uniform in [2k, 200k] (seeded), one point per triangle (centroid,
    outward normal, panel area); for Gni and for Gnj the systems
    diag x + K(area/e1 .* x) = b with 8 right-hand sides U[-1, 1] each, 20
    GMRES iterations (fmmb_gmres, restart 30).  All 64 x 8 systems share the
    launches of one forest plan (fmmb_set_geometry_batch), every right-hand
    side replayed as a CUDA graph; one depth for the forest from
    fmmb_autotune_lmax_batch.  p = 10, mixed precision."""
    import torch
    import old_fmm_bem_b200 as ob
    from old_fmm_bem_b200 import geometry
    probs = geometry.bem_batch_problems(64, seed=17)
    off = np.cumsum([0] + [p[0].shape[1] for p in probs]).astype(np.int32)
    x = np.ascontiguousarray(np.concatenate([p[0] for p in probs], axis=1))
    nrm = np.ascontiguousarray(np.concatenate([p[1] for p in probs], axis=1))
    weight = (np.concatenate([p[2] for p in probs]) / geometry.E1).astype(np.float32)
    n, nrhs, iters = x.shape[1], 8, 20
    bbox = (-1.0001, -1.0001, -1.0001, 2.0002)
    xd, nd, wd = torch.from_numpy(x).cuda(), torch.from_numpy(nrm).cuda(), torch.from_numpy(weight).cuda()
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    rng = np.random.default_rng(23)
    b = torch.from_numpy(rng.uniform(-1, 1, nrhs * n)).cuda()
    res = {}
    total_ms = 0.0
    with ClockSampler(int(os.environ.get("LOCAL_RANK", 0))) as clk:
        for name, kernel in (("gni", ob.LAPLACE_GNI), ("gnj", ob.LAPLACE_GNJ)):
            tn, sn = (nd, None) if kernel == ob.LAPLACE_GNI else (None, nd)
            kw = dict(kernel=kernel, p=P_ORDER, precision=ob.MIXED, semantics=ob.SEM_ACCURATE, exclude_self=True)
            if args.lmax:
                lmax, tune = args.lmax, None
            else:
                lmax, tune = ob.autotune_lmax_batch(off, xd, off, xd, target_normals=tn, source_normals=sn,
                                                    bbox=bbox, lmin=3, lmax=6, reps=1, nrhs=nrhs, **kw)
            plan = ob.Plan(lmax=lmax, nrhs=nrhs, **kw)
            plan.set_stream(stream)
            t0 = time.perf_counter()
            plan.set_geometry_batch(off, xd, off, xd, tn, sn, bbox=bbox)
            torch.cuda.synchronize()
            tree_s = time.perf_counter() - t0
            X = torch.zeros(nrhs * n, dtype=torch.float64, device="cuda")
            box = {}

            def solve():
                X.zero_()
                box["out"] = plan.gmres(b, X, wd, diag=geometry.BEM_DIAG, precond=1 / geometry.BEM_DIAG, restart=30,
                                        max_iter=iters)

            per_step = []
            ms = _timed(solve, stream, max(1, min(args.steps, 3)), max(3, min(args.warmup, 3)), flush, per_step)
            _, it, resid = box["out"]
            # one matvec against the per-problem FP64 direct sum (first right-hand side, 1024 targets of
            # each of the four largest problems)
            q1 = (weight * rng.uniform(-1, 1, n)).astype(np.float32)
            q8 = np.tile(q1, nrhs)
            pot, _ = plan.evaluate(q8, f64=True)
            errs = []
            for k in np.argsort(np.diff(off))[-4:]:
                i0 = int(off[k])
                i1 = min(int(off[k + 1]), i0 + 1024)
                vd, _ = plan.direct(q8, i0, i1)
                errs.append(float(np.linalg.norm(pot[i0:i1] - vd) / np.linalg.norm(vd)))
            matvecs = iters + 1  # the initial residual and one per iteration
            res[name] = {"lmax": lmax, "autotune_ms_per_matvec": tune, "tree_build_s": tree_s, "solve_ms": ms,
                         "solve_ms_per_step": per_step,
                         "iterations": it, "matvecs": matvecs, "matvec_ms": ms / matvecs,
                         "max_rel_resid": float(np.max(resid)), "median_rel_resid": float(np.median(resid)),
                         "rel_err_vs_fp64_direct": float(np.sqrt(np.mean(np.square(errs)))),
                         "gpu_launches_per_matvec": plan.stats()["launches"]}
            total_ms += ms
            plan.close()
    pts = 2 * n * nrhs * (iters + 1)
    print(json.dumps({"metric": "batched BEM GMRES: FMM matvec Mpts/s (64 unit-sphere problems, 8 RHS, Gni + Gnj)",
                      "value": pts / (total_ms * 1e-3) / 1e6, "unit": "Mpts/s", "n_gpus": 1,
                      "steps": max(1, min(args.steps, 3)), "ms_per_step": total_ms, "dtype": "f32+fp16x3+f64",
                      "data": "synthetic",
                      "config": {"workload": f"64 geodesic unit spheres, {n} centroid points in all "
                                             f"({int(np.diff(off).min())}..{int(np.diff(off).max())} per problem), "
                                             "Gni and Gnj BEM systems (diag (e1+e2)/(2e1(e1-e2)), weights area/e1, "
                                             "e1=4, e2=20), 8 RHS U[-1,1], 20 GMRES iterations, p=10 mixed; step = "
                                             "both solves", "l2": "flushed between steps"},
                      "results": res, "clocks": clk.summary()}))



def run_c4_matvec(args):
    """The batched matvec of batch64 alone: the same 64 problems and forest
    plan (Gni, p = 10, mixed, depth --lmax or 3) with 1 and with 8 right-hand
    sides; CUDA-event time per evaluate (3 warm-up, 5 timed, L2 flushed)."""
    import torch
    import old_fmm_bem_b200 as ob
    from old_fmm_bem_b200 import geometry
    probs = geometry.bem_batch_problems(64, seed=17)
    off = np.cumsum([0] + [p[0].shape[1] for p in probs]).astype(np.int32)
    x = torch.from_numpy(np.ascontiguousarray(np.concatenate([p[0] for p in probs], axis=1))).cuda()
    nrm = torch.from_numpy(np.ascontiguousarray(np.concatenate([p[1] for p in probs], axis=1))).cuda()
    n = int(off[-1])
    bbox = (-1.0001, -1.0001, -1.0001, 2.0002)
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    lmax = args.lmax or 3
    res = {}
    for nrhs in (1, 8):
        plan = ob.Plan(kernel=ob.LAPLACE_GNI, p=P_ORDER, lmax=lmax, nrhs=nrhs, precision=ob.MIXED,
                       semantics=ob.SEM_ACCURATE, exclude_self=True)
        plan.set_stream(stream)
        plan.set_geometry_batch(off, x, off, x, nrm, None, bbox=bbox)
        q = torch.from_numpy(np.random.default_rng(5).uniform(-1, 1, nrhs * n).astype(np.float32)).cuda()
        pot = torch.zeros(nrhs * n, dtype=torch.float32, device="cuda")
        ms = _timed(lambda: plan.evaluate(q, pot), stream, 5, 3, flush)
        res[f"rhs{nrhs}"] = {"ms_per_evaluate": ms, "mpts_s": nrhs * n / (ms * 1e-3) / 1e6,
                             "launches": plan.stats()["launches"]}
        plan.close()
    print(json.dumps({"metric": "batched BEM matvec Mpts/s (64 unit-sphere problems, Gni, p=10, 1 and 8 RHS)",
                      "value": res["rhs8"]["mpts_s"], "unit": "Mpts/s", "n_gpus": 1, "steps": 5,
                      "dtype": "f32+fp16x3+f64", "data": "synthetic",
                      "config": {"workload": f"64 geodesic unit spheres, {n} centroids, Gni, depth {lmax}",
                                 "l2": "flushed between steps"}, "results": res}))


def run_c5(args):
    """Complex Helmholtz e^{ikr}/(4 pi r): 1,048,576 points uniform on the unit
    sphere, complex charges with parts U[-1, 1], k = 5, p = 16; one step = the
    matvec and its adjoint w.r.t. the charges (A^T w, the transposed plan);
    mixed (FP32 complex P2P) and FP64 forms, octree depth from
    fmmb_autotune_lmax for each; rel err of the potential against the FP64
    complex direct sum (fmmb_direct_f64) on 1,024 targets."""
    import torch
    import old_fmm_bem_b200 as ob
    from oracle import helmholtz_oracle as ho
    n, k, p = 1 << 20, 5.0, 16
    x, q = ho.sphere_points(n, 29)
    w = ho.sphere_points(n, 31)[1]
    bbox = (-1.0001, -1.0001, -1.0001, 2.0002)
    xd = torch.from_numpy(x).cuda()
    qd = torch.from_numpy(q).cuda()
    wd = torch.from_numpy(w).cuda()
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device="cuda")
    stream = torch.cuda.current_stream()
    steps = max(1, min(args.steps, 3))
    res = {}
    sel = np.sort(np.random.default_rng(3).choice(n, 1024, replace=False))
    with ClockSampler(int(os.environ.get("LOCAL_RANK", 0))) as clk:
        for name, prec in (("mixed", ob.MIXED), ("fp64", ob.FP64)):
            kw = dict(kernel=ob.HELMHOLTZ_G, p=p, precision=prec, semantics=ob.SEM_ACCURATE, exclude_self=True)
            lmax, tune = (args.lmax, None) if args.lmax else _autotune_helm(ob, xd, bbox, kw, k)
            plan = ob.Plan(lmax=lmax, wavenumber=k, **kw)
            t0 = time.perf_counter()
            plan.set_geometry(xd, xd, bbox=bbox)
            torch.cuda.synchronize()
            setup_s = time.perf_counter() - t0
            pot = torch.zeros(n, dtype=torch.complex128, device="cuda")
            adj = torch.zeros(n, dtype=torch.complex128, device="cuda")
            plan.evaluate_transpose(wd, adj, f64=True)  # builds the transposed plan
            t_f = _timed(lambda: plan.evaluate(qd, pot, f64=True), stream, steps, 2, flush)
            t_fa = _timed(lambda: (plan.evaluate(qd, pot, f64=True), plan.evaluate_transpose(wd, adj, f64=True)),
                          stream, steps, 2, flush)
            # accuracy on 1,024 targets against the FP64 direct sum (a plan over those targets)
            dp = ob.Plan(kernel=ob.HELMHOLTZ_G, p=4, lmax=2, semantics=ob.SEM_ACCURATE, exclude_self=True, wavenumber=k)
            dp.set_geometry(np.ascontiguousarray(x[:, sel]), x, bbox=bbox)
            vd, _ = dp.direct(q)
            dp.close()
            v = pot.cpu().numpy()[sel]
            st = plan.stats()
            ph = _phases(plan, stream, flush)
            fl = 6 * (((p + 1) * (p + 2) // 2) ** 2 + (p * (p + 1) // 2) ** 2)  # even and odd block, 3 real products
            m2l_tf = fl * st["m2l_pairs"] / (ph["m2l"] * 1e-3) / 1e12
            res[name] = {"lmax": lmax, "autotune_ms": tune, "setup_s": setup_s, "matvec_ms": t_f,
                         "matvec_plus_adjoint_ms": t_fa, "phase_ms": ph, "stats": st,
                         "m2l_roofline": {"kernel": "m2l_parity (M2L)", "bound": "fp64 tensor",
                                          "achieved": m2l_tf, "peak": 37.0, "unit": "TFLOP/s",
                                          "frac": m2l_tf / 37.0,
                                          "note": f"{fl} flops of the even and odd blocks, three real products "
                                                  f"each, per box pair ({st['m2l_pairs']} pairs) over the M2L phase "
                                                  "time (P2P overlapped on the side stream); peak = nominal FP64 of "
                                                  "a B200"},
                         "rel_err_vs_fp64_direct": float(np.linalg.norm(v - vd) / np.linalg.norm(vd))}
            plan.close()
    m = res["mixed"]
    print(json.dumps({"metric": "FMM matvec Mpts/s (complex Helmholtz G, 1,048,576 points on the unit sphere, k=5, "
                                "p=16)",
                      "value": n / (m["matvec_ms"] * 1e-3) / 1e6, "unit": "Mpts/s", "n_gpus": 1, "steps": steps,
                      "ms_per_step": m["matvec_ms"], "dtype": "c64 P2P + f64", "data": "synthetic",
                      "config": {"workload": "complex Helmholtz e^{ikr}/(4 pi r), 1,048,576 points uniform on the unit "
                                             "sphere, q with re/im U[-1,1], k=5 (kD=10), p=16; adjoint = A^T w",
                                 "l2": "flushed between steps"},
                      "results": res, "mixed_speedup_over_fp64": res["fp64"]["matvec_ms"] / m["matvec_ms"],
                      "clocks": clk.summary()}))


def _autotune_helm(ob, xd, bbox, kw, k):
    """fmmb_autotune_lmax for the Helmholtz plan (depths 3..5)."""
    import ctypes
    lib = ob.load()
    cfg = ob._Config()
    lib.fmmb_config_init(ctypes.byref(cfg))
    cfg.kernel, cfg.p, cfg.precision, cfg.semantics = kw["kernel"], kw["p"], kw["precision"], kw["semantics"]
    cfg.exclude_self, cfg.wavenumber = 1, k
    best = ctypes.c_int(-1)
    ms = np.zeros(3, np.float32)
    bb = np.asarray(bbox, np.float32)
    ptr = [xd[i].data_ptr() for i in range(3)]
    n = xd.shape[1]
    rc = lib.fmmb_autotune_lmax(ctypes.byref(cfg), n, *ptr, None, None, None, n, *ptr, None, None, None,
                                bb.ctypes.data, 3, 5, 1, ctypes.byref(best), ms.ctypes.data)
    if rc != 0:
        raise RuntimeError(lib.fmmb_last_error().decode())
    return best.value, {l: float(ms[l - 3]) for l in range(3, 6)}


def run_c3_matvec(args):
    """One matvec of the headline workload alone: the mixed Laplace G
    evaluate with its field on the 1,048,576 clustered points at p = 12,
    depth --lmax (default 6, the autotuner's choice there), phases serialised
    (the near field after the far field) so that each kernel's CUDA-event
    time is its own; --warmup untimed and --steps timed evaluates, L2 flushed
    between them.  The launch order of one evaluate is fixed (P2P first half,
    P2M, M2M, M2L, P2P second half, L2L, L2P), which is what a profiler's
    launch skip counts on."""
    import torch
    import old_fmm_bem_b200 as ob
    x, q, _ = c3_problem(C3_SEED)
    n = x.shape[1]
    lmax = args.lmax or 6
    flush = torch.empty(L2_FLUSH_BYTES // 4, dtype=torch.float32, device="cuda")
    stream = torch.cuda.Stream()
    xd = torch.from_numpy(x).cuda()
    qd = torch.from_numpy(q).cuda()
    pot = torch.zeros(n, dtype=torch.float64, device="cuda")
    grad = torch.zeros(3 * n, dtype=torch.float64, device="cuda")
    plan = ob.Plan(kernel=ob.LAPLACE_G, p=C3_P, lmax=lmax, precision=ob.MIXED, semantics=ob.SEM_ACCURATE,
                   exclude_self=True)
    plan.set_stream(stream)
    plan.set_geometry(xd, xd, bbox=(0.0, 0.0, 0.0, 1.0))
    plan.set_overlap(False)

    def step():
        plan.evaluate(qd, pot, grad, f64=True)

    ms = _timed(step, stream, args.steps, args.warmup, flush)
    ph = np.array(list(_phases(plan, stream, flush).values()))
    st = plan.stats()
    plan.close()
    print(json.dumps({"metric": "FMM matvec Mpts/s (Laplace G with field, 1,048,576 clustered points, p=12, "
                                "phases serialised)",
                      "value": n / (ms * 1e-3) / 1e6, "unit": "Mpts/s", "n_gpus": 1, "steps": args.steps,
                      "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True,
                      "dtype": "f32+fp16x3+f64", "data": "synthetic",
                      "config": {"workload": "the headline point set, one mixed evaluate with field", "lmax": lmax,
                                 "l2": "flushed between steps"},
                      "phase_ms_last": dict(zip(["p2p", "p2m", "m2m", "m2l", "l2l", "l2p", "total"],
                                                [float(v) for v in ph])),
                      "stats": st}))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--precision", default="mixed", choices=["mixed", "fp64"])
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline")
    ap.add_argument("--lmax", type=int, default=0,
                    help="batch64 / helmholtz1m / c3_matvec: this octree depth instead of the autotuner's")
    ap.add_argument("--fd", type=int, default=64, help="adjoint1m: finite-difference coordinates (0: none)")
    ap.add_argument("--config", default="adjoint1m", choices=["bem", "uniform32k", "adjoint1m", "c3_matvec",
                                                           "batch64", "batch64_matvec", "helmholtz1m"],
                    help="adjoint1m: the headline, Laplace G forward + backward on 1,048,576 clustered points, p=12 "
                         "(default); c3_matvec: one mixed evaluate of that workload, phases serialised; "
                         "bem: the Gnj BEM matvec on a 245,760-point icosphere; uniform32k: FP64 Laplace G "
                         "on 32,768 uniform points; batch64: GMRES on 64 "
                         "BEM problems x 8 right-hand sides; batch64_matvec: its matvec alone, 1 and 8 "
                         "right-hand sides; helmholtz1m: complex Helmholtz, "
                         "1,048,576 sphere points, k=5, p=16")
    args = ap.parse_args()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    if world > 1 and args.impl == "ours":
        import datetime

        import torch
        torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", 0)))
        torch.distributed.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    if args.impl == "reference":
        if args.config == "bem":
            run_reference_c2(args, rank, world)
        else:
            run_reference(args, rank, world)
    elif args.config == "uniform32k":
        run_c1(args)
    elif args.config == "adjoint1m":
        run_headline(args, rank, world)
    elif args.config == "c3_matvec":
        run_c3_matvec(args)
    elif args.config == "batch64":
        run_c4(args)
    elif args.config == "batch64_matvec":
        run_c4_matvec(args)
    elif args.config == "helmholtz1m":
        run_c5(args)
    else:
        run_ours(args, rank, world)  # bem
    if world > 1 and args.impl == "ours":
        import torch
        torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
