#!/usr/bin/env python
"""Benchmark: RPY M.f applies per right-hand side, reported as ns per particle
per right-hand side (lower is better), FP32-batched operator on one GB300.

Workload (default "large"): N = 1e6 particles uniform in a periodic box
L = 480, radius a = 1, xi = 0.3, rc = 10, mesh K = 256, B-spline order p = 6,
R = 16 right-hand sides i.i.d. N(0,1).  A step is one drop-in style apply
with new positions: positions -> B-spline records + tile sort + cell list,
then M = M_recip + M_real + M_self applied to all 16 right-hand sides in one
48-component mesh pass.  Inputs are seeded synthetic data (the reference
ships no dataset).  Every timed step reads and writes buffers far larger
than the 129 MB L2 (the FP32 mesh alone is 3.2 GB), so no flush is needed.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl gb300|reference]

--impl reference times the reference's CPU path for the same workload on
the host cores (the reference compiled from its sources where available,
else the oracle's C restatement of it) and prints the same JSON line.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "RPY M·f applies/s/RHS (ns/particle), FP32-batched vs FP64, rel-L2 ≤1e-5"
UNIT = "ns/particle/RHS"

WORKLOADS = {
    "large": dict(N=1_000_000, L=480.0, K=256, p=6, R=16, xi=0.3, rc=10.0, a=1.0),
    "multi_rhs": dict(N=200_000, L=250.0, K=160, p=6, R=16, xi=0.3, rc=10.0, a=1.0),
    "scale_up": dict(N=100_000, L=220.0, K=128, p=6, R=1, xi=0.3, rc=10.0, a=1.0),
    # 64 systems, N log-uniform in [500, 50000], phi = 0.05, K = next 2^a3^b5^c >= 0.6 L,
    # p in {4, 6, 8}, R = 4 (one CUDA-graph launch vs a per-system loop)
    "uneven_batch": dict(count=64, R=4, xi=0.3, rc=10.0, a=1.0),
}

# DRAM traffic per launch over algorithmic bytes, (dram__bytes_read.sum +
# dram__bytes_write.sum) / algorithmic bytes, from one-kernel ncu captures of small
# cases of the same kernels (FP32, 48 or 24 components; inputs larger than L2):
# spread and interpolation at N = 2e5, K = 160, R = 16, tile 16x8x4; the fused
# z-FFT/influence kernel at K = 256, R = 8.  A full launch's traffic is estimated
# as the ratio times its algorithmic bytes (the spread and z-FFT traffic grows in
# proportion; the interpolation's halo re-reads grow with the mesh, so its
# estimate is a lower bound).
NCU_TRAFFIC_RATIO = {"spread": 1.019, "influence": 0.982, "interp": 1.802}


def algorithmic_bytes(w, s=4):
    """Bytes each kernel must move at minimum (per launch)."""
    K, N, C = w["K"], w["N"], 3 * w["R"]
    Kr, Kc = K ** 3, K * K * (K // 2 + 1)
    return {
        "spread": C * s * Kr + s * C * N,          # mesh written once, forces read
        "influence": C * 4 * s * Kc + 2 * s * Kc,  # complex mesh read+write, table once
        "interp": C * s * Kr + s * C * N,          # mesh read once, result written
    }


def peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as fh:
            d = json.load(fh)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6800.0, "fallback"


class Clocks:
    """nvidia-smi samples during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.fh = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index), "--query-gpu=" + self.FIELDS,
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=self.fh, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        self.fh.close()
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        with open(self.path) as fh:
            for line in fh:
                parts = [x.strip() for x in line.split(",")]
                if len(parts) < 9:
                    continue
                try:
                    sm.append(float(parts[1]))
                    smax.append(float(parts[2]))
                except ValueError:
                    continue
                for nm, v in zip(names, parts[5:9]):
                    if v.lower().startswith("active"):
                        reasons.add(nm)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(smax),
                "reasons": sorted(reasons), "samples": len(sm)}


def synth(w, seed):
    rng = np.random.default_rng(seed)
    pos = rng.uniform(0.0, w["L"], size=(w["N"], 3))
    f = rng.standard_normal((w["R"], 3 * w["N"])).astype(np.float32)
    return pos, f


def dist_env():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return ws, rank, local


def _ref_lib_available():
    import oracle
    oracle.build(reference=True)
    return os.path.exists(oracle.REF_COLORED_SO)


def _real_self_time(w, pos, f1, nth, reps):
    """The real-space + self part (absent from the reference): the oracle's
    FP64 restatement of Beenakker's sum, best of `reps`."""
    import oracle
    best = None
    for _ in range(reps):
        t0 = time.perf_counter()
        oracle.real_self(pos, w["L"], w["xi"], w["rc"], f1, radius=w["a"], nthreads=nth)
        dt = time.perf_counter() - t0
        best = dt if best is None else min(best, dt)
    return best


def _reference_recip_time(w, pos, f1, nth, reps, colored=True):
    """The reference's own compute_spme (old-version/spme.c:560-726) on `nth`
    OpenMP threads, one right-hand side of the full system with new positions
    (its P build included), best of `reps`; returns (seconds, its phase timers)."""
    import oracle
    ref = oracle.Reference(w["xi"], w["K"], w["p"], w["N"], w["L"], nthreads=nth,
                           colored=colored)
    best, phases = None, {}
    try:
        for _ in range(reps):
            v = np.zeros((1, 3 * w["N"]))
            t0 = time.perf_counter()
            _, ph = ref.compute_with_timers(pos, 1, 1.0, f1, 3 * w["N"], 0.0, v, 3 * w["N"])
            dt = time.perf_counter() - t0
            if best is None or dt < best:
                best, phases = dt, ph
    finally:
        ref.close()
    return best, phases


def cpu_baseline_time(w, nth=None, single_thread=True):
    """CPU baseline of the full operator on the host cores, one right-hand side of
    the whole system per rep (a step's work at R = 1):
    * reciprocal part: the reference's own compute_spme, compiled unmodified from
      its sources (coloured OpenMP spread), all cores, best of 2; the FFT phases
      (the project's DFTI shim standing in for MKL) reported separately from the
      reference's own timers; once more on 1 thread;
    * real-space + self part: the oracle's restatement (the reference has none).
    Where the reference build is absent, the oracle's restatement of the
    reciprocal path stands in (kind "port")."""
    import oracle
    oracle.build(reference=True)
    pos, f = synth(w, seed=99)
    f1 = f[:1].astype(np.float64)
    nth = nth or (os.cpu_count() or 1)
    N = w["N"]
    t_rs = _real_self_time(w, pos, f1, nth, 2)
    out = {"unit": UNIT, "cores": nth}
    if _ref_lib_available():
        t_rec, ph = _reference_recip_time(w, pos, f1, nth, 2)
        out.update({
            "kind": "reference",
            "value": (t_rec + t_rs) * 1e9 / N,
            "sample": f"1 right-hand side of the full N={N} system per rep, best of 2: the "
                      "reference's compute_spme compiled unmodified (coloured OpenMP spread, "
                      "project DFTI shim for MKL) + the oracle's real-space/self sum (absent "
                      "from the reference)",
            "reference_recip_ns": t_rec * 1e9 / N,
            "port_real_self_ns": t_rs * 1e9 / N,
            "reference_phases_s": ph,
            "fft_phase_ns": (ph.get("forward_fft", 0.0) + ph.get("backward_fft", 0.0)) * 1e9 / N,
        })
        if single_thread:
            # the reference's reciprocal path alone on 1 thread (one rep, ~10-20 s at
            # N = 1e6); the real-space restatement is not the reference's code
            t1, ph1 = _reference_recip_time(w, pos, f1, 1, 1)
            out["single_thread"] = {
                "cores": 1, "reference_recip_ns": t1 * 1e9 / N, "reference_phases_s": ph1,
                "fft_phase_ns": (ph1.get("forward_fft", 0.0) + ph1.get("backward_fft", 0.0))
                * 1e9 / N}
    else:
        best = None
        for _ in range(2):
            t0 = time.perf_counter()
            oracle.recip(pos, w["L"], w["xi"], w["K"], w["p"], f1, radius=w["a"], nthreads=nth)
            dt = time.perf_counter() - t0
            best = dt if best is None else min(best, dt)
        out.update({"kind": "port", "value": (best + t_rs) * 1e9 / N,
                    "sample": f"1 right-hand side of the full N={N} system per rep, best of 2; "
                              "the oracle's FP64 restatement of the reference path + real-space/"
                              "self (reference build absent)",
                    "port_recip_ns": best * 1e9 / N, "port_real_self_ns": t_rs * 1e9 / N})
    return out


def cpu_baseline_batch(systems, nth=None):
    """CPU baseline of the uneven batch on the host cores: the reference's own
    compute_spme (compiled unmodified, coloured OpenMP spread, all cores) on each
    system inside its domain (p in {4, 6}, even K, 4p < K), plus the oracle's
    real-space/self sum it lacks; one right-hand side per system, one rep.
    None when the reference build is absent."""
    if not _ref_lib_available():
        return None
    nth = nth or (os.cpu_count() or 1)
    total, parts, used = 0.0, 0, 0
    for k, s in enumerate(systems):
        if not (s["p"] in (4, 6) and s["K"] % 2 == 0 and 4 * s["p"] < s["K"]):
            continue
        rng = np.random.default_rng(500 + k)
        pos = rng.uniform(0.0, s["L"], size=(s["N"], 3))
        f1 = rng.standard_normal((1, 3 * s["N"]))
        wk = {"N": s["N"], "L": s["L"], "K": s["K"], "p": s["p"], "xi": s["xi"],
              "rc": s["rc"], "a": s["radius"]}
        t_rec, _ = _reference_recip_time(wk, pos, f1, nth, 1)
        total += t_rec + _real_self_time(wk, pos, f1, nth, 1)
        parts += s["N"]
        used += 1
    if used == 0:
        return None
    return {"value": total * 1e9 / parts, "unit": UNIT, "cores": nth, "kind": "reference",
            "sample": f"{used} of {len(systems)} systems (those in the reference's domain: p in "
                      "{4, 6}, even K, 4p < K; the GPU value covers all systems), 1 right-hand "
                      "side each, one rep: the reference's compute_spme compiled unmodified "
                      "(coloured OpenMP spread, project DFTI shim for MKL) + the oracle's "
                      "real-space/self sum (absent from the reference)",
            "systems": used, "particles": parts}


def host_side_child(args):
    """Child-process half of host_side: the CPU baseline and/or the FP64 oracle of
    the first two right-hand sides of synth(w, seed), written to args.host_side."""
    w = WORKLOADS[args.workload]
    out = {}
    if args.workload == "uneven_batch":
        from spme_gb300.batch import uneven_systems
        systems = uneven_systems(count=w["count"], xi=w["xi"], rc=w["rc"], radius=w["a"],
                                 seed=args.host_seed)
        out["cpu"] = json.dumps(cpu_baseline_batch(systems))
    else:
        if not args.no_cpu_baseline:
            out["cpu"] = json.dumps(cpu_baseline_time(w))
        if not args.no_oracle_check:
            import oracle
            pos, f = synth(w, seed=args.host_seed)
            nth = os.cpu_count() or 1
            f2 = f[:2].astype(np.float64)
            o_rec = oracle.recip(pos, w["L"], w["xi"], w["K"], w["p"], f2, radius=w["a"],
                                 nthreads=nth)
            o_rs = oracle.real_self(pos, w["L"], w["xi"], w["rc"], f2, radius=w["a"],
                                    nthreads=nth)
            out["full"], out["real_self"] = o_rec + o_rs, o_rs
    np.savez(args.host_side, **out)
    return 0


def host_side(workload, seed, want_cpu, want_oracle):
    """(cpu_baseline, oracle refs) computed in a child process (see host_side_child)."""
    fd, path = tempfile.mkstemp(suffix=".npz")
    os.close(fd)
    cmd = [sys.executable, os.path.abspath(__file__), "--workload", workload, "--host-side",
           path, "--host-seed", str(seed)]
    if not want_cpu:
        cmd.append("--no-cpu-baseline")
    if not want_oracle:
        cmd.append("--no-oracle-check")
    try:
        subprocess.run(cmd, check=True)
        with np.load(path) as z:
            cpu = json.loads(str(z["cpu"])) if "cpu" in z.files else None
            oref = ({"full": z["full"], "real_self": z["real_self"]}
                    if "full" in z.files else None)
    finally:
        os.unlink(path)
    return cpu, oref


def run_reference(args, w):
    """The reference's CPU path on the host cores for the same workload: per step
    one right-hand side of the full system with new positions (the reference's
    compute_spme, plus the oracle's real-space/self sum it lacks)."""
    ws, rank, _ = dist_env()
    if rank != 0:
        return 0
    import oracle
    have_ref = _ref_lib_available()
    pos, f = synth(w, seed=7)
    f1 = f[:1].astype(np.float64)
    nth = os.cpu_count() or 1
    N = w["N"]
    ref = (oracle.Reference(w["xi"], w["K"], w["p"], N, w["L"], nthreads=nth, colored=True)
           if have_ref else None)
    times, phases = [], {}
    for k in range(args.warmup + args.steps):
        v = np.zeros((1, 3 * N))
        t0 = time.perf_counter()
        if ref is not None:
            _, ph = ref.compute_with_timers(pos, 1, 1.0, f1, 3 * N, 0.0, v, 3 * N)
        else:
            ph = {}
            oracle.recip(pos, w["L"], w["xi"], w["K"], w["p"], f1, radius=w["a"], nthreads=nth)
        oracle.real_self(pos, w["L"], w["xi"], w["rc"], f1, radius=w["a"], nthreads=nth)
        dt = time.perf_counter() - t0
        if k >= args.warmup:
            times.append(dt)
            for key, val in ph.items():
                phases[key] = phases.get(key, 0.0) + val / args.steps
    if ref is not None:
        ref.close()
    ms = 1e3 * statistics.mean(times)
    value = ms * 1e6 / N
    kind = "reference" if have_ref else "port"
    sample = ("each step: 1 right-hand side of the full system with new positions: the "
              "reference's compute_spme compiled unmodified (coloured OpenMP spread, project "
              "DFTI shim for MKL) + the oracle's real-space/self sum (absent from the reference)"
              if have_ref else
              "each step: 1 right-hand side of the full system, the oracle's FP64 restatement "
              "of the reference path + real-space/self (reference build absent)")
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT,
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic: positions U[0,L), forces N(0,1), seeded",
        "config": config_of(w, args),
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": nth, "kind": kind,
                         "sample": sample},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "reference_phases_s_per_step": phases,
    }
    print(json.dumps(line), flush=True)
    return 0


def config_of(w, args):
    return {"workload": f"uniform spheres N={w['N']}, L={w['L']}, K={w['K']}, p={w['p']}, "
                        f"R={w['R']}, xi={w['xi']}, rc={w['rc']}, a={w['a']}",
            "N": w["N"], "L": w["L"], "K": w["K"], "p": w["p"], "R": w["R"], "xi": w["xi"],
            "rc": w["rc"], "radius": w["a"], "terms": "recip+real+self",
            "l2": "inputs larger than L2 (FP32 mesh 3.2 GB per pass); no flush",
            "parallelism": f"replicas x{args.gpus}" if args.gpus > 1 else "single GPU"}


def run_gb300(args, w):
    import torch

    import spme_gb300

    ws, rank, local = dist_env()
    torch.cuda.set_device(local)
    dist = None
    if ws > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl")

    N, R = w["N"], w["R"]
    pos, f = synth(w, seed=1000 + rank)
    # the CPU baseline and the FP64 oracle of the first two right-hand sides of the
    # timed inputs run in a child process before any GPU work here, so that their
    # OpenMP threads and large host arrays never live in the timed process
    cpu_base, oref = None, None
    want_cpu = rank == 0 and ws == 1 and not args.no_cpu_baseline
    want_oracle = rank == 0 and not args.no_fp64 and not args.no_oracle_check
    if want_cpu or want_oracle:
        cpu_base, oref = host_side(args.workload, 1000 + rank, want_cpu, want_oracle)
    # a dedicated (non-default) stream: the engine launches on it and the CUDA
    # events below are recorded on it
    stream = torch.cuda.Stream()
    torch.cuda.set_stream(stream)
    eng = spme_gb300.Engine(N, w["L"], w["xi"], w["K"], w["p"], radius=w["a"], rcut=w["rc"],
                            precision="fp32", max_nrhs=R, terms=spme_gb300.TERM_ALL)
    pos_d = torch.tensor(pos, device="cuda")
    f_d = torch.tensor(f, device="cuda")
    u_d = torch.zeros_like(f_d)
    tune = None
    if args.tile:
        tile = tuple(int(v) for v in args.tile.split(","))
        eng.set_tile(*tile)
        tune = {"tile": list(tile), "fixed": True}
    elif not args.no_autotune:
        # tile shape measured on this device (outside the timed region, not cached)
        from spme_gb300.autotune import autotune
        tile, timings = autotune(eng, pos_d, f_d, reps=2, use_cache=False)
        tune = {"tile": list(tile),
                "ms_per_candidate": {"x".join(map(str, k)): round(v, 3) for k, v in timings.items()}}
    eng.set_stream(stream.cuda_stream)

    def step():
        eng.set_positions(pos_d)
        eng.apply(f_d, u_d)

    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    eng.set_profiling(1)
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    clocks = Clocks(local)
    clocks.start()
    l0 = eng.launch_count()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record(stream)
    for _ in range(args.steps):
        step()
    ev1.record(stream)
    torch.cuda.synchronize()
    launches = eng.launch_count() - l0
    ck = clocks.stop()
    ms = ev0.elapsed_time(ev1) / args.steps
    stages = eng.stage_times()  # last timed step, real-space overlapped as in production
    # one extra serialized step attributes time to every stage alone
    eng.set_profiling(2)
    step()
    torch.cuda.synchronize()
    stages_serial = eng.stage_times()
    eng.set_profiling(0)
    if dist:
        t = torch.tensor([ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
        dist.barrier()
    value = ms * 1e6 / (N * R)  # per-rank work fixed (weak scaling): time per unit on each

    # end to end through the public API with pinned host buffers
    pos_h = torch.tensor(pos).pin_memory().numpy()
    f_h = torch.tensor(f).pin_memory().numpy()
    u_h = torch.zeros(f.shape, dtype=torch.float32).pin_memory().numpy()
    eng.set_stream(None)  # the engine's own stream for the host-pointer API
    for _ in range(max(1, args.warmup)):
        eng.set_positions(pos_h)
        eng.apply(f_h, u_h)
    e2e_times = []
    for _ in range(args.steps):
        t0 = time.perf_counter()
        eng.set_positions(pos_h)
        eng.apply(f_h, u_h)
        e2e_times.append(time.perf_counter() - t0)
    e2e_ms = 1e3 * statistics.mean(e2e_times)
    # the mean is reported; the median shows the steady state apart from host-side
    # stalls (copies over the shared host link)
    e2e_median_ms = 1e3 * statistics.median(e2e_times)
    if dist:
        t = torch.tensor([e2e_ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e2e_ms = float(t.item())

    # FP64 plain single-RHS path and accuracy of the FP32 batch against it
    extra = {}
    if rank == 0 and not args.no_fp64:
        e64 = spme_gb300.Engine(N, w["L"], w["xi"], w["K"], w["p"], radius=w["a"],
                                rcut=w["rc"], precision="fp64", max_nrhs=1,
                                terms=spme_gb300.TERM_ALL)
        e64.set_stream(stream.cuda_stream)
        p64 = torch.tensor(pos, device="cuda")
        f64 = torch.tensor(f[:1].astype(np.float64), device="cuda")
        u64 = torch.zeros_like(f64)
        e64.set_positions(p64)
        e64.apply(f64, u64)
        torch.cuda.synchronize()
        a0, a1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        reps = 3
        a0.record(stream)
        for _ in range(reps):
            e64.set_positions(p64)
            e64.apply(f64, u64)
        a1.record(stream)
        torch.cuda.synchronize()
        ms64 = a0.elapsed_time(a1) / reps
        ref = u64[0].double()
        got = u_d[0].double()
        rel = float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref))
        ns64 = ms64 * 1e6 / N
        kmax = np.pi * w["K"] / w["L"]
        acc = {"rel_l2_fp32_vs_fp64": rel,
               "spme_truncation_recip": float(np.exp(-kmax ** 2 / (4 * w["xi"] ** 2))),
               "spme_truncation_real": float(np.exp(-(w["xi"] * w["rc"]) ** 2))}
        if oref is not None:
            def rel_np(a, b):
                return float(np.linalg.norm(a - b) / np.linalg.norm(b))
            acc["rel_l2_fp32_vs_oracle"] = rel_np(u_d[:2].double().cpu().numpy(), oref["full"])
            acc["rel_l2_fp64_vs_oracle"] = rel_np(u64[:1].cpu().numpy(), oref["full"][:1])
            # the FP32 real-space + self part alone
            ers = spme_gb300.Engine(N, w["L"], w["xi"], w["K"], w["p"], radius=w["a"],
                                    rcut=w["rc"], precision="fp32", max_nrhs=2,
                                    terms=spme_gb300.TERM_REAL | spme_gb300.TERM_SELF)
            ers.set_stream(stream.cuda_stream)
            ers.set_positions(p64)
            urs = torch.zeros_like(f_d[:2])
            ers.apply(f_d[:2].contiguous(), urs)
            torch.cuda.synchronize()
            acc["rel_l2_fp32_real_self_vs_oracle"] = rel_np(urs.double().cpu().numpy(),
                                                            oref["real_self"])
            acc["oracle_rhs_checked"] = 2
            ers.close()
        # the FP64 real-space sum timed alone (one more apply, stages serialized)
        e64.set_profiling(2)
        e64.set_positions(p64)
        e64.apply(f64, u64)
        torch.cuda.synchronize()
        rs64_ms = e64.stage_times().get("realspace", 0.0)
        e64.set_profiling(0)
        extra = {"fp64_plain": {"value": ns64, "unit": UNIT, "ms_per_apply": ms64,
                                "terms": "recip+real+self", "nrhs": 1,
                                "realspace_ms": rs64_ms},
                 "fp32_batched_speedup_vs_fp64_plain": ns64 / value,
                 "accuracy": acc}
        e64.close()

    if rank != 0:
        if dist:
            dist.destroy_process_group()
        return 0

    peak, peak_kind = peaks()
    alg = algorithmic_bytes(w)
    kern = {}
    for k in ("spread", "influence", "interp"):
        t_ms = stages.get(k, 0.0)
        if t_ms > 0:
            gbs = alg[k] / (t_ms * 1e-3) / 1e9
            kern[k] = {"ms": t_ms, "alg_bytes": alg[k], "achieved_gbs": gbs,
                       "frac": gbs / peak}
    for k in ("pack", "realspace", "fft_fwd", "fft_bwd", "unpack"):
        if k in stages:
            kern[k] = {"ms": stages[k]}
    for k, v in stages_serial.items():
        kern.setdefault(k, {})["ms_serialized"] = v
    # real-space sum: arithmetic of the pair applications (9 FMA per pair and
    # right-hand side: r.f, then F f + G r (r.f)) over the expected number of
    # ordered pairs within rc, N (N - 1) (4/3) pi rc^3 / L^3, against the
    # measured FMA peak (FP32 batched engine, FP64 plain path)
    pairs = N * (N - 1) * (4.0 / 3.0) * np.pi * w["rc"] ** 3 / w["L"] ** 3
    rs = {"pairs_expected": pairs, "flops_per_pair_rhs": 18}
    try:
        peak32, peak64 = spme_gb300.fma_peak("fp32"), spme_gb300.fma_peak("fp64")
        rs.update({"fp32_fma_peak_tflops": peak32 / 1e12, "fp64_fma_peak_tflops": peak64 / 1e12})
    except Exception:
        peak32 = peak64 = None
    t32 = stages_serial.get("realspace", 0.0)
    if t32 > 0:
        f32 = pairs * R * 18 / (t32 * 1e-3)
        rs["fp32"] = {"ms": t32, "tflops": f32 / 1e12,
                      "frac_of_measured_peak": f32 / peak32 if peak32 else None}
    t64 = extra.get("fp64_plain", {}).get("realspace_ms", 0.0) if extra else 0.0
    if t64 > 0:
        f64 = pairs * 1 * 18 / (t64 * 1e-3)
        rs["fp64"] = {"ms": t64, "nrhs": 1, "tflops": f64 / 1e12,
                      "frac_of_measured_peak": f64 / peak64 if peak64 else None}
    dom = max(("spread", "influence", "interp"), key=lambda k: kern.get(k, {}).get("ms", 0.0))
    roof = None
    if dom in kern:
        tr = NCU_TRAFFIC_RATIO[dom] * alg[dom]
        roof = {"kernel": dom, "bound": "hbm", "achieved": kern[dom]["achieved_gbs"],
                "peak": peak, "unit": "GB/s", "frac": kern[dom]["achieved_gbs"] / peak,
                "traffic": tr, "traffic_source": "small-case ncu ratio x algorithmic bytes",
                "peak_kind": peak_kind}
    h2d = pos.nbytes + f.nbytes
    d2h = f.nbytes
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": ws, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": False, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32",
        "data": "synthetic: positions U[0,L) and forces N(0,1), seeded",
        "config": config_of(w, args),
        "roofline": roof,
        "cpu_baseline": cpu_base,
        "e2e": {"value": e2e_ms * 1e6 / (N * R), "unit": UNIT, "h2d_bytes_per_step": h2d,
                "d2h_bytes_per_step": d2h, "ms_per_step": e2e_ms,
                "ms_per_step_median": e2e_median_ms},
        "clocks": ck,
        "gpu_launches": launches,
        "kernels": kern,
        "realspace_arithmetic": rs,
        "autotune": tune,
    }
    line.update(extra)
    if ws == 1 and args.workload == "large" and not args.no_secondary:
        line["secondary_workloads"] = run_secondary(args)
    print(json.dumps(line), flush=True)
    if dist:
        dist.destroy_process_group()
    return 0


def run_secondary(args):
    """The single-right-hand-side system, the mid-size 16-right-hand-side system
    and the uneven batch, each in a child process (its own engines and memory),
    summarised in the main line."""
    out = {}
    for wl in ("scale_up", "multi_rhs", "uneven_batch"):
        cmd = [sys.executable, os.path.abspath(__file__), "--workload", wl, "--steps",
               str(max(5, args.steps)), "--warmup", "3", "--no-secondary"]
        if args.no_cpu_baseline:
            cmd.append("--no-cpu-baseline")
        try:
            r = subprocess.run(cmd, capture_output=True, text=True, timeout=600)
            d = json.loads([x for x in r.stdout.splitlines() if x.startswith("{")][-1])
        except Exception as exc:  # reported, never fatal for the main line
            out[wl] = {"error": str(exc)[:200]}
            continue
        keep = ("value", "unit", "ms_per_step", "config", "e2e", "kernels", "per_system_loop",
                "engines_graph", "speedup_vs_loop", "speedup_vs_engines_graph",
                "stages_ms_serialized", "gpu_launches", "autotune", "fp64_plain",
                "fp32_batched_speedup_vs_fp64_plain", "accuracy", "cpu_baseline", "clocks")
        out[wl] = {k: d[k] for k in keep if k in d}
    return out


def run_batch(args, w):
    """Uneven batch: the native batch (one persistent launch per stage over all
    systems, one cuFFT plan per distinct K, the step one CUDA-graph launch)
    against the same systems through one engine each (a per-system loop, and
    the engines as branches of one captured graph)."""
    import torch

    from spme_gb300.batch import SystemBatch, uneven_systems

    ws, rank, local = dist_env()
    torch.cuda.set_device(local)
    systems = uneven_systems(count=w["count"], xi=w["xi"], rc=w["rc"], radius=w["a"],
                             seed=1234 + rank)
    R = w["R"]
    cpu_base = (host_side(args.workload, 1234 + rank, True, False)[0]
                if rank == 0 and ws == 1 and not args.no_cpu_baseline else None)
    rng = np.random.default_rng(77 + rank)
    pos = [torch.tensor(rng.uniform(0, s["L"], (s["N"], 3)), device="cuda") for s in systems]
    f = [torch.tensor(rng.standard_normal((R, 3 * s["N"])), dtype=torch.float32, device="cuda")
         for s in systems]
    u = [torch.zeros_like(x) for x in f]
    b = SystemBatch(systems, nrhs=R)  # autotunes the batch's tile and concurrency in bind
    b.bind(pos, f, u)
    units = sum(s["N"] for s in systems) * R
    stream = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def timed(fn):
        for _ in range(args.warmup):
            fn()
        torch.cuda.synchronize()
        e0.record(stream)
        for _ in range(args.steps):
            fn()
        e1.record(stream)
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / args.steps

    loop_ms = timed(b.run_loop)
    b.capture_engines_graph()
    graph_ms = timed(b.run_engines_graph)
    l0 = b.batch.launch_count()
    clocks = Clocks(local)
    clocks.start()
    ms = timed(b.run)
    ck = clocks.stop()
    launches = (b.batch.launch_count() - l0) // (args.steps + args.warmup)
    # one serialized step attributes time to every stage
    b.batch.set_graphs(False)
    b.batch.set_profiling(True)
    b.run()
    torch.cuda.synchronize()
    stages = b.batch.stage_times()
    b.batch.set_profiling(False)
    if rank != 0:
        return 0
    line = {
        "metric": METRIC, "value": ms * 1e6 / units, "unit": UNIT, "n_gpus": ws,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms,
        "higher_is_better": False, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic: positions U[0,L) and forces N(0,1), seeded",
        "config": {"workload": f"uneven batch of {w['count']} systems, N log-uniform in "
                               f"[500, 50000], phi=0.05, K=next smooth >= 0.6 L, p in {{4,6,8}}, "
                               f"R={R}, xi={w['xi']}, rc={w['rc']}",
                   "systems": len(systems), "particles": units // R,
                   "distinct_K": len({s["K"] for s in systems}),
                   "l2": "whole batch larger than L2"},
        "gpu_launches": launches,
        "stages_ms_serialized": stages,
        "per_system_loop": {"value": loop_ms * 1e6 / units, "unit": UNIT, "ms_per_step": loop_ms},
        "engines_graph": {"value": graph_ms * 1e6 / units, "unit": UNIT, "ms_per_step": graph_ms},
        "speedup_vs_loop": loop_ms / ms,
        "speedup_vs_engines_graph": graph_ms / ms,
        "autotune": ({"tile": list(b.tuned[0]), "overlap": b.tuned[1]} if b.tuned else None),
        "cpu_baseline": cpu_base,
        "clocks": ck,
    }
    print(json.dumps(line), flush=True)
    b.close()
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--workload", default="large", choices=sorted(WORKLOADS))
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-fp64", action="store_true")
    ap.add_argument("--no-oracle-check", action="store_true",
                    help="skip the FP64 oracle check of the timed result (outside the timed region)")
    ap.add_argument("--no-autotune", action="store_true")
    ap.add_argument("--no-secondary", action="store_true",
                    help="skip the mid-size and uneven-batch workloads after the large one")
    ap.add_argument("--host-side", default=None, help=argparse.SUPPRESS)
    ap.add_argument("--host-seed", type=int, default=0, help=argparse.SUPPRESS)
    ap.add_argument("--tile", default=None,
                    help="fixed mesh tile 'tx,ty,tz' instead of autotuning (e.g. for profiling)")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    w = WORKLOADS[args.workload]
    if args.host_side:
        return host_side_child(args)
    if args.workload == "uneven_batch":
        if args.impl == "reference":
            print(json.dumps({"impl": "reference", "unavailable":
                              "the uneven-batch workload is not a reference configuration"}))
            return 0
        return run_batch(args, w)
    if args.impl == "reference":
        return run_reference(args, w)
    return run_gb300(args, w)


if __name__ == "__main__":
    sys.exit(main())
