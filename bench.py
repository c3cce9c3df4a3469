#!/usr/bin/env python
"""
Benchmark: atom-steps/s of the 1,000,000-sphere Hertz isotropic-compression run
(gran/hertz/history kn 2e5, kt 2/7 kn, gamman 50, gammat 25, xmu 0.5;
fix nve/sphere; Cundall damping 0.7/0.7; fix deform/pressure on x, y, z with
target 1.0, gain 1e-3, couple xyz, max/rate 1e-4, remap x; dt 5e-5; neighbor
skin 0.1), seeded packing of diameters U[0.8, 1.2] at solid fraction 0.45,
density 2.5, at rest.  W warm-up steps then K timed steps of one run.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

One JSON line on stdout (rank 0).  `value` is whole-job atom-steps/s with the
state resident in HBM; `e2e` is the same metric through the public Python API
starting from host arrays (upload, setup, K steps with the per-step pressure
read-back the reference's host servo does, download).  `--impl reference`
times the CPU restatement of the reference path (the reference itself, Python
+ Taichi 1.7.4, cannot be installed here) on all host cores.

Multi-GPU: the path does not shard (one packing, one box); N GPUs run N
independent replicas (weak scaling), no collective on the data path.
"""

from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "atom-steps/s, 1M-sphere Hertz servo: mixed vs FP64 GPU at ≤1e-6 pressure err"
UNIT = "atom-steps/s"
KN = 2.0e5
PAIR = dict(kn=KN, kt=KN * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=0.5, dampflag=1)
DT = 5.0e-5
SKIN = 0.1
CUNDALL = (0.7, 0.7)
PGAIN = 1.0e-3
DEFORM = dict(axes={d: {"style": "pressure", "ptarget": 1.0, "pgain": PGAIN} for d in "xyz"}, couple="xyz",
              max_rate=1.0e-4, remap="x")
# published number for the same 1M isotropic-compression run (reference README, FP32, Taichi Vulkan on a
# Radeon 890M): the nearest published figure to this metric
PUBLISHED_FP32 = 2548.10e6
WORKLOAD = ("1M-sphere isotropic compression: gran/hertz/history kn=2e5 kt=2/7kn gn=50 gt=25 xmu=0.5, "
            "nve/sphere, damping/cundall 0.7 0.7, deform/pressure x/y/z pressure 1.0 pgain 1e-3 couple xyz "
            "max/rate 1e-4 remap x, dt 5e-5, skin 0.1, d~U[0.8,1.2] rho 2.5 phi 0.45 at rest")


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=200)
    ap.add_argument("--warmup", type=int, default=100)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--n", type=int, default=1_000_000)
    ap.add_argument("--seed", type=int, default=2)
    ap.add_argument("--precision", default="both", choices=["both", "mixed", "fp64"])
    ap.add_argument("--cpu-budget", type=float, default=12.0, help="seconds of CPU baseline work")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--workload", default="config2",
                    choices=["config2", "dense", "ensemble", "adjoint", "triaxial", "e2e"],
                    help="config2: the 1M-sphere servo run (default); ensemble: the batched-instances run; "
                         "e2e: the config-2 end-to-end job alone (for launch lists)")
    ap.add_argument("--instances", type=int, default=512, help="ensemble: number of instances")
    ap.add_argument("--no-dense", action="store_true", help="skip the contact-dense 1M-sphere line")
    ap.add_argument("--dense-reps", type=int, nargs=3, default=[4, 4, 4],
                    help="dense: copies of the compressed 15,625-sphere cell along x, y, z")
    return ap.parse_args()


# ----------------------------------------------------------------- clocks


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled while a region runs."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int, period_ms: int = 50):
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None
        try:
            self.p = subprocess.Popen(["nvidia-smi", f"--id={gpu_index}", f"--query-gpu={self.Q}",
                                       "--format=csv,noheader,nounits", f"-lms={period_ms}"],
                                      stdout=self.f, stderr=subprocess.DEVNULL)
        except OSError:
            self.p = None

    def stop(self) -> dict:
        if self.p is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.12)
        self.p.terminate()
        self.p.wait(timeout=10)
        self.f.flush()
        rows = [r.split(", ") for r in Path(self.f.name).read_text().strip().splitlines() if r.strip()]
        os.unlink(self.f.name)
        sm = [float(r[1]) for r in rows if len(r) >= 9 and r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in rows if len(r) >= 9 and r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = sorted({names[k] for r in rows if len(r) >= 9 for k in range(4) if r[5 + k].strip() == "Active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(sm)}


# ----------------------------------------------------------------- GPU arm


def box_of(p):
    """Lower and upper corners of a packing's periodic box (`L` a cube edge or three edges, `lo` optional)."""
    L = np.broadcast_to(np.asarray(p["L"], dtype=np.float64), (3,))
    lo = np.asarray(p.get("lo", np.zeros(3)), dtype=np.float64)
    return [float(a) for a in lo], [float(a) for a in lo + L]


def make_sim(G, p, n, precision, host=None):
    """The config-2 system; `host` (optional) holds x, v as pinned float64 tensors to upload from."""
    lo, hi = box_of(p)
    dom = G.Domain(boxlo=lo, boxhi=hi, boundary=("p", "p", "p"))
    atom = G.AtomSystem(max_atoms=n)
    if host is not None:
        atom.add_particles(x=host["x"], radius=host["radius"], density=p["density"], v=host["v"])
    else:
        atom.add_particles(x=p["x"], radius=p["radius"], density=p["density"], v=p["v"])
    nl = G.NeighborList(domain=dom, skin=SKIN, max_atoms=n, max_neighbors_per_atom=32)
    hist = G.ContactHistory(max_atoms=n, max_neighbors=32)
    pair = G.GranHertzHistory(domain=dom, **PAIR)
    sim = G.Simulation(domain=dom, atom=atom, neighbor=nl, history=hist, pair=pair, dt=DT, precision=precision)
    sim.add_fix(G.FixNVESphere(domain=dom))
    sim.add_fix(G.FixDampingCundall(domain=dom, gamma_lin=CUNDALL[0], gamma_ang=CUNDALL[1]))
    sim.add_fix(G.FixDeformPressure(domain=dom, **DEFORM))
    return sim


def list_stats(sim):
    import torch
    nnb = sim.neighbor.nnb.double().mean().item()
    t = sim.history.touch
    bits = sum(((t >> k) & 1).sum().item() for k in range(sim.neighbor.slots))
    return nnb, bits / max(sim.atom.nlocal, 1)


def algorithmic_bytes(kernel: str, precision: str, n_nb: float, n_c: float, flagged: float) -> float:
    """Bytes per atom a launch must move through HBM.

    fused_a (A), every atom: the position's Verlet stream plus the skin check's reference words.
      mixed: reads and writes the position (high and low FP32 words, 24 + 24), reads the velocity (24),
             m (kinetic term, 4), the offset at the last build (12) and the packed cell (4)       =  92
             plus per flagged atom (`flagged` = fraction) the angular velocity, force, torque, 1/m and
             1/I read (24 + 24 + 8) and both velocities written (48): 104
      FP64:  reads x, v (48), x at the last build (24); writes x (24)                       =  96
             plus per flagged atom omega, force, torque, 1/m and 1/I read (24 + 48 + 16) and v, omega
             written (48): 136
      A's records also carry per-build constants and padding in their fourth lanes for C's gathers,
      which move with them (layout_bytes: 112 + 104 mixed / 122 + 160 FP64 per flagged atom); those
      are not counted here.
    fused_c (C): the contact kernel's per-atom bytes, S + 4 n_nb + 52 n_c (own state read once and
      force written once, S = 84 mixed / 140 FP64; 4 per neighbor index; 4 partner + 48 shear per
      touching slot)."""
    if kernel == "fused_a":
        return (92.0 + 104.0 * flagged) if precision == "mixed" else (96.0 + 136.0 * flagged)
    if kernel == "fused_c":
        return (84.0 if precision == "mixed" else 140.0) + 4.0 * n_nb + 52.0 * n_c
    return 0.0


def layout_bytes(kernel: str, precision: str, flagged: float) -> float:
    """Bytes per atom A's record layout makes it read and write (see algorithmic_bytes)."""
    if kernel == "fused_a":
        return (112.0 + 104.0 * flagged) if precision == "mixed" else (122.0 + 160.0 * flagged)
    return 0.0


KERNEL_NAMES = {("fused_a", "mixed"): "k_a32", ("fused_a", "fp64"): "k_a64", ("fused_c", "mixed"): "k_cf",
                ("fused_c", "fp64"): "k_cf", ("fused_s", "mixed"): "k_s", ("fused_s", "fp64"): "k_s"}
TRAFFIC_FILE = ROOT / "profiles" / "ncu_traffic_config2_1M.json"


def ncu_traffic(kernel: str, precision: str):
    """DRAM bytes (read + write) per launch of a kernel of this workload, from the committed ncu capture
    (profiles/ncu_traffic_config2_1M.json, which names its command); None when absent."""
    if not TRAFFIC_FILE.exists():
        return None
    d = json.loads(TRAFFIC_FILE.read_text())
    k = d.get("kernels", {}).get(f"{KERNEL_NAMES[(kernel, precision)]}/{precision}")
    if not k:
        return None
    return {"bytes": k["dram_bytes_read"] + k["dram_bytes_write"], "source": f"ncu: {d.get('command', '')}"}


FP64_COUNTS_FILE = ROOT / "profiles" / "fp64_pipe_config2.json"


def fp64_peak_dfma_per_s() -> float:
    """The FP64 pipe's DFMA rate on this GPU, measured now (tmps_probe_fp64: eight independent DFMA chains
    per thread, eight blocks of 256 threads per SM; best of five timed launches)."""
    import torch
    from taichimps_gb300 import _device
    L = _device.lib()
    sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    blocks, threads, iters = 8 * sms, 256, 4096
    out = torch.empty(blocks * threads, dtype=torch.float64, device="cuda")
    st = _device.stream()
    for _ in range(2):
        L.tmps_probe_fp64(blocks, threads, iters, out.data_ptr(), st)
    best = None
    s = torch.cuda.current_stream()
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(s)
        L.tmps_probe_fp64(blocks, threads, iters, out.data_ptr(), st)
        e1.record(s)
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1)
        best = ms if best is None else min(best, ms)
    return 8.0 * iters * blocks * threads / (best * 1e-3)


def fp64_roofline(kernel: str, n: int, kernel_ms, peak: float):
    """FP64-pipe roofline of an FP64-form kernel: its FP64 instructions per atom (DFMA + DMUL + DADD, from
    the committed ncu counts, profiles/fp64_pipe_config2.json) x atoms / its CUDA-event time, against the
    DFMA rate measured by fp64_peak_dfma_per_s."""
    if not FP64_COUNTS_FILE.exists() or not kernel_ms or not peak:
        return None
    d = json.loads(FP64_COUNTS_FILE.read_text())
    k = d.get("kernels", {}).get(kernel)
    if not k:
        return None
    ach = k["fp64_inst_per_atom"] * n / (kernel_ms * 1e-3)
    return {"kernel": kernel, "bound": "fp64 pipe", "achieved": ach, "peak": peak, "unit": "FP64 inst/s",
            "frac": ach / peak, "fp64_inst_per_atom": k["fp64_inst_per_atom"],
            "pipe_active_pct_ncu": k.get("pipe_active_pct"), "kernel_ms": kernel_ms,
            "peak_source": "measured now: tmps_probe_fp64 (DFMA)", "counts_source": f"ncu: {d.get('command', '')}"}


def max_over_ranks(ms: float, world: int, device: str = "cuda") -> float:
    """The timed region of a replica run ends when the slowest rank's does: the maximum over ranks
    (the only collective of the replica path), then a barrier."""
    if world <= 1:
        return ms
    import torch
    t = torch.tensor([ms], dtype=torch.float64, device=device)
    torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    torch.distributed.barrier()
    return float(t.item())


def replica_seed(seed: int, rank: int) -> int:
    """Each rank runs its own packing (independent replicas, no data-path exchange)."""
    return seed + rank


def run_gpu_arm(args, p, precision, rank, world):
    """W warm-up + K timed steps of one run through Simulation (the fused step), one precision."""
    import torch
    import taichimps_gb300 as G
    from taichimps_gb300 import _device, _lib

    L = _lib.load()
    n = len(p["x"])
    K, W = args.steps, args.warmup
    sim = make_sim(G, p, n, precision)
    sim.run(W)                      # setup (build + setup forces) + W warm-up steps
    torch.cuda.synchronize()
    if world > 1:
        torch.distributed.barrier()
    names = ["fused_a", "fused_c", "fused_s"]
    clocks = ClockSampler(torch.cuda.current_device())
    # the timed run continues the warm-up run: the engine is re-entered without a second setup;
    # steps run as replays of a captured CUDA graph (chunks of eng.chunk steps)
    eng = sim.last_engine
    # the timed steps are whole graph replays: chunks of the largest divisor of K up to 64 steps
    eng.chunk = max(c for c in range(1, min(64, K) + 1) if K % c == 0)
    eng.begin()
    # a chunk's first run is plain launches, its second captures the graph (untimed, warm-up)
    eng.run(2 * eng.chunk)
    torch.cuda.synchronize()
    l0 = L.tmps_launch_count()
    g0 = eng.graph_kernel_launches
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    eng.run(K)
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1)
    clk = clocks.stop()
    # graph replays do not pass through the host entry points, so count the launches the graph holds
    launches = (L.tmps_launch_count() - l0) + (eng.graph_kernel_launches - g0)
    cull = eng.cull_stats()
    flagged = eng.flagged_count() / max(sim.atom.nlocal, 1)
    # per-kernel CUDA-event timings: the next K steps launched one by one (same run, same state)
    _device.TIMED = {k: [] for k in names}
    eng.run(K)
    torch.cuda.synchronize()
    timed = {k: [a.elapsed_time(b) for a, b in v] for k, v in _device.TIMED.items()}
    _device.TIMED = None
    eng.finish()
    ms = max_over_ranks(ms, world)
    sim.check_device_status()
    n_nb, n_c = list_stats(sim)
    sim.domain.pull()
    pressure = sim.fixes[-1].last_pressure()
    kern = {k: (sum(v) / len(v) if v else None) for k, v in timed.items()}
    return dict(sim=sim, n=n, ms=ms, launches=launches, clocks=clk, kern_ms=kern, n_nb=n_nb, n_c=n_c,
                pressure=pressure, builds=sim.neighbor.build_count, rebuilds_timed=eng.rebuilds,
                steps_run=sim.timestep, cull=cull, flagged=flagged, rows=eng.rows)


def run_e2e(args, p, precision):
    """The same metric through the public API, from pinned host arrays: upload and setup
    (Simulation.run builds the list and evaluates the setup forces), K steps whose servo pressure tensor
    lands in pinned host memory every step (the per-step read-back of the reference's host servo path,
    FixDeformPressure.record_pressure), then the download of positions and velocities.  The whole job
    runs once untimed first (allocator and graph warm-up), then three times timed; the median counts."""
    import torch
    import taichimps_gb300 as G

    n = len(p["x"])
    K = args.steps
    host = {k: torch.from_numpy(np.ascontiguousarray(p[k])).pin_memory() for k in ("x", "radius", "v")}

    def job():
        sim = make_sim(G, p, n, precision, host=host)
        fix = sim.fixes[-1]
        fix.record_pressure(K + 1)
        sim.run(K)
        pressures = fix.pressure_history(range(1, K + 1))
        x = sim.atom.x.to_numpy()
        v = sim.atom.v.to_numpy()
        return x, v, pressures

    job()
    times = []
    for _ in range(3):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        x, v, pressures = job()
        torch.cuda.synchronize()
        times.append(time.perf_counter() - t0)
    dt = statistics.median(times)
    assert np.isfinite(x).all() and np.isfinite(v).all() and np.isfinite(pressures).all()

    # where a job's time goes: one more job, synchronised after each public call (so the phases add up
    # to a little more than an unsynchronised job)
    phases = {}

    def lap(name, t0):
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        phases[name] = round((t1 - t0) * 1e3, 4)
        return t1

    torch.cuda.synchronize()
    t = time.perf_counter()
    sim = make_sim(G, p, n, precision, host=host)
    t = lap("system from pinned arrays (Domain, AtomSystem.add_particles, list, pair, fixes)", t)
    fix = sim.fixes[-1]
    fix.record_pressure(K + 1)
    sim.run(K)
    t = lap("Simulation.run: neighbor build, setup forces, K fused steps, hand-back", t)
    fix.pressure_history(range(1, K + 1))
    t = lap("pressure_history", t)
    sim.atom.x.to_numpy()
    sim.atom.v.to_numpy()
    lap("x, v to_numpy", t)
    up = n * (3 * 8 + 8 + 3 * 8)                # positions, radius, velocities (mass and inertia are formed on the device)
    down = n * 2 * 3 * 8 + K * 48               # final x, v; per step the pressure tensor
    return {"value": n * K / dt, "unit": UNIT, "h2d_bytes_per_step": up / K, "d2h_bytes_per_step": down / K,
            "seconds": dt, "precision": precision,
            "includes": "upload, neighbor build + setup forces, K steps, per-step pressure to host, download "
                        "(median of three timed jobs after an untimed one)", "job_seconds": times,
            "phases_ms": phases}


# ----------------------------------------------------------------- CPU (oracle)


def oracle_sim(O, p, nthreads):
    O.set_threads(nthreads)
    lo, hi = box_of(p)
    dom = O.OracleDomain.make(lo, hi)
    at = O.OracleAtoms(x=p["x"], radius=p["radius"], density=p["density"], v=p["v"])
    nl = O.OracleNeighbor(dom, skin=SKIN, max_neighbors=32)
    hist = O.OracleHistory(32)
    pair = O.OraclePair("hertz/history", **PAIR)
    fixes = [O.OracleCundall(*CUNDALL), O.OracleDeform(dom, **DEFORM)]
    return O.OracleSim(dom, at, nl, hist, pair, DT, fixes=fixes)


def cpu_baseline(p, budget_s, max_steps):
    from oracle import oracle as O
    O.build()
    cores = os.cpu_count() or 1
    sim = oracle_sim(O, p, cores)
    sim.setup(max_steps)
    t0 = time.perf_counter()
    steps = 0
    while steps < max_steps and (time.perf_counter() - t0) < budget_s:
        sim.step()
        steps += 1
    dt = time.perf_counter() - t0
    n = sim.atoms.n
    return {"value": n * steps / dt, "unit": UNIT, "cores": cores, "kind": "port",
            "sample": f"{steps} steps of the same {n}-sphere run after setup ({dt:.1f} s of CPU work), oracle "
                      f"(C restatement, OpenMP {cores} threads)"}, sim


def reference_arm(args, rank, world):
    """--impl reference: the CPU restatement of the reference path on all host cores."""
    if rank != 0:
        return None
    from oracle import oracle as O
    from taichimps_gb300.packing import config2
    O.build()
    p = config2(seed=args.seed, n=args.n)
    cores = os.cpu_count() or 1
    sim = oracle_sim(O, p, cores)
    K, W = args.steps, args.warmup
    sim.setup(W + K)
    for _ in range(W):
        sim.step()
    t0 = time.perf_counter()
    for _ in range(K):
        sim.step()
    dt = time.perf_counter() - t0
    n = sim.atoms.n
    v = n * K / dt
    return {"metric": METRIC, "value": v, "unit": UNIT, "impl": "reference", "n_gpus": world, "steps": K,
            "warmup": W, "ms_per_step": 1e3 * dt / K, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic: seeded FCC-site packing (taichimps_gb300.packing)",
            "config": {"workload": WORKLOAD, "n_atoms": n},
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
                             "sample": f"{W}+{K} steps of the full {n}-sphere run; the reference (Python + "
                                       "Taichi 1.7.4) is not installable offline, so its CPU path is timed "
                                       "through the project's C restatement (oracle/)"},
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}


# ----------------------------------------------------------------- ensemble

ENSEMBLE_METRIC = "atom-steps/s, batched ensemble of independent servo packings vs looped single solves"


def ensemble_instance(G, seed, k, precision):
    """Instance k of the ensemble: sphere count log-uniform [500, 16000], kn log-uniform [1e4, 1e6], xmu
    U[0.1, 0.8], kt 2/7 kn, gamman 50 (gammat 25, dampflag 1: not given, as in the other runs), d U[0.8, 1.2],
    rho 2.5, phi 0.45, isotropic pressure servo to 1.0 (gain 1e-3, max/rate 1e-4, couple xyz, remap x)."""
    from taichimps_gb300.packing import make_packing_box
    rng = np.random.default_rng([seed, k])
    n = int(round(math.exp(rng.uniform(math.log(500), math.log(16000)))))
    kn = float(math.exp(rng.uniform(math.log(1e4), math.log(1e6))))
    xmu = float(rng.uniform(0.1, 0.8))
    pk = make_packing_box(n, 0.8, 1.2, 0.45, seed * 1_000_003 + k)
    dom = G.Domain(boxlo=[0.0] * 3, boxhi=[float(v) for v in pk["L"]], boundary=("p", "p", "p"))
    atom = G.AtomSystem(max_atoms=n)
    atom.add_particles(x=pk["x"], radius=pk["radius"], density=2.5, v=pk["v"])
    nl = G.NeighborList(domain=dom, skin=SKIN, max_atoms=n, max_neighbors_per_atom=16, slots="auto")
    hist = G.ContactHistory(max_atoms=n, max_neighbors=16)
    pair = G.GranHertzHistory(domain=dom, kn=kn, kt=kn * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=xmu, dampflag=1)
    sim = G.Simulation(domain=dom, atom=atom, neighbor=nl, history=hist, pair=pair, dt=DT, precision=precision)
    sim.add_fix(G.FixNVESphere(domain=dom))
    sim.add_fix(G.FixDeformPressure(domain=dom, **DEFORM))
    return sim


def run_ensemble(args):
    """Both arms on the same instances: W warm-up steps (with the setup) through the arm, then K timed steps
    continuing the run (run ... pre no): the batched engine, then every instance looped on its own."""
    import torch
    import taichimps_gb300 as G
    K, W, m = args.steps, args.warmup, args.instances
    prec = "mixed" if args.precision == "both" else args.precision
    batch = [ensemble_instance(G, args.seed, k, prec) for k in range(m)]
    natoms = sum(s.atom.nlocal for s in batch)
    eng = G.BatchedEngine(batch, precision=prec)
    eng.run(W)
    for s in batch:
        s.run_pre = False
    torch.cuda.synchronize()
    r0 = eng.graph_replays
    t0 = time.perf_counter()
    eng.run(K)
    torch.cuda.synchronize()
    t_batch = time.perf_counter() - t0
    launches_batch = 3 * eng.chunk * (eng.graph_replays - r0)
    shape = {"groups_per_warp_a_c": list(eng.launch_shape), "tuning_us_per_launch": eng.tuning}
    del eng, batch
    torch.cuda.empty_cache()
    looped = [ensemble_instance(G, args.seed, k, prec) for k in range(m)]
    for s in looped:
        s.run(W)
        s.run_pre = False
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for s in looped:
        s.run(K)
    torch.cuda.synchronize()
    t_loop = time.perf_counter() - t0
    sizes = [s.atom.nlocal for s in looped]
    return {"metric": ENSEMBLE_METRIC, "value": natoms * K / t_batch, "unit": UNIT, "n_gpus": 1, "steps": K,
            "warmup": W, "ms_per_step": 1e3 * t_batch / K, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32/f64 mixed" if prec == "mixed" else "f64",
            "data": "synthetic: seeded FCC-site packings per instance in a lattice-shaped periodic box "
                    "(taichimps_gb300.packing.make_packing_box)",
            "config": {"workload": f"{m} independent periodic packings, gran/hertz/history with per-instance kn "
                                   "(log-uniform 1e4..1e6) and xmu (U 0.1..0.8), isotropic pressure servo to 1.0, "
                                   "dt 5e-5", "instances": m, "total_atoms": natoms,
                       "atoms_min": min(sizes), "atoms_max": max(sizes), "precision": prec},
            "looped_single_solves": {"value": natoms * K / t_loop, "seconds": t_loop,
                                     "how": "Simulation.run of each instance in turn (its own fused step, CUDA "
                                            "graphs), same steps"},
            "speedup_vs_looped": t_loop / t_batch, "batched_seconds": t_batch,
            "gpu_launches_batched": launches_batch, "launch_shape": shape}


# ----------------------------------------------------------------- dense state

DENSE_WORKLOAD = ("1M-sphere contact-dense servo run: a 15,625-sphere cell compressed to p = 1 "
                  "(packing.dense_cell) tiled 4x4x4, at rest; the config-2 physics (gran/hertz/history kn=2e5 "
                  "kt=2/7kn gn=50 gt=25 xmu=0.5, nve/sphere, damping/cundall 0.7 0.7, deform/pressure x/y/z "
                  "pressure 1.0 pgain 1e-3 couple xyz max/rate 1e-4 remap x, dt 5e-5, skin 0.1)")
DENSE_TRAFFIC_FILE = ROOT / "profiles" / "ncu_traffic_dense_1M.json"


def contact_bytes(precision: str, n_nb: float, n_c: float) -> float:
    """Algorithmic bytes per atom of one contact-kernel launch: S + 4 n_nb + 52 n_c, S the atom's own
    state read once and its force and torque written once (84 mixed, 140 FP64), 4 per neighbor-list
    entry, 4 (partner) + 48 (shear read and written) per touching entry."""
    return (84.0 if precision == "mixed" else 140.0) + 4.0 * n_nb + 52.0 * n_c


# the contact-dense state's two contact kernels, timed together, and what holds them
PAIR_KERNELS = "k_pair_contacts + k_pair_gather"
# (profiles/pair_kernels_dense_ncu.md)
DENSE_BOUND = {"mixed": "latency of the gathers", "fp64": "fp64 pipe"}


def dense_traffic(kernel: str, precision: str):
    if not DENSE_TRAFFIC_FILE.exists():
        return None
    d = json.loads(DENSE_TRAFFIC_FILE.read_text())
    k = d.get("kernels", {}).get(f"{kernel}/{precision}")
    if not k:
        return None
    return {"bytes": k["dram_bytes_read"] + k["dram_bytes_write"], "source": f"ncu: {d.get('command', '')}",
            "n_atoms": d.get("n_atoms")}


def run_dense(args, rank, world, forms):
    """The contact kernel where contacts exist: the same physics on the tiled compressed packing, W warm-up
    and K timed steps per form, the contact kernel's time against its algorithmic bytes at the measured
    neighbor and contact counts.  The FP64 form is the reference for the mixed form's pressure here."""
    import torch
    from taichimps_gb300.packing import dense_config2
    p = dense_config2(reps=tuple(args.dense_reps))
    p["density"] = 2.5
    runs = {}
    for prec in forms:
        runs[prec] = run_gpu_arm(args, p, prec, rank, world)
        del runs[prec]["sim"]
        torch.cuda.empty_cache()
    if rank != 0:
        return None
    peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
    peak = peaks.get("hbm_gbs", 6806.5)
    scal = lambda t: (t[0] + t[1] + t[2]) / 3.0
    out = {"workload": DENSE_WORKLOAD, "n_atoms": runs[forms[0]]["n"], "steps": args.steps, "warmup": args.warmup,
           "forms": {}}
    for prec, r in runs.items():
        n = r["n"]
        kb = contact_bytes(prec, r["n_nb"], r["n_c"])
        c_ms = r["kern_ms"].get("fused_c")
        ach = kb * n / (c_ms * 1e-3) / 1e9 if c_ms else None
        name = PAIR_KERNELS if r["rows"] else KERNEL_NAMES[("fused_c", prec)]
        tr = dense_traffic(name, prec)
        out["forms"][prec] = {
            "value": world * n * args.steps / (r["ms"] * 1e-3), "ms_per_step": r["ms"] / args.steps,
            "kernel_ms": r["kern_ms"], "neighbors_per_atom": r["n_nb"], "contacts_per_atom": r["n_c"],
            "flagged_atoms_frac": r["flagged"], "rebuilds_in_timed_steps": r["rebuilds_timed"],
            "mean_pressure": scal(r["pressure"]), "pressure": list(map(float, r["pressure"])),
            "gpu_launches": r["launches"], "clocks": r["clocks"],
            "contact_kernel": {"kernel": name, "bound": DENSE_BOUND[prec], "achieved": ach,
                               "peak": peak, "unit": "GB/s", "frac": (ach / peak) if ach else None,
                               "bytes_per_atom": kb, "algorithmic_bytes_per_launch": kb * n,
                               "bytes_formula": "S + 4 n_nb + 52 n_c, S = 84 mixed / 140 FP64",
                               "kernel_ms": c_ms, "traffic": tr["bytes"] if tr else None,
                               "traffic_source": tr["source"] if tr else None}}
    if len(runs) == 2:
        m, f = out["forms"]["mixed"], out["forms"]["fp64"]
        out["speedup_mixed_vs_fp64"] = m["value"] / f["value"]
        out["mixed_mean_pressure_rel_err_vs_fp64"] = rel(m["mean_pressure"], f["mean_pressure"])
    return out


# ----------------------------------------------------------------- main


def oracle_pressure(p, steps):
    """Mean pressure of the oracle after the same number of steps (same run, FP64, all cores)."""
    from oracle import oracle as O
    O.build()
    sim = oracle_sim(O, p, os.cpu_count() or 1)
    sim.run(steps)
    return sim.last_pressure


def rel(a, b):
    a, b = float(a), float(b)
    return abs(a - b) / abs(b) if b != 0.0 else (0.0 if a == 0.0 else float("inf"))


TRIAXIAL_METRIC = "atom-steps/s, triaxial test (pair granular, rolling resistance) with logging every 100 steps"
E_MOD, POISSON = 5.0e6, 0.3
KN_EQUIV = (4.0 / 3.0) * E_MOD / (2.0 * (1.0 - POISSON ** 2))  # hertz/material's 4/3 E* (same elastic form)


def triaxial_packing(n, seed):
    """The config-2 procedure at this size, at the stiffness of hertz/material E 5e6, nu 0.3."""
    from taichimps_gb300.packing import compress_packing
    # strain capacity cycles x cycle_steps x dt x max_rate = 0.18 (0.4 -> 0.57 needs ~0.11)
    return compress_packing(n, seed=seed, kn=KN_EQUIV, max_rate=5e-4, dt=2e-4, cycles=40, cycle_steps=45000,
                            relax_cycles=6, phi0=0.4, jitter=0.25, precision="mixed")


def triaxial_sim(G, pk, precision):
    """pair granular hertz/material (E 5e6, coeff_restitution 0.5, nu 0.3), mindlin (kt from G*, xt 1,
    friction 0.5), rolling epsd (k_roll 1e3, gamma_roll 50, mu_roll 0.1); nve/sphere; deform/pressure:
    x and y pressure 1.0 (gain 0.1, max/rate 1e-2), z erate -1e-3, remap x; dt 5e-5."""
    n = len(pk["radius"])
    dom = G.Domain(boxlo=[float(a) for a in pk["lo"]], boxhi=[float(a) for a in pk["lo"] + pk["L"]],
                   boundary=("p", "p", "p"))
    atom = G.AtomSystem(max_atoms=n)
    atom.add_particles(x=pk["x"], radius=pk["radius"], density=pk["density"])
    nl = G.NeighborList(domain=dom, skin=0.1, max_atoms=n, max_neighbors_per_atom=32)
    hist = G.ContactHistory(max_atoms=n, max_neighbors=32)
    pair = G.PairGranular(domain=dom, normal="hertz/material", normal_coeffs=[E_MOD, 0.5, POISSON],
                          damping="coeff_restitution", tangential="mindlin", tangential_coeffs=[None, 1.0, 0.5],
                          rolling="epsd", rolling_coeffs=[1e3, 50.0, 0.1])
    sim = G.Simulation(domain=dom, atom=atom, neighbor=nl, history=hist, pair=pair, dt=5e-5, precision=precision)
    sim.add_fix(G.FixNVESphere(domain=dom))
    fx = G.FixDeformPressure(domain=dom, axes={"x": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1},
                                               "y": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1},
                                               "z": {"style": "erate", "rate": -1e-3}},
                             max_rate=1e-2, remap="x")
    sim.add_fix(fx)
    return sim, fx


def triaxial_log(G, sim, fx, steps, every):
    """Runs `steps` steps; every `every` steps logs the deviatoric stress q = p_zz - (p_xx + p_yy)/2,
    the volumetric strain eps_v = 1 - V / V0 (compression positive) and the coordination number."""
    import torch
    n = sim.atom.nlocal
    cn = G.ComputeContactAtom(max_atoms=n)
    dom = sim.domain
    dom.pull()
    v0 = float(np.prod(np.array(dom.boxhi) - np.array(dom.boxlo)))
    fx.record_pressure(8)
    log = []
    t_run = 0.0
    for k in range(steps // every):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        sim.run(every)
        torch.cuda.synchronize()
        t_run += time.perf_counter() - t0
        sim.run_pre = False
        P = fx.pressure_history([sim.timestep])[0]
        dom.pull()
        vol = float(np.prod(np.array(dom.boxhi) - np.array(dom.boxlo)))
        counts = cn.compute(sim.atom, dom, sim.neighbor)
        log.append((sim.timestep, float(P[2] - 0.5 * (P[0] + P[1])), 1.0 - vol / v0,
                    float(np.mean(counts))))
    return np.array(log), t_run


def run_triaxial(args):
    import torch
    import taichimps_gb300 as G
    n, steps = args.n, args.steps
    t0 = time.perf_counter()
    pk = triaxial_packing(n, args.seed)
    t_pack = time.perf_counter() - t0
    out = {}
    for prec in ("mixed", "fp64"):
        sim, fx = triaxial_sim(G, pk, prec)
        log, t_run = triaxial_log(G, sim, fx, steps, 100)
        out[prec] = {"log": log, "t": t_run}
        del sim, fx
        torch.cuda.empty_cache()
    m, f = out["mixed"]["log"], out["fp64"]["log"]
    qs = max(np.abs(f[:, 1]).max(), 1e-300)
    dev = lambda a, b, k: float(np.abs(a[:, k] - b[:, k]).max())
    first = lambda a, b, k, j: float(np.abs(a[:j, k] - b[:j, k]).max())
    return {"metric": TRIAXIAL_METRIC, "value": n * steps / out["mixed"]["t"], "unit": "atom-steps/s", "n_gpus": 1,
            "steps": steps, "warmup": 0, "ms_per_step": 1e3 * out["mixed"]["t"] / steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32/f64 mixed",
            "data": "synthetic: seeded packing compressed to p = 1 by the quenched isotropic servo at the "
                    "hertz/material stiffness (taichimps_gb300.packing.compress_packing)",
            "config": {"workload": f"triaxial test, {n} spheres, pair granular hertz/material + mindlin + rolling "
                                   f"epsd, x/y pressure 1.0, z erate -1e-3, {steps} steps, log every 100",
                       "n_atoms": n, "phi": pk["phi"], "pressure_start": [float(a) for a in pk["pressure"][:3]]},
            "fp64_atom_steps_per_s": n * steps / out["fp64"]["t"], "mixed_over_fp64": out["fp64"]["t"] / out["mixed"]["t"],
            "pack_s": t_pack,
            "mixed_vs_fp64": {"q_max_abs_dev_over_max_q": dev(m, f, 1) / qs,
                              "q_first_10_logs_over_max_q": first(m, f, 1, 10) / qs,
                              "eps_v_max_abs_dev": dev(m, f, 2), "cn_max_abs_dev": dev(m, f, 3)},
            "log_every": 100,
            "log_fp64": [[int(a), b, c, d] for a, b, c, d in f[::10]],
            "log_mixed": [[int(a), b, c, d] for a, b, c, d in m[::10]]}


ADJOINT_METRIC = "seconds per gradient of a stress-curve loss (forward + adjoint), triaxial calibration run"


def run_adjoint(args):
    """The calibration run's gradient: a packing compressed by the quenched isotropic servo
    (packing.compress_packing), then x/y pressure servo at 1.0 and z erate -1e-3 with remap x,
    gran/hertz/history kn 1e5, kt 2/7 kn, gamman 50, gammat 25, xmu 0.5, dt 5e-5; the loss is the
    squared difference of the deviatoric stress every 50 steps from the curve of kn 1.3e5, xmu 0.4.
    Times the forward (with checkpoints every 100 steps) and the reverse (recompute + adjoint)."""
    import torch
    from taichimps_gb300.adjoint import AdjointRun, stress_curve
    from taichimps_gb300.packing import compress_packing
    n, steps = args.n, args.steps
    t0 = time.perf_counter()
    pk = compress_packing(n, seed=args.seed)
    t_pack = time.perf_counter() - t0
    axes = {"x": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1},
            "y": {"style": "pressure", "ptarget": 1.0, "pgain": 0.1},
            "z": {"style": "erate", "rate": -1e-3}}
    run = AdjointRun(pk["x"], pk["radius"], pk["density"], pk["lo"], pk["lo"] + pk["L"], dt=5e-5, steps=steps,
                     axes=axes, max_rate=1e-2, sample_every=50, checkpoint_every=100)
    base = dict(kn=1.0e5, kt=1.0e5 * 2.0 / 7.0, gamman=50.0, gammat=25.0, xmu=0.5)
    target = run.forward(**dict(base, kn=1.3e5, xmu=0.4)).clone()
    T = lambda a: torch.tensor(a, dtype=torch.float64, requires_grad=True)
    ps = {k: T(v) for k, v in base.items()}
    r = torch.tensor(pk["radius"], dtype=torch.float64, device="cuda", requires_grad=True)
    times = []
    for rep in range(2):  # the second is timed (the first compiles nothing but warms the allocator)
        for v in ps.values():
            v.grad = None
        r.grad = None
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        q = stress_curve(run, ps["kn"], ps["kt"], ps["gamman"], ps["gammat"], ps["xmu"], r)
        torch.cuda.synchronize()
        t1 = time.perf_counter()
        loss = ((q - target) ** 2).sum()
        loss.backward()
        torch.cuda.synchronize()
        times.append((t1 - t0, time.perf_counter() - t1))
    t_f, t_b = times[-1]
    grads = {k: float(v.grad) for k, v in ps.items()}
    return {"metric": ADJOINT_METRIC, "value": t_f + t_b, "unit": "s", "n_gpus": 1, "steps": steps, "warmup": 1,
            "ms_per_step": 1e3 * (t_f + t_b) / steps, "higher_is_better": False, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64",
            "data": "synthetic: seeded packing compressed to p = 1 by the quenched isotropic servo "
                    "(taichimps_gb300.packing.compress_packing)",
            "config": {"workload": f"triaxial calibration gradient, {n} spheres, {steps} steps, q every 50 steps, "
                                   "checkpoints every 100", "n_atoms": n, "phi": pk["phi"],
                       "pressure_start": [float(a) for a in pk["pressure"][:3]]},
            "forward_s": t_f, "reverse_s": t_b, "pack_s": t_pack, "rebuilds": run.rebuilds,
            "loss": float(loss), "grad": dict(grads, radius_norm=float(r.grad.norm())),
            "forward_atom_steps_per_s": n * steps / t_f, "gradient_atom_steps_per_s": n * steps / (t_f + t_b)}


def main():
    args = parse()
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.workload == "triaxial":
        if args.impl != "ours" or world > 1:
            print(json.dumps({"impl": args.impl, "unavailable": "the triaxial workload runs on one GPU, ours only"}))
            return
        import torch
        torch.cuda.set_device(local)
        print(json.dumps(run_triaxial(args)), flush=True)
        return
    if args.workload == "adjoint":
        if args.impl != "ours" or world > 1:
            print(json.dumps({"impl": args.impl, "unavailable": "the reference has no differentiable path"}))
            return
        import torch
        torch.cuda.set_device(local)
        print(json.dumps(run_adjoint(args)), flush=True)
        return
    if args.workload == "ensemble":
        if args.impl != "ours" or world > 1:
            print(json.dumps({"impl": args.impl, "unavailable": "the ensemble workload runs on one GPU, ours only"}))
            return
        import torch
        torch.cuda.set_device(local)
        print(json.dumps(run_ensemble(args)), flush=True)
        return
    if args.workload == "dense":
        if args.impl != "ours":
            print(json.dumps({"impl": args.impl, "unavailable": "the dense line is part of the default run"}))
            return
        import torch
        torch.cuda.set_device(local)
        if world > 1:
            torch.distributed.init_process_group("nccl", device_id=torch.device("cuda", local))
        forms = ["mixed", "fp64"] if args.precision == "both" else [args.precision]
        out = run_dense(args, rank, world, forms)
        if out is not None:
            print(json.dumps(out), flush=True)
        if world > 1:
            torch.distributed.destroy_process_group()
        return
    if args.workload == "e2e":
        if args.impl != "ours" or rank != 0:
            if rank == 0:
                print(json.dumps({"impl": args.impl, "unavailable": "the e2e job is part of the default run"}))
            return
        import torch
        from taichimps_gb300.packing import config2
        torch.cuda.set_device(local)
        prec = "mixed" if args.precision == "both" else args.precision
        out = run_e2e(args, config2(seed=args.seed, n=args.n), prec)
        print(json.dumps({"workload": "e2e: " + WORKLOAD, "n_atoms": args.n, "steps": args.steps, "e2e": out}),
              flush=True)
        return
    if args.impl == "reference":
        out = reference_arm(args, rank, world)
        if out is not None:
            print(json.dumps(out), flush=True)
        return
    import torch
    from taichimps_gb300.packing import config2
    torch.cuda.set_device(local)
    if world > 1:
        torch.distributed.init_process_group("nccl", device_id=torch.device("cuda", local))
    p = config2(seed=replica_seed(args.seed, rank), n=args.n)
    forms = ["mixed", "fp64"] if args.precision == "both" else [args.precision]
    runs = {}
    for prec in forms:
        runs[prec] = run_gpu_arm(args, p, prec, rank, world)
        del runs[prec]["sim"]
        torch.cuda.empty_cache()
    if rank != 0:
        if world > 1:
            torch.distributed.destroy_process_group()
        return
    head = forms[0]
    r = runs[head]
    n, K, W = r["n"], args.steps, args.warmup
    values = {k: world * n * K / (v["ms"] * 1e-3) for k, v in runs.items()}
    value = values[head]
    peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
    peak = peaks.get("hbm_gbs", 6806.5)
    kern = r["kern_ms"]
    dom_name = max(("fused_a", "fused_c"), key=lambda k: kern.get(k) or 0.0)
    bytes_atom = algorithmic_bytes(dom_name, head, r["n_nb"], r["n_c"], r["flagged"])
    achieved = bytes_atom * n / (kern[dom_name] * 1e-3) / 1e9 if kern.get(dom_name) else None
    traffic = ncu_traffic(dom_name, head)
    c_bytes = algorithmic_bytes("fused_c", head, r["n_nb"], r["n_c"], r["flagged"])
    c_traffic = ncu_traffic("fused_c", head)
    e2e = None if args.no_e2e else run_e2e(args, p, head)
    dense = None if args.no_dense else run_dense(args, rank, world, forms)
    fp64_peak = fp64_peak_dfma_per_s() if "fp64" in runs else None
    cpu = None
    p_oracle = None
    if not args.no_cpu:
        # a bounded sample: as many steps as --cpu-budget seconds of CPU work allow (~10-15 s)
        cpu, _ = cpu_baseline(p, args.cpu_budget, 1_000_000)
        # the oracle runs as many steps as each GPU form ran in all (warm-up, graph capture, timed
        # replays and the per-kernel timing pass); every form runs the same count
        steps_run = {v["steps_run"] for v in runs.values()}
        assert len(steps_run) == 1, steps_run
        p_oracle = oracle_pressure(p, steps_run.pop())
    scal = lambda t: (t[0] + t[1] + t[2]) / 3.0
    forms_out = {}
    for k, v in runs.items():
        kb = {kk: algorithmic_bytes(kk, k, v["n_nb"], v["n_c"], v["flagged"]) for kk in ("fused_a", "fused_c")}
        forms_out[k] = {
            "value": values[k], "ms_per_step": v["ms"] / K, "kernel_ms": v["kern_ms"],
            "kernel_gbs": {kk: (kb[kk] * n / (v["kern_ms"][kk] * 1e-3) / 1e9 if v["kern_ms"].get(kk) else None)
                           for kk in kb},
            "mean_pressure": scal(v["pressure"]), "pressure": list(map(float, v["pressure"])),
            "mean_pressure_rel_err_vs_oracle": None if p_oracle is None else rel(scal(v["pressure"]), scal(p_oracle)),
            "gpu_launches": v["launches"], "rebuilds_in_timed_steps": v["rebuilds_timed"],
            "groups_culled": {"groups": v["cull"][0], "culled_after_timed_steps": v["cull"][1]},
            "flagged_atoms_frac": v["flagged"],
            "kernel_bytes_per_atom": kb,
            "kernel_bytes_note": "algorithmic bytes (see algorithmic_bytes); fused_c on this contact-free state "
                                 "moves far fewer (its bound check), so its GB/s figure is nominal"}
        if k == "fp64":
            forms_out[k]["fp64_roofline"] = fp64_roofline("k_a64", n, v["kern_ms"].get("fused_a"), fp64_peak)
    out = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": K, "warmup": W,
        "ms_per_step": r["ms"] / K, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": value / PUBLISHED_FP32,
        "dtype": "f32/f64 mixed" if head == "mixed" else "f64",
        "data": "synthetic: seeded FCC-site packing, d~U[0.8,1.2], phi 0.45, at rest (taichimps_gb300.packing.config2)",
        "config": {"workload": WORKLOAD, "n_atoms": n, "precision": head, "parallelism": f"replicas{world}",
                   "l2": "inputs larger than L2: ~0.4 GB of per-atom and neighbor state per replica",
                   "neighbors_per_atom": r["n_nb"], "contacts_per_atom": r["n_c"], "neighbor_builds": r["builds"]},
        "roofline": {"kernel": KERNEL_NAMES[(dom_name, head)], "bound": "hbm", "achieved": achieved, "peak": peak,
                     "unit": "GB/s", "frac": (achieved / peak) if achieved else None,
                     "traffic": traffic["bytes"] if traffic else None,
                     "traffic_source": traffic["source"] if traffic else None,
                     "algorithmic_bytes_per_launch": bytes_atom * n, "bytes_per_atom": bytes_atom,
                     "layout_bytes_per_atom": layout_bytes(dom_name, head, r["flagged"]),
                     "kernel_ms": kern[dom_name], "peak_source": "measured (MEASURED_PEAKS.json hbm_gbs)"},
        # the contact kernel on this contact-free state: its bound check rules out most groups, so it
        # moves a small part of the nominal S + 4 n_nb + 52 n_c bytes per atom (traffic) and its time
        # is latency; no roofline fraction is claimed here -- the contact-dense line ("dense") carries
        # the contact kernel's roofline on the bytes it moves
        "contact_kernel": {"kernel": KERNEL_NAMES[("fused_c", head)], "bound": "latency (contact-free state)",
                           "frac": None, "nominal_bytes_per_atom": c_bytes, "kernel_ms": kern.get("fused_c"),
                           "traffic": c_traffic["bytes"] if c_traffic else None},
        "speedup_mixed_vs_fp64": (values["mixed"] / values["fp64"]) if len(values) == 2 else None,
        "oracle_mean_pressure": None if p_oracle is None else scal(p_oracle),
        "pressure_compared_after_steps": r["steps_run"],
        "forms": forms_out,
        "cpu_baseline": cpu, "e2e": e2e, "gpu_launches": r["launches"], "clocks": r["clocks"],
        "dense": dense,
    }
    print(json.dumps(out), flush=True)
    if world > 1:
        torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
