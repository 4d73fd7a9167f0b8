"""Benchmark of the tet-DG RHS hot path on B200: DOF-stage-updates/s of LSERK4 stages.

Default workload: 3-D scalar Burgers, nodal DG order N=4 (Np=35, Nfp=15) on a periodic 64^3 x 6
Kuhn-cube mesh (K = 1,572,864 tets), 16 x-slab partitions, u0 = 0.5 + 8 seeded random Fourier modes.  One
"step" is one LSERK4 stage over all K elements: the fused volume + Lax-Friedrichs surface + LIFT + stage update
kernel.  Four forms run from the same initial state: plain FP64 (rhsStage, reference-contract layout), plain
FP32, mixed (rhsStageMixed: compensated FP32 state, FP32 products on the element's higher-order part,
compact affine geometry and compressed face maps) and mixed_tc (the same stage with its products on the tensor
cores, three-part BF16 operands, FP32 accumulation).  `value` is the chosen form: the fastest one whose
relative L2 error against the FP64 run stays <= 1e-6 at t_final (after the warm-up and timed stages).

Usage: python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference] [--n 64] [--order 4]
Under torchrun (N > 1) every rank runs an independent replica (the path shards by partition; one GPU per
replica) and the time is the max over ranks.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, HERE)

METRIC = "DOF-stage-updates/s on 1 B200, chosen vs plain FP64 at L2 err≤1e-6; %HBM"
UNIT = "DOF-stage-updates/s"
FALLBACK_HBM_GBS = 6650.0


def peaks():
    try:
        with open(os.path.join(HERE, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


def peaks_bf16():
    """Dense bf16 tensor rate in TFLOP/s: the driver-measured burst figure, else the pool's fallback."""
    try:
        with open(os.path.join(HERE, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return float(d["bf16_tflops"]), "measured"
    except Exception:
        return 1590.0, "fallback"


def b_alg_mixed(N: int) -> float:
    """Algorithmic bytes per DOF-stage of the mixed stage: hi, lo and resu read and written (FP32), plus the
    compact per-element geometry (8 floats) and connectivity (5 int32) spread over the Np nodes."""
    Np = (N + 1) * (N + 2) * (N + 3) // 6
    return 6 * 4 + (8 * 4 + 5 * 4) / Np


def b_alg_tcm(N: int, halo_per_elem: float) -> float:
    """Algorithmic bytes per DOF-stage of the tensor-core mixed stage: hi, lo and resu read and written (FP32),
    the compact per-element geometry (8 floats), the tile-local connectivity (4 int32) and the tile's halo list
    (8 bytes per face whose neighbour lies outside the tile), spread over the Np nodes."""
    Np = (N + 1) * (N + 2) * (N + 3) // 6
    return 6 * 4 + (8 * 4 + 4 * 4 + 8 * halo_per_elem) / Np


def b_alg_f64_compact(N: int) -> float:
    """Algorithmic bytes per DOF-stage of the FP64 stage on the compact layout: u and resu read, u and resu
    written (FP64), plus the per-element geometry (25 doubles) and compact connectivity (5 int32) spread over the
    Np nodes."""
    Np = (N + 1) * (N + 2) * (N + 3) // 6
    return 4 * 8 + (25 * 8 + 5 * 4) / Np


def kuhn_halo_per_elem(n: int, slabs: int, tile: int = 128) -> float:
    """Faces per element whose neighbour lies outside the element's tile (tiles of `tile` consecutive elements
    of one x-slab partition) on the periodic n^3 x 6 Kuhn mesh: the halo the tensor-core stage gathers."""
    from dgkernel_b200 import mesh as M
    _, _, _, _, EToVp, EToP = M.kuhn_mesh(n, slabs)
    EToE, _ = M.ti_connect3d(EToVp)
    K = EToE.shape[0]
    Kp = K // slabs
    e = np.arange(K)
    first = (e // Kp) * Kp + ((e % Kp) // tile) * tile  # first element of each element's tile
    last = np.minimum(first + tile, (e // Kp + 1) * Kp)
    outside = (EToE < first[:, None]) | (EToE >= last[:, None])
    return float(outside.sum()) / K


def b_alg_per_dof(N: int, elem_bytes: int) -> float:
    """Algorithmic bytes per DOF-stage of the fused stage kernel in the reference-contract layout:
    u read + resu read + resu write + u write, 9 per-node metrics, and per face point nx, ny, nz, Fscale plus
    one int32 gather index, spread over the Np nodes (neighbour traces assumed L2 hits)."""
    Np = (N + 1) * (N + 2) * (N + 3) // 6
    Nfp = (N + 1) * (N + 2) // 2
    r = 4 * Nfp / Np
    return 4 * elem_bytes + 9 * elem_bytes + r * (4 * elem_bytes + 4)


class ClockSampler:
    """SM clocks and throttle reasons sampled while running: NVML reads every 2 ms from a thread (short timed
    regions still get samples), else nvidia-smi every 100 ms."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")
    NAMES = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")

    def __init__(self, index: int, period_s: float = 0.002):
        self.index, self.period, self.rows, self.proc, self.nv = index, period_s, [], None, None
        self.stop = threading.Event()

    def _nvml_index(self):
        vis = os.environ.get("CUDA_VISIBLE_DEVICES", "")
        ids = [v for v in vis.split(",") if v.strip()]
        if ids and all(v.strip().isdigit() for v in ids) and self.index < len(ids):
            return int(ids[self.index])
        return self.index

    def __enter__(self):
        try:
            import pynvml as nv
            nv.nvmlInit()
            self.nv, self.h = nv, nv.nvmlDeviceGetHandleByIndex(self._nvml_index())
            self.masks = (nv.nvmlClocksEventReasonHwSlowdown, nv.nvmlClocksEventReasonHwThermalSlowdown,
                          nv.nvmlClocksEventReasonSwThermalSlowdown, nv.nvmlClocksEventReasonSwPowerCap)
            self.smax = nv.nvmlDeviceGetMaxClockInfo(self.h, nv.NVML_CLOCK_SM)
            self.t = threading.Thread(target=self._poll, daemon=True)
            self.t.start()
            return self
        except Exception:
            self.nv = None
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None
        return self

    def _poll(self):
        nv = self.nv
        while not self.stop.is_set():
            try:
                sm = nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM)
                rs = nv.nvmlDeviceGetCurrentClocksEventReasons(self.h)
                self.rows.append([str(self.index), str(sm), str(self.smax), "", ""] +
                                 ["Active" if rs & m else "Not Active" for m in self.masks])
            except Exception:
                return
            time.sleep(self.period)

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([c.strip() for c in line.split(",")])

    def __exit__(self, *a):
        self.stop.set()
        if self.nv is not None:
            self.t.join(timeout=1)
            try:
                self.nv.nvmlShutdown()
            except Exception:
                pass
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"], "samples": 0}
        sm = [float(r[1]) for r in self.rows if r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if r[2].replace(".", "").isdigit()]
        reasons = sorted({self.NAMES[i] for r in self.rows for i in range(4)
                          if len(r) > 5 + i and r[5 + i] == "Active"})
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": reasons, "samples": len(self.rows), "source": "nvml" if self.nv else "nvidia-smi"}


def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import datetime
        import torch
        import torch.distributed as dist
        if torch.cuda.is_available():
            torch.cuda.set_device(local)
            dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
        else:  # host-only ranks (the reference arm's plumbing, tests): gloo
            dist.init_process_group("gloo", timeout=datetime.timedelta(seconds=300))
    return world, rank, local


def max_over_ranks(x: float, world: int) -> float:
    if world == 1:
        return x
    import torch
    import torch.distributed as dist
    dev = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], device=dev, dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def barrier(world: int):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


def time_stages(prob, steps: int, stream):
    """Run `steps` stages on `stream`, CUDA events on that stream, synchronize on both sides."""
    import torch
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record(stream)
    prob.run_stages(steps)
    e1.record(stream)
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / steps  # ms per stage


def cpu_baseline(N: int, steps: int, seconds: float = 12.0, n: int = 16, slabs: int = 16, serial_stages: int = 0):
    """Oracle port (C restatement of the OKL loops, OpenMP over the @outer partition loop) on the host cores:
    order N, `slabs` x-slab partitions of an n^3 x 6 Kuhn mesh, set up by the oracle's own numpy restatement of
    the reference's setup chain (no GPU involved).  Times `steps` stages (or as many as fit in `seconds` when
    steps is 0) with one thread per partition up to the host's cores, then `serial_stages` stages on 1 thread
    (the OCCA Serial mode)."""
    from oracle import burgers_ref as BR
    from oracle import oracle as O
    t0 = time.perf_counter()
    ref = BR.Problem(N, n, slabs, "modes")
    rs = O.RunState(ref)
    setup_s = time.perf_counter() - t0
    u = np.ascontiguousarray(ref.u0, dtype=np.float64).copy()
    resu = np.zeros_like(u)
    P = len(rs.K)
    threads = max(1, min(os.cpu_count() or 1, P))
    rs.run(u, resu, ref.dt, 1, 0, 0, threads)  # warm-up stage
    done, t0 = 0, time.perf_counter()
    while True:
        rs.run(u, resu, ref.dt, 1, done % 5, 0, threads)
        done += 1
        el_t = time.perf_counter() - t0
        if (steps and done >= steps) or (not steps and el_t >= seconds):
            break
    value = u.size * done / el_t
    out = {"value": value, "unit": UNIT, "cores": threads, "kind": "port",
           "sample": f"order {N}, {n}^3x6 Kuhn mesh ({ref.K:,} tets, {P} x-slab partitions), {done} LSERK4 stages of "
                     f"exchange + LF RHS + update, C restatement of the OKL loops (gcc -O3 -fopenmp, "
                     f"-ffp-contract=off), OpenMP over partitions, {threads} threads of {os.cpu_count()} host cores",
           "seconds": el_t, "setup_s": setup_s}
    if serial_stages:
        t0 = time.perf_counter()
        rs.run(u, resu, ref.dt, serial_stages, done % 5, 0, 1)
        ser = time.perf_counter() - t0
        out["serial"] = {"value": u.size * serial_stages / ser, "unit": UNIT, "cores": 1, "stages": serial_stages,
                         "seconds": ser}
    return out


def run_reference(args, world, rank):
    """The reference arm: the oracle port of the reference's OKL loops on the host cores, on the same workload as
    our arm (order, mesh, partitions, u0), `steps` stages after one warm-up stage; plus a Serial (1 core)
    sample."""
    if rank != 0:
        return
    base = cpu_baseline(args.order, args.steps, n=args.n, slabs=args.slabs, serial_stages=1)
    Np = (args.order + 1) * (args.order + 2) * (args.order + 3) // 6
    out = {"impl": "reference", "metric": METRIC, "value": base["value"], "unit": UNIT, "n_gpus": args.gpus,
           "steps": args.steps, "warmup": args.warmup, "ms_per_step": base["seconds"] / max(1, args.steps) * 1e3,
           "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
           "config": {"workload": f"3-D Burgers tet-DG, order {args.order} (Np={Np}), periodic {args.n}^3x6 Kuhn "
                                  f"mesh (K={6 * args.n ** 3}), {args.slabs} x-slab partitions, u0 = 0.5 + 8 seeded "
                                  f"Fourier modes; one step = one LSERK4 stage (the reference's CPU path: OpenMP "
                                  f"over partitions, one warm-up stage; Serial 1-core sample in cpu_baseline.serial)"},
           "cpu_baseline": base, "e2e": {"value": base["value"], "unit": UNIT, "h2d_bytes_per_step": 0,
                                         "d2h_bytes_per_step": 0}}
    print(json.dumps(out), flush=True)


def run_ensemble(args, world, rank, local):
    """Batching workload: 256 independent order-3 instances, n_i ~ U{6..24} (seeded), FP32 compensated state (mixed
    stage), one persistent launch per stage, stages replayed from a captured CUDA graph, autotuned shape."""
    import torch
    from dgkernel_b200.burgers import BurgersEnsemble, ensemble_sizes
    from dgkernel_b200 import autotune as T
    torch.cuda.set_device(local)
    stream = torch.cuda.Stream()
    t0 = time.time()
    E = BurgersEnsemble(3, ensemble_sizes(256), stream=stream.cuda_stream)
    setup_s = time.time() - t0
    best = T.autotune(E)
    E.run_stages(5)
    E.run_stages(5)
    g = E.capture_steps(2)
    reps = max(1, args.steps // 10)
    E.run_graph(g, 1)
    # The instances are inviscid and unlimited: past t ~ 0.17 (about 200 stages) the finest ones form shocks and
    # leave the stable range.  The timed stages therefore run in blocks of at most 100 (10 graph replays), each
    # from the same smooth state restored on the device outside the timed region (stage work does not depend on
    # the values).
    E.runner.ExecuteKernel("joinState")  # the FP64 array u keeps the smooth start (the stages touch only hi, lo)
    barrier(world)
    torch.cuda.synchronize()
    elapsed, ok = 0.0, True
    with ClockSampler(local) as clk:
        left = reps
        while left > 0:
            nrep = min(10, left)
            E.runner.ExecuteKernel("splitState")
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            E.run_graph(g, nrep)
            e1.record(stream)
            torch.cuda.synchronize()
            elapsed += e0.elapsed_time(e1)
            left -= nrep
        ok = bool(np.isfinite(E.get("u")).all())
    ms = max_over_ranks(elapsed / (10 * reps), world)
    if rank == 0:
        out = {"metric": "DOF-stage-updates/s, batching form (256 order-3 instances)", "value": world * E.dofs / (ms * 1e-3),
               "unit": UNIT, "n_gpus": world, "steps": 10 * reps, "warmup": 10, "ms_per_step": ms,
               "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32x2+f32",
               "data": "synthetic",
               "config": {"workload": f"256 independent 3-D Burgers instances, order 3, n_i^3 x 6 Kuhn meshes with "
                                      f"n_i ~ U{{6..24}} (K = {E.K}), one partition per instance, seeded "
                                      f"random-mode u0 per instance; one step = one LSERK4 stage of all instances",
                          "launch": "one persistent mixed-stage launch per stage, 10-stage CUDA graph replayed",
                          "timed_blocks": "blocks of <= 100 stages, each from the same smooth state (restored "
                                          "untimed): the inviscid instances form shocks after ~200 stages",
                          "tuned_shape": best, "setup_s": setup_s, "finite": ok},
               "clocks": clk.summary(), "gpu_launches": 10 * reps}
        print(json.dumps(out), flush=True)
    g.Free()
    E.free()


def oz_ops_per_element(N: int, S: int = 6) -> float:
    """Integer multiply-adds x 2 per element and stage of the exact-digit precision kernel as issued (digit
    products p + q <= S - 1 over 128 matrix rows and the padded K of the volume, 3 rup32(Np), and LIFT,
    rup32(4 Nfp))."""
    Np = (N + 1) * (N + 2) * (N + 3) // 6
    Nfp = (N + 1) * (N + 2) // 2
    r32 = lambda x: (x + 31) // 32 * 32
    return 2.0 * 128 * (3 * r32(Np) + r32(4 * Nfp)) * S * (S + 1) / 2


def run_precision(args, world, rank, local):
    """Precision workload: order 7, 32^3 x 6 Kuhn mesh, u0 = 0.5 + 0.25 sin(pi x) cos(pi y) sin(pi z), to t = 0.2:
    the precision form (both element-local products as exact 8-bit-digit GEMMs on the tensor cores, six digits
    per operand joined in FP64, compensated FP32 state) against the plain FP64 run of the same mesh, with L2 and
    Linf errors at t_final; the same at order 4 beside it."""
    import torch
    from dgkernel_b200.burgers import BurgersProblem, MIXED
    torch.cuda.set_device(local)
    stream = torch.cuda.Stream()
    n = 32 if args.n == 64 else args.n
    ops_peak = 2.0 * peaks_bf16()[0]  # dense int8 rate = twice the bf16 rate on B200
    per_order = {}
    for order in (7, 4):
        res = {}
        for name, dt in (("f64", np.float64), ("tc", MIXED)):
            P = BurgersProblem(order, n, 1, dt, "smooth", stream=stream.cuda_stream,
                               tensor=True if dt == MIXED else None)
            nst = max(5 * int(np.ceil(args.t_final / P.dt)), args.warmup + 5)
            P.run_stages(args.warmup)
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            with ClockSampler(local) as clk:
                e0.record(stream)
                P.run_stages(nst - args.warmup)
                e1.record(stream)
                torch.cuda.synchronize()
            res[name] = {"ms": e0.elapsed_time(e1) / (nst - args.warmup), "u": P.get("u"), "dofs": P.dofs,
                         "stages": nst, "clk": clk.summary(), "K": P.K}
            P.free()
        ref, tc = res["f64"]["u"], res["tc"]["u"]
        fin = bool(np.isfinite(tc).all())
        ops = oz_ops_per_element(order) * res["tc"]["K"] / (res["tc"]["ms"] * 1e-3) / 1e12
        per_order[order] = {
            "tc_value": world * res["tc"]["dofs"] / (res["tc"]["ms"] * 1e-3), "tc_ms_per_step": res["tc"]["ms"],
            "fp64_value": world * res["f64"]["dofs"] / (res["f64"]["ms"] * 1e-3), "fp64_ms_per_step": res["f64"]["ms"],
            "speedup_vs_fp64": res["f64"]["ms"] / res["tc"]["ms"],
            "stages": res["tc"]["stages"], "finite": fin,
            "l2_err_vs_fp64": float(np.linalg.norm(tc - ref) / np.linalg.norm(ref)) if fin else None,
            "linf_err_vs_fp64": float(np.max(np.abs(tc - ref)) / np.max(np.abs(ref))) if fin else None,
            "int8_tops": ops, "tensor_frac": ops / ops_peak,
            "clocks": res["tc"]["clk"]}
    if rank == 0:
        m = per_order[7]
        out = {"metric": "DOF-stage-updates/s, precision form (order 7, 32^3x6)", "value": m["tc_value"], "unit": UNIT,
               "n_gpus": world, "steps": m["stages"], "warmup": args.warmup, "ms_per_step": m["tc_ms_per_step"],
               "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
               "dtype": "i8 digits x6 (exact int32 acc, f64 join), f32x2 state",
               "data": "synthetic",
               "config": {"workload": f"3-D Burgers, order 7 (Np=120), periodic {n}^3x6 Kuhn mesh, u0 = 0.5 + 0.25 "
                                      f"sin cos sin, to t = {args.t_final}; order 4 on the same mesh beside it",
                          "orders": {str(k): {kk: vv for kk, vv in v.items() if kk != "clocks"}
                                     for k, v in per_order.items()}},
               "roofline": {"bound": "tensor", "achieved": m["int8_tops"], "peak": ops_peak, "unit": "TOPS (int8)",
                            "frac": m["tensor_frac"], "traffic": None, "kernel": "rhs_stage_oz_kernel",
                            "peak_kind": "twice the measured bf16 dense rate",
                            "ops_per_element": oz_ops_per_element(7)},
               "clocks": m["clocks"], "gpu_launches": m["stages"]}
        print(json.dumps(out), flush=True)


def run_learned(args, world, rank, local):
    """Learned-sensor workload: shock-forming u0 = 0.5 + sin sin sin, order 4, 48^3 x 6, to t = 0.5 with artificial
    viscosity.  The sensor network is trained first (library kernels) on (modal features, PP activation) pairs
    from PP runs on random-mode fields.  The judge is the PP-sensor FP64 viscosity stage.  The timed form is the
    composite: the tensor-core mixed stage with the sensor over every element and the BR1 viscous term only where
    it is not zero, run with the PP sensor, the network (PP fallback in the low-confidence band) and the network
    reading outputs below the band as smooth; each run's stage rate and relative L1 error against the judge at
    t_final are reported, beside the plain FP64 stage's rate on the same mesh."""
    import torch
    from dgkernel_b200.burgers import BurgersProblem, MIXED
    from dgkernel_b200 import sensor as SN
    torch.cuda.set_device(local)
    stream = torch.cuda.Stream()
    n = args.n if args.n != 64 else 48
    t0 = time.time()
    X, Y = [], []
    for seed, nn in ((300, 24), (301, 24), (302, 32), (303, 32)):  # two resolutions: shocks as the target mesh sees them
        P = BurgersProblem(4, nn, 1, np.float64, "modes", seed=seed, viscosity="pp", mode_sigma=0.2, eps0=2.0,
                           stream=stream.cuda_stream)
        x, y = SN.collect_pairs(P, 0.6, every=40)
        X.append(x)
        Y.append(y)
        P.free()
    X, Y = np.concatenate(X), np.concatenate(Y)
    npairs, active = len(Y), float((Y > 0).mean())
    Xb, Yb = SN.balance(X, Y, 0.6)
    data_s = time.time() - t0
    t0 = time.time()
    net = SN.SensorNet(35, seed=13)
    hist = net.fit(torch.tensor(Xb, device="cuda"), torch.tensor(Yb, device="cuda"), epochs=60, batch=8192)
    train_s = time.time() - t0
    params = net.numpy()

    def timed_run(P):
        nst = 5 * int(np.ceil(0.5 / P.dt))
        P.run_stages(args.warmup)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        with ClockSampler(local) as clk:
            e0.record(stream)
            P.run_stages(nst - args.warmup)
            e1.record(stream)
            torch.cuda.synchronize()
        return {"u": P.get("u"), "ms": e0.elapsed_time(e1) / (nst - args.warmup), "dofs": P.dofs, "stages": nst,
                "clk": clk.summary()}

    runs = {}
    J = BurgersProblem(4, n, 1, np.float64, "shock", viscosity="pp", eps0=2.0, stream=stream.cuda_stream)
    runs["fp64_pp"] = timed_run(J)
    dt = J.dt
    J.free()
    for sensor in ("pp", "mlp0", "mlp"):
        P = BurgersProblem(4, n, 1, MIXED, "shock", mma=True, learned=sensor, eps0=2.0, stream=stream.cuda_stream)
        assert abs(P.dt - dt) <= 1e-12 * dt
        if sensor != "pp":
            P.set_sensor(sensor, params)
        runs[sensor] = timed_run(P)
        P.free()
    # the plain FP64 stage (no viscosity) on the same mesh: the per-DOF rate the composite is compared with
    F = BurgersProblem(4, n, 1, np.float64, "shock", stream=stream.cuda_stream)
    F.run_stages(args.warmup)
    fp64_ms = time_stages(F, 20, stream)
    F.free()
    ref = runs["fp64_pp"]["u"]
    l1 = {k: (float(np.abs(v["u"] - ref).sum() / np.abs(ref).sum()) if np.all(np.isfinite(v["u"])) else None)
          for k, v in runs.items() if k != "fp64_pp"}
    dofs = runs["mlp0"]["dofs"]
    rate = {k: world * dofs / (v["ms"] * 1e-3) for k, v in runs.items()}
    fp64_rate = world * dofs / (fp64_ms * 1e-3)
    # roofline of the composite stage on the bytes every stage moves: the tensor-core stage (state, geometry,
    # tile-local connectivity, halo lists) and the sensor pass (the state read once, eps / active row / h / N
    # per element); the sparse passes' bytes vary with the active set and are not counted
    Np = 35
    hbm, peak_kind = peaks()
    b_alg = b_alg_tcm(4, kuhn_halo_per_elem(n, 1)) + 8 + (8 + 4 + 8) / Np
    achieved = b_alg * dofs / (runs["mlp0"]["ms"] * 1e-3) / 1e9
    if rank == 0:
        m = runs["mlp0"]
        out = {"metric": "DOF-stage-updates/s, learned-sensor form (order 4, 48^3x6 shock)", "value": rate["mlp0"],
               "unit": UNIT, "n_gpus": world, "steps": m["stages"], "warmup": args.warmup, "ms_per_step": m["ms"],
               "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
               "dtype": "f32x2+f32 (bf16x3 products) + f64 sparse viscosity, sensor f64/f16",
               "data": "synthetic",
               "config": {"workload": f"3-D Burgers, order 4, {n}^3 x 6 Kuhn mesh ({6 * n ** 3} tets), u0 = 0.5 + sin "
                                      "sin sin, to t = 0.5 with BR1 artificial viscosity eps = eps0 sigma h / N (eps0 "
                                      "2); composite stage: tensor-core mixed stage + sensor over every element + "
                                      "viscous term where it is not zero",
                          "chosen_sensor": "mlp0 (network; outputs below the confidence band read as smooth; PP "
                                           "fallback inside the band)",
                          "ms_per_stage": {k: v["ms"] for k, v in runs.items()},
                          "dof_stage_per_s": rate, "plain_fp64_stage_ms": fp64_ms,
                          "plain_fp64_dof_stage_per_s": fp64_rate,
                          "vs_plain_fp64": {k: rate[k] / fp64_rate for k in rate},
                          "l1_err_vs_pp_fp64": l1, "stages": m["stages"], "training_pairs": npairs,
                          "active_fraction": active, "balanced_pairs": int(len(Yb)),
                          "train_loss": [hist[0], hist[-1]], "data_s": data_s, "train_s": train_s},
               "roofline": {"bound": "hbm", "achieved": achieved, "peak": hbm, "unit": "GB/s", "frac": achieved / hbm,
                            "traffic": None, "peak_kind": peak_kind, "b_alg_per_dof": b_alg,
                            "kernel": "composite stage (sensor pass + tensor-core stage; sparse passes not counted)"},
               "clocks": m["clk"], "gpu_launches": 7 * m["stages"]}
        print(json.dumps(out), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=400)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--n", "--cubes", dest="n", type=int, default=64, help="cubes per axis of the Kuhn mesh")
    ap.add_argument("--order", type=int, default=4)
    ap.add_argument("--slabs", type=int, default=16)
    ap.add_argument("--e2e-steps", type=int, default=8)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--t-final", type=float, default=0.2, help="precision workload: final time (0.2)")
    ap.add_argument("--workload", default="burgers", choices=["burgers", "ensemble", "learned", "precision"],
                    help="burgers: order 4, 64^3x6 (default); precision: order 7, 32^3x6; ensemble: 256 order-3 "
                         "instances; learned: order 4, 48^3x6 shock with the learned sensor")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    world, rank, local = dist_setup(args)
    try:
        if args.impl == "reference":
            return run_reference(args, world, rank)
        if args.workload == "ensemble":
            return run_ensemble(args, world, rank, local)
        if args.workload == "learned":
            return run_learned(args, world, rank, local)
        if args.workload == "precision":
            return run_precision(args, world, rank, local)
        return run_burgers(args, world, rank, local)
    finally:
        if world > 1:
            import torch.distributed as dist
            dist.destroy_process_group()


def volume_microbench(prob, stream, hbm, local, launches: int = 20, warmup: int = 3):
    """The standalone volume derivative (`differentiate`: Dr/Ds/Dt applied to u, then the nine per-node metrics)
    on the benchmark mesh, FP64, in HBM GB/s by the reference's own formula 13 * 8 B * Np * K / t (U, nine
    metrics, three outputs; tetnudg/tet_nudg_mesh_physical_derivative_test.go:544-547).  Every launch streams
    13 arrays of K Np doubles, far larger than L2.  Checked against the analytic derivative of the initial
    field (a size-independent property: the interpolation error of the order-N nodal field)."""
    import torch
    from dgkernel_b200.burgers import random_modes, DEFAULT_SEED
    prob.differentiate(warmup)
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local) as clk:
        e0.record(stream)
        prob.differentiate(launches)
        e1.record(stream)
        torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / launches
    Np, K = prob.el.Np, prob.K
    nbytes = 13 * 8 * Np * K
    gbs = nbytes / (ms * 1e-3) / 1e9
    X, Y, Z = prob.get("X"), prob.get("Y"), prob.get("Z")
    ux = np.zeros_like(X)
    for kx, ky, kz, a, phi in random_modes(DEFAULT_SEED):
        ux -= a * np.pi * kx * np.sin(np.pi * (kx * X + ky * Y + kz * Z) + phi)
    got = prob.get("DuDx")
    err = float(np.linalg.norm(got - ux) / np.linalg.norm(ux))
    return {"value": gbs, "unit": "GB/s", "ms_per_launch": ms, "launches": launches, "bytes_per_launch": nbytes,
            "formula": "13 * 8 B * Np * K / t (tet_nudg_mesh_physical_derivative_test.go:544-547)",
            "hbm_frac": gbs / hbm, "dof_per_s": Np * K / (ms * 1e-3), "kernel": "diff_dmma_kernel",
            "dudx_rel_err_vs_analytic": err, "clocks": clk.summary()}


def run_burgers(args, world, rank, local):
    """The default line (order 4, 64^3 x 6): plain FP64, plain FP32 and the mixed forms from one u0; the chosen
    form."""
    import torch
    from dgkernel_b200.burgers import BurgersProblem, RK4A, RK4B, MIXED
    torch.cuda.set_device(local)
    stream = torch.cuda.Stream()
    hbm, peak_kind = peaks()
    results = {}
    finals = {}
    # mixed_tc: the mixed stage with its element-local products on the tensor cores (orders 1..4)
    # f64c: the FP64 stage on the compact layout (the control that separates layout from precision)
    forms = [("f64", np.float64, {}), ("f64c", np.float64, {"compact": True}), ("f32", np.float32, {}),
             ("mixed", MIXED, {})]
    if args.order <= 4:
        forms.append(("mixed_tc", MIXED, {"mma": True}))
    kernels = {"f64": "rhs_stage_dmma_kernel", "f64c": "rhs_stage_dmma_kernel (compact)", "f32": "rhs_stage_dmma_kernel (float)",
               "mixed": "rhs_stage_mixed_kernel", "mixed_tc": "rhs_stage_tcm_kernel"}
    micro = None
    for name, dt, kw in forms:
        if name == "f64":
            kw = dict(kw, derivatives=True)
        prob = BurgersProblem(args.order, args.n, args.slabs, dt, "modes", stream=stream.cuda_stream, **kw)
        if name == "f64":
            micro = volume_microbench(prob, stream, hbm, local)
        prob.run_stages(args.warmup)
        barrier(world)
        with ClockSampler(local) as clk:
            ms = time_stages(prob, args.steps, stream)
        ms = max_over_ranks(ms, world)
        finals[name] = prob.get("u").astype(np.float64)
        results[name] = {"ms": ms, "dofs": prob.dofs, "clocks": clk.summary(), "prob": prob,
                         "b_alg": b_alg_tcm(args.order, kuhn_halo_per_elem(args.n, args.slabs))
                         if name == "mixed_tc" else b_alg_mixed(args.order) if name == "mixed" else
                         b_alg_f64_compact(args.order) if name == "f64c" else
                         b_alg_per_dof(args.order, 8 if name == "f64" else 4),
                         "kernel": kernels[name]}
        if name != "f64":
            prob.free()
    ref = finals["f64"]
    errs = {k: float(np.linalg.norm(v - ref) / np.linalg.norm(ref)) for k, v in finals.items()}
    dofs = results["f64"]["dofs"]
    thr = {k: world * dofs / (v["ms"] * 1e-3) for k, v in results.items()}
    eligible = [k for k in thr if errs[k] <= 1e-6]
    chosen = max(eligible, key=lambda k: thr[k])
    ch = results[chosen]

    # end to end through the runner's ExecuteKernel with the chosen form's state copied from and to pinned host
    # memory every stage (the copy pattern of examples/3d_scalar_burgers_equation.go:269-270)
    prob = results["f64"]["prob"]
    if chosen != "f64":
        prob.free()
        dt_kw = {k: (d, kw) for k, d, kw in forms}[chosen]
        prob = BurgersProblem(args.order, args.n, args.slabs, dt_kw[0], "modes", stream=stream.cuda_stream,
                              **dt_kw[1])
    r = prob.runner
    state = ("uhi", "ulo", "resu") if chosen.startswith("mixed") else ("u", "resu")
    hdt = torch.float64 if chosen in ("f64", "f64c") else torch.float32
    hosts = {nm: torch.empty(dofs, dtype=hdt, pin_memory=True).numpy() for nm in state}
    for nm, h in hosts.items():
        r.CopyFromDevice(nm, h)
        r.Bindings[nm].host = h
    kc = r.KernelConfigs["rhsStage"]
    params = [r.Param(p.name).Copy() if p.name in state else r.Param(p.name) for p in kc.params]
    r.ConfigureKernel("stageE2E", *params)
    r.BuildKernel(prob.op_id(), "stageE2E")
    r.ExecuteKernel("stageE2E", RK4A[0], RK4B[0], prob.dt)
    barrier(world)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    for s in range(args.e2e_steps):
        r.ExecuteKernel("stageE2E", RK4A[s % 5], RK4B[s % 5], prob.dt)
    torch.cuda.synchronize()
    e2e_s = max_over_ranks((time.perf_counter() - t0) / args.e2e_steps, world)
    e2e_bytes = sum(h.nbytes for h in hosts.values())
    prob.free()

    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline(args.order, 0)
    if rank == 0:
        bpd = ch["b_alg"]
        achieved = bpd * dofs / (ch["ms"] * 1e-3) / 1e9
        traffic = None
        try:
            with open(os.path.join(HERE, "profiles", "traffic.json")) as f:
                tj = json.load(f)
            key = f"rhs_stage_N{args.order}_{chosen}"
            if key in tj:
                traffic = tj[key]["dram_bytes_per_dof"] * dofs
        except Exception:
            pass
        Np = (args.order + 1) * (args.order + 2) * (args.order + 3) // 6
        f64 = results["f64"]
        plain_ach = f64["b_alg"] * dofs / (f64["ms"] * 1e-3) / 1e9
        out = {
            "metric": METRIC, "value": thr[chosen], "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": ch["ms"], "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": {"f64": "f64", "f64c": "f64", "f32": "f32", "mixed": "f32x2+f32",
                                                  "mixed_tc": "f32x2+f32 (bf16x3 products, f32 acc)"}[chosen],
            "data": "synthetic",
            "config": {"workload": f"3-D Burgers tet-DG, order {args.order} (Np={Np}), periodic {args.n}^3x6 Kuhn "
                                   f"mesh (K={dofs // Np}), {args.slabs} x-slab partitions, u0 = 0.5 + 8 seeded "
                                   f"Fourier modes; one step = one LSERK4 stage", "chosen": chosen,
                       "t_final_stages": args.warmup + args.steps,
                       "l2": "inputs larger than L2 (every stage streams GBs of state, metrics and face data)",
                       "parallelism": f"replicas x{world}" if world > 1 else "1 GPU"},
            "forms": {k: {"value": thr[k], "ms_per_step": results[k]["ms"], "l2_err_vs_fp64": errs[k],
                          "b_alg_per_dof": results[k]["b_alg"],
                          "hbm_frac": results[k]["b_alg"] * dofs / (results[k]["ms"] * 1e-3) / 1e9 / hbm}
                      for k in thr},
            "chosen_vs_plain_fp64": {"speedup": thr[chosen] / thr["f64"], "l2_err": errs[chosen]},
            # the same FP64 arithmetic on the compact layout: what the layout buys and what precision adds
            "chosen_vs_compact_fp64": {"speedup": thr[chosen] / thr["f64c"], "compact_fp64_vs_plain_fp64":
                                       thr["f64c"] / thr["f64"]} if "f64c" in thr else None,
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": hbm, "unit": "GB/s",
                         "frac": achieved / hbm, "traffic": traffic, "peak_kind": peak_kind,
                         "b_alg_per_dof": bpd, "kernel": ch["kernel"]},
            "plain_fp64_roofline": {"bound": "hbm", "achieved": plain_ach, "peak": hbm, "unit": "GB/s",
                                    "frac": plain_ach / hbm, "b_alg_per_dof": f64["b_alg"],
                                    "kernel": f64["kernel"]},
            "microbench": micro,
            "cpu_baseline": cpu,
            "e2e": {"value": world * dofs / e2e_s, "unit": UNIT, "h2d_bytes_per_step": e2e_bytes,
                    "d2h_bytes_per_step": e2e_bytes,
                    "path": f"Runner.ExecuteKernel (C ABI) with Copy() of {', '.join(state)}"},
            "clocks": ch["clocks"],
            "gpu_launches": args.steps,
        }
        print(json.dumps(out), flush=True)


if __name__ == "__main__":
    main()
