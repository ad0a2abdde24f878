#!/usr/bin/env python
"""Benchmark of the network-to-conductance hot path on B200.

Workload (one "step"): the single large CNT network of 25,000 CNTs in a 6 um
cube (~2.5 M points), seeded; the full hot path of one observation window:
contact grid -> tunnelling contacts -> Hoshen-Kopelman clusters -> percolation
-> unit-resistor DEA -> backbone -> real-resistor DEA along x -> effective
resistance.  The real-resistor solves stop at 1e-8 relative residual (FP64
check of |b - A x| / |b| reported); the unit-resistor solve that classifies
the backbone stops at 1e-12 in both arms, because at 1e-8 the backbone depends
on the CG iterate rather than on the network (see `TOL_UNIT`).
Metric: networks solved per second.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
  python bench.py --hybrid [--steps K] [--warmup W]   # hybrid CNT/GNP contact + cluster stages

`ours`: `value` times the device path with the network already resident in
HBM; `e2e` times the same step through the C ABI from pinned host buffers
(upload of the window-trimmed network + solve + read-back of R), with two
contexts in a pipeline (step k + 1's upload overlaps step k's device work;
`e2e.sequential_value` is the same without the overlap).  The
`reference` arm runs the upstream program (oracle/_ref/ref_dump, built from
the upstream sources) on the same network files, written by numpy alone
(cicy_geom_b200.netgen: the reference process never loads libcicy_b200.so),
with one process per host core.  Multi-GPU runs are independent replicas (one
network per rank).
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

# Unit-resistor pass tolerance, the same in both arms.  Upstream solves it to the one input
# tolerance, and its backbone threshold (1e-9 of the largest element current,
# Backbone_Network.cpp:227) then classifies elements on an unconverged iterate: on this
# network upstream's own backbone has 53,904 element points at 1e-8, 39,778 at 1e-10 and
# 39,767 at 1e-12.  At 1e-12 the dead-branch currents stay below 0.013 of the threshold and
# the live ones above 380 times it, so any solver's iterate gives the same backbone.
SIDE, N_CNTS, TOL, TOL_UNIT = 6.0, 25000, 1e-8, 1e-12
METRIC = "networks solved/s at 1e-8 residual (25k-CNT 6um network, full hot path)"
DATA = "synthetic (seeded CNT polylines of the workload's length, radius and step statistics; one independent network per GPU)"
REF_BIN = os.path.join(ROOT, "oracle", "_ref", "ref_dump")
PRECONDS = {"jacobi": 0, "learned": 1, "chain": 2, "mg": 3}
MG_DRAM_BYTES_PER_ROW = 594.0  # ncu: k_mg_pcg_sm DRAM read + write per launch / free rows (8k-CNT network: 545 and 642 B)
KERNELS = {0: "k_pcg (grid-wide persistent PCG)", 1: "PCG resident in registers or one cluster (k_pcg_cta, k_pcg_cluster)",
           2: "k_mg_pcg (chain-aggregation multigrid PCG)"}


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--precision", default="fp64", choices=["fp64", "mixed"])
    ap.add_argument("--precond", default="mg", choices=["jacobi", "chain", "learned", "mg"])
    ap.add_argument("--unsmoothed", action="store_true", help="multigrid without the smoothed level-1 prolongator")
    ap.add_argument("--no-comparison", action="store_true", help="skip the per-preconditioner comparison and the SpMV measurement")
    ap.add_argument("--mc", type=int, default=256, help="Monte-Carlo realisations for the batched-solve measurement (0: skip)")
    # a smaller network of the same generator, for profiler captures (the bench line names the size it ran)
    ap.add_argument("--side", type=float, default=SIDE)
    ap.add_argument("--cnts", type=int, default=N_CNTS)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--hybrid", action="store_true",
                    help="time the hybrid CNT/GNP contact and cluster stages instead (4 um, 8,000 CNTs, 1,500 GNPs)")
    return ap.parse_args()


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


def workload_config(rank: int, side: float = SIDE, cnts: int = N_CNTS):
    from cicy_geom_b200.network import NetworkConfig
    from cicy_geom_b200.replicas import seed

    return NetworkConfig(side=side, n_cnts=cnts, seed=seed(rank), tolerance=TOL, tolerance_unit=TOL_UNIT)


def workload(rank: int, side: float = SIDE, cnts: int = N_CNTS):
    from cicy_geom_b200.network import generate_cnt_network

    cfg = workload_config(rank, side, cnts)
    raw = generate_cnt_network(cfg)
    return cfg, raw, raw.extract_window(cfg)


def config_dict(side: float = SIDE, cnts: int = N_CNTS) -> dict:
    """The workload as both arms name it (identical dicts)."""
    return {"workload": f"single CNT network: {cnts:,} CNTs, {side:g} um cube, seeded polylines (seed 2,000,000 + rank); "
                        f"unit-resistor pass to {TOL_UNIT:g}, real-resistor pass to {TOL:g} relative residual",
            "l2": "GPU arm: 256 MB buffer written between steps (L2 flush); CPU arm: one process per network",
            "parallelism": "independent networks (GPU arm: one per GPU; CPU arm: one per host process)"}


class ClockSampler:
    """SM clocks and throttle reasons sampled during the timed region.

    NVML is read every 100 ms by a separate process (read-only queries; the
    same counters nvidia-smi prints; faster polling was seen to slow the
    timed steps' host synchronisations on some boxes); without NVML,
    nvidia-smi at its 100 ms floor.  Rows: sm MHz, max sm MHz, power W, hw_slowdown,
    hw_thermal_slowdown, sw_thermal_slowdown, sw_power_cap (bools).
    """

    NAMES = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]

    def __init__(self, index: int):
        self.index = index
        self.rows = []
        self.proc = None
        self.stop = threading.Event()
        self.source = None

    # NVML polled from a separate process, so its driver calls never queue behind or in front of
    # this process's launches and synchronisations
    NVML_LOOP = (
        "import sys, time\n"
        "import pynvml as N\n"
        "N.nvmlInit()\n"
        "h = N.nvmlDeviceGetHandleByIndex(int(sys.argv[1]))\n"
        "bits = [N.nvmlClocksEventReasonHwSlowdown, N.nvmlClocksEventReasonHwThermalSlowdown,\n"
        "        N.nvmlClocksEventReasonSwThermalSlowdown, N.nvmlClocksEventReasonSwPowerCap]\n"
        "mx = N.nvmlDeviceGetMaxClockInfo(h, N.NVML_CLOCK_SM)\n"
        "while True:\n"
        "    r = N.nvmlDeviceGetCurrentClocksEventReasons(h)\n"
        "    v = [N.nvmlDeviceGetClockInfo(h, N.NVML_CLOCK_SM), mx, N.nvmlDeviceGetPowerUsage(h) / 1000.0]\n"
        "    print(', '.join([str(x) for x in v] + ['Active' if r & b else 'Not Active' for b in bits]), flush=True)\n"
        "    time.sleep(0.1)\n")

    def __enter__(self):
        try:
            import pynvml  # noqa: F401

            self.proc = subprocess.Popen([sys.executable, "-c", self.NVML_LOOP, str(self.index)], stdout=subprocess.PIPE,
                                         stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
            t0 = time.time()
            while not self.rows and time.time() - t0 < 30.0 and self.proc.poll() is None:
                time.sleep(0.02)
            if self.rows:
                self.rows.clear()
                self.source = "nvml 100 ms (separate process)"
                return self
            self.proc.terminate()
            self.proc = None
        except Exception:
            self.proc = None
        q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={q}", "--format=csv,noheader,nounits",
                                          "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
            # nvidia-smi's start-up takes the driver for a while: let it finish before the timed region
            t0 = time.time()
            while not self.rows and time.time() - t0 < 5.0 and self.proc.poll() is None:
                time.sleep(0.05)
            self.rows.clear()
            self.source = "nvidia-smi 100 ms"
        except FileNotFoundError:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) != 7:
                continue
            try:
                self.rows.append([float(parts[0]), float(parts[1]), float(parts[2])] +
                                 [p.lower().startswith("active") for p in parts[3:]])
            except ValueError:
                pass

    def __exit__(self, *a):
        self.stop.set()
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()
        elif self.source:
            self.t.join(timeout=1.0)

    def summary(self):
        rows = list(self.rows)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        reasons = sorted({self.NAMES[i] for r in rows for i in range(4) if r[3 + i]})
        return {"sm_mhz": statistics.median(r[0] for r in rows), "sm_max_mhz": max(r[1] for r in rows), "reasons": reasons,
                "samples": len(rows), "power_w_median": statistics.median(r[2] for r in rows), "source": self.source}


def pinned_network(net):
    """Copy the window network's arrays into pinned host memory; return (keep-alive, cicy_network)."""
    import ctypes as C

    import torch

    from cicy_geom_b200 import _abi

    a = net.arrays()
    keep = {}

    def pin(name, dt, ct):
        arr = np.ascontiguousarray(a[name], dtype=dt)
        t = torch.empty(arr.shape, dtype={np.float64: torch.float64, np.int32: torch.int32, np.int64: torch.int64}[dt],
                        pin_memory=True)
        t.numpy()[...] = arr
        keep[name] = t
        return C.cast(t.data_ptr(), C.POINTER(ct)), arr.nbytes

    v = _abi.Network()
    nbytes = 0
    v.n_points = len(a["x"])
    for f, dt, ct in [("x", np.float64, C.c_double), ("y", np.float64, C.c_double), ("z", np.float64, C.c_double),
                      ("flag", np.int32, C.c_int32), ("structure_ptr", np.int64, C.c_int64), ("structure_idx", np.int64, C.c_int64),
                      ("radii", np.float64, C.c_double), ("cnts_inside", np.int32, C.c_int32),
                      ("boundary_cnt_ptr", np.int64, C.c_int64), ("boundary_cnt_idx", np.int32, C.c_int32),
                      ("boundary_pts_ptr", np.int64, C.c_int64), ("boundary_pts_idx", np.int64, C.c_int64)]:
        p, b = pin(f, dt, ct)
        setattr(v, f, p)
        nbytes += b
    v.n_cnts = len(a["radii"])
    v.n_inside = len(a["cnts_inside"])
    v.window = _abi.Cuboid(*[float(t) for t in a["window"]])
    return keep, v, nbytes


def cpu_baseline_reference(cfg, raw):
    """Upstream program on this network, one thread, hot path only (bounded sample: one network)."""
    from cicy_geom_b200.network import write_read_network_files

    if not os.path.exists(REF_BIN):
        return None
    with tempfile.TemporaryDirectory(prefix="cicy_bench_") as d:
        write_read_network_files(d, raw, cfg)
        r = subprocess.run([REF_BIN, "time", d, repr(TOL_UNIT)], capture_output=True, text=True, timeout=900)
        if r.returncode != 0:
            return None
        t = json.loads(r.stdout.strip().splitlines()[-1])
    return {"value": 1.0 / t["hot_s"], "unit": "networks/s", "cores": 1, "kind": "reference",
            "sample": f"one full network (grid {t['grid_s']:.2f}s, HK {t['hk_s']:.2f}s, unit DEA {t['unit_dea_s']:.2f}s, "
                      f"real DEA {t['real_dea_s']:.2f}s), upstream code, 1 thread", "hot_s": t["hot_s"], "R": t["R"]}


def _run_ref_processes(d, shares, timeout=1800):
    """One upstream process per entry of `shares` (its number of hot-path runs), all at
    once; returns the per-run JSON records."""
    procs = [subprocess.Popen([REF_BIN, "time", d, repr(TOL_UNIT), str(k)], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL,
                              text=True) for k in shares if k > 0]
    recs = []
    t0 = time.time()
    for p in procs:
        out, _ = p.communicate(timeout=max(1.0, timeout - (time.time() - t0)))
        if p.returncode != 0:
            raise RuntimeError(f"ref_dump exited with {p.returncode}")
        recs += [json.loads(x) for x in out.strip().splitlines() if x.startswith("{")]
    return recs


def run_reference(args):
    """The upstream program on this arm's network, timed on the host cores.

    The network files are written by numpy alone (cicy_geom_b200.netgen), so this
    process never loads libcicy_b200.so.  Warm-up: `warmup` runs as concurrent
    processes.  Timed: `steps` runs spread over P = min(cores, steps) concurrent
    processes, each repeating the hot path (contact grid, clusters, electrical
    analysis) on fresh objects; value = steps / (last hot-path end - first
    hot-path start) on the system-wide monotonic clock."""
    from cicy_geom_b200 import netgen

    rank, world, _ = dist_env()
    if rank != 0:
        return 0
    if not os.path.exists(REF_BIN):
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/ref_dump was not built (run __graft_entry__.build())"}))
        return 0
    cfg = workload_config(0, args.side, args.cnts)
    cores = os.cpu_count() or 1
    with tempfile.TemporaryDirectory(prefix="cicy_ref_") as d:
        netgen.write_network_files(d, cfg)
        for i in range(0, args.warmup, cores):
            _run_ref_processes(d, [1] * min(cores, args.warmup - i))
        p = max(1, min(cores, args.steps))
        shares = [args.steps // p + (1 if k < args.steps % p else 0) for k in range(p)]
        recs = _run_ref_processes(d, shares)
    window = max(r["t_end"] for r in recs) - min(r["t_start"] for r in recs)
    hot = [r["hot_s"] for r in recs]
    value = len(recs) / window
    R = recs[0]["R"]
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "networks/s", "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": window / len(recs) * 1e3, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": DATA, "config": config_dict(args.side, args.cnts),
            "cpu_baseline": {"value": value, "unit": "networks/s", "cores": p, "kind": "reference",
                             "sample": f"{len(recs)} hot-path runs (contact grid + clusters + electrical analysis) of the upstream "
                                       f"program on this network, {p} concurrent single-threaded processes "
                                       f"({', '.join(str(k) for k in shares)} runs each), {window:.1f} s from the first hot-path "
                                       f"start to the last end; median run {statistics.median(hot):.2f} s"},
            "e2e": {"value": value, "unit": "networks/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "R_x": R[0], "gpu_launches": 0}
    print(json.dumps(line))
    return 0


def cg_bytes(nodes, reserved, nnz_lower, iters, s_val=8, s_v=8):
    """Algorithmic bytes of one CG launch: iterations x (SpMV + vector traffic)."""
    n = nodes - reserved
    nnz_full = n + 2 * nnz_lower
    b_spmv = nnz_full * (s_val + 4) + 4 * (n + 1) + s_v * n + s_v * n
    return iters * (b_spmv + 12 * s_v * n)


def direct_voltage_error(S, x):
    """max |x - x_d| / max |x_d| over the rows connected to a prescribed node, x_d
    the FP64 sparse direct solve (SuperLU) of the same system; rows of floating
    islands (singular, no prescribed node) are left out."""
    import scipy.sparse as sp
    from scipy.sparse.csgraph import connected_components
    from scipy.sparse.linalg import spsolve

    from cicy_geom_b200.learned import full_csr

    A = full_csr(S).tocsr()
    n = A.shape[0]
    C = A.tocoo()
    off = C.row != C.col
    nc, comp = connected_components(sp.coo_matrix((np.ones(off.sum()), (C.row[off], C.col[off])), shape=(n, n)), directed=False)
    rs = np.asarray(A.sum(axis=1)).ravel()
    g = np.zeros(nc, bool)
    g[comp[rs > 1e-9 * A.diagonal()]] = True
    idx = np.nonzero(g[comp])[0]
    xd = spsolve(A[idx][:, idx].tocsc(), np.asarray(S["b"])[idx])
    return float(np.max(np.abs(x[idx] - xd)) / np.max(np.abs(xd)))


def solver_comparison(cfg, net, device, steps=3, warmup=2):
    """The same network step with each preconditioner and precision (device-resident,
    CUDA events): upstream Jacobi-PCG ("plain CG"), chain block-Jacobi, learned,
    multigrid in FP64, and Jacobi, chain and learned in mixed precision; per run
    the real-pass voltages' error against an FP64 direct solve of the same system."""
    import ctypes as C

    import torch

    from cicy_geom_b200._abi import Result, check, lib
    from cicy_geom_b200.device import Context

    out = {}
    runs = [("jacobi", "jacobi", 0), ("chain", "chain", 0), ("learned", "learned", 0), ("mg", "mg", 0),
            ("mg_unsmoothed", "mg", 0), ("jacobi_mixed", "jacobi", 1), ("chain_mixed", "chain", 1), ("learned_mixed", "learned", 1)]
    for name, pk, prec in runs:
        ctx = Context(device)
        # bounded: a stalled run stops early
        ctx.set_solver(precision=prec, preconditioner=PRECONDS[pk], max_iter_factor=20, smoothed=name != "mg_unsmoothed")
        ctx.upload(net)
        params = cfg.params()
        res = Result()
        stream = torch.cuda.ExternalStream(ctx.stream(), device=device)
        for _ in range(warmup):
            check(lib().cicy_network_to_conductance(ctx.handle, C.byref(params), C.byref(res)), "warm-up", ctx.handle)
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(steps):
            check(lib().cicy_network_to_conductance(ctx.handle, C.byref(params), C.byref(res)), name, ctx.handle)
        e1.record(stream)
        torch.cuda.synchronize()
        t = e0.elapsed_time(e1) * 1e-3 / steps
        sv = res.solves[: res.n_solves]
        real = [i for i in range(res.n_solves) if sv[i].pass_ >= 0]
        verr = None
        if real:
            S = ctx.system(real[0])
            verr = direct_voltage_error(S, np.asarray(S["voltages"])[S["reserved"]:])
        out[name] = {"precision": "mixed" if prec else "fp64", "networks_per_s": 1.0 / t, "ms_per_step": t * 1e3,
                     "cg_iterations": [int(x.iterations) for x in sv], "cg_ms": [round(x.seconds * 1e3, 3) for x in sv],
                     "fallback": [int(x.fallback) for x in sv], "max_rel_residual": max(x.rel_residual for x in sv),
                     "R_x": res.resistances[0], "real_pass_voltage_error_vs_fp64_direct": verr}
        ctx.close()
    for name, _, _ in runs:
        out[name]["R_x_rel_diff_vs_mg_fp64"] = abs(out[name]["R_x"] - out["mg"]["R_x"]) / abs(out["mg"]["R_x"])
    out["speedup_vs_jacobi"] = {k: out[k]["networks_per_s"] / out["jacobi"]["networks_per_s"] for k, _, _ in runs if k != "jacobi"}
    return out


def contact_search_roofline(ctx, net, res, stage_acc, steps, hbm):
    """Contact grid + tunnelling contacts + HK labels of the timed steps (device
    events of the two stages, cicy_result.stage_seconds) against the algorithmic
    bytes B_contact = N_p (24 xyz + 4 CNT id) + N_s (4 write + 4 read) + 4 (R + 1)
    + 16 N_k and B_label = 8 N_k + 8 N_c per network."""
    import ctypes as C

    from cicy_geom_b200._abi import lib

    nr, ns = C.c_int64(), C.c_int64()
    lib().cicy_get_sectioned_domain(ctx.handle, C.byref(nr), C.byref(ns), None, None)
    a = net.arrays()
    n_p, n_c = len(a["x"]), len(a["radii"])
    n_k = int(res.n_point_contacts)
    b = n_p * 28 + ns.value * 8 + 4 * (nr.value + 1) + 16 * n_k + 8 * n_k + 8 * n_c
    t = (stage_acc[0] + stage_acc[1]) / steps
    return {"stages": "cicy_contact_grid + cicy_clusters", "seconds_per_network": t, "points_per_s": n_p / t,
            "bound": "hbm", "algorithmic_bytes": b, "achieved": b / t / 1e9, "peak": hbm, "unit": "GB/s", "frac": b / t / 1e9 / hbm,
            "points": n_p, "slots": ns.value, "regions": nr.value, "point_contacts": n_k,
            "note": "stage time includes the host reads of the sizes (scan totals) between kernels; the largest kernel is "
                    "k_pairs (one thread per region slot)"}


def network_construction(cfg, device, args, R_step, reps=5):
    """The step's window network built on the device (cicy_ctx_generate_cnt_network +
    cicy_ctx_extract_window: generator and Shells + Cutoff_Wins trim in one context)
    against the host route the timed step's inputs take (host generator, host trim,
    upload from host memory).  Both routes' calls return with their device work
    complete, so host wall clock times them (best of `reps`).  The device-built
    network then runs the hot path with the step's solver settings; its R_x is
    compared with the step's."""
    import time as _t

    from cicy_geom_b200.device import Context
    from cicy_geom_b200.network import generate_cnt_network

    with Context(device) as ctx:
        ctx.set_solver(precision=1 if args.precision == "mixed" else 0, preconditioner=PRECONDS[args.precond], smoothed=not args.unsmoothed)
        ctx.generate_network(cfg)  # warm-up: buffers grow to this network's size
        dev = []
        for _ in range(reps):
            t0 = _t.perf_counter()
            ctx.generate_network(cfg)
            dev.append(_t.perf_counter() - t0)
        host = []
        for _ in range(2):
            t0 = _t.perf_counter()
            net = generate_cnt_network(cfg).extract_window(cfg)
            ctx.upload(net)
            host.append(_t.perf_counter() - t0)
        ctx.generate_network(cfg)
        r = ctx.network_to_conductance(cfg.params())
    R = float(r.resistances[0])
    return {"device_seconds": min(dev), "host_seconds": min(host), "speedup": min(host) / min(dev),
            "R_x_device_built": R, "R_x_rel_diff_vs_step": abs(R - R_step) / abs(R_step) if R_step else None,
            "note": "device: generator + window trim on the device; host: generator, Shells + Cutoff_Wins on the host, upload "
                    "(the route of the timed step's inputs); wall clock around synchronous calls, best of the repeats"}


def spmv_roofline(ctx, device, hbm, target_bytes=320e6, reps=20):
    """cicy_spmv_csr on copies of the unit-pass system laid out block-diagonally
    until the matrix is larger than L2 (126 MB); algorithmic bytes
    12 nnz + 4 (n+1) + 16 n per call over the CUDA-event time."""
    import ctypes as C

    import scipy.sparse as sp
    import torch

    from cicy_geom_b200._abi import lib
    from cicy_geom_b200.learned import full_csr

    A1 = full_csr(ctx.system(0))
    one = 12 * A1.nnz + 4 * A1.shape[0] + 16 * A1.shape[0]
    copies = max(1, int(np.ceil(target_bytes / one)))
    A = sp.block_diag([A1] * copies, format="csr")
    n, nnz = A.shape[0], A.nnz
    dev = torch.device(f"cuda:{device}")
    rp = torch.tensor(A.indptr.astype(np.int32), device=dev)
    ci = torch.tensor(A.indices.astype(np.int32), device=dev)
    va = torch.tensor(A.data, device=dev)
    x = torch.randn(n, dtype=torch.float64, device=dev)
    y = torch.empty(n, dtype=torch.float64, device=dev)
    st = torch.cuda.current_stream(dev)
    args = [C.c_void_p(t.data_ptr()) for t in (rp, ci, va, x, y)]
    for _ in range(3):
        lib().cicy_spmv_csr(n, *args, C.c_void_p(st.cuda_stream))
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(st)
    for _ in range(reps):
        lib().cicy_spmv_csr(n, *args, C.c_void_p(st.cuda_stream))
    e1.record(st)
    torch.cuda.synchronize()
    t = e0.elapsed_time(e1) * 1e-3 / reps
    bytes_ = 12 * nnz + 4 * (n + 1) + 16 * n
    return {"kernel": "k_spmv_csr (cicy_spmv_csr, FP64 CSR)", "bound": "hbm", "rows": n, "nnz": nnz,
            "workload": f"{copies} block-diagonal copies of the 25k-CNT unit-pass system (> L2)",
            "achieved": bytes_ / t / 1e9, "peak": hbm, "unit": "GB/s", "frac": bytes_ / t / 1e9 / hbm, "us_per_call": t * 1e6,
            "traffic": None}


MC_REF_SAMPLE = range(8, 16)  # realisations timed with the upstream program (~45 s of single-core work)


def mc_reference_sample(cfgs, device_seconds, cores=None, timeout=900):
    """Upstream program (oracle/_ref/ref_dump, hot path: grid + HK + electrical)
    on a fixed sample of the Monte-Carlo realisations, one process per host core,
    against this library's per-network device time of the same realisations."""
    from cicy_geom_b200.network import generate_cnt_network, write_read_network_files

    if not os.path.exists(REF_BIN):
        return None
    sample = [cfgs[k] for k in MC_REF_SAMPLE if k < len(cfgs)]
    cores = min(cores or os.cpu_count() or 1, len(sample))
    with tempfile.TemporaryDirectory(prefix="cicy_mc_") as base:
        dirs = []
        for c in sample:
            d = os.path.join(base, str(c.seed))
            os.makedirs(d)
            write_read_network_files(d, generate_cnt_network(c), c)
            dirs.append(d)
        hot, pending, running = {}, list(zip(sample, dirs)), []
        t0 = time.perf_counter()
        while pending or running:
            while pending and len(running) < cores:
                c, d = pending.pop(0)
                running.append((c, subprocess.Popen([REF_BIN, "time", d, repr(c.tolerance_unit)], stdout=subprocess.PIPE,
                                                    stderr=subprocess.DEVNULL, text=True)))
            time.sleep(0.05)
            for item in list(running):
                c, p = item
                if p.poll() is not None:
                    running.remove(item)
                    try:
                        hot[c.seed] = json.loads(p.stdout.read().strip().splitlines()[-1])["hot_s"]
                    except Exception:
                        hot[c.seed] = float("nan")
            if time.perf_counter() - t0 > timeout:
                for _, p in running:
                    p.kill()
                return None
        wall = time.perf_counter() - t0
    seeds = [c.seed for c in sample]
    ref_sum = sum(hot[s] for s in seeds)
    dev = [device_seconds.get(s) for s in seeds]
    ours = sum(dev) if all(v is not None for v in dev) else None
    return {"kind": "reference", "cores": cores, "realisations": seeds, "reference_hot_seconds": [hot[s] for s in seeds],
            "reference_networks_per_s_per_core": len(seeds) / ref_sum, "reference_networks_per_s": len(seeds) / wall,
            "reference_wall_seconds": wall, "ours_device_seconds": dev,
            "ours_networks_per_s": len(seeds) / ours if ours else None,
            "sample": f"realisations {MC_REF_SAMPLE.start}-{MC_REF_SAMPLE.stop - 1} of the sweep (seeds {seeds[0]}-{seeds[-1]}), "
                      f"whole hot path per network; upstream: one process per host core ({cores}); ours: the per-network device "
                      f"path, one network after another on one GPU (cicy_result.stage_seconds total)"}


def batched_monte_carlo(count, device, reps=3):
    """Monte-Carlo sweep: `count` seeded realisations (cube side U[2,5] um, CNT
    volume fraction U[0.5%,3%]), each run through the device path to its
    real-resistor system; then all systems solved at 1e-8 (|r| <= 1e-8
    min(|r0|, |b|), FP64-verified) by one graph-captured launch per solver:
    learned-preconditioned CG in mixed precision and in FP64 (one CTA per
    system, launch shape from the autotuner), plain Jacobi-CG the same way
    (the baseline), and the chain-aggregation multigrid (one cluster per
    system).  The multigrid is also compared with the sum of the per-network
    multigrid solve times of the same systems."""
    import time as _t

    from cicy_geom_b200 import batch as BT

    t0 = _t.time()
    cfgs = BT.monte_carlo_configs(count)
    systems, info = BT.realisation_systems(cfgs, device=device)
    prep = _t.time() - t0
    if not systems:
        return {"realisations": count, **info, "systems": 0}
    bs = BT.BatchSolver(systems, tol=TOL, device=device, learned=True)
    ns = len(systems)

    def measure(tune=False, runs=reps, solver=None):
        b = solver or bs
        shape = b.autotune() if tune else None
        t = min(b.solve() for _ in range(runs))
        it, rel, fl = b.results()
        return {"seconds": t, "systems_per_s": ns / t, "launch": shape, "iterations_total": int(it.sum()), "iterations_max": int(it.max()),
                "converged": int((fl == 1).sum()), "max_rel_residual": float(rel.max())}

    out = {}
    bs.set_solver("learned", 1)
    out["learned_mixed"] = measure(tune=True)
    bs.set_solver("learned", 0)
    out["learned_fp64"] = measure(tune=True)
    # the same preconditioner without training (every coupling weight 0.8, the initial
    # parameters) and without the learned term (chain blocks only)
    from cicy_geom_b200.learned import init_params

    bu = BT.BatchSolver(systems, tol=TOL, device=device, learned=init_params(0))
    bu.set_solver("learned", 0)
    out["untrained_constant_fp64"] = measure(tune=True, solver=bu)
    untrained_gnn_seconds = bu.gnn_seconds
    bu.close()
    # the network trained on 2,000 Laplacians of this generator (disjoint seeds)
    from cicy_geom_b200.learned import monte_carlo_params

    bmc = BT.BatchSolver(systems, tol=TOL, device=device, learned=monte_carlo_params())
    bmc.set_solver("learned", 0)
    out["learned_mc2000_fp64"] = measure(tune=True, solver=bmc)
    mc_gnn_seconds = bmc.gnn_seconds
    bmc.close()
    bs.set_solver("chain", 0)
    out["chain_fp64"] = measure(tune=True)
    # the plain GPU Jacobi-CG baseline, one CTA per system and with the largest systems on clusters:
    # the faster is the baseline
    bs.set_solver("jacobi", 0)
    bs.set_shape(1024, 2)
    jac = {}
    for rows in (0, out["learned_mixed"]["launch"]["cluster_split_rows"] or 32768):
        bs.set_split(rows)
        jac[rows] = measure(runs=1)
        jac[rows]["cluster_split_rows"] = rows
    out["jacobi_fp64"] = min(jac.values(), key=lambda v: v["seconds"])
    out["jacobi_fp64_variants"] = list(jac.values())
    bs.set_split(0)
    setup = bs.enable_multigrid()
    bs.set_method(1)
    out["multigrid"] = measure()
    bs.close()
    jac = out["jacobi_fp64"]["seconds"]
    # preconditioner set-up outside the timed launch: the graph network's forward (learned)
    # and the hierarchies (multigrid); the chain factors are built inside the launch
    setup_outside = {"learned_mixed": bs.gnn_seconds, "learned_fp64": bs.gnn_seconds, "multigrid": setup,
                     "untrained_constant_fp64": untrained_gnn_seconds, "chain_fp64": 0.0, "learned_mc2000_fp64": mc_gnn_seconds}
    for k in ("learned_mixed", "learned_fp64", "multigrid", "untrained_constant_fp64", "chain_fp64", "learned_mc2000_fp64"):
        out[k]["speedup_vs_jacobi"] = jac / out[k]["seconds"]
        t = out[k]["seconds"] + setup_outside[k]
        out[k]["setup_seconds_outside_launch"] = setup_outside[k]
        out[k]["systems_per_s_with_setup"] = ns / t
        out[k]["speedup_vs_jacobi_with_setup"] = jac / t
    def gain(arm, training):
        g = out["untrained_constant_fp64"]["seconds"] / out[arm]["seconds"]
        return {"iterations": out["untrained_constant_fp64"]["iterations_total"] / max(out[arm]["iterations_total"], 1),
                "iterations_max": out["untrained_constant_fp64"]["iterations_max"] / max(out[arm]["iterations_max"], 1),
                "seconds": g,
                "note": ("gains under 10 % over the untrained network (all coupling weights 0.8)" if g < 1.1 else
                         "gains 10 % or more over the untrained network"),
                "training": training}

    out["trained_gain_over_untrained"] = gain("learned_fp64", "the shipped parameters: 24 seeded networks of 2-3 um, one real "
                                                               "system each (python -m cicy_geom_b200.learned)")
    out["mc2000_gain_over_untrained"] = gain("learned_mc2000_fp64", "2,000 real-resistor Laplacians of this generator on seeds "
                                                                    "5,000,000 + k (python -m cicy_geom_b200.learned --monte-carlo 2000 "
                                                                    "--steps 4000), evaluated here on the 256 fresh seeds 3,000,000 + k")
    seq = sum(s["seconds_ref"] for s in systems)
    n = [s["A"].shape[0] for s in systems]
    dev = info.pop("device_seconds", {})
    ref = mc_reference_sample(cfgs, dev)
    return {"realisations": count, **info, "systems": ns, "unknowns_total": int(sum(n)), "unknowns_max": int(max(n)), **out,
            "per_network_pipeline": {"networks_per_s_device": len(dev) / sum(dev.values()) if dev else None,
                                     "realisations": len(dev), "device_seconds_total": sum(dev.values()) if dev else None},
            "cpu_baseline_sample": ref,
            "gnn_forward_seconds": bs.gnn_seconds, "multigrid_setup_seconds": setup,
            "multigrid_sequential_solve_seconds": seq, "multigrid_speedup_vs_sequential": seq / out["multigrid"]["seconds"],
            "generation_and_assembly_seconds": prep,
            "construction": info.get("construction"),
            "generation_and_assembly_note": "per realisation, in one context: the network generated and window-trimmed on the "
                                            "device, contacts, clusters, both DEA passes, and the real-resistor systems copied "
                                            "to the host for the batched solves",
            "sample": "cube side U[2,5] um, CNT volume fraction U[0.5%,3%], seeds 3,000,000+k; solve stage only "
                      "(generation, contacts, clusters, assembly and the unit-resistor pass run per network before it); "
                      "learned/Jacobi: one CTA per system, the largest systems on 16-CTA clusters when the autotuner picks it, in one "
                      "graph launch; multigrid: one cluster of 16, 8 or 4 CTAs per system"}


def sharded_monte_carlo(count, device, rank, world):
    """Monte-Carlo sweep split over the ranks (replicas.shard: the realisations,
    largest first, dealt round-robin): each rank builds its realisations' systems
    on its GPU (device generator and window trim) and solves them in one
    multigrid batch launch.  The sweep's time is the slowest rank's; its
    throughput is all ranks' systems over that time.  Every rank takes the same
    reductions, also when its own shard fails, so no rank waits on another."""
    import time as _t

    from cicy_geom_b200 import batch as BT
    from cicy_geom_b200 import replicas

    t_prep = t_solve = 0.0
    ns, failed, err = 0, False, None
    try:
        all_cfgs = BT.monte_carlo_configs(count)
        cfgs = replicas.shard(all_cfgs, [c.n_cnts for c in all_cfgs], rank, world)
        t0 = _t.perf_counter()
        systems, _ = BT.realisation_systems(cfgs, device=device)
        t_prep = _t.perf_counter() - t0
        if systems:
            bs = BT.BatchSolver(systems, tol=TOL, device=device)
            try:
                setup = bs.enable_multigrid()
                bs.set_method(1)
                t_solve = setup + min(bs.solve() for _ in range(3))
                _, _, fl = bs.results()
                failed = bool((fl != 1).any())
            finally:
                bs.close()
        ns = len(systems)
    except Exception as e:  # noqa: BLE001
        failed, err = True, f"{type(e).__name__}: {e}"
    import torch

    dev = f"cuda:{device}" if torch.cuda.is_available() else None  # NCCL reduces device tensors, gloo host tensors
    t_solve_max, n_total, any_failed = replicas.sweep_totals(t_solve, ns, failed, world, device=dev)
    t_prep_max, _, _ = replicas.sweep_totals(t_prep, 0, False, world, device=dev)
    out = {"realisations": count, "ranks": world, "systems": int(n_total), "solver": "multigrid batch (one launch per rank)",
           "solve_seconds_incl_setup_max_over_ranks": t_solve_max, "systems_per_s": n_total / t_solve_max if t_solve_max else None,
           "preparation_seconds_max_over_ranks": t_prep_max, "failed_on_some_rank": any_failed,
           "shard": "realisations sorted by CNT count, dealt round-robin; no data-path collective"}
    if err:
        out["error_on_rank_0" if rank == 0 else "error"] = err
    return out


def run_ours(args):
    import ctypes as C

    import torch

    from cicy_geom_b200._abi import Result, check, lib
    from cicy_geom_b200.device import Context

    from cicy_geom_b200 import replicas

    rank, world, local = replicas.env()
    replicas.init(world, gpu=torch.cuda.is_available())
    torch.cuda.set_device(local)
    cfg, raw, net = workload(rank, args.side, args.cnts)
    params = cfg.params()
    ctx = Context(local)
    ctx.set_solver(precision=1 if args.precision == "mixed" else 0, preconditioner=PRECONDS[args.precond], smoothed=not args.unsmoothed)
    stream = torch.cuda.ExternalStream(ctx.stream(), device=local)
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device=f"cuda:{local}")  # 256 MB > L2
    ctx.upload(net)
    res = Result()
    L = lib()

    def step():
        check(L.cicy_network_to_conductance(ctx.handle, C.byref(params), C.byref(res)), "cicy_network_to_conductance", ctx.handle)

    for _ in range(args.warmup):
        step()
    # ---- device-resident timing ----
    def barrier():
        replicas.barrier(world)
        torch.cuda.synchronize()

    per_kernel = {}  # kernel kind -> [device seconds, launches, algorithmic bytes]
    stage_acc = [0.0] * 6  # grid, clusters, unit DEA, backbone, real DEA, total (device events per step)
    cg_time, iters, resid = 0.0, [], []
    launches0 = ctx.kernel_launches()
    with ClockSampler(local) as clk:
        barrier()
        ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ev0.record(stream)
        for _ in range(args.steps):
            with torch.cuda.stream(stream):
                flush.zero_()
            step()
            for j in range(6):
                stage_acc[j] += res.stage_seconds[j]
            for s in res.solves[: res.n_solves]:
                cg_time += s.seconds
                acc = per_kernel.setdefault(int(s.kernel), [0.0, 0, 0, 0])
                acc[0] += s.seconds
                acc[1] += 1
                acc[2] += cg_bytes(s.nodes, s.reserved, s.nnz_lower, s.iterations)
                acc[3] += s.nodes - s.reserved
                iters.append(int(s.iterations))
                resid.append(float(s.rel_residual))
        ev1.record(stream)
        barrier()
    launches = ctx.kernel_launches() - launches0
    t_dev = ev0.elapsed_time(ev1) * 1e-3
    R = list(res.resistances)
    # ---- end to end through the C ABI from pinned host buffers ----
    keep, hnet, h2d = pinned_network(net)
    out_host = torch.empty(3, dtype=torch.float64, pin_memory=True)
    barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        with torch.cuda.stream(stream):
            flush.zero_()
        check(L.cicy_upload_network(ctx.handle, C.byref(hnet)), "cicy_upload_network", ctx.handle)
        step()
        out_host.numpy()[:] = np.array(res.resistances)
    e1.record(stream)
    barrier()
    t_seq = e0.elapsed_time(e1) * 1e-3
    # ---- end to end, pipelined: two contexts, as a serving loop runs them ----
    # One host thread uploads step k + 1's network into one context (host checks, pinned H2D
    # copies on that context's stream) while this thread runs step k on the other context and
    # reads its resistances back.  All device work of the steps is issued by this thread, one
    # step after the other, so kernels of the two contexts never run at the same time; every
    # step's copies and read-back are inside the timed region.
    ctx2 = Context(local)
    ctx2.set_solver(precision=1 if args.precision == "mixed" else 0, preconditioner=PRECONDS[args.precond], smoothed=not args.unsmoothed)
    ctx2.upload(net)
    res2 = Result()
    check(L.cicy_network_to_conductance(ctx2.handle, C.byref(params), C.byref(res2)), "cicy_network_to_conductance", ctx2.handle)
    stream2 = torch.cuda.ExternalStream(ctx2.stream(), device=local)
    ctxs, streams, results = [ctx, ctx2], [stream, stream2], [res, res2]
    free = [threading.Semaphore(1), threading.Semaphore(1)]
    ready = [threading.Semaphore(0), threading.Semaphore(0)]
    up_err = []

    def uploader():
        try:
            for k in range(args.steps):
                i = k % 2
                free[i].acquire()
                check(L.cicy_upload_network(ctxs[i].handle, C.byref(hnet)), "cicy_upload_network", ctxs[i].handle)
                ready[i].release()
        except Exception as e:  # noqa: BLE001
            up_err.append(e)
            for r_ in ready:
                r_.release()

    barrier()
    e0.record(stream)
    th = threading.Thread(target=uploader)
    th.start()
    for k in range(args.steps):
        i = k % 2
        ready[i].acquire()
        if up_err:
            break
        with torch.cuda.stream(streams[i]):
            flush.zero_()
        check(L.cicy_network_to_conductance(ctxs[i].handle, C.byref(params), C.byref(results[i])), "cicy_network_to_conductance",
              ctxs[i].handle)
        out_host.numpy()[:] = np.array(results[i].resistances)
        free[i].release()
    th.join()
    if up_err:
        raise up_err[0]
    last = torch.cuda.Event()
    last.record(streams[(args.steps - 1) % 2])
    stream.wait_event(last)
    e1.record(stream)
    barrier()
    t_e2e = e0.elapsed_time(e1) * 1e-3
    ctx2.close()
    t_dev, t_e2e, t_seq = replicas.max_over_ranks([t_dev, t_e2e, t_seq], world, device=f"cuda:{local}")
    # N > 1: the Monte-Carlo sweep split over the ranks (every rank takes part in its reductions)
    mc_sharded = sharded_monte_carlo(args.mc, local, rank, world) if args.mc > 0 and world > 1 else None
    if rank == 0:
        peaks = {}
        pk_path = os.path.join(ROOT, "MEASURED_PEAKS.json")
        if os.path.exists(pk_path):
            peaks = json.load(open(pk_path))
        hbm = peaks.get("hbm_gbs", 6650.0)
        top = max(per_kernel, key=lambda k: per_kernel[k][0]) if per_kernel else 0
        k_sec, k_launch, k_bytes, k_rows = per_kernel.get(top, [0.0, 0, 0, 0])
        achieved = (k_bytes / k_launch) / (k_sec / k_launch) / 1e9 if k_launch and k_sec > 0 else 0.0
        # DRAM bytes per launch of the multigrid kernel: 215-233 B per free row in an ncu capture of
        # the 8k-CNT network's two passes (the system read once, L2-resident across iterations),
        # scaled by the rows of this workload's launches
        traffic = MG_DRAM_BYTES_PER_ROW * k_rows / k_launch if top == 2 and k_launch else None
        line = {
            "metric": METRIC,
            "value": world * args.steps / t_dev,
            "unit": "networks/s",
            "n_gpus": world,
            "steps": args.steps,
            "warmup": args.warmup,
            "ms_per_step": t_dev / args.steps * 1e3,
            "higher_is_better": True,
            "scaling": "weak",
            "vs_baseline": None,
            "dtype": "f64" if args.precision == "fp64" else "f32/f64 mixed",
            "data": DATA,
            "config": config_dict(args.side, args.cnts),
            "points_in_window": len(net.arrays()["x"]),
            "solver_settings": {"precision": args.precision, "preconditioner": args.precond, "tolerance_real": TOL,
                                "tolerance_unit": TOL_UNIT, "mg_level1_prolongator": "piecewise constant" if args.unsmoothed else "smoothed"},
            "roofline": {"kernel": KERNELS[top], "bound": "hbm", "achieved": achieved, "peak": hbm,
                         "unit": "GB/s", "frac": achieved / hbm, "traffic": traffic,
                         "traffic_note": "bytes per launch scaled by rows from an ncu capture of the same kernel on the "
                                         "8k-CNT network (DRAM read + write, 594 B per free row: the system, the hierarchy and "
                                         "the dense coarsest inverse read once into shared memory and L2); the algorithmic bytes "
                                         "per launch are several times larger because the system stays on chip across iterations",
                         "algorithmic_bytes_per_launch": k_bytes / k_launch if k_launch else None,
                         "launches_per_step": k_launch / args.steps, "share_of_step": k_sec / t_dev,
                         "note": "algorithmic bytes = iterations x (SpMV + 12 vector passes) of the solves this kernel ran; "
                                 "the systems live in shared memory / L2, so the kernel is latency-bound (one cluster or "
                                 "grid barrier per reduction); peak is the measured HBM copy bandwidth (of measured)"},
            "contact_search": contact_search_roofline(ctx, net, res, stage_acc, args.steps, hbm),
            "e2e": {"value": world * args.steps / t_e2e, "unit": "networks/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": 24,
                    "pipeline": "two contexts: step k + 1's upload (host checks, pinned H2D copies) overlaps step k's device work "
                                "and read-back; one thread issues all device work, so the contexts' kernels never overlap",
                    "sequential_value": world * args.steps / t_seq},
            "gpu_launches": int(launches),
            "clocks": clk.summary(),
            "solver": {"cg_iterations": iters[: len(iters) // max(args.steps, 1)], "max_rel_residual": max(resid) if resid else None,
                       "cg_seconds_per_step": cg_time / args.steps,
                       "kernels": {KERNELS[k]: {"seconds_per_step": v[0] / args.steps, "launches_per_step": v[1] / args.steps}
                                   for k, v in per_kernel.items()}},
            "R_x": R[0],
        }
        # the measured step above is the result; a failing extra section is recorded, not fatal
        def extra(key, fn):
            try:
                line[key] = fn()
            except Exception as e:  # noqa: BLE001
                line[key] = {"error": f"{type(e).__name__}: {e}"}
                print(f"bench: {key} failed: {e}", file=sys.stderr)

        if not args.no_comparison and world == 1:
            extra("solver_comparison", lambda: solver_comparison(cfg, net, local))
            extra("spmv", lambda: spmv_roofline(ctx, local, hbm))
        if world == 1:
            extra("network_construction", lambda: network_construction(cfg, local, args, R[0]))
        if args.mc > 0 and world == 1:
            extra("batched_monte_carlo", lambda: batched_monte_carlo(args.mc, local))
        if mc_sharded is not None:
            line["batched_monte_carlo_sharded"] = mc_sharded
        if not args.no_cpu_baseline and world == 1:
            cb = None
            try:
                cb = cpu_baseline_reference(cfg, raw)
            except Exception as e:  # noqa: BLE001
                print(f"bench: cpu_baseline failed: {e}", file=sys.stderr)
            if cb:
                line["cpu_baseline"] = {k: cb[k] for k in ("value", "unit", "cores", "kind", "sample")}
                line["R_x_reference"] = cb["R"][0]
                line["R_x_rel_diff"] = abs(R[0] - cb["R"][0]) / abs(cb["R"][0])
                line["R_x_note"] = (f"both arms: unit-resistor pass to {TOL_UNIT:g}, real-resistor pass to {TOL:g}; "
                                    "the reference runs upstream's Jacobi-PCG, this arm the multigrid PCG")
        print(json.dumps(line))
    replicas.finish(world)
    return 0


HYBRID_SIDE, HYBRID_CNTS, HYBRID_GNPS, HYBRID_SEED = 4.0, 8000, 1500, 4_200_001
GNP_DUMP = os.path.join(ROOT, "oracle", "_ref", "gnp_dump")


def run_hybrid(args):
    """Hybrid CNT/GNP sample (4 um cube, 8,000 CNTs, 1,500 GNPs of side U[0.5, 1]
    um and thickness 10 nm, seeded): one step is the whole GNP_CNT_mix path of
    window 0 on the device (cicy_geom_b200.hybrid): window extraction, contact
    grid, CNT / GNP / CNT-GNP contacts and labels, mixed percolation and the
    electrical stage (unit-resistor DEA, CNT+GNP backbone, real-resistor DEA
    along x, R_x).  Stages are timed on the host around the synchronous C-ABI
    calls (their host<->device copies included).  The upstream program
    (oracle/_ref/gnp_dump, flow mode) runs the same stages on one host core; its
    resistance is compared with this one."""
    from cicy_geom_b200.hybrid import hybrid_network_to_conductance
    from cicy_geom_b200.network import NetworkConfig, generate_cnt_network, generate_gnps, write_gnp_file, write_read_network_files
    from oracle.dumpio import read_dump

    side = HYBRID_SIDE
    # unit pass to 1e-12 on both sides (the backbone's 1e-9 current threshold), real pass to 1e-10
    cfg = NetworkConfig(side=side, n_cnts=HYBRID_CNTS, seed=HYBRID_SEED, resistances=(1, 0, 0), tolerance_unit=TOL_UNIT)
    ov_gnp = cfg.gs_min / np.sqrt(8.0)  # Input_Reader.cpp:1368
    d = tempfile.mkdtemp(prefix="cicy_hybrid_")
    write_read_network_files(d, generate_cnt_network(cfg), cfg)
    write_gnp_file(d, generate_gnps(HYBRID_GNPS, side, HYBRID_SEED + 1))
    from cicy_geom_b200.device import Context

    times, R = [], None
    precond = {"jacobi": 0, "learned": 1, "chain": 2, "mg": 3}[args.precond]
    with Context(0) as ctx:
        ctx.set_solver(1 if args.precision == "mixed" else 0, precond)
        for step in range(args.warmup + args.steps):
            tm = {}
            r, _, st = hybrid_network_to_conductance(d, cfg, ov_gnp, timings=tm, ctx=ctx)
            R = list(r.resistances)
            if step >= args.warmup:
                times.append(tm)
            sv = [(int(x.nodes), int(x.iterations)) for x in r.solves[: r.n_solves]]
    stage_ms = {k: 1e3 * statistics.median(t[k] for t in times) for k in times[0]}
    step_s = statistics.median(sum(t.values()) for t in times)
    line = {"metric": "hybrid CNT/GNP networks solved per second (4 um, 8,000 CNTs, 1,500 GNPs, whole path to R_x)", "value": 1.0 / step_s,
            "unit": "networks/s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * step_s,
            "higher_is_better": True, "dtype": "f64", "data": "synthetic (seeded CNT polylines and GNPs)",
            "config": {"workload": "hybrid 4um 8000 CNTs + 1500 GNPs, window 0 = the sample, R along x; unit-resistor pass to 1e-12, "
                                   "real-resistor pass to 1e-10 relative residual"},
            "solver_settings": {"precision": args.precision, "preconditioner": args.precond},
            "stage_ms": stage_ms, "R_x": R[0], "solves": sv, "percolated": int(st["mixed"]["n_percolated"]),
            "timing": "host wall clock around synchronous C-ABI calls, median over steps"}
    if os.path.exists(GNP_DUMP):
        r = subprocess.run([GNP_DUMP, d, os.path.join(d, "ref.bin"), repr(cfg.vdw), repr(cfg.tunnel), repr(cfg.gs_min),
                            repr(2 * cfg.radius + cfg.tunnel), repr(float(ov_gnp)), "-1", "flow", repr(cfg.step), "electrical_time",
                            repr(TOL_UNIT)],
                           capture_output=True, timeout=1800)
        if r.returncode == 0:
            z = read_dump(os.path.join(d, "ref.bin"))
            ref = [float(x) for x in z["flow_seconds"]]
            line["cpu_baseline"] = {"value": 1.0 / sum(ref), "unit": "networks/s", "cores": 1, "kind": "reference",
                                    "sample": "upstream's GNP_CNT_mix stages on the same files (window extraction, Generate_contact_grid, "
                                              "Determine_clusters_and_percolation, Perform_analysis_on_clusters along x), one thread",
                                    "stage_seconds": ref}
            line["R_x_reference"] = float(z["flow_resistances"][0])
            line["R_x_rel_diff"] = abs(R[0] - line["R_x_reference"]) / abs(line["R_x_reference"])
        else:
            line["cpu_baseline_error"] = r.stderr.decode(errors="replace")[-300:]
    print(json.dumps(line))
    return 0


def main():
    args = parse()
    if args.hybrid:
        return run_hybrid(args)
    if args.impl == "reference":
        return run_reference(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
