#!/usr/bin/env python
"""Full-step throughput of the B200 tree code (one JSON line on rank 0).

The line is the result with the main figures of each form; the whole record
(sweeps, learned form, ensembles, precision, block steps, with their parameters)
goes to stderr as one JSON line, and to --report FILE.

Workload (the large Plummer configuration): N = 2^24 equal-mass Plummer
sphere (seeded, the reference's plummer.h algorithm), float32, eps = 0.005,
NLEAF = 16, NCRIT = 64, levelSplit = 5, dt = 1/128, fixed-theta FP32 walk.
The headline uses theta = 0.6, the largest opening angle of the
configuration's sweep {0.3, 0.4, 0.5, 0.6}; every theta of the sweep is
measured too (throughput and median / p99 force error against the FP64
direct sum), and the metric's bar is median |da|/|a| <= 1e-3.  A step is the reference's full step (treecode.cu:137-168): box +
keys + sort + octree + multipoles + groups + walk + leapfrog move + energies,
replayed as captured CUDA graphs; inputs stay resident in HBM (the particle
state, 1.3 GB, is larger than the 126 MB L2, so no flush is needed).

  value   : N x n_gpus / (device time per step), Mparticles/s
  e2e     : the same through the C ABI from pinned host buffers: every step
            copies pos+vel host->device, runs the step, scatters the
            accelerations back to caller order and copies them device->host
  roofline: the walk kernel (FP32 FMA bound, no tensor cores): algorithmic
            flops = 20 per direct + 64 per quadrupole interaction
            (treecode.cu:149-158) / walk time from CUDA events recorded on the
            handle's stream inside the timed region; peak = this GPU's FP32
            FMA throughput measured by bonsai_fp32_peak
  hbm_roofline: the other stages (build, multipoles, groups, gathers,
            move) against HBM bandwidth: algorithmic bytes per particle and
            per cell / their event time, beside the reference's IOCOUNT
            build accounting (32 B per particle per level)
  cpu_baseline / --impl reference: the CPU restatement of the reference
            algorithm (oracle/, OpenMP over the host cores), on a bounded
            sample: full-N build, multipoles and groups, the walk of a sample
            of groups extrapolated to all groups.

Multi-GPU (torchrun): independent replicas, one per GPU (the single-system
step has no exchange step); max of the device times over ranks.  Beside it,
`batching_split`: the batching ensemble's systems partitioned over the ranks
by estimated work, each rank advancing only its own systems, no data-path
collective, per-system energies gathered to rank 0 at the end (strong
scaling of the fixed 512-system ensemble).
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

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

METRIC = "Mparticles/s per full step at N=2^24, median |δa|/|a|≤1e-3; learned-θ vs fixed-θ"
UNIT = "Mparticles/s"
# the walk's DRAM traffic (read + write) per launch from one ncu capture of the
# same workload at N = 2^22, theta 0.6 (profiles/walk_k_walk_plummer_4M.md);
# scaled by the particle count for other N (the walk's misses grow with N)
WALK_DRAM_BYTES_2P22 = 225.7e6 + 71.6e6


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--particles", type=int, default=1 << 24, dest="n")
    ap.add_argument("--theta", type=float, default=0.6)
    ap.add_argument("--relative-alpha", type=float, default=0.0,
                    help="run the headline steps in the relative opening mode with this alpha (0: fixed theta)")
    ap.add_argument("--sweep", default="0.3,0.4,0.5,0.6,0.7,0.8,0.9,1.0",
                    help="thetas of the sweep reported beside the headline")
    ap.add_argument("--learned-target", type=float, default=1e-3,
                    help="per-group error target of the learned opening angles (0: skip the learned form)")
    ap.add_argument("--precision-n", type=int, default=1 << 26,
                    help="particles of the precision form (composite galaxy; 0: skip)")
    ap.add_argument("--field-n", type=int, default=1 << 25,
                    help="particles of the learned form's clustered field (0: skip)")
    ap.add_argument("--autotune", type=int, default=1, help="report the autotuned headline configuration (0: skip)")
    ap.add_argument("--octree-n", type=int, default=20000000,
                    help="particles of the octree-build comparison with the reference's published build (0: skip)")
    ap.add_argument("--block-levels", type=int, default=3, help="levels of the block time step block (<0: skip)")
    ap.add_argument("--batch-systems", type=int, default=512,
                    help="systems of the batching form reported beside the headline (0: skip)")
    ap.add_argument("--batch-steps", type=int, default=32)
    ap.add_argument("--batch-autotune", type=int, default=1, help="autotune the ensemble's nLeaf/nCrit/layout (0: keep 16/64)")
    ap.add_argument("--batch-ds", type=int, default=1, help="also time the ensemble with double-single positions (0: skip)")
    ap.add_argument("--split-emulate", type=int, default=0,
                    help="on one GPU, run the split batching form's ranks one after another (a check of the split)")
    ap.add_argument("--eps", type=float, default=0.005)
    ap.add_argument("--nleaf", type=int, default=16)
    ap.add_argument("--ncrit", type=int, default=64)
    ap.add_argument("--level-split", type=int, default=5)
    ap.add_argument("--dt", type=float, default=1.0 / 128)
    ap.add_argument("--seed", type=int, default=19810614)
    ap.add_argument("--e2e-steps", type=int, default=20,
                    help="pipelined end-to-end steps (the first upload and the last download are not overlapped)")
    ap.add_argument("--error-samples", type=int, default=4096)
    ap.add_argument("--report", default="", help="also write the whole record (JSON) to this file")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--cpu-group-fraction", type=float, default=1.0 / 512)
    return ap.parse_args()


# Algorithmic HBM bytes of the non-walk stages (keys, the PH permutation counted
# once, state gather, tree, multipoles, groups, kick-drift-kick), per particle
# and per cell; the reference's own build accounting (IOCOUNT,
# treebuild/treebuild.cu:646-650) is 32 B per particle per level.
HBM_BYTES_PER_PARTICLE = {"keys": 28, "sort": 24, "gather_pos_vel": 64, "tree": 8, "multipoles": 16, "groups": 8,
                          "kdk": 80}
HBM_BYTES_PER_CELL = {"tree": 16, "multipoles": 72}
HBM_BYTES_PER_GROUP = 8
HBM_FALLBACK_GBS = 6650.0


def hbm_peak():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "MEASURED_PEAKS.json hbm_gbs (measured copy bandwidth)"
    except (OSError, KeyError, ValueError):
        return HBM_FALLBACK_GBS, "fallback 6.65 TB/s (earlier copy measurement on this pool)"


def hbm_roofline(n, info, stage_ms):
    """The non-walk stages of one step against HBM bandwidth."""
    per_step = (n * sum(HBM_BYTES_PER_PARTICLE.values()) + info["ncells"] * sum(HBM_BYTES_PER_CELL.values())
                + HBM_BYTES_PER_GROUP * info["ngroups"])
    peak, src = hbm_peak()
    achieved = per_step / (stage_ms * 1e-3) / 1e9
    ref_bytes = 32.0 * n * info["nlevels"]
    return {"bound": "hbm", "stages": "box+keys+sorts+tree+multipoles+groups+gathers+move+energies",
            "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak, "peak_source": src,
            "stage_ms": stage_ms, "algorithmic_bytes_per_step": per_step,
            "bytes_per_particle": HBM_BYTES_PER_PARTICLE, "bytes_per_cell": HBM_BYTES_PER_CELL,
            "cells": info["ncells"], "groups": info["ngroups"], "levels": info["nlevels"],
            "reference_build_bytes": ref_bytes, "reference_build_gbs": ref_bytes / (stage_ms * 1e-3) / 1e9,
            "reference_build_accounting": "IOCOUNT: 32 B per particle per level (treebuild/treebuild.cu:646-650)"}


def workload(a):
    alpha = getattr(a, "relative_alpha", 0.0)
    how = ("fixed-theta FP32" if not alpha else
           "relative opening test alpha=%g (safety angle 2.0, theta the first evaluation's fallback), FP32"
           % alpha)
    return ("plummer N=%d theta=%g eps=%g nleaf=%d ncrit=%d levelSplit=%d dt=1/%d seed=%d, %s"
            % (a.n, a.theta, a.eps, a.nleaf, a.ncrit, a.level_split, round(1 / a.dt), a.seed, how))


# ---------------------------------------------------------------------------
# distributed plumbing (replicas)
# ---------------------------------------------------------------------------
class Dist:
    def __init__(self, backend):
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.rank = int(os.environ.get("RANK", "0"))
        self.local = int(os.environ.get("LOCAL_RANK", "0"))
        self.pg = None
        self.backend = backend
        if self.world > 1:
            import datetime
            import torch.distributed as dist
            os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
            dist.init_process_group(backend, timeout=datetime.timedelta(seconds=600))
            self.pg = dist

    def barrier(self):
        if self.pg:
            if self.backend == "nccl":  # the rank's own GPU, not one NCCL infers
                self.pg.barrier(device_ids=[self.local])
            else:
                self.pg.barrier()

    def max(self, x: float) -> float:
        if not self.pg:
            return x
        import torch
        dev = "cuda" if self.pg.get_backend() == "nccl" else "cpu"
        t = torch.tensor([x], dtype=torch.float64, device=dev)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())

    def close(self):
        if self.pg:
            self.pg.destroy_process_group()


# ---------------------------------------------------------------------------
# clocks during the timed region
# ---------------------------------------------------------------------------
class ClockSampler:
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.rows = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "-i", str(self.index), "--query-gpu=" + self.Q,
                                          "--format=csv,noheader,nounits", "-lms", "200"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.th = threading.Thread(target=self._read, daemon=True)
            self.th.start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([c.strip() for c in line.split(",")])

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.th.join(timeout=2)
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in self.rows:
            try:
                sm.append(float(r[1]))
                mx = float(r[2])
                for k, nm in enumerate(names):
                    if r[5 + k].lower() == "active":
                        reasons.add(nm)
            except (ValueError, IndexError):
                continue
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


# ---------------------------------------------------------------------------
# CPU restatement of the reference (oracle/), bounded sample
# ---------------------------------------------------------------------------
def cpu_reference_step(O, pos, vel, a, rng, full=False):
    """One step of the reference algorithm on the host cores.  full: the walk
    covers every group (a measured step); otherwise it runs on a random
    sample of cpu_group_fraction of the groups and is extrapolated.  Returns
    (seconds per full step (measured, or estimated), description)."""
    t0 = time.perf_counter()
    S = O.OracleStep(pos, theta=a.theta, eps=a.eps, nleaf=a.nleaf, ncrit=a.ncrit, level_split=a.level_split)
    S.build()
    t1 = time.perf_counter()
    S.multipoles()
    t2 = time.perf_counter()
    S.groups()
    t3 = time.perf_counter()
    G = len(S.gbeg)
    if full:
        gs, sel = G, None
    else:
        gs = max(1, int(round(G * a.cpu_group_fraction)))
        sel = np.sort(rng.choice(G, gs, replace=False)).astype(np.int32)
    S.forces(gsel=sel)
    t4 = time.perf_counter()
    acc = np.zeros_like(pos)
    if full:
        acc[S.ph_perm] = S.acc
    p2, v2 = pos.copy(), vel.copy()
    O.move(p2, v2, acc, a.dt, True, a.eps)
    t5 = time.perf_counter()
    frac = 1.0 if full else S.gnp[sel].sum() / float(pos.shape[0])
    walk_full = (t4 - t3) / frac
    total = (t1 - t0) + (t2 - t1) + (t3 - t2) + walk_full + (t5 - t4)
    if full:
        desc = ("full-N box+keys+sort+tree %.2fs, multipoles %.2fs, groups %.2fs, walk of all %d groups %.2fs, "
                "move %.2fs (measured, nothing extrapolated)" % (t1 - t0, t2 - t1, t3 - t2, G, t4 - t3, t5 - t4))
    else:
        desc = ("full-N box+keys+sort+tree %.2fs, multipoles %.2fs, groups %.2fs; walk of %d/%d groups "
                "(%.3f%% of particles) %.2fs extrapolated to %.1fs; move %.2fs"
                % (t1 - t0, t2 - t1, t3 - t2, gs, G, 100 * frac, t4 - t3, walk_full, t5 - t4))
    return total, desc, S


def reference_gpu_make_groups(O, pos, a, reps=10):
    """The reference's own GPU group formation (code/makeGroups.cu: PH keys,
    Thrust sort_by_key, segment scans, groups), the one hot-path CUDA file that
    builds for sm_100a unmodified (oracle/build_ref.sh -> oracle/_ref/ref_groups),
    timed with CUDA events on the same input; its domain box comes from the
    oracle (buildTree.cu does not build for sm_100)."""
    import tempfile
    exe = os.path.join(ROOT, "oracle", "_ref", "ref_groups")
    if not os.path.exists(exe):
        return {"unavailable": "oracle/_ref/ref_groups not built (oracle/build_ref.sh needs the reference tree)"}
    try:
        import torch
        if not torch.cuda.is_available():
            return {"unavailable": "no GPU"}
    except ImportError:
        return {"unavailable": "no torch to probe for a GPU"}
    box, _ = O.bbox(pos)
    n = pos.shape[0]
    with tempfile.TemporaryDirectory() as dd:
        inp = os.path.join(dd, "in.f32")
        np.ascontiguousarray(pos, np.float32).tofile(inp)
        args = [exe, inp, str(n)] + ["%.9g" % float(b) for b in box] + [str(a.level_split), str(a.ncrit), str(reps)]
        r = subprocess.run(args, capture_output=True, text=True)
    lines = [l for l in r.stdout.splitlines() if l.startswith("REFGROUPS ")]
    if r.returncode != 0 or not lines:
        return {"unavailable": "ref_groups exited %d" % r.returncode}
    info = json.loads(lines[-1][len("REFGROUPS "):])
    # best of the calls: the reference allocates its temporaries inside every
    # call, and those host-side allocations vary from call to call
    return {"value": n / info["ms_min"] / 1e3, "unit": "Mparticles/s", "ms": info["ms_min"],
            "ms_median": info["ms_median"], "reps": info["reps"], "groups": info["groups"], "n": n,
            "what": "code/makeGroups.cu unmodified for sm_100a (PH keys, Thrust sort_by_key, segment scans, "
                    "groups; its own temporary allocations included), levelSplit %d, nCrit %d"
                    % (a.level_split, a.ncrit)}


def reference_gpu_walk(S, a, reps=3):
    """The reference's own multipoles and tree walk (code/computeMultipoles.cu,
    code/computeForces.cu: the "modified reference" with mechanical sm_100a
    shims, oracle/_ref/ref_walk), timed with CUDA events around
    Treecode<float>::computeMultipoles and ::computeForces on the tree of the
    CPU restatement's step S (the reference's comparison-partition octree and
    groups, which the reference's CDP build cannot produce on sm_100)."""
    import tempfile
    from oracle import ref_walk as RW
    if not RW.available():
        return {"unavailable": "oracle/_ref/ref_walk not built (oracle/build_ref.sh needs the reference tree)"}
    try:
        import torch
        if not torch.cuda.is_available():
            return {"unavailable": "no GPU"}
    except ImportError:
        return {"unavailable": "no torch to probe for a GPU"}
    T = S.tree
    tree = {"cell_data": T.cell_data(), "size": S.size4, "mono": S.mono4, "quad0": S.quad0, "quad1": S.quad1,
            "l1": (int(T.level_beg[1]), int(T.level_end[1])),
            "groups": np.stack([S.gbeg, S.gnp], 1).astype(np.int32), "ipos": S.ipos, "jpos": S.jpos}
    if int(np.max(S.gnp)) > 64:
        return {"unavailable": "groups larger than the reference walk's 64 particles"}
    eps2 = float(np.float32(np.float32(a.eps) * np.float32(a.eps)))
    with tempfile.TemporaryDirectory() as dd:
        inp = os.path.join(dd, "tree.in")
        RW.write_input(inp, tree, a.theta, eps2, a.ncrit)
        info = RW.time_walk(inp, reps)
    if "unavailable" in info:
        return info
    n = S.pos4.shape[0]
    flops = (20.0 * info["direct_mean"] + 64.0 * info["approx_mean"]) * n
    return {"walk_ms": info["walk_ms_min"], "walk_ms_median": info["walk_ms_median"],
            "multipoles_ms": info["multipoles_ms_min"], "walk_tflops": flops / (info["walk_ms_min"] * 1e-3) / 1e12,
            "interactions_per_particle": {"approx": info["approx_mean"], "direct": info["direct_mean"],
                                          "max_approx": info["approx_max"], "max_direct": info["direct_max"]},
            "cells": info["cells"], "groups": info["groups"], "reps": info["reps"],
            "what": "code/computeForces.cu + code/computeMultipoles.cu with mechanical sm_100a shims (sync "
                    "shuffles, bounds-checked loads for textures, __syncwarp at warp exchanges), the reference's "
                    "launch (104 blocks x 128 threads, NI=2), on the comparison-partition tree of the same input; "
                    "CUDA events around the public Treecode calls, best of %d" % info["reps"]}


def bench_config(a, world):
    """The workload description, the same in both arms."""
    return {"workload": workload(a), "n_per_gpu": a.n, "parallelism": "replicas x%d" % world,
            "l2": "no flush: particle state 1.3 GB > 126 MB L2"}


# what the result line keeps of the whole record: these keys as they are, of each
# form its main figures, of the sweep a row per theta.  A line of all of it is over
# 20 KB, more than readers of a log's tail get.
LINE_KEYS = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
             "vs_baseline", "dtype", "data", "config", "e2e", "gpu_launches", "clocks", "roofline", "cpu_baseline",
             "accuracy", "stages_ms", "status")
FORM_KEYS = ("value", "ms_per_step", "ms_per_big_step", "ms", "theta", "median_rel_force_err", "gain_at_equal_median",
             "vs_best_fixed_meeting_target", "vs_published", "ds_cost", "frac", "unavailable")
MAX_LINE = 4000


def result_line(record):
    """The result line (a string of at most MAX_LINE characters) of a whole record."""
    def short(x):
        if isinstance(x, float):
            return float("%.7g" % x)
        if isinstance(x, dict):
            return {k: short(v) for k, v in x.items()}
        return [short(v) for v in x] if isinstance(x, (list, tuple)) else x

    line = {k: record[k] if k in ("value", "ms_per_step") else short(record[k]) for k in LINE_KEYS if k in record}
    forms = {}
    for name, form in record.items():
        if name in LINE_KEYS or not isinstance(form, dict):
            continue
        kept = {k: short(form[k]) for k in FORM_KEYS if isinstance(form.get(k), (int, float, str))}
        if kept:
            forms[name] = kept
    if record.get("theta_sweep"):
        forms["theta_sweep"] = [short([r["theta"], r["value"], r["median_rel_force_err"]]) for r in record["theta_sweep"]]
    for part in ({"forms": forms}, {}):
        text = json.dumps(dict(line, **part))
        if len(text) <= MAX_LINE:
            break
    return text


def run_reference(a):
    d = Dist("gloo")
    if d.rank != 0:
        d.close()
        return
    from oracle import oracle as O
    O.build()
    pos, vel = O.plummer_float4(a.n, a.seed)
    # the reference's GPU kernels first, before the OpenMP work (whose spinning
    # threads would slow the reference's host-side allocations)
    ref_gpu = reference_gpu_make_groups(O, pos, a)
    rng = np.random.default_rng(1)
    # warm-up: sampled steps (the walk of cpu_group_fraction of the groups,
    # extrapolated), reported beside the measurement as an estimate
    est = []
    est_desc = ""
    for s in range(a.warmup):
        t, est_desc, _ = cpu_reference_step(O, pos, vel, a, rng)
        est.append(t)
    # timed: one full step, every group walked -- the whole configuration,
    # so one step is what fits the run; steps = full steps timed
    tm, desc, S = cpu_reference_step(O, pos, vel, a, rng, full=True)
    ref_walk = reference_gpu_walk(S, a)
    v = a.n / tm / 1e6
    cores = O.num_threads()
    line = {"metric": METRIC, "value": v, "unit": UNIT, "n_gpus": a.gpus, "steps": 1, "warmup": a.warmup,
            "steps_requested": a.steps,
            "ms_per_step": tm * 1e3, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic: seeded Plummer sphere (plummer.h algorithm)",
            "config": bench_config(a, a.gpus), "impl": "reference",
            "cpu_baseline": {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
                             "sample": "one full step, nothing sampled: " + desc},
            "cpu_sampled_estimate": ({"value": a.n / statistics.mean(est) / 1e6, "unit": UNIT, "steps": len(est),
                                      "extrapolated": True, "sample": "warm-up steps: " + est_desc}
                                     if est else None),
            "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "reference_gpu_make_groups": ref_gpu,
            "reference_gpu_walk": ref_walk}
    print(json.dumps(line), flush=True)
    d.close()


# ---------------------------------------------------------------------------
# the B200 path
# ---------------------------------------------------------------------------
def run_ours(a):
    import ctypes

    import torch

    d = Dist("nccl")
    torch.cuda.set_device(d.local)
    import bonsai2_b200 as B
    from bonsai2_b200.treecode import _p

    L = B.load()
    n = a.n
    # pinned host staging (host_mem<T> of the reference, cudamem.h:64-96)
    nbytes = n * 16
    hp = L.bonsai_host_alloc(nbytes)
    hv = L.bonsai_host_alloc(nbytes)
    ha = L.bonsai_host_alloc(nbytes)
    if not (hp and hv and ha):
        raise RuntimeError("pinned allocation failed")
    pos = np.ctypeslib.as_array((ctypes.c_float * (4 * n)).from_address(hp)).reshape(n, 4)
    vel = np.ctypeslib.as_array((ctypes.c_float * (4 * n)).from_address(hv)).reshape(n, 4)
    accb = np.ctypeslib.as_array((ctypes.c_float * (4 * n)).from_address(ha)).reshape(n, 4)
    p0, v0 = B.plummer(n, a.seed)
    pos[:] = p0
    vel[:] = v0

    peak = ctypes.c_double(0.0)
    rc = L.bonsai_fp32_peak(d.local, ctypes.byref(peak))
    if rc:
        raise B.BonsaiError(rc, "bonsai_fp32_peak")

    t = B.Treecode(eps=a.eps, theta=a.theta, ncrit=a.ncrit, nleaf=a.nleaf, level_split=a.level_split, dt=a.dt,
                   device=d.local)
    t.alloc(n)
    if a.relative_alpha:
        from bonsai2_b200 import learned as Lr
        Lr.set_relative_bound(t, Lr.THETA_BOUND)
        Lr.set_theta_mode(t, 3, a.relative_alpha, a.relative_alpha)
    if L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n):
        raise RuntimeError("set_particles")
    nkern = L.bonsai_graph_kernel_count(t.handle)
    t.step(a.warmup, graph=True)
    assert t.synchronize() == 0
    E0 = t.computeEnergies()

    # ---- timed region: K graph steps, events on the handle's stream ----
    phase = np.zeros(4 * a.steps + 1, np.float32)
    d.barrier()
    torch.cuda.synchronize()
    clk = ClockSampler(d.local)
    clk.start()
    rc = L.bonsai_step_timed(t.handle, a.steps, _p(phase))
    torch.cuda.synchronize()
    clocks = clk.stop()
    d.barrier()
    if rc:
        raise B.BonsaiError(rc, "bonsai_step_timed")
    status = t.synchronize()
    region_ms = d.max(float(phase[4 * a.steps]))
    ms = region_ms / a.steps
    ph = phase[:4 * a.steps].reshape(a.steps, 4)
    walk_ms = float(ph[:, 1].mean())
    E1 = t.computeEnergies()
    hbm = hbm_roofline(n, t.tree_info(), float(ph[:, 0].mean()) + float(ph[:, 2].mean()))
    st = np.zeros(4, np.uint64)
    L.bonsai_get_stats(t.handle, _p(st))
    n_app, n_dir = float(st[0]), float(st[1])
    flops = 20.0 * n_dir + 64.0 * n_app
    achieved = flops / (walk_ms * 1e-3) / 1e12
    value = n * d.world / (ms * 1e-3) / 1e6

    # ---- accuracy at the final positions: an eager force evaluation vs FP64 direct sum ----
    t.buildTree(a.nleaf)
    t.computeMultipoles()
    t.makeGroups(a.level_split, a.ncrit)
    t.computeForces(False)
    acc = t.get_acc().astype(np.float64)
    rng = np.random.default_rng(4096 + d.rank)
    samp = rng.choice(n, min(a.error_samples, n), replace=False).astype(np.int32)
    ref = t.direct_fp64(samp, include_self=True)
    err = np.linalg.norm(acc[samp, :3] - ref[:, :3], axis=1) / np.linalg.norm(ref[:, :3], axis=1)

    # ---- e2e through the C ABI with host buffers, pipelined ----
    # every step uploads its inputs from pinned host memory and downloads its
    # accelerations; the asynchronous calls let step k+1's upload and step k's
    # download overlap compute.  Events: the handle's stream before the first
    # upload, the download stream after the last download.
    stream = torch.cuda.ExternalStream(L.bonsai_stream(t.handle))
    h2d_s, d2h_s = ctypes.c_void_p(), ctypes.c_void_p()
    L.bonsai_copy_streams(t.handle, ctypes.byref(h2d_s), ctypes.byref(d2h_s))
    d2h_stream = torch.cuda.ExternalStream(d2h_s.value)
    e2e = float("nan")
    if a.e2e_steps > 0:
        for rep in range(2):  # first round warms the staging buffers
            rc = L.bonsai_synchronize(t.handle)
            d.barrier()
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            for s in range(a.e2e_steps):
                rc |= L.bonsai_set_particles_async(t.handle, _p(pos), _p(vel), n)
                rc |= L.bonsai_step(t.handle, 1, 1)
                rc |= L.bonsai_get_particles_async(t.handle, None, None, _p(accb))
            e1.record(d2h_stream)
            e1.synchronize()
            if rc or L.bonsai_synchronize(t.handle):
                raise B.BonsaiError(rc, "e2e steps")
        e2e = d.max(e0.elapsed_time(e1) / a.e2e_steps)
    e2e_value = n * d.world / (e2e * 1e-3) / 1e6

    t.close()
    # the forms beside the headline run on a single GPU only (under torchrun
    # every rank reports the replicated headline and leaves together)
    solo = d.rank == 0 and d.world == 1
    # the batching ensemble split across the ranks (every rank takes part)
    split = None
    if a.batch_systems > 0 and d.world > 1:
        split = batching_split_form(B, L, a, d)
    elif solo and a.batch_systems > 0 and a.split_emulate > 1:
        split = batching_split_form(B, L, a, d, emulate_world=a.split_emulate)
    sweep = theta_sweep(B, L, pos, vel, a, d.local) if (solo and a.sweep) else None
    learned = learned_theta(B, L, pos, vel, a, d.local, sweep) if (solo and a.learned_target > 0) else None
    batching = batching_form(B, L, a, d.local) if (solo and a.batch_systems > 0) else None
    tuned = autotuned_headline(B, L, pos, vel, a, d.local) if (solo and a.autotune) else None
    octree = octree_build_form(B, L, a, d.local) if (solo and a.octree_n > 0) else None
    grouping = group_formation_form(B, L, pos, vel, a, d.local) if solo else None
    blocks = block_steps_form(B, L, pos, vel, a, d.local) if (solo and a.block_levels >= 0) else None
    precision = precision_form(B, L, a, d.local) if (solo and a.precision_n > 0) else None
    field = learned_field_form(B, L, a, d.local) if (solo and a.field_n > 0) else None

    cpu = None
    if d.rank == 0 and d.world == 1 and not a.no_cpu_baseline:
        from oracle import oracle as O
        O.build()
        tcpu, desc, _ = cpu_reference_step(O, p0, v0, a, np.random.default_rng(1))
        cpu = {"value": n / tcpu / 1e6, "unit": UNIT, "cores": O.num_threads(), "kind": "port",
               "sample": "one step: " + desc}

    if d.rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": d.world, "steps": a.steps,
            "warmup": a.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32",
            "data": "synthetic: seeded Plummer sphere (plummer.h algorithm), N per GPU",
            "config": bench_config(a, d.world),
            "execution": "captured CUDA graphs",
            "roofline": {"bound": "fp32", "achieved": achieved, "peak": float(peak.value), "unit": "TFLOP/s",
                         "frac": achieved / float(peak.value),
                         "traffic": WALK_DRAM_BYTES_2P22 * n / 4194304 if abs(a.theta - 0.6) < 1e-6 else None,
                         "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum of k_walk at N=2^22, "
                                           "theta 0.6, scaled by N",
                         "kernel": "k_walk", "peak_source": "measured FP32 FMA probe (bonsai_fp32_peak)",
                         "flops_per_launch": flops},
            "hbm_roofline": hbm,
            "cpu_baseline": cpu,
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": 2 * nbytes,
                    "d2h_bytes_per_step": nbytes, "ms_per_step": e2e, "steps": a.e2e_steps,
                    "api": "bonsai_set_particles_async + bonsai_step + bonsai_get_particles_async, pinned host "
                           "buffers, pipelined (copies overlap other steps' compute)"},
            "gpu_launches": int(nkern) * a.steps,
            "clocks": clocks,
            "accuracy": {"median_rel_force_err": float(np.median(err)), "p99_rel_force_err": float(np.percentile(err, 99)),
                         "samples": int(samp.shape[0]), "oracle": "FP64 direct sum (bonsai_direct_fp64)"},
            "stages_ms": {"build_multipoles_groups": float(ph[:, 0].mean()), "walk": walk_ms,
                          "move_energies": float(ph[:, 2].mean())},
            "interactions_per_particle": {"approx": n_app / n, "direct": n_dir / n, "max_approx": int(st[2]),
                                          "max_direct": int(st[3])},
            "energy": {"E_start": float(E0[3]), "E_end": float(E1[3]),
                       "rel_drift": abs(float(E1[3]) - float(E0[3])) / abs(float(E0[3])),
                       "steps_between": a.steps},
            "status": int(status),
            "theta_sweep": sweep,
            "learned_theta": learned,
            "batching": batching,
            "batching_split": split,
            "autotuned_headline": tuned,
            "octree_build": octree,
            "group_formation": grouping,
            "block_time_steps": blocks,
            "precision_form": precision,
            "learned_form_clustered_field": field,
        }
        if learned:
            learned["vs_fixed_headline"] = learned["value"] / value
            learned["double_single"]["vs_fixed_headline"] = learned["double_single"]["value"] / value
        whole = json.dumps(line)
        if a.report:
            with open(a.report, "w") as f:
                f.write(whole + "\n")
        print(whole, file=sys.stderr, flush=True)
        print(result_line(line), flush=True)
    for hptr in (hp, hv, ha):
        L.bonsai_host_free(hptr)
    d.close()


def theta_sweep(B, L, pos, vel, a, device):
    """Throughput and accuracy for every theta of the sweep (3 timed graph
    steps each; error of an eager force evaluation at the initial positions
    on 2048 seeded samples against the FP64 direct sum)."""
    from bonsai2_b200.treecode import _p
    out = []
    n = pos.shape[0]
    rng = np.random.default_rng(2048)
    samp = np.ascontiguousarray(rng.choice(n, min(2048, n), replace=False).astype(np.int32))
    ref = None
    for th in [float(x) for x in a.sweep.split(",") if x]:
        t = B.Treecode(eps=a.eps, theta=th, ncrit=a.ncrit, nleaf=a.nleaf, level_split=a.level_split, dt=a.dt,
                       device=device)
        t.alloc(n)
        L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n)
        t.buildTree(a.nleaf)
        t.computeMultipoles()
        t.makeGroups(a.level_split, a.ncrit)
        t.computeForces(False)
        acc = t.get_acc().astype(np.float64)
        if ref is None:
            ref = t.direct_fp64(samp, include_self=True)
        err = np.linalg.norm(acc[samp, :3] - ref[:, :3], axis=1) / np.linalg.norm(ref[:, :3], axis=1)
        L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n)
        t.step(2, graph=True)
        t.synchronize()
        ph = np.zeros(4 * 3 + 1, np.float32)
        rc = L.bonsai_step_timed(t.handle, 3, _p(ph))
        if rc:
            raise B.BonsaiError(rc, "sweep")
        st = np.zeros(4, np.uint64)
        L.bonsai_get_stats(t.handle, _p(st))
        walk = float(np.median(ph[:12].reshape(3, 4)[:, 1]))
        ms = float(ph[12]) / 3
        out.append({"theta": th, "value": n / (ms * 1e-3) / 1e6, "ms_per_step": ms, "walk_ms": walk,
                    "walk_tflops": (20.0 * float(st[1]) + 64.0 * float(st[0])) / (walk * 1e-3) / 1e12,
                    "approx_per_particle": float(st[0]) / n, "direct_per_particle": float(st[1]) / n,
                    "median_rel_force_err": float(np.median(err)), "p99_rel_force_err": float(np.percentile(err, 99))})
        t.close()
    return out


def learned_theta(B, L, pos, vel, a, device, sweep):
    """The learned form: per-group opening bounds from the MLP (relative
    accuracy mode, bonsai2_b200.learned), trained on a Plummer sphere of
    another seed and calibrated there (one shift of the output range, by
    bisection to 0.9 x the target median error; untimed setup), then timed on
    the bench system like the headline and judged against the FP64 direct
    sum; compared with the fixed angles of the sweep at equal median and
    equal p99 error, with the fastest fixed angle that meets the target, and
    with the relative mode's single-parameter form (tau = alpha A_g) at the
    same median.  Float and double-single positions."""
    from bonsai2_b200 import learned as Lr
    n = pos.shape[0]
    t0 = time.perf_counter()
    ptr, vtr = B.plummer(n, a.seed + 1)
    X, y, _ = Lr.relative_training_set(ptr, vtr, eps=a.eps, target=a.learned_target, max_groups=8192,
                                       nleaf=a.nleaf, ncrit=a.ncrit, level_split=a.level_split, device=device)
    w, loss = Lr.train(X, y, epochs=3000, lr=3e-3, lo=Lr.YLO, hi=Lr.YHI, device=device)
    c, lo, hi, e_cal = Lr.calibrate_relative(ptr, vtr, w, a.eps, a.learned_target, nleaf=a.nleaf, ncrit=a.ncrit,
                                             level_split=a.level_split, device=device)
    t_train = time.perf_counter() - t0
    del ptr, vtr
    rng = np.random.default_rng(2048)
    samp = np.ascontiguousarray(np.sort(rng.choice(n, min(2048, n), replace=False)).astype(np.int32))
    t = B.Treecode(eps=a.eps, theta=a.theta, device=device)
    t.alloc(n)
    t.h_ptclPos[:] = pos
    t.h_ptclVel[:] = vel
    t.ptcl_h2d()
    ref = t.direct_fp64(samp, include_self=True)
    t.close()
    kw = dict(theta=a.theta, eps=a.eps, device=device, nleaf=a.nleaf, ncrit=a.ncrit, level_split=a.level_split,
              dt=a.dt, steps=a.steps)
    out = compare_to_sweep(measure(B, L, pos, vel, samp, ref, weights=w, y_range=(lo, hi), **kw), sweep,
                           a.learned_target)
    out["unit"] = UNIT
    out["target"] = a.learned_target
    out["mode"] = ("relative: a cell passing the geometric test at theta %.2f is opened when M l^3 > tau_g ds^5, "
                   "tau_g = A_g 10^y_g (A_g: the group's mean |a| of the previous evaluation, y_g: the network)"
                   % Lr.THETA_BOUND)
    out["training"] = {"system": "Plummer N=%d seed %d" % (n, a.seed + 1), "pairs": int(X.shape[0]),
                       "final_loss": loss, "seconds": t_train,
                       "label": "cost-optimal y per group for a geometric-mean error of 0.9 x target (allocation)",
                       "calibration_shift": c, "y_range": [lo, hi], "median_err_on_training_system": e_cal}
    out["double_single"] = compare_to_sweep(
        measure(B, L, pos, vel, samp, ref, weights=w, y_range=(lo, hi), precision=1, **kw), sweep, a.learned_target)
    # the relative mode without the network: one alpha for every group,
    # bisected on the bench system itself to the learned form's median
    alpha = relative_alpha_at(B, L, pos, vel, samp, ref, out["median_rel_force_err"], **kw)
    out["relative_single_alpha"] = compare_to_sweep(
        measure(B, L, pos, vel, samp, ref, alpha=alpha, **kw), sweep, a.learned_target)
    out["relative_single_alpha"]["alpha"] = alpha
    out["calibrated_on_bench_system"] = calibrated_here(B, L, Lr, pos, vel, samp, ref, w, a.eps, a.learned_target,
                                                        sweep, kw)
    return out


def calibrated_here(B, L, Lr, pos, vel, samp, ref, w, eps, target, sweep, kw, fraction=0.9):
    """The same network with its one output shift bisected on the bench
    system itself, against 1024 direct-sum samples drawn independently of the
    judging samples -- the one knob set on the judged system, as the fixed
    angle it is compared with is picked from a sweep on that system.  Float
    and double-single positions; the untimed setup is reported."""
    t0 = time.perf_counter()
    c, lo, hi, e_cal = Lr.calibrate_relative(pos, vel, w, eps, target, fraction=fraction, samples=1024, seed=7,
                                             nleaf=kw.get("nleaf", 16), ncrit=kw.get("ncrit", 64),
                                             level_split=kw.get("level_split", 5), device=kw["device"])
    t_cal = time.perf_counter() - t0
    out = compare_to_sweep(measure(B, L, pos, vel, samp, ref, weights=w, y_range=(lo, hi), **kw), sweep, target)
    out["double_single"] = compare_to_sweep(
        measure(B, L, pos, vel, samp, ref, weights=w, y_range=(lo, hi), precision=1, **kw), sweep, target)
    out["calibration"] = {"shift": c, "y_range": [lo, hi], "fraction_of_target": fraction,
                          "median_err_on_calibration_samples": e_cal, "samples": 1024, "sample_seed": 7,
                          "seconds": t_cal}
    return out


def compare_to_sweep(r, sweep, target):
    """Fixed-angle throughput at the same median and p99 error (log-log
    interpolation over the sweep), and the fastest fixed angle of the sweep
    whose median error meets the target."""
    if not sweep:
        return r
    em = at_equal(sweep, "value", "median_rel_force_err", r["median_rel_force_err"])
    ep = at_equal(sweep, "value", "p99_rel_force_err", r["p99_rel_force_err"])
    r["fixed_theta_value_at_equal_median"] = em
    r["fixed_theta_value_at_equal_p99"] = ep
    r["gain_at_equal_median"] = r["value"] / em if em else None
    r["gain_at_equal_p99"] = r["value"] / ep if ep else None
    ok = [q for q in sweep if q["median_rel_force_err"] <= target]
    if ok:
        best = max(ok, key=lambda q: q["value"])
        r["best_fixed_meeting_target"] = {"theta": best["theta"], "value": best["value"],
                                          "median_rel_force_err": best["median_rel_force_err"]}
        r["vs_best_fixed_meeting_target"] = r["value"] / best["value"]
    return r


def relative_alpha_at(B, L, pos, vel, samp, ref, median, *, theta, eps, device, nleaf, ncrit, level_split, **_):
    """The single alpha whose relative walk (tau = alpha A_g) has the given
    median error on this system (bisection in log alpha)."""
    from bonsai2_b200 import learned as Lr
    from bonsai2_b200.treecode import _p
    n = pos.shape[0]
    t = B.Treecode(eps=eps, theta=theta, ncrit=ncrit, nleaf=nleaf, level_split=level_split, device=device)
    t.alloc(n)
    L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n)
    Lr.set_relative_bound(t, Lr.THETA_BOUND)
    refn = np.linalg.norm(ref[:, :3], axis=1)

    def med(la):
        Lr.set_theta_mode(t, 3, 10.0 ** la, 10.0 ** la)
        Lr.run_relative(t, nleaf, ncrit, level_split, evaluations=3)
        acc = t.get_acc()[samp].astype(np.float64)
        return float(np.median(np.linalg.norm(acc[:, :3] - ref[:, :3], axis=1) / refn))

    lo, hi = -4.0, -0.5
    for _ in range(10):
        mid = 0.5 * (lo + hi)
        if med(mid) > median:
            hi = mid
        else:
            lo = mid
    t.close()
    return float(10.0 ** lo)


def measure(B, L, pos, vel, samp, ref, *, theta, eps, device, nleaf=16, ncrit=64, level_split=5, dt=1.0 / 128,
            steps=3, precision=0, weights=None, y_range=None, alpha=None):
    """One configuration on one system: force evaluations judged at the
    sample particles against ref (FP64 direct sum), then `steps` timed graph
    steps from the same initial state.  weights: the learned form (theta
    mode 1, output range y_range); alpha: the relative mode with one
    parameter (theta mode 3).  Both read the previous evaluation's
    accelerations (and the learned form the previous walk's statistics), so
    their accuracy is taken at the seventh evaluation of the same positions
    (the first is the fixed-angle fallback; the bounds settle within ~5), the
    steady state the timed steps run in, and the timing after one untimed
    step.  pos may be float64 (loaded as double-single in precision 1,
    rounded to float in precision 0)."""
    from bonsai2_b200 import learned as Lr
    from bonsai2_b200.treecode import _p
    n = pos.shape[0]
    t = B.Treecode(eps=eps, theta=theta, ncrit=ncrit, nleaf=nleaf, level_split=level_split, dt=dt, device=device)
    t.set_precision(precision)
    relative = weights is not None or alpha is not None
    if relative:
        Lr.set_relative_bound(t, Lr.THETA_BOUND)
    if weights is not None:
        Lr.set_weights(t, weights)
        Lr.set_theta_mode(t, 1, *(y_range or (Lr.YLO, Lr.YHI)))
    elif alpha is not None:
        Lr.set_theta_mode(t, 3, alpha, alpha)

    def load():
        if pos.dtype == np.float64:
            t.set_particles_f64(pos, vel)
        else:
            t.alloc(n) if t.nPtcl != n else None
            t.nPtcl = n
            L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n)

    load()
    # relative modes: judged at their steady state (the bounds of one
    # evaluation follow from the previous one's accelerations and walk
    # statistics; they settle within ~5 evaluations after a load)
    Lr.run_relative(t, nleaf, ncrit, level_split, evaluations=7 if relative else 1)
    acc = t.get_acc()[samp].astype(np.float64)
    err = np.linalg.norm(acc[:, :3] - ref[:, :3], axis=1) / np.linalg.norm(ref[:, :3], axis=1)
    if relative:
        cnt = Lr.group_interactions(t)
        tau = Lr.group_scale(t)
    load()
    t.step(1, graph=True)
    t.synchronize()
    ph = np.zeros(4 * steps + 1, np.float32)
    rc = L.bonsai_step_timed(t.handle, steps, _p(ph))
    if rc:
        raise B.BonsaiError(rc, "measure")
    st = np.zeros(4, np.uint64)
    L.bonsai_get_stats(t.handle, _p(st))
    status = t.synchronize()
    t.close()
    walk = float(np.median(ph[:4 * steps].reshape(steps, 4)[:, 1]))
    ms = float(ph[4 * steps]) / steps
    out = {"theta": theta, "value": n / (ms * 1e-3) / 1e6, "ms_per_step": ms, "walk_ms": walk,
           "walk_tflops": (20.0 * float(st[1]) + 64.0 * float(st[0])) / (walk * 1e-3) / 1e12,
           "approx_per_particle": float(st[0]) / n, "direct_per_particle": float(st[1]) / n,
           "median_rel_force_err": float(np.median(err)), "p99_rel_force_err": float(np.percentile(err, 99)),
           "status": int(status)}
    if relative:
        out["theta"] = Lr.THETA_BOUND
        out["groups_walked"] = int(cnt.shape[0])
        out["group_scale_range"] = [float(np.percentile(tau, 10)), float(np.percentile(tau, 90))]
    return out


def at_equal(sweep, value_key, err_key, e):
    """Fixed-angle throughput interpolated (log-log) at error e, or None."""
    pts = sorted(((s[err_key], s[value_key]) for s in sweep), key=lambda x: x[0])
    for (e0, v0), (e1, v1) in zip(pts, pts[1:]):
        if e0 <= e <= e1 and e1 > e0:
            f = (np.log(e) - np.log(e0)) / (np.log(e1) - np.log(e0))
            return float(np.exp(np.log(v0) + f * (np.log(v1) - np.log(v0))))
    return None


def precision_form(B, L, a, device):
    """The precision form: the composite galaxy (NFW-like halo, exponential
    disk, Hernquist bulge; log-normal masses; radii ~1e-3 to 200), double-
    single positions against float positions at the same angle, both judged
    against the FP64 direct sum on the exact positions (8192 samples).  Then
    the same galaxy moved to (1e4, -7e3, 5e3) at 2^22 particles: float
    positions lose the bulge's separations there, double-single ones do not."""
    n = a.precision_n
    pos, vel = B.galaxy(n, seed=a.seed)
    rng = np.random.default_rng(8192)
    samp = np.ascontiguousarray(np.sort(rng.choice(n, 8192, replace=False)).astype(np.int32))
    eps = 0.01

    def reference(p, sm):
        # FP64 direct sum on the exact (double) positions
        t = B.Treecode(eps=eps, theta=a.theta, device=device)
        t.set_precision(1)
        t.set_particles_f64(p, vel[:p.shape[0]])
        r = t.direct_fp64(sm, include_self=True)
        t.close()
        return r

    ref = reference(pos, samp)
    out = {"config": "composite galaxy N=%d (60%% NFW r_s=10 cut 200, 30%% exp. disk R_d=3 z_d=0.3, 10%% Hernquist "
                     "a=0.5; log-normal masses sigma 0.5), theta %.2f, eps %.3f, 8192 samples" % (n, a.theta, eps)}
    for prec, key in ((1, "double_single"), (0, "fp32")):
        out[key] = measure(B, L, pos, vel, samp, ref, theta=a.theta, eps=eps, device=device, precision=prec)
    out["ds_cost"] = out["fp32"]["value"] / out["double_single"]["value"]
    m = min(n, 1 << 22)
    small = pos[:m].copy() if m < n else pos.copy()
    small_samp = np.ascontiguousarray(np.sort(np.random.default_rng(4096).choice(m, 4096, replace=False)).astype(np.int32))
    small[:, :3] += np.array([1.0e4, -7.0e3, 5.0e3])
    ref_far = reference(small, small_samp)
    far = {}
    for prec, key in ((1, "double_single"), (0, "fp32")):
        r = measure(B, L, small, vel[:m], small_samp, ref_far, theta=a.theta, eps=eps, device=device, precision=prec,
                    steps=1)
        far[key] = {"median_rel_force_err": r["median_rel_force_err"], "p99_rel_force_err": r["p99_rel_force_err"]}
    # the FP64 checker walk on the same lists: the truncation error alone
    t = B.Treecode(eps=eps, theta=a.theta, device=device)
    t.set_precision(1)
    t.set_particles_f64(small, vel[:m])
    t.buildTree(16)
    t.computeMultipoles()
    t.makeGroups(5, 64)
    a64, _ = t.compute_forces_fp64()
    t.close()
    e64 = np.linalg.norm(a64[small_samp, :3] - ref_far[:, :3], axis=1) / np.linalg.norm(ref_far[:, :3], axis=1)
    far["fp64_walk"] = {"median_rel_force_err": float(np.median(e64)), "p99_rel_force_err": float(np.percentile(e64, 99))}
    out["shifted_to_1e4"] = dict(far, particles=m, shift=[1.0e4, -7.0e3, 5.0e3])
    return out


def learned_field_form(B, L, a, device):
    """The learned form on the clustered field (64 Plummer subclusters plus
    a 20 % uniform background): the network is trained and calibrated on a
    field of another seed (untimed), then learned and fixed angles are timed
    on the bench field and judged against the FP64 direct sum (2048 samples);
    throughput at equal median and p99 error, and against the fastest fixed
    angle that meets the target."""
    from bonsai2_b200 import learned as Lr
    n = a.field_n
    eps = 0.001
    pos, vel = B.clustered_field(n, seed=a.seed)
    t0 = time.perf_counter()
    ptr, vtr = B.clustered_field(n, seed=a.seed + 1)
    X, y, _ = Lr.relative_training_set(ptr, vtr, eps=eps, target=a.learned_target, max_groups=8192, device=device)
    w, loss = Lr.train(X, y, epochs=3000, lr=3e-3, lo=Lr.YLO, hi=Lr.YHI, device=device)
    # field realisations differ more than Plummer seeds: calibrate to 0.8 x target
    c, lo, hi, e_cal = Lr.calibrate_relative(ptr, vtr, w, eps, a.learned_target, fraction=0.8, device=device)
    t_train = time.perf_counter() - t0
    del ptr, vtr
    rng = np.random.default_rng(2048)
    samp = np.ascontiguousarray(np.sort(rng.choice(n, 2048, replace=False)).astype(np.int32))
    t = B.Treecode(eps=eps, theta=0.5, device=device)
    t.alloc(n)
    t.h_ptclPos[:] = pos
    t.h_ptclVel[:] = vel
    t.ptcl_h2d()
    ref = t.direct_fp64(samp, include_self=True)
    t.close()
    kw = dict(theta=0.5, eps=eps, device=device)
    sweep = [measure(B, L, pos, vel, samp, ref, **dict(kw, theta=th)) for th in (0.4, 0.5, 0.6, 0.7, 0.8, 0.9, 1.0)]
    lrn = compare_to_sweep(measure(B, L, pos, vel, samp, ref, weights=w, y_range=(lo, hi), **kw), sweep,
                           a.learned_target)
    alpha = relative_alpha_at(B, L, pos, vel, samp, ref, lrn["median_rel_force_err"], nleaf=16, ncrit=64,
                              level_split=5, **kw)
    rel = compare_to_sweep(measure(B, L, pos, vel, samp, ref, alpha=alpha, **kw), sweep, a.learned_target)
    rel["alpha"] = alpha
    here = calibrated_here(B, L, Lr, pos, vel, samp, ref, w, eps, a.learned_target, sweep, kw)
    return {"config": "clustered field N=%d: 64 Plummer subclusters (masses log-uniform over 2 decades, scale radii "
                      "log-uniform 0.01-0.2, centres uniform in the unit cube) + 20%% uniform background; eps %.3f; "
                      "2048 samples" % (n, eps),
            "learned": lrn, "relative_single_alpha": rel, "calibrated_on_bench_field": here,
            "fixed_theta_sweep": sweep,
            "gain_at_equal_median": lrn.get("gain_at_equal_median"),
            "gain_at_equal_p99": lrn.get("gain_at_equal_p99"),
            "training": {"system": "clustered field seed %d" % (a.seed + 1), "pairs": int(X.shape[0]),
                         "final_loss": loss, "seconds": t_train, "target": a.learned_target,
                         "calibration_shift": c, "calibration_fraction": 0.8, "y_range": [lo, hi],
                         "median_err_on_training_field": e_cal}}


# the reference's one published number: the standalone octree build of a
# float32 Plummer sphere, N = 20,000,000, NLEAF 16, sm_35 (treebuild/readme:32-40)
PUBLISHED_OCTREE_MPTCL_S = 58.7943
PUBLISHED_OCTREE_SHAPE = {"nodes": 596463, "leaves": 4041848, "cells": 4638311, "levels": 15}


def octree_build_form(B, L, a, device):
    """The octree build alone (box, both keys, tree-key sort, gather into tree
    order, cells, levels, leaves: bonsai_build_tree) on the configuration of
    the reference's published build, timed with CUDA events over 5 builds
    after a warm-up build; tree shape beside the published one."""
    import torch
    from bonsai2_b200.treecode import _p
    n = a.octree_n
    p, v = B.plummer(n, a.seed)
    t = B.Treecode(eps=a.eps, theta=a.theta, nleaf=16, device=device)
    t.alloc(n)
    L.bonsai_set_particles(t.handle, _p(p), _p(v), n)
    t.buildTree(16)
    st = torch.cuda.ExternalStream(L.bonsai_stream(t.handle))
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    reps = 5
    e0.record(st)
    for _ in range(reps):
        t.buildTree(16)
    e1.record(st)
    e1.synchronize()
    info = t.tree_info()
    t.close()
    ms = e0.elapsed_time(e1) / reps
    value = n / (ms * 1e-3) / 1e6
    return {"particles": n, "nleaf": 16, "ms": ms, "value": value, "unit": "Mparticles/s",
            "published_value": PUBLISHED_OCTREE_MPTCL_S, "vs_published": value / PUBLISHED_OCTREE_MPTCL_S,
            "published_hardware": "sm_35 (K20+), treebuild_scan.cu PreferEqual", "note": "different GPU generations",
            "shape": {"nodes": info["nnodes"], "leaves": info["nleaves"], "cells": info["ncells"],
                      "levels": info["nlevels"]},
            "published_shape": PUBLISHED_OCTREE_SHAPE}


def group_formation_form(B, L, pos, vel, a, device):
    """Group formation alone on the headline system (PH-key sort, segments,
    groups, state gather into PH order: bonsai_make_groups after a build),
    timed with CUDA events over 5 calls; the reference arm times the
    reference's own makeGroups (code/makeGroups.cu, which also computes the PH
    keys) on the same input."""
    import torch
    from bonsai2_b200.treecode import _p
    n = pos.shape[0]
    t = B.Treecode(eps=a.eps, theta=a.theta, ncrit=a.ncrit, nleaf=a.nleaf, level_split=a.level_split, device=device)
    t.alloc(n)
    L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n)
    st = torch.cuda.ExternalStream(L.bonsai_stream(t.handle))
    reps, ms = 5, 0.0
    for r in range(reps + 1):  # a build before every call (groups reorder the state); the first is a warm-up
        t.buildTree(a.nleaf)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        t.makeGroups(a.level_split, a.ncrit)
        e1.record(st)
        e1.synchronize()
        if r > 0:
            ms += e0.elapsed_time(e1) / reps
    ng = t.tree_info()["ngroups"]
    t.close()
    return {"ms": ms, "value": n / (ms * 1e-3) / 1e6, "unit": "Mparticles/s", "groups": ng,
            "note": "PH keys are computed with the tree keys in the build (k_keys); the reference arm's "
                    "reference_gpu_make_groups times code/makeGroups.cu on the same input"}


def autotuned_headline(B, L, pos, vel, a, device):
    """The headline system with nLeaf / nCrit / walk layout from the
    autotuner (nLeaf {8, 16, 32} x nCrit {32, 64, 128} x 2 layouts, 2 timed
    graph steps each, untimed setup), then measured like the sweep: throughput
    and error against the FP64 direct sum.  Reported beside the headline, which
    keeps the reference's nLeaf 16 / nCrit 64."""
    from bonsai2_b200.treecode import _p
    n = pos.shape[0]
    t = B.Treecode(eps=a.eps, theta=a.theta, ncrit=a.ncrit, nleaf=a.nleaf, level_split=a.level_split, dt=a.dt,
                   device=device)
    t.alloc(n)
    L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n)
    t0 = time.perf_counter()
    r = t.autotune(nleaf=(8, 16, 32), ncrit=(32, 64, 128), steps=2)
    secs = time.perf_counter() - t0
    t.close()
    rng = np.random.default_rng(2048)
    samp = np.ascontiguousarray(np.sort(rng.choice(n, 2048, replace=False)).astype(np.int32))
    u = B.Treecode(eps=a.eps, theta=a.theta, device=device)
    u.alloc(n)
    u.h_ptclPos[:] = pos
    u.h_ptclVel[:] = vel
    u.ptcl_h2d()
    ref = u.direct_fp64(samp, include_self=True)
    u.close()
    out = measure(B, L, pos, vel, samp, ref, theta=a.theta, eps=a.eps, device=device, nleaf=r["nleaf"],
                  ncrit=r["ncrit"], level_split=a.level_split, dt=a.dt, steps=3)
    out.update({"nleaf": r["nleaf"], "ncrit": r["ncrit"], "walk_layout": r["layout"], "autotune_seconds": secs,
                "candidates_ms": r["ms"].tolist()})
    return out


def block_steps_form(B, L, pos, vel, a, device):
    """Block time steps on the headline system: levels 0..K (dt/2^k),
    eta 0.05, one big step of dt timed after one untimed big step; compared
    with what the finest substep would cost for every particle (2^K plain
    steps) and reported with the level histogram and the energy change over
    the step."""
    from bonsai2_b200.treecode import _p
    import torch
    n = pos.shape[0]
    K = a.block_levels
    t = B.Treecode(eps=a.eps, theta=a.theta, ncrit=a.ncrit, nleaf=a.nleaf, level_split=a.level_split, dt=a.dt,
                   device=device)
    t.alloc(n)
    L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n)
    t.set_block_steps(K, 0.05)
    t.block_step(1)
    e0 = t.computeEnergies()
    st = torch.cuda.ExternalStream(L.bonsai_stream(t.handle))
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    ev0.record(st)
    t.block_step(1)
    ev1.record(st)
    ev1.synchronize()
    status = t.synchronize()
    e1 = t.computeEnergies()
    lev = t.levels()
    t.close()
    ms = ev0.elapsed_time(ev1)
    return {"levels": K, "eta": 0.05, "ms_per_big_step": ms, "substeps": 1 << K,
            "value": n / (ms * 1e-3) / 1e6, "unit": "Mparticles per big step per s",
            "level_histogram": np.bincount(lev, minlength=K + 1).tolist(),
            "energy_rel_change": abs(float(e1[3]) - float(e0[3])) / abs(float(e0[3])), "status": int(status)}


def batching_form(B, L, a, device):
    """The batching form: an ensemble of independent Plummer spheres (N per
    system log-uniform in [2^10, 2^18], seeded; theta 0.5, eps 0.01), every
    stage one launch over all systems, the step replayed as captured graphs;
    nLeaf / nCrit / walk layout from the autotuner (untimed setup); then
    batch_steps timed steps.  Three systems are re-run alone for the same
    steps and compared bit for bit; forces are judged on 2048 samples against
    the FP64 direct sum inside each sample's system."""
    from bonsai2_b200.ensemble import plummer_ensemble, system_sizes
    from bonsai2_b200.treecode import _p
    counts = system_sizes(a.batch_systems, 1 << 10, 1 << 18, seed=2024)
    pos, vel = plummer_ensemble(counts, base_seed=a.seed)
    n = pos.shape[0]
    prm = dict(eps=0.01, theta=0.5, ncrit=64, nleaf=16, level_split=a.level_split, dt=1.0 / 64, device=device)
    t = B.Treecode(**prm)
    t.set_systems(counts)
    L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n)
    t0 = time.perf_counter()
    if a.batch_autotune:
        tune = t.autotune(nleaf=(8, 16, 32), ncrit=(16, 32, 64, 128), steps=2)
    else:
        tune = {"nleaf": 16, "ncrit": 64, "layout": 0}
    t_tune = time.perf_counter() - t0
    nl, nc, lay = tune["nleaf"], tune["ncrit"], tune["layout"]
    # accuracy at the initial positions
    t.buildTree(nl)
    t.computeMultipoles()
    t.makeGroups(a.level_split, nc)
    t.computeForces(False)
    acc = t.get_acc().astype(np.float64)
    rng = np.random.default_rng(2048)
    samp = np.ascontiguousarray(rng.choice(n, 2048, replace=False).astype(np.int32))
    ref = t.direct_fp64(samp, include_self=True)
    err = np.linalg.norm(acc[samp, :3] - ref[:, :3], axis=1) / np.linalg.norm(ref[:, :3], axis=1)
    # timed steps from the initial state
    L.bonsai_set_particles(t.handle, _p(pos), _p(vel), n)
    nkern = L.bonsai_graph_kernel_count(t.handle)
    ph = np.zeros(4 * a.batch_steps + 1, np.float32)
    rc = L.bonsai_step_timed(t.handle, a.batch_steps, _p(ph))
    if rc:
        raise B.BonsaiError(rc, "batching steps")
    status = t.synchronize()
    ms = float(ph[4 * a.batch_steps]) / a.batch_steps
    steps_ph = ph[:4 * a.batch_steps].reshape(a.batch_steps, 4)
    fin = np.empty((n, 4), np.float32)
    L.bonsai_get_particles(t.handle, _p(fin), None, None)
    t.close()
    # the same ensemble with double-single positions, every system moved to its
    # own offset far from the origin (uniform in [-1e4, 1e4]^3), the same tuned
    # parameters: its throughput and its cost against float positions
    ds = None
    if a.batch_ds:
        shift = np.repeat(np.random.default_rng(7).uniform(-1.0e4, 1.0e4, (len(counts), 3)), counts, axis=0)
        p64 = pos.astype(np.float64)
        p64[:, :3] += shift
        w = B.Treecode(**dict(prm, nleaf=nl, ncrit=nc))
        w.set_walk_layout(lay)
        w.set_systems(counts)
        w.set_precision(1)
        w.set_particles_f64(p64, vel)
        w.step(2, graph=True)  # warm-up and graph capture
        w.set_particles_f64(p64, vel)
        ph2 = np.zeros(4 * a.batch_steps + 1, np.float32)
        rc = L.bonsai_step_timed(w.handle, a.batch_steps, _p(ph2))
        if rc:
            raise B.BonsaiError(rc, "batching steps, double-single")
        st2 = w.synchronize()
        w.close()
        ms2 = float(ph2[4 * a.batch_steps]) / a.batch_steps
        ds = {"value": n / (ms2 * 1e-3) / 1e6, "unit": UNIT, "ms_per_step": ms2, "cost_vs_float": ms2 / ms,
              "status": int(st2), "offsets": "each system moved by U(-1e4, 1e4)^3"}
    off = np.concatenate([[0], np.cumsum(counts)])
    same = []
    for s in (0, int(np.argmax(counts)), len(counts) - 1):
        u = B.Treecode(**dict(prm, nleaf=nl, ncrit=nc))
        u.set_walk_layout(lay)
        b, e = int(off[s]), int(off[s + 1])
        u.alloc(e - b)
        ps, vs = np.ascontiguousarray(pos[b:e]), np.ascontiguousarray(vel[b:e])
        L.bonsai_set_particles(u.handle, _p(ps), _p(vs), e - b)
        u.step(a.batch_steps, graph=True)
        u.synchronize()
        one = np.empty((e - b, 4), np.float32)
        L.bonsai_get_particles(u.handle, _p(one), None, None)
        u.close()
        same.append(bool(np.array_equal(one.view(np.uint32), fin[b:e].view(np.uint32))))
    return {"value": n / (ms * 1e-3) / 1e6, "unit": UNIT, "ms_per_step": ms, "systems": int(len(counts)),
            "particles": int(n), "n_min": int(counts.min()), "n_max": int(counts.max()), "steps": a.batch_steps,
            "stages_ms": {"build_multipoles_groups": float(steps_ph[:, 0].mean()),
                          "walk": float(steps_ph[:, 1].mean()), "move_energies": float(steps_ph[:, 2].mean())},
            "kernels_per_step": int(nkern), "autotuned": {"nleaf": nl, "ncrit": nc, "walk_layout": lay,
                                                          "seconds": t_tune},
            "median_rel_force_err": float(np.median(err)), "p99_rel_force_err": float(np.percentile(err, 99)),
            "bit_identical_to_alone": same, "status": int(status), "double_single": ds,
            "config": "512 Plummer spheres, N_s = floor(2^U(10,18)) seed 2024, theta 0.5, eps 0.01, dt 1/64"}


def batching_split_form(B, L, a, d, emulate_world=0):
    """The batching form split across the ranks: the ensemble's systems are
    partitioned by estimated work (bonsai2_b200.ensemble.partition_systems),
    every rank generates and advances only its own systems as an ensemble of
    its own (nLeaf 16, nCrit 64, the half-warp layout on every rank, so that
    each system's result equals the one-process run), with no data-path
    collective; the device time is the max over ranks, and the only exchange is
    the final gather of per-system energies to rank 0.  Fixed total work
    (strong scaling).  emulate_world > 1 runs that many ranks one after another
    in this process on one GPU (a check of the split, not a scaling number)."""
    from bonsai2_b200.ensemble import gather_systems, partition_systems, plummer_ensemble, shard, system_sizes
    from bonsai2_b200.treecode import _p
    counts = system_sizes(a.batch_systems, 1 << 10, 1 << 18, seed=2024)
    world = emulate_world if emulate_world > 1 else d.world
    parts = partition_systems(counts, world)
    ranks = range(world) if emulate_world > 1 else [d.rank]
    prm = dict(eps=0.01, theta=0.5, ncrit=64, nleaf=16, level_split=a.level_split, dt=1.0 / 64,
               device=d.local)
    ms_rank, energies, sys_rank = [], [], []
    for r in ranks:
        mine = parts[r]
        cr = counts[mine].astype(np.int32)
        pos, vel = plummer_ensemble(cr, seeds=a.seed + mine)
        nr = int(cr.sum())
        t = B.Treecode(**prm)
        t.set_systems(cr)
        L.bonsai_set_particles(t.handle, _p(pos), _p(vel), nr)
        t.step(max(a.warmup, 1), graph=True)  # warm-up and graph capture
        L.bonsai_set_particles(t.handle, _p(pos), _p(vel), nr)
        ph = np.zeros(4 * a.batch_steps + 1, np.float32)
        if emulate_world <= 1:
            d.barrier()
        rc = L.bonsai_step_timed(t.handle, a.batch_steps, _p(ph))
        st = t.synchronize()
        if rc or st:
            raise B.BonsaiError(rc or st, "split batching steps")
        ms_rank.append(float(ph[4 * a.batch_steps]) / a.batch_steps)
        t.computeEnergies()
        energies.append(t.system_energies())
        sys_rank.append(mine)
        t.close()
    if emulate_world > 1:
        ms = max(ms_rank)
        E = gather_systems(None, np.concatenate(sys_rank), np.concatenate(energies), len(counts))
        per_rank = ms_rank
    else:
        ms = d.max(ms_rank[0])
        E = gather_systems(d.pg, sys_rank[0], energies[0], len(counts))
        per_rank = [None] * d.world
        if d.pg:
            d.pg.all_gather_object(per_rank, ms_rank[0])
        else:
            per_rank = ms_rank
    if d.rank != 0:
        return None
    W = [float(np.sum(counts[p] * np.log2(np.maximum(counts[p], 2)))) for p in parts]
    n = int(counts.sum())
    return {"value": n / (ms * 1e-3) / 1e6, "unit": UNIT, "ms_per_step": ms, "scaling": "strong",
            "ranks": world, "emulated_on_one_gpu": emulate_world > 1, "systems": int(len(counts)), "particles": n,
            "systems_per_rank": [int(len(p)) for p in parts],
            "particles_per_rank": [int(counts[p].sum()) for p in parts],
            "estimated_work_imbalance": max(W) / (sum(W) / len(W)),
            "ms_per_step_per_rank": per_rank, "steps": a.batch_steps,
            "energies_gathered": int(E.shape[0]), "total_energy_sum": float(E[:, 3].sum()),
            "config": "512 Plummer spheres, N_s = floor(2^U(10,18)) seed 2024, theta 0.5, eps 0.01, dt 1/64, "
                      "nLeaf 16, nCrit 64; systems partitioned by N log2 N (longest first)"}


def main():
    a = parse()
    if a.impl == "reference":
        run_reference(a)
    else:
        run_ours(a)


if __name__ == "__main__":
    main()
