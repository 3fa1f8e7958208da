"""Benchmark of the PDAC time step on B200: cell-updates/s.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl engine|reference]

One "step" is one full PDAC time step (boundary, fieldn, tilde, iter with all
its outer sweeps, ygas, htilde, ftem) of the whole domain; the metric is
cells x steps / device seconds.  Default workload: the 3D Cartesian plume on
the 256 x 256 x 192 grid (20 m cells, 5 x 5 vent at 1000 K and 150 m/s, three
particle classes, MUSCL), FP64; its resident fields (about 20 GB) are far
larger than L2.  --workload plume2d_128x192 selects the 2D cylindrical plume
(10 m cells, two classes), whose working set fits in L2, so L2 is flushed (a
256 MiB write) between its timed steps.  Inputs are synthetic, generated by
pdac_b200.configs.  Each step is timed on the engine's stream with CUDA
events.  The *_rk3_* workloads run the same decks through the explicit
SSP-RK3 solver (time_integration = 1: boundary, initialize_fieldn,
explicit_iter, ygas), the 3D one at dt = 1 ms.

An FP64 line also carries "mixed": the same deck in the mixed-precision
form (PDAC_PREC_MIXED, FP32 face fluxes) over the same steps from the same
initial state, with its device time over the timed steps, its ratio to the
FP64 value and its relative L-inf error per field against the FP64 state
after the last step (left out with --no-mixed-arm, or when the device cannot
hold a second engine).  --precision mixed reports the other way round
("vs_fp64").

With --gpus N (under torchrun) every rank advances its own replica of the
domain (the single-domain corrector does not shard; "replicas only"), the
timed region is bracketed by a barrier and device syncs, and the time is the
max over ranks.

--impl reference times the reference algorithm on the host, rank 0 only: the
CPU oracle (a C++ restatement of the reference Fortran) on the same full grid
and deck as the GPU arm, in the GPU's colour order with its 3D cell loops on
every host thread, over the GPU arm's warm-up steps (untimed) and then as
many of its timed steps, in order, as fit in about a minute.  The explicit-
solver workloads (whose oracle runs on one thread) use one replica per host
core on a 64 x 64 x 48 domain of the same deck instead, and say so.
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

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)
# hardware work queues of this process (read when CUDA starts): the
# ensemble's members run on one stream each, and the default of 8 queues
# serialises streams that share one (35.6 vs 30.1 M cell-updates/s on the
# 64-member ensemble)
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

UNIT = "cell-updates/s"
WORKLOADS = {
    # name: (deck builder, keyword arguments of the full workload, of the CPU sample, L2 handling)
    "plume3d_256x256x192": ("plume_3d", {}, {"nx": 64, "ny": 64, "nz": 48}, "inputs larger than L2 (~20 GB resident)"),
    "plume2d_128x192": ("plume_2d", {}, {}, "flushed between timed steps (256 MiB write)"),
    # a reduced 3D case of the same deck, small enough for full ncu captures
    "plume3d_128x128x96": ("plume_3d", {"nx": 128, "ny": 128, "nz": 96}, {"nx": 64, "ny": 64, "nz": 48},
                           "inputs larger than L2 (~2.6 GB resident)"),
    # the same decks advanced by the explicit SSP-RK3 solver (time_integration = 1)
    "plume3d_rk3_256x256x192": ("plume_3d_rk3", {}, {"nx": 64, "ny": 64, "nz": 48},
                                "inputs larger than L2 (~25 GB resident)"),
    "plume2d_rk3_128x192": ("plume_2d_rk3", {}, {}, "flushed between timed steps (256 MiB write)"),
    "plume3d_rk3_128x128x96": ("plume_3d_rk3", {"nx": 128, "ny": 128, "nz": 96}, {"nx": 64, "ny": 64, "nz": 48},
                               "inputs larger than L2 (~3.2 GB resident)"),
    # the large 3D deck over synthetic topography (8 seeded Gaussian hills) with immersed boundaries,
    # five particle classes, and a reduced case of it
    "plume3d_hills_384x384x256": ("plume_3d_hills", {}, {"nx": 64, "ny": 64, "nz": 48},
                                  "inputs larger than L2 (~90 GB resident)"),
    "plume3d_hills_128x128x96": ("plume_3d_hills", {"nx": 128, "ny": 128, "nz": 96}, {"nx": 64, "ny": 64, "nz": 48},
                                 "inputs larger than L2 (~4 GB resident)"),
    # 64 independent 2D cylindrical members on uneven grids (pdac_b200.ensemble), stepped together
    "ensemble2d_64": ("ensemble", {"n": 64, "seed": 0}, {"members": 2},
                      "inputs larger than L2 (~3 GB resident over the members)"),
}
WORKLOAD = "plume3d_256x256x192"


def explicit(workload):
    return "_rk3_" in workload


def is_ensemble(workload):
    return WORKLOADS[workload][0] == "ensemble"


def metric(workload, precision="fp64"):
    if is_ensemble(workload):
        return "cell-updates/s (%s semi-implicit step, batched ensemble)" % (
            "FP64" if precision == "fp64" else "mixed-precision")
    return "cell-updates/s (%s %s step)" % ("FP64" if precision == "fp64" else "mixed-precision",
                                           "explicit SSP-RK3" if explicit(workload) else "semi-implicit")


# per-field comparison of a mixed-precision run with the FP64 run of the same
# steps: max |mixed - fp64| / max |fp64| over all cells (relative L-inf)
COMPARED_FIELDS = ("p", "ep", "rlk", "ug", "vg", "wg", "us", "vs", "ws", "tg", "ts", "ygc")


def field_errors(mixed, fp64):
    import numpy as np
    out = {}
    for k in COMPARED_FIELDS:
        if k not in fp64:
            continue
        a, b = np.asarray(mixed[k], dtype=np.float64), np.asarray(fp64[k], dtype=np.float64)
        scale = float(np.max(np.abs(b)))
        out[k] = float(np.max(np.abs(a - b))) / scale if scale > 0 else float(np.max(np.abs(a - b)))
    return out


def make_case(workload=None, sample=False, precision=0):
    from pdac_b200 import configs
    from pdac_b200.setup_state import Case
    builder, kw, kw_sample, _ = WORKLOADS[workload or WORKLOAD]
    return Case(getattr(configs, builder)(**(kw_sample if sample else kw)), precision=precision)


def sample_name(workload):
    kw = WORKLOADS[workload][2]
    if not kw:
        return workload
    return f"{workload} deck on a {kw['nx']} x {kw['ny']} x {kw['nz']} domain"


# ---------------------------------------------------------------------------
# CPU arms (oracle); run in spawned processes before any GPU work
# ---------------------------------------------------------------------------
def _oracle_worker(args):
    """Advance `warm` steps untimed, then time `steps` steps of the oracle."""
    warm, steps, order, workload = args
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle
    case = make_case(workload, sample=True)
    o = pyoracle.Oracle(case, order=order)
    for s in range(1, warm + 1):
        o.step(s)
    nits = []
    t0 = time.perf_counter()
    for s in range(warm + 1, warm + steps + 1):
        nits.append(o.step(s))
    dt = time.perf_counter() - t0
    return case.ncell * steps / dt, dt, nits


def cpu_steps(workload, steps):
    """Timed oracle steps of a bounded CPU sample (about 10-30 s of work)."""
    return min(steps, 5) if WORKLOADS[workload][2] else steps


def cpu_baseline(workload, warm, steps):
    """Single-thread oracle: the steps the GPU arm times (2D) or the first
    timed steps of the reduced-domain sample (3D)."""
    import multiprocessing as mp
    ctx = mp.get_context("spawn")
    k = cpu_steps(workload, steps)
    with ctx.Pool(1) as pool:
        v, dt, nits = pool.map(_oracle_worker, [(warm, k, 1, workload)])[0]
    return dict(value=v, unit=UNIT, cores=1, kind="port",
                sample=f"steps {warm + 1}-{warm + k} of {sample_name(workload)}, "
                       f"CPU oracle (C++ restatement of the reference), lexicographic sweep order, 1 thread, "
                       f"{dt:.1f} s, mean nit {sum(nits) / len(nits):.1f}")


def _replicas(workload):
    """One replica per host core, bounded by available host memory."""
    cores = os.cpu_count() or 1
    try:
        import psutil
        avail = psutil.virtual_memory().available
    except Exception:
        return cores
    per = 2.0e9 if WORKLOADS[workload][2] else 0.2e9  # oracle footprint of one replica, generous
    return max(1, min(cores, int(0.6 * avail / per)))


def _full_oracle_worker(args):
    """The oracle on the full workload, coloured sweep order, on `threads`
    host threads: `warm` untimed steps (the GPU arm's warm-up steps), then
    the GPU arm's timed steps in order until `steps` of them or `budget_s`
    seconds of timed work (at least one step)."""
    warm, steps, workload, threads, budget_s = args
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle
    used = pyoracle.set_threads(threads)
    case = make_case(workload)
    o = pyoracle.Oracle(case, order=pyoracle.ORDER_COLORED)
    t0 = time.perf_counter()
    for s in range(1, warm + 1):
        o.step(s)
    warm_s = time.perf_counter() - t0
    nits, times = [], []
    for s in range(warm + 1, warm + steps + 1):
        t = time.perf_counter()
        nits.append(o.step(s))
        times.append(time.perf_counter() - t)
        if sum(times) >= budget_s:
            break
    return case.ncell, nits, times, warm_s, used


def full_grid_fits(workload):
    """Whether the oracle (about 2.2 kB a cell) and the set-up (0.3 kB a
    cell) of the full workload fit in 80 % of the available host memory."""
    _, kw, _, _ = WORKLOADS[workload]
    case_cells = kw.get("nx", 256) * kw.get("ny", 256) * kw.get("nz", 192)
    try:
        import psutil
        return 2.6e3 * case_cells < 0.8 * psutil.virtual_memory().available
    except Exception:
        return True


# timed seconds of the reference arm's oracle steps (after the warm-up steps)
REFERENCE_BUDGET_S = 45.0


def reference_arm(args):
    """The reference algorithm on the host cores, on the GPU arm's workload.

    Semi-implicit workloads: the CPU oracle (C++ restatement of the reference
    Fortran) on the FULL grid and deck of the GPU arm, in the GPU's colour
    order (the same outer-sweep counts step by step), with its 3D cell loops
    on every host thread; it advances the GPU arm's warm-up steps untimed and
    then times the GPU arm's timed steps in order, as many as fit in
    REFERENCE_BUDGET_S seconds (at least one).  Explicit-solver workloads,
    whose oracle runs on one thread, and full grids that do not fit in host
    memory: one oracle replica per host core on a reduced domain of the same
    deck (the line says so)."""
    import multiprocessing as mp
    workload = args.workload
    cores = os.cpu_count() or 1
    steps = max(1, args.steps)
    ctx = mp.get_context("spawn")
    if not explicit(workload) and full_grid_fits(workload):
        with ctx.Pool(1) as pool:
            ncell, nits, times, warm_s, used = pool.map(
                _full_oracle_worker, [(args.warmup, steps, workload, cores, REFERENCE_BUDGET_S)])[0]
        k = len(nits)
        wall = sum(times)
        value = ncell * k / wall
        threads = used if make_case(workload).is3d else 1
        sample = (f"steps {args.warmup + 1}-{args.warmup + k} of {workload} (the first {k} of the GPU arm's "
                  f"{steps} timed steps, after its {args.warmup} warm-up steps, {warm_s:.0f} s untimed), full "
                  f"{ncell}-cell grid, CPU oracle (C++ restatement of the reference) in the GPU's colour order, "
                  f"{threads} host thread(s), nit {nits}, s/step {[round(t, 1) for t in times]}")
        config = {"workload": workload, "cells": ncell, "order": "colored (as the GPU)", "nit": nits,
                  "host_threads": threads, "l2": "n/a (host)"}
        cores_used = threads
    else:
        cores = _replicas(workload)
        steps = cpu_steps(workload, steps)
        with ctx.Pool(cores) as pool:
            res = pool.map(_oracle_worker, [(args.warmup, steps, 1, workload)] * cores)
            wall = max(r[1] for r in res)  # timed steps only, slowest replica
        ncell = make_case(workload, sample=True).ncell
        value = cores * ncell * steps / wall
        nits = [n for r in res for n in r[2]]
        k = steps
        sample = (f"steps {args.warmup + 1}-{args.warmup + steps} of {sample_name(workload)} per replica, "
                  f"{cores} replicas (one per host core), CPU oracle, lexicographic order, "
                  f"mean nit {sum(nits) / len(nits):.1f} (a reduced domain, not the GPU arm's grid)")
        config = {"workload": workload, "cells": ncell, "replicas": cores, "order": "lexicographic",
                  "l2": "n/a (host)", "same_grid_as_gpu_arm": False}
        cores_used = cores
    line = {
        "metric": metric(workload, args.precision), "value": value, "unit": UNIT, "n_gpus": args.gpus, "steps": k,
        "warmup": args.warmup, "ms_per_step": 1000.0 * wall / k, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": config,
        "impl": "reference",
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores_used, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------
# clocks sampling during the timed region
# ---------------------------------------------------------------------------
class Clocks:
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index):
        self.index = index
        self.rows = []
        self.proc = None

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--id={self.index}", f"--query-gpu={self.Q}",
                                          "--format=csv,noheader,nounits", "-lms", "100"],
                                         stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm = [float(r[1]) for r in self.rows if len(r) > 2 and r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if len(r) > 2 and r[2].replace(".", "").isdigit()]
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        reasons = set()
        for r in self.rows:
            for q, n in enumerate(names):
                if len(r) > 5 + q and r[5 + q].lower() == "active":
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm)}


def measured_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return d["hbm_gbs"], "measured"
    return 6650.0, "fallback"


def profiled_traffic(workload, kernel, algorithmic_bytes):
    """DRAM bytes per launch of `kernel` from a committed ncu capture, and
    how it was obtained: the capture's own figure on a captured workload; on
    another the DRAM/algorithmic ratio times this launch's algorithmic bytes
    where that ratio was found the same at two sizes; else None."""
    p = os.path.join(ROOT, "profiles", "traffic.json")
    if not os.path.exists(p):
        return None, "no capture"
    d = json.load(open(p)).get(kernel)
    if not d:
        return None, "no capture"
    own = d["workloads"].get(workload)
    if own:
        return own["bytes_per_launch"], f"ncu on {workload}, mean over {own['launches']} launches"
    if d["proportional"]:
        return (d["dram_per_algorithmic"] * algorithmic_bytes,
                f"{d['dram_per_algorithmic']:.2f} x algorithmic bytes, the DRAM/algorithmic ratio of ncu captures "
                f"({d['evidence']})")
    return None, f"not scaled from {', '.join(d['workloads'])}: {d['why_not']}"


# ---------------------------------------------------------------------------
# engine arm
# ---------------------------------------------------------------------------
def engine_arm(args):
    import numpy as np
    import torch

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    else:
        torch.cuda.set_device(0)

    workload = args.workload
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = cpu_baseline(workload, args.warmup, args.steps)

    from pdac_b200 import roofline
    from pdac_b200.engine import Engine

    from pdac_b200 import abi
    prec = abi.PREC_MIXED if args.precision == "mixed" else abi.PREC_FP64
    case = make_case(workload, precision=prec)
    free_before = torch.cuda.mem_get_info()[0]
    eng = Engine(case)
    engine_bytes = free_before - torch.cuda.mem_get_info()[0]
    ncell = case.ncell
    nfluid = case.fluid_count()
    dims = 3 if case.is3d else 2
    small = not case.is3d  # working set fits in L2: flush it between timed steps
    flush = torch.empty(256 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda") if small else None

    def barrier():
        torch.cuda.synchronize()
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    # warm-up steps (untimed), then the launch shapes tuned on the warmed-up
    # state (pdac_gpu_autotune: the state is left as it was)
    for s in range(1, args.warmup + 1):
        eng.step(s)
    tuning = eng.autotune() if not args.no_autotune else None
    barrier()
    eng.reset_stats(profile_corrector=False)  # production path: the sweep loop runs on the device
    nits = []
    step_ms = []
    with Clocks(local) as clk:
        barrier()
        for q in range(args.steps):
            if flush is not None:
                flush.zero_()
            torch.cuda.synchronize()
            eng.mark(0)
            nits.append(eng.step(args.warmup + q + 1))
            eng.mark(1)
            step_ms.append(eng.elapsed(0, 1))
        barrier()
    timed_stats = eng.stats()
    phase_ms = eng.phase_times()  # device time of each phase in the last timed step
    # per-kernel times of the corrector come from the next steps, run with the
    # host sweep loop and CUDA events around every colour phase's kernels
    prof_steps = min(args.steps, 3)
    eng.reset_stats(profile_corrector=True)
    prof_nits = [eng.step(args.warmup + args.steps + q + 1) for q in range(prof_steps)]
    stats = eng.stats()
    total_ms = sum(step_ms)
    vs_fp64 = mixed_arm = None
    # (a second engine beside the first: only where the device holds both)
    room = torch.cuda.mem_get_info()[0] > 1.2 * engine_bytes + (2 << 30)
    if room and (prec == abi.PREC_MIXED or not args.no_mixed_arm):
        # the other precision over the same steps from the same initial state,
        # launch shapes tuned after the same warm-up steps: its device time
        # over the timed steps and the mixed form's error per field
        nall = args.warmup + args.steps + prof_steps
        other_prec = abi.PREC_FP64 if prec == abi.PREC_MIXED else abi.PREC_MIXED
        other = Engine(make_case(workload, precision=other_prec))
        other_ms = 0.0
        for s in range(1, nall + 1):
            if s == args.warmup + 1 and not args.no_autotune:
                other.autotune()
            if flush is not None:
                flush.zero_()
            other.mark(0)
            other.step(s)
            other.mark(1)
            if args.warmup < s <= args.warmup + args.steps:
                other_ms += other.elapsed(0, 1)
        mine_state, other_state = eng.download(), other.download()
        mt_mine, mt_other = eng.mass_totals(), other.mass_totals()
        other.close()
        other_value = ncell * args.steps / (other_ms / 1000.0)
        mine_value = ncell * args.steps / (total_ms / 1000.0)
        if prec == abi.PREC_MIXED:
            mix_state, ref_state, mt_mix, mt_ref = mine_state, other_state, mt_mine, mt_other
            vs_fp64 = {"fp64_value": other_value, "ratio": mine_value / other_value}
        else:
            mix_state, ref_state, mt_mix, mt_ref = other_state, mine_state, mt_other, mt_mine
            mixed_arm = {"value": other_value, "ratio_to_fp64": other_value / mine_value,
                         "dtype": "f32 flux passes, f64 state and updates"}
        cmp = {"steps_compared": nall, "field_rel_linf": field_errors(mix_state, ref_state),
               "mass_totals_rel": [abs(a - b) / abs(b) if b else abs(a - b) for a, b in zip(mt_mix, mt_ref)]}
        (vs_fp64 if vs_fp64 is not None else mixed_arm).update(cmp)
    if dist is not None:
        t = torch.tensor([total_ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms = float(t.item())
    value = world * ncell * args.steps / (total_ms / 1000.0)

    # end-to-end through the C ABI: upload from pinned host memory, step,
    # download, every step
    e2e_case = make_case(workload, precision=prec)
    e2 = Engine(e2e_case, upload=False)
    if tuning is not None:
        e2.set_tuning(tuning)
    host = {k: torch.from_numpy(v).pin_memory().numpy() for k, v in e2e_case.state.items()}
    nbytes = sum(v.nbytes for v in host.values())
    import ctypes as C
    view = abi.make_state_view(host)
    L = e2.L
    # every step's inputs go up from the pinned host arrays and its result
    # comes back into them; between two steps one pdac_gpu_exchange_state
    # does both (the previous step's download and this step's upload, field
    # by field on the two copy engines), so the timed windows are: the first
    # upload with step 1, each exchange with the next step, the last download
    vp = C.byref(view)
    for s in range(1, args.warmup + 1):
        assert (L.pdac_gpu_upload_state(e2.h, vp) if s == 1 else L.pdac_gpu_exchange_state(e2.h, vp, vp)) == 0
        e2.step(s)
    assert L.pdac_gpu_download_state(e2.h, vp) == 0
    barrier()
    e2e_ms = 0.0
    for q in range(args.steps + 1):
        if flush is not None:
            flush.zero_()
        torch.cuda.synchronize()
        e2.mark(2)
        if q == 0:
            st = L.pdac_gpu_upload_state(e2.h, vp)
        elif q < args.steps:
            st = L.pdac_gpu_exchange_state(e2.h, vp, vp)
        else:
            st = L.pdac_gpu_download_state(e2.h, vp)
        if q < args.steps:
            e2.step(args.warmup + q + 1)
        e2.mark(3)
        e2e_ms += e2.elapsed(2, 3)
        assert st == 0
    if dist is not None:
        t = torch.tensor([e2e_ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e2e_ms = float(t.item())
    e2e_value = world * ncell * args.steps / (e2e_ms / 1000.0)

    peak, peak_kind = measured_peaks()
    mean_nit = sum(nits) / len(nits)
    measured_on = (f"steps {args.warmup + args.steps + 1}-{args.warmup + args.steps + prof_steps} "
                   f"(nit {prof_nits}), CUDA events on the engine stream")
    if explicit(workload):
        # explicit solver: the kernel group (flux passes, stage kernels,
        # gas-enthalpy wavefronts, final solve) that took the most device time
        calls = max(stats["rk3_calls"], 1)
        group = max(stats["rk3_ms"], key=stats["rk3_ms"].get)
        names = {"flux": "flux passes (k_rk3_mflux, k_tilde_flux*, k_htilde_flux*)", "stage": "k_rk3_stage",
                 "wave": "k_rk3_wave_pre/tile/post (gas-enthalpy wavefront)", "final": "k_rk3_final_rhs/phys/solve"}
        gbytes = roofline.rk3_group_bytes(case.nsolid, case.ngas, dims, nfluid)
        kname = names[group]
        bytes_per_launch = gbytes[group]
        avg_launch_s = stats["rk3_ms"][group] / 1000.0 / calls
        achieved = bytes_per_launch / avg_launch_s / 1e9
        rdetail = {"unit_of_launch": "one kernel group of one explicit_iter", "launches": calls,
                   "group_ms_per_explicit_iter": {k: v / calls for k, v in stats["rk3_ms"].items()},
                   "group_algorithmic_bytes": gbytes, "measured_on": measured_on}
    else:
        # roofline of the dominant kernel: the residual test or the inner loop of
        # the corrector's colour phases, whichever took more device time
        phases = max(stats["corr_launches"], 1)
        sweeps_cells = nfluid * (stats["corr_launches"] // 3)  # fluid cells of all timed sweeps
        tested = stats["tested_cells"]  # of which the active set tested
        unconv = stats["work_cells"]
        if stats["inner_ms"] >= stats["resid_ms"]:
            kname, kms = "k_inner_team", stats["inner_ms"]
            kbytes = roofline.inner_bytes(case.nsolid, case.ngas, dims, unconv)
        else:
            kname, kms = "k_resid_scan", stats["resid_ms"]
            kbytes = roofline.resid_bytes(case.nsolid, dims, tested - unconv, unconv, ncell, phases)
        bytes_per_launch = kbytes / phases
        avg_launch_s = kms / 1000.0 / phases
        achieved = bytes_per_launch / avg_launch_s / 1e9
        rdetail = {"launches": phases,
                   "route": "kernel timed in launches (host sweep loop, the steps of measured_on); the timed steps run "
                            "the same cell bodies inside one launch of the sweep loop",
                   "corrector_ms": {"resid": stats["resid_ms"], "inner": stats["inner_ms"]},
                   "unconverged_cell_visits": unconv, "tested_cell_visits": tested,
                   "fluid_cell_visits": sweeps_cells, "measured_on": measured_on}

    traffic, traffic_basis = profiled_traffic(workload, kname, bytes_per_launch)
    if rank == 0:
        line = {
            "metric": metric(workload, args.precision), "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None,
            "dtype": "f64" if prec == abi.PREC_FP64 else "f32 flux passes, f64 state and updates", "data": "synthetic",
            "config": {"workload": workload, "cells": ncell, "fluid_cells": nfluid, "nsolid": case.nsolid,
                       "mean_nit": mean_nit, "nit": nits, "parallelism": f"replicas{world}",
                       "l2": WORKLOADS[workload][3], "precision": args.precision,
                       "launch_shapes": tuning if tuning is not None else "defaults (--no-autotune)"},
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": nbytes, "d2h_bytes_per_step": nbytes,
                    "copies": "whole state up and down every step from pinned host memory; between steps one "
                              "pdac_gpu_exchange_state (download and upload overlapped field by field)"},
            "gpu_launches": timed_stats["launches"],
            "roofline": {"bound": "hbm", "kernel": kname, "achieved": achieved, "peak": peak,
                         "peak_kind": peak_kind, "unit": "GB/s", "frac": achieved / peak,
                         "traffic": traffic, "traffic_basis": traffic_basis,
                         "algorithmic_bytes_per_launch": bytes_per_launch,
                         "avg_launch_us": avg_launch_s * 1e6, **rdetail},
            "last_step_phase_ms": phase_ms,
            "clocks": clk.summary(),
            "cpu_baseline": cpu,
        }
        if vs_fp64 is not None:
            line["vs_fp64"] = vs_fp64
        if mixed_arm is not None:
            line["mixed"] = mixed_arm
        print(json.dumps(line), flush=True)
    eng.close()
    e2.close()
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()


# ---------------------------------------------------------------------------
# ensemble workload: many independent 2D members stepped together
# ---------------------------------------------------------------------------
def ensemble_decks(workload):
    from pdac_b200 import ensemble
    kw = WORKLOADS[workload][1]
    return ensemble.member_decks(kw["n"], seed=kw["seed"])


def _ensemble_oracle_worker(args):
    """Oracle steps of the given members, one after the other: `warm`
    untimed steps each, then `steps` timed steps each."""
    members, warm, steps, workload = args
    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import pyoracle
    from pdac_b200.setup_state import Case
    decks = ensemble_decks(workload)
    cells, wall, nits = 0, 0.0, []
    for m in members:
        case = Case(decks[m])
        o = pyoracle.Oracle(case, order=1)
        for s in range(1, warm + 1):
            o.step(s)
        t0 = time.perf_counter()
        for s in range(warm + 1, warm + steps + 1):
            nits.append(o.step(s))
        wall += time.perf_counter() - t0
        cells += case.ncell * steps
    return cells, wall, nits


def ensemble_cpu_baseline(workload, warm, steps):
    """Single-thread oracle on the first members of the ensemble."""
    import multiprocessing as mp
    nm = WORKLOADS[workload][2]["members"]
    k = min(steps, 5)
    with mp.get_context("spawn").Pool(1) as pool:
        cells, wall, nits = pool.map(_ensemble_oracle_worker, [(list(range(nm)), warm, k, workload)])[0]
    return dict(value=cells / wall, unit=UNIT, cores=1, kind="port",
                sample=f"steps {warm + 1}-{warm + k} of members 0-{nm - 1} of {workload}, CPU oracle "
                       f"(C++ restatement of the reference), lexicographic sweep order, 1 thread, {wall:.1f} s, "
                       f"mean nit {sum(nits) / len(nits):.1f}")


def ensemble_reference_arm(args):
    """The reference algorithm on the host cores: the ensemble's members
    spread over one process per core (largest first), each member advanced
    `steps` timed steps after the warm-up; time = slowest process."""
    import multiprocessing as mp
    from pdac_b200 import ensemble
    workload = args.workload
    decks = ensemble_decks(workload)
    cells = [d["nx"] * d["nz"] for d in decks]
    cores = min(os.cpu_count() or 1, len(decks))
    steps = max(1, min(args.steps, 5))
    warm = args.warmup
    parts = [p for p in ensemble.split(cells, cores) if p]
    with mp.get_context("spawn").Pool(len(parts)) as pool:
        res = pool.map(_ensemble_oracle_worker, [(p, warm, steps, workload) for p in parts])
    wall = max(r[1] for r in res)
    total = sum(r[0] for r in res)
    value = total / wall
    nits = [n for r in res for n in r[2]]
    line = {
        "metric": metric(workload), "value": value, "unit": UNIT, "n_gpus": args.gpus, "steps": steps,
        "warmup": warm, "ms_per_step": 1000.0 * wall / steps, "higher_is_better": True,
        "scaling": "strong", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
        "config": {"workload": workload, "members": len(decks), "cells": sum(cells), "processes": len(parts),
                   "order": "lexicographic", "l2": "n/a (host)"},
        "impl": "reference",
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": len(parts), "kind": "port",
                         "sample": f"all {len(decks)} members, steps {warm + 1}-{warm + steps} each, spread over "
                                   f"{len(parts)} processes (one per host core), CPU oracle, "
                                   f"mean nit {sum(nits) / len(nits):.1f}"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def ensemble_arm(args):
    import torch
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
    else:
        torch.cuda.set_device(0)
    workload = args.workload
    cpu = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        cpu = ensemble_cpu_baseline(workload, args.warmup, args.steps)

    from pdac_b200 import abi, ensemble, roofline
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    import ctypes as C

    decks = ensemble_decks(workload)
    all_cells = [d["nx"] * d["nz"] for d in decks]
    mine = ensemble.split(all_cells, world)[rank]  # no exchange between ranks
    prec = abi.PREC_MIXED if args.precision == "mixed" else abi.PREC_FP64
    cases = [Case(decks[m], precision=prec) for m in mine]
    engines = [Engine(c) for c in cases]
    batch = ensemble.Batch(engines)
    my_cells = sum(c.ncell for c in cases)
    total_cells = sum(all_cells)

    def barrier():
        torch.cuda.synchronize()
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize()

    for s in range(1, args.warmup + 1):
        batch.step(s)
    barrier()
    for e in engines:
        e.reset_stats(profile_corrector=False)
    nits, step_ms = [], []
    with Clocks(local) as clk:
        barrier()
        for q in range(args.steps):
            nits.append(batch.step(args.warmup + q + 1))
            step_ms.append(batch.elapsed())
        barrier()
    launches = sum(e.stats()["launches"] for e in engines)
    total_ms = sum(step_ms)
    if dist is not None:
        t = torch.tensor([total_ms, float(launches)], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms = float(t[0].item())
        t = torch.tensor([float(launches)], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.SUM)
        launches = int(t.item())
    value = total_cells * args.steps / (total_ms / 1000.0)

    vs_fp64 = None
    if prec == abi.PREC_MIXED:
        # the FP64 batch of the same members over the same steps: its device
        # time over the timed steps and the mixed members' error per field
        # (the largest over the members)
        nall = args.warmup + args.steps
        ref_engines = [Engine(Case(decks[m])) for m in mine]
        rb = ensemble.Batch(ref_engines)
        ref_ms = 0.0
        for s in range(1, nall + 1):
            rb.step(s)
            if s > args.warmup:
                ref_ms += rb.elapsed()
        errs = {}
        for e, r in zip(engines, ref_engines):
            for k, v in field_errors(e.download(), r.download()).items():
                errs[k] = max(errs.get(k, 0.0), v)
        rb.close()
        for r in ref_engines:
            r.close()
        if dist is not None:
            t = torch.tensor([ref_ms], device="cuda")
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ref_ms = float(t.item())
        ref_value = total_cells * args.steps / (ref_ms / 1000.0)
        vs_fp64 = {"fp64_value": ref_value, "ratio": value / ref_value, "steps_compared": nall,
                   "field_rel_linf_max_over_members": errs}

    # the same members and steps through the plain single-context path, one
    # member after the other (no batch): the speed-up of batching
    def one_by_one(member_cases):
        seq = [Engine(c) for c in member_cases]
        for s in range(1, args.warmup + 1):
            for e in seq:
                e.step(s)
        ms = 0.0
        for q in range(args.steps):
            for e in seq:
                e.mark(0)
                e.step(args.warmup + q + 1)
                e.mark(1)
                ms += e.elapsed(0, 1)
        for e in seq:
            e.close()
        if dist is not None:
            t = torch.tensor([ms], device="cuda")
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms

    seq_ms = one_by_one(cases)
    seq_value = total_cells * args.steps / (seq_ms / 1000.0)
    if vs_fp64 is not None:
        # the plain FP64 form: the same members in FP64, one after the other
        plain_ms = one_by_one([Case(decks[m]) for m in mine])
        plain_value = total_cells * args.steps / (plain_ms / 1000.0)
        vs_fp64["fp64_unbatched_value"] = plain_value
        vs_fp64["ratio_to_fp64_unbatched"] = value / plain_value

    # the survey's step byte model: every fluid cell read and written in
    # every pass and every outer sweep, summed over this rank's members
    step_bytes = 0.0
    for c, col in zip(cases, zip(*nits)):
        mean_nit = sum(col) / len(col)
        step_bytes += c.fluid_count() * roofline.step_bytes_per_cell(c.nsolid, c.ngas, mean_nit, 2)
    my_ms = sum(step_ms) / args.steps
    achieved = step_bytes / (my_ms / 1000.0) / 1e9

    # end to end through the public API: every member's state uploaded from
    # pinned host memory, one batch step, every member's state downloaded;
    # the host calls are synchronous, so events on torch's stream bracket them
    hosts = [{k: torch.from_numpy(v).pin_memory().numpy() for k, v in c.state.items()} for c in cases]
    views = [abi.make_state_view(h) for h in hosts]
    nbytes = sum(v.nbytes for h in hosts for v in h.values())
    e2_engines = [Engine(c, upload=False) for c in cases]
    e2 = ensemble.Batch(e2_engines)
    L = e2_engines[0].L

    # every member's inputs go up and its result comes back every step; between
    # two steps one pdac_gpu_exchange_state per member does both (download and
    # upload overlapped field by field), so the timed windows are: the first
    # uploads with step 1, each round of exchanges with the next step, the last
    # downloads
    def e2e_window(q, s, last):
        st = 0
        for e, v in zip(e2_engines, views):
            vp = C.byref(v)
            if q == 0:
                st |= L.pdac_gpu_upload_state(e.h, vp)
            elif q < last:
                st |= L.pdac_gpu_exchange_state(e.h, vp, vp)
            else:
                st |= L.pdac_gpu_download_state(e.h, vp)
        if q < last:
            e2.step(s)
        assert st == 0

    for q in range(args.warmup + 1):
        e2e_window(q, q + 1, args.warmup)
    barrier()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e2e_ms = 0.0
    for q in range(args.steps + 1):
        torch.cuda.synchronize()
        a.record()
        e2e_window(q, args.warmup + q + 1, args.steps)
        b.record()
        b.synchronize()
        e2e_ms += a.elapsed_time(b)
    if dist is not None:
        t = torch.tensor([e2e_ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e2e_ms = float(t.item())
    e2e_value = total_cells * args.steps / (e2e_ms / 1000.0)

    peak, peak_kind = measured_peaks()
    if rank == 0:
        flat = [n for row in nits for n in row]
        line = {
            "metric": metric(workload, args.precision), "value": value, "unit": UNIT, "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None,
            "dtype": "f64" if prec == abi.PREC_FP64 else "f32 flux passes, f64 state and updates", "data": "synthetic",
            "config": {"workload": workload, "members": len(decks), "cells": total_cells,
                       "members_on_rank0": len(mine), "cells_on_rank0": my_cells,
                       "grids": "nx U{64..256} x nz U{96..384}, 10 m cells, 2D cylindrical",
                       "mean_nit": sum(flat) / len(flat), "max_nit": max(flat),
                       "parallelism": f"members split over {world} rank(s) by cell count, no exchange",
                       "host_threads_per_rank": len(mine), "l2": WORKLOADS[workload][3],
                       "unbatched_value": seq_value, "unbatched_ms_per_step": seq_ms / args.steps,
                       "unbatched": "the same members and steps, one pdac_gpu_step after the other"},
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": nbytes * world,
                    "d2h_bytes_per_step": nbytes * world,
                    "copies": "every member's state up and down every step from pinned host memory; between "
                              "steps one pdac_gpu_exchange_state per member"},
            "gpu_launches": launches,
            "roofline": {"bound": "hbm", "kernel": "whole ensemble step (every kernel of every member, concurrent)",
                         "achieved": achieved, "peak": peak, "peak_kind": peak_kind, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": None,
                         "algorithmic_bytes_per_launch": step_bytes, "avg_launch_us": my_ms * 1000.0,
                         "unit_of_launch": "one batch step of rank 0's members",
                         "byte_model": "roofline.step_bytes_per_cell at each member's mean nit (every fluid cell "
                                       "every pass and outer sweep)"},
            "clocks": clk.summary(),
            "cpu_baseline": cpu,
        }
        if vs_fp64 is not None:
            line["vs_fp64"] = vs_fp64
        print(json.dumps(line), flush=True)
    batch.close()
    e2.close()
    for e in engines + e2_engines:
        e.close()
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--workload", default=WORKLOAD, choices=sorted(WORKLOADS))
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="engine", choices=["engine", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-autotune", action="store_true",
                    help="keep the default launch shapes instead of tuning them after the warm-up steps")
    ap.add_argument("--precision", default="fp64", choices=["fp64", "mixed"],
                    help="mixed: the flux passes in FP32 (PDAC_PREC_MIXED), compared with FP64 in the same run")
    ap.add_argument("--no-mixed-arm", action="store_true",
                    help="FP64 runs: leave out the mixed-precision form that otherwise runs "
                         "over the same steps and is reported beside the FP64 value (\"mixed\")")
    args = ap.parse_args()
    if args.impl == "reference":
        if int(os.environ.get("RANK", "0")) != 0:
            return
        (ensemble_reference_arm if is_ensemble(args.workload) else reference_arm)(args)
        return
    (ensemble_arm if is_ensemble(args.workload) else engine_arm)(args)


if __name__ == "__main__":
    main()
