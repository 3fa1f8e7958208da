"""The workloads whose speed this framework is judged by.

Every case is a burst of a run's time loop as a host program drives it: the
host owns the state arrays (the module arrays of the reference, here pinned
host memory), hands them to the device, advances K time steps on the device
and reads the whole state back, as it does between two outputs, restarts or
couplings (``pdac_gpu_upload_state``, K x ``pdac_gpu_step``,
``pdac_gpu_download_state``; ``pdac_gpu_batch_step`` for an ensemble).

The state a burst starts from is a few steps into the eruption, where the
corrector does its typical number of outer sweeps; the vent velocity,
temperature and volume fractions come from the seed.  The decks are the
builders of ``pdac_b200.configs`` (2D cylindrical plume, 3D plume over flat
ground, 3D plume over hills with immersed boundaries), over

  solver     "semi" (semi-implicit, the default) and "rk3" (explicit SSP-RK3)
  precision  "fp64" and "mixed" (FP32 face fluxes)
  nsolid     1, 2, 3 or 5 particle classes
  les        the Smagorinsky sub-grid model (the reference's default) or none
  members    0: one domain; else an ensemble of that many 2D members stepped
             as one batch, their grids those pdac_b200.ensemble draws from
             the case's grid_seed

Sizes run from 24 x 33 cells, where a step is launches and latency, to the
256 x 256 x 192 plume of the default benchmark.
"""
import math
import os
import random
import tempfile

import torch

from pdac_b200 import abi, configs, ensemble
from pdac_b200.engine import Engine, PdacError
from pdac_b200.setup_state import Case

# steps run before a burst's state is taken
WARM_STEPS = 3

DIAMETERS = {1: (100.0,), 2: (50.0, 500.0), 3: (30.0, 250.0, 1000.0),
             5: (20.0, 63.2, 200.0, 632.0, 2000.0)}
DENSITY = 2500.0


def _case(name, deck, nx, ny, nz, nsolid, steps, solver="semi", precision="fp64", les=False, members=0, grid_seed=0):
    c = dict(deck=deck, nx=nx, ny=ny, nz=nz, nsolid=nsolid, steps=steps, solver=solver, precision=precision,
             les=les, members=members, grid_seed=grid_seed)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest calls: a coarse axisymmetric run for a first look
        _case("2d_coarse", "plume2d", 24, 1, 33, 2, 3),
        # the 2D cylindrical workload of the benchmark, an everyday run
        _case("2d_plume", "plume2d", 128, 1, 192, 2, 10),
        # a fine 2D run on a ragged grid with the default sub-grid model
        _case("2d_fine_les", "plume2d", 251, 1, 383, 2, 5, les=True),
        # the same 2D workload on the explicit solver
        _case("2d_rk3", "plume2d", 128, 1, 192, 2, 10, solver="rk3"),
        # a small 3D run with one particle class and the sub-grid model
        _case("3d_small_les", "plume3d", 49, 45, 41, 1, 5, les=True),
        # an ordinary 3D run
        _case("3d_mid", "plume3d", 128, 128, 96, 3, 4),
        # an ordinary 3D run with mixed-precision fluxes, odd sizes
        _case("3d_mid_mixed", "plume3d", 131, 117, 101, 2, 4, precision="mixed"),
        # five classes over topography with immersed boundaries
        _case("3d_hills", "hills3d", 128, 128, 96, 5, 3),
        # an ordinary 3D run on the explicit solver
        _case("3d_rk3", "plume3d", 128, 128, 96, 3, 4, solver="rk3"),
        # a large explicit run with mixed-precision fluxes
        _case("3d_rk3_large_mixed", "plume3d", 224, 208, 161, 3, 3, solver="rk3", precision="mixed"),
        # an ensemble of independent 2D runs in one batch
        _case("ensemble2d_24", "plume2d", 0, 0, 0, 2, 2, members=24),
        # the benchmark's 3D workload, the largest
        _case("3d_large", "plume3d", 256, 256, 192, 3, 4),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: each family as often as listed."""
    family = rng.choice(["2d", "2d", "2d", "2drk3", "3d", "3d", "3d", "3d", "3drk3", "3drk3", "hills", "ensemble"])
    mixed = "mixed" if rng.random() < 0.25 else "fp64"
    if family in ("2d", "2drk3"):
        nx, nz = _logint(rng, 20, 256), _logint(rng, 30, 384)
        semi = family == "2d"
        return _case(None, "plume2d", nx, 1, nz, rng.choice([1, 2, 2, 3]), rng.randint(2, 10),
                     solver="semi" if semi else "rk3", precision=mixed, les=semi and rng.random() < 0.35)
    if family == "ensemble":
        return _case(None, "plume2d", 0, 0, 0, 2, rng.randint(1, 3), precision=mixed, members=_logint(rng, 4, 24),
                     grid_seed=rng.randint(1, 10 ** 6))
    if family == "hills":
        nx = _logint(rng, 64, 128)
        return _case(None, "hills3d", nx, nx + rng.randint(-6, 0), _logint(rng, 60, 96), 5, rng.randint(2, 3),
                     precision=mixed)
    cells = math.exp(rng.uniform(math.log(4.0e4), math.log(5.0e6)))
    base = (cells / 0.75) ** (1.0 / 3.0)
    nx = max(24, int(base * rng.uniform(0.85, 1.15)))
    ny = max(24, int(base * rng.uniform(0.85, 1.15)))
    nz = max(24, int(cells / (nx * ny)))
    semi = family == "3d"
    return _case(None, "plume3d", nx, ny, nz, rng.choice([1, 2, 3, 3]), rng.randint(2, 4),
                 solver="semi" if semi else "rk3", precision=mixed, les=semi and rng.random() < 0.35)


def _deck(case, seed):
    """The case's deck with the vent's velocity, temperature and volume
    fractions drawn from the seed."""
    rng = random.Random(1000003 * (seed + 1))
    ns = case["nsolid"]
    dia = DIAMETERS[ns]
    rk3 = case["solver"] == "rk3"
    t_gas = rng.uniform(950.0, 1150.0)
    scale = rng.uniform(0.85, 1.15)
    if case["deck"] == "plume2d":
        d = (configs.plume_2d_rk3 if rk3 else configs.plume_2d)(
            nx=case["nx"], nz=case["nz"], diameters=dia, density=DENSITY, t_gas=t_gas,
            w_gas=rng.uniform(80.0, 120.0), ep_solid=tuple([0.02 / ns * scale] * ns))
    elif case["deck"] == "plume3d":
        d = (configs.plume_3d_rk3 if rk3 else configs.plume_3d)(
            nx=case["nx"], ny=case["ny"], nz=case["nz"], diameters=dia, density=DENSITY, t_gas=t_gas,
            w_gas=rng.uniform(120.0, 160.0), ep_solid=tuple([0.02 / ns * scale] * ns))
    else:
        d = configs.plume_3d_hills(
            nx=case["nx"], ny=case["ny"], nz=case["nz"], diameters=dia, density=DENSITY, t_gas=t_gas,
            w_gas=rng.uniform(100.0, 130.0), ep_total=0.03 * scale,
            dem_dir=os.path.join(tempfile.gettempdir(), f"pdac_b200_dem_{os.getuid()}"))
    if case["les"]:
        d.set("model", iturb=1, modturbo=1)
    return d


def _members(case, seed):
    """The ensemble's decks: grids from the case, vents from the seed."""
    decks = []
    for m in range(case["members"]):
        grid = ensemble.member_params(m, case["grid_seed"])
        vent = ensemble.member_params(m, seed)
        decks.append(configs.plume_2d(**{**vent, "nx": grid["nx"], "nz": grid["nz"]}))
    return decks


def _pinned(sizes):
    """Pinned arrays for the states of several runs: each state array of all
    runs in one piece, and every run's own part of them."""
    whole, parts = {}, [{} for _ in sizes]
    for k in sizes[0]:
        whole[k] = torch.empty(sum(s[k] for s in sizes), dtype=torch.float64, pin_memory=True).numpy()
        at = 0
        for part, s in zip(parts, sizes):
            part[k] = whole[k][at:at + s[k]]
            at += s[k]
    return whole, parts


def _download(engine, host):
    """The whole state into the host's own arrays."""
    view = abi.make_state_view(host)
    st = engine.L.pdac_gpu_download_state(engine.h, view)
    if st != 0:
        raise PdacError(st, "download_state")


def prepare(case, seed):
    """The device-resident run (or the ensemble's members and their batch),
    a few steps in, the host's state arrays that the burst starts from and
    the ones it is read back into."""
    prec = abi.PREC_MIXED if case["precision"] == "mixed" else abi.PREC_FP64
    cases = [Case(d, precision=prec) for d in (_members(case, seed) if case["members"] else [_deck(case, seed)])]
    sizes = [{k: v.size for k, v in c.state.items()} for c in cases]
    _, hosts = _pinned(sizes)
    result, outs = _pinned(sizes)
    engines = []
    for c, host in zip(cases, hosts):
        for k, v in c.state.items():
            host[k][:] = v
        c.state = None  # the host's copy from here on is the pinned one
        e = Engine(c, upload=False)
        e.upload(host)
        engines.append(e)
    batch = ensemble.Batch(engines) if case["members"] else None
    for _ in range(WARM_STEPS):
        batch.step() if batch else engines[0].step()
    for e, host in zip(engines, hosts):
        _download(e, host)
    return dict(batch=batch, engines=engines, hosts=hosts, outs=outs, result=result, steps=case["steps"])


def run(state):
    """One burst: the host's state up, K steps, the whole state down.
    Returns every state array as the host holds it (an ensemble's members one
    after the other)."""
    engines, batch = state["engines"], state["batch"]
    for e, host in zip(engines, state["hosts"]):
        e.upload(host)
    for s in range(state["steps"]):
        sweep = WARM_STEPS + 1 + s
        if batch:
            batch.step(sweep)
        else:
            engines[0].step(sweep)
    for e, out in zip(engines, state["outs"]):
        _download(e, out)
    return state["result"]


def _cells(case):
    """Cells of the case's domains."""
    if case["members"]:
        grids = [ensemble.member_params(m, case["grid_seed"]) for m in range(case["members"])]
        return sum(g["nx"] * g["nz"] for g in grids)
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    """What the steps cannot do without: the state read and written once per
    step, and per cell and step the face fluxes of every conserved quantity
    of every phase (upwind, gradients, limiter: ~40 operations per face), the
    interphase terms and one solution of the coupled momentum system per face
    (one outer sweep)."""
    d3 = case["deck"] != "plume2d"
    d, ns, ng = (3 if d3 else 2), case["nsolid"], 2
    ph = 1 + ns
    doubles = 8 + ns * 3 - 1 + d * ph + 2 * ng
    stages = 3 if case["solver"] == "rk3" else 1
    per_face = 40 * (2 * ph + d * ph + ng)
    flops = stages * d * per_face + d * (2 * ph ** 3 // 3 + 4 * ph * ph) + 200 * ph
    n = _cells(case) * case["steps"]
    return {"bytes": n * 2 * 8 * doubles, "flops": n * flops}


def exact(case, seed):
    """None: a step's result is where a Gauss-Seidel iteration in a stated
    cell order stops at a stated tolerance, so it has no value of its own in
    another arithmetic; the steps already run in 64 bits (the mixed mode's
    fluxes are FP32 by its definition)."""
    return None
