"""The 3D flux and stress passes split into simple cells and the rest, against
the oracle.

A simple cell's stencils stay inside the mesh and meet no wall and no
boundary-layer cell; its pass reads plain offsets and no flags. The others go
through the general pass as a list. The meshes have none, one and many simple
cells, rows that end inside a warp, walls inside the mesh (a staircase of
hills) and one to five classes. Bound: the 1e-12 of the path's other explicit
passes.
"""
import numpy as np
import pytest

import pyoracle
from helpers import rel_linf

pytestmark = pytest.mark.gpu

TOL = 1e-12
MESHES = [((5, 5, 5), 2, 0), ((6, 7, 10), 1, 1), ((7, 6, 9), 3, 2), ((35, 9, 11), 2, 3), ((12, 34, 10), 3, 4),
          ((11, 10, 33), 5, 5), ((40, 37, 13), 4, 6)]


def _rough(case, seed):
    """A state with velocities of both signs and gradients everywhere."""
    rng = np.random.default_rng(seed)
    for name in ("ug", "vg", "wg", "us", "vs", "ws"):
        case.state[name][:] += rng.uniform(-20.0, 20.0, case.state[name].size)
    for name in ("rgp", "tg", "sieg", "ep", "p"):
        case.state[name][:] *= rng.uniform(0.98, 1.0, case.state[name].size)
    case.state["rlk"][:] += rng.uniform(0.0, 2.0, case.state["rlk"].size)
    return case


def _case(mesh, ns, seed):
    from pdac_b200 import configs
    from pdac_b200.setup_state import Case
    nx, ny, nz = mesh
    return _rough(Case(configs.plume_3d(nx=nx, ny=ny, nz=nz, vent_cells=2, diameters=tuple(np.geomspace(30, 1000, ns)),
                                        ep_solid=tuple([0.02 / ns] * ns))), seed)


def _check(eng, ora, names, what):
    for name in names:
        a, b = eng.get(name), ora.get("mf3" if name == "mf" else name)
        assert rel_linf(a, b) <= TOL, f"{what}: {name} {rel_linf(a, b):.2e}"


def _passes(case):
    from pdac_b200.engine import Engine
    eng, ora = Engine(case), pyoracle.Oracle(case)
    dt = case.deck["dt"]
    for x in (eng, ora):
        x.boundary(1)
        x.fieldn()
        x.tilde(dt)
    _check(eng, ora, ("mf", "rug", "rvg", "rwg", "rus", "rvs", "rws"), "tilde")
    for x in (eng, ora):
        x.htilde(dt)
    _check(eng, ora, ("rhg", "rhs"), "htilde")
    for x in (eng, ora):
        x.ygas(dt)
    _check(eng, ora, ("ygc",), "ygas")
    eng.close()


@pytest.mark.parametrize("mesh,ns,seed", MESHES)
def test_flux_passes_match_the_oracle(mesh, ns, seed):
    _passes(_case(mesh, ns, seed))


@pytest.mark.parametrize("immb", [0, 1])
def test_flux_passes_over_hills(tmp_path, immb):
    from pdac_b200 import configs
    from pdac_b200.setup_state import Case
    _passes(_rough(Case(configs.small_3d_topo(tmp_path, immb=immb, nx=24, ny=21, nz=19)), 7))
