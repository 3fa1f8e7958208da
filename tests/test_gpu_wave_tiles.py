"""The explicit solver's gas-enthalpy wavefront over its tile layouts, against
the oracle.

The columns (j, k) are dealt out to tiles: one tile for a 2D mesh of up to 256
columns, several beyond that and in 3D (16 x 4 columns each); in a batch,
where blocks that wait for one another are not allowed, a mesh of several
tiles takes one launch per hyperplane. The meshes end inside and at the edge
of a tile, have fewer columns than one, and rows shorter than a tile's skew.
Engine and oracle compute the same bits here while no cell fails the caloric
inversion; the bound is the 1e-9 of the path's other parity tests.
"""
import numpy as np
import pytest

import pyoracle
from helpers import compare_state

pytestmark = pytest.mark.gpu

FIELDS = ("p", "ep", "rog", "rgp", "tg", "sieg", "cg", "ug", "wg", "rlk", "ts", "sies", "us", "ws", "ygc")
MESHES = [(5, 6), (7, 258), (9, 259), (6, 34), (20, 33), ((5, 5, 5),), ((6, 18, 6),), ((9, 19, 7),), ((12, 37, 15),),
          ((5, 35, 23),), ((21, 16, 10),)]


def _case(mesh):
    from pdac_b200 import configs
    from pdac_b200.setup_state import Case
    if len(mesh) == 2:
        return Case(configs.plume_2d_rk3(nx=mesh[0], nz=mesh[1], vent_radius=20.0))
    nx, ny, nz = mesh[0]
    return Case(configs.plume_3d_rk3(nx=nx, ny=ny, nz=nz, vent_cells=2))


@pytest.mark.parametrize("mesh", MESHES)
def test_wavefront_tiles_match_the_oracle(mesh):
    from pdac_b200 import ensemble
    from pdac_b200.engine import Engine
    case = _case(mesh)
    ora, alone, member = pyoracle.Oracle(case), Engine(case), Engine(case)
    batch = ensemble.Batch([member])
    for sweep in (1, 2, 3):
        ora.step(sweep)
        alone.step(sweep)
        batch.step(sweep)
    want, got, inb = ora.get_state(), alone.download(), member.download()
    errs, bad = compare_state(got, want, FIELDS + (("vg", "vs") if case.is3d else ()), 1e-9, case.nsolid, case.ncell)
    assert not bad, bad
    for name in got:
        assert np.array_equal(got[name], inb[name]), name
    batch.close()
    alone.close()
    member.close()


def test_several_columns_per_thread():
    """A mesh of more columns than the device holds threads for: each thread
    takes several in turn; same bits as a launch per hyperplane."""
    from pdac_b200 import configs, ensemble
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    case = Case(configs.plume_3d_rk3(nx=7, ny=262, nz=243, vent_cells=3))
    alone, member = Engine(case), Engine(case)
    batch = ensemble.Batch([member])
    for sweep in (1, 2):
        alone.step(sweep)
        batch.step(sweep)
    got, inb = alone.download(), member.download()
    for name in got:
        assert np.array_equal(got[name], inb[name]), name
    batch.close()
    alone.close()
    member.close()
