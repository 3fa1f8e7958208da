"""Every form of the explicit solver's gas-enthalpy wavefront against a launch
per hyperplane, bit for bit, with the form that ran asserted.

Tiles hold 16 x 4 columns (j, k) in 3D, in 2D all of them (up to 256) or 64.
The meshes end inside and at the edge of a tile and have rows shorter than a
tile's skew; the last ones have more columns than the device finds threads for,
which refuses tiles and by itself takes one launch over all hyperplanes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LAUNCHES, PLANES, TILES, TILES_64 = 1, 2, 3, 4
MESHES = [(9, 35, 23), (7, 68, 36), (6, 18, 18), (12, 130, 70), (5, 2060), (9, 1030), (23, 258), (40, 67),
          (6, 262, 243), (5, 640, 620)]


def _case(mesh):
    from pdac_b200 import configs
    from pdac_b200.setup_state import Case
    if len(mesh) == 2:
        return Case(configs.plume_2d_rk3(nx=mesh[0], nz=mesh[1], vent_radius=20.0))
    nx, ny, nz = mesh
    return Case(configs.plume_3d_rk3(nx=nx, ny=ny, nz=nz, vent_cells=2))


def _tiles(mesh, form):
    """The columns of a tile and the number of tiles; None: refused."""
    if len(mesh) == 3:
        if form == TILES_64:
            return None
        m = -(-(mesh[1] - 2) // 16) * -(-(mesh[2] - 2) // 4)
        return (16, 4, m) if m * 64 < 57000 else None
    nk = mesh[1] - 2
    if form == TILES and nk <= 256:
        return (1, -(-nk // 32) * 32, 1)
    return (1, 64, -(-nk // 64))


@pytest.mark.parametrize("mesh", MESHES)
def test_forms_give_the_bits_of_a_launch_per_hyperplane(mesh):
    from pdac_b200.engine import Engine, PdacError
    case = _case(mesh)
    want = None
    for form in (LAUNCHES, PLANES, TILES, TILES_64, 0):
        e = Engine(case)
        lay = None
        if form in (TILES, TILES_64):
            lay = _tiles(mesh, form)
            if lay is None:
                with pytest.raises(PdacError):
                    e.set_forms(wave=form)
                e.close()
                continue
        if form:
            e.set_forms(wave=form)
        else:
            lay = _tiles(mesh, TILES)
        f = e.forms()
        if form == LAUNCHES:
            assert f["wave_tiles"] == f["wave_blocks"] == 0
        elif lay is None:
            assert f["wave_tiles"] == 0 and f["wave_blocks"] > 0
        else:
            assert (f["wave_tj"], f["wave_tk"], f["wave_tiles"], f["wave_blocks"]) == lay + (0,)
        for sweep in (1, 2):
            e.step(sweep)
        got = e.download()
        e.close()
        if form == LAUNCHES:
            want = got
        for name in want:
            assert np.array_equal(got[name], want[name]), f"form {form}: {name}"
