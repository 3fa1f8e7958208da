"""2D meshes through every form of the sweep loop, for every phase count with
kernels of its own and one without: cluster, cooperative grid, graph of launches
(alone and as a member of a batch) and the host loop, bit for bit, with the form
that ran asserted.  A 3D mesh takes the graph, which a small batch no longer
shows for 2D.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CLUSTER, GRID, GRAPH, HOST = 1, 2, 3, 4
MESHES = [("2d", (13, 33)), ("2d", (97, 61)), ("3d", (14, 13, 12))]


def _case(kind, mesh, ns):
    from pdac_b200 import configs
    from pdac_b200.setup_state import Case
    kw = dict(diameters=tuple(np.geomspace(30.0, 1000.0, ns)) if ns > 1 else (100.0,), ep_solid=tuple([0.02 / ns] * ns))
    if kind == "2d":
        return Case(configs.plume_2d(nx=mesh[0], nz=mesh[1], vent_radius=20.0, **kw))
    return Case(configs.plume_3d(nx=mesh[0], ny=mesh[1], nz=mesh[2], vent_cells=2, **kw))


@pytest.mark.parametrize("ns", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("kind,mesh", MESHES)
def test_forms_agree(kind, mesh, ns):
    from pdac_b200.engine import Engine, PdacError
    from pdac_b200.ensemble import Batch
    case = _case(kind, mesh, ns)
    host = Engine(case)
    host.reset_stats(True)
    engines = {HOST: host}
    for form in (CLUSTER, GRID, GRAPH):
        e = Engine(case)
        if form == CLUSTER and kind == "3d":
            with pytest.raises(PdacError):
                e.set_forms(sweep=form)
            e.close()
            continue
        e.set_forms(sweep=form)
        # a form stands through new launch shapes; the grid in few blocks
        e.set_tuning(dict(tile_shape=0, tile_kchunk=2, inner_grid=37, test_grid=5, coop_cells_per_block=300))
        engines[form] = e
    auto = Engine(case)
    members = {form: Engine(case) for form in (GRID, GRAPH)}  # both take the graph there
    for form, e in members.items():
        e.set_forms(sweep=form)
    batch = Batch(list(members.values()))
    for sweep in (1, 2, 3):
        nit = host.step(sweep)
        want = host.download()
        assert batch.step(sweep) == [nit, nit]
        for form, e in engines.items():
            if e is not host:
                assert e.step(sweep) == nit, form
            assert e.forms()["sweep"] == form
        assert auto.step(sweep) == nit and auto.forms()["sweep"] == (CLUSTER if kind == "2d" else GRID)
        for e in [auto, *engines.values(), *members.values()]:
            got = e.download()
            for name in want:
                assert np.array_equal(got[name], want[name]), f"step {sweep}: {name}"
    batch.close()
    for e in [auto, *engines.values(), *members.values()]:
        e.close()
