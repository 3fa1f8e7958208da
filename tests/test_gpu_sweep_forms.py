"""The forms of iter's sweep loop against each other on the GPU.

The sweep loop runs on one thread-block cluster (small 2D meshes), on a
cooperative grid or as a graph of launches; a mesh stepped with profiling on
takes the launches.  Every form runs the same cells in the same colour order,
so after each step the sweep counts, the unconverged cells and every state
array are equal, bit for bit.  The meshes put the active set's last word, the
colours' first cells and the worklists (shorter and longer than one round of
the warps) at odd places; 364 x 361 lies above the cluster's limit and 359 x
363 just below it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MESHES = [
    ("2d", 5, 7, 1, 2), ("2d", 13, 33, 1, 2), ("2d", 31, 65, 2, 3), ("2d", 97, 129, 3, 2), ("2d", 364, 361, 2, 2),
    ("2d", 41, 50, 4, 2), ("2d", 37, 43, 5, 2), ("2d", 359, 363, 1, 2),
    ("3d", (6, 5, 7), None, 1, 2), ("3d", (11, 13, 9), None, 3, 3), ("3d", (33, 31, 35), None, 2, 3),
    ("3d", (17, 16, 15), None, 4, 2), ("3d", (20, 18, 17), None, 5, 2), ("3d", (66, 61, 70), None, 3, 2),
]


def _deck(kind, a, b, ns):
    from pdac_b200 import configs
    dia = tuple(np.geomspace(30.0, 1000.0, ns))
    if kind == "2d":
        return configs.plume_2d(nx=a, nz=b, vent_radius=20.0 if a < 20 else 50.0, diameters=dia,
                                ep_solid=tuple([0.02 / ns] * ns))
    nx, ny, nz = a
    return configs.plume_3d(nx=nx, ny=ny, nz=nz, vent_cells=2 if nx < 30 else 5, diameters=dia,
                            ep_solid=tuple([0.02 / ns] * ns))


@pytest.mark.parametrize("kind,a,b,ns,steps", MESHES)
def test_sweep_loop_forms_agree(kind, a, b, ns, steps):
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    case = Case(_deck(kind, a, b, ns))
    one, launches, grid = Engine(case), Engine(case), Engine(case)
    launches.reset_stats(True)  # profiling: a launch per colour phase
    # the grid with one block per 32 cells in 3D, with few blocks in 2D, and
    # other launch grids
    grid.set_tuning(dict(tile_shape=0, tile_kchunk=2, inner_grid=37, test_grid=5,
                         coop_cells_per_block=32 if kind == "3d" else 4096))
    for sweep in range(1, steps + 1):
        nits = [e.step(sweep) for e in (one, launches, grid)]
        assert nits[0] == nits[1] == nits[2], f"step {sweep}: sweeps {nits}"
        want = launches.download()
        cells = launches.unconverged_cells()
        for e in (one, grid):
            got = e.download()
            for name in want:
                assert np.array_equal(got[name], want[name]), f"step {sweep}: {name}"
            assert np.array_equal(e.unconverged_cells(), cells)
    for e in (one, launches, grid):
        e.close()


@pytest.mark.parametrize("cells_per_block", [300, 4000, 40000])
def test_grids_of_few_blocks_agree(cells_per_block):
    """Worklists of many rounds of a grid's warps, whose expected long and
    short cells alternate, and of a few rounds."""
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    case = Case(_deck("3d", (33, 31, 35), None, 2))
    one, grid = Engine(case), Engine(case)
    grid.set_tuning(dict(tile_shape=0, tile_kchunk=2, inner_grid=37, test_grid=5, coop_cells_per_block=cells_per_block))
    for sweep in (1, 2):
        assert one.step(sweep) == grid.step(sweep)
        got, want = grid.download(), one.download()
        for name in want:
            assert np.array_equal(got[name], want[name]), f"step {sweep}: {name}"
    one.close()
    grid.close()


@pytest.mark.parametrize("kind,a,b,ns", [("2d", 97, 129, 2), ("2d", 23, 31, 5), ("3d", (33, 31, 35), None, 2)])
def test_forms_agree_on_a_loop_that_ends_unconverged(kind, a, b, ns):
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    deck = _deck(kind, a, b, ns)
    deck.set("numeric", maxout=3)
    deck.set("control", cstop=0)
    case = Case(deck)
    one, launches = Engine(case), Engine(case)
    launches.reset_stats(True)
    for sweep in (1, 2):
        assert one.step(sweep) == launches.step(sweep) == 4
        cells = launches.unconverged_cells()
        assert cells.size > 0 and np.array_equal(one.unconverged_cells(), cells)
        got, want = one.download(), launches.download()
        for name in want:
            assert np.array_equal(got[name], want[name]), f"step {sweep}: {name}"
    one.close()
    launches.close()


def test_two_threads_step_their_own_contexts():
    """Two host threads stepping a context each: a cooperative grid of one is
    in flight at a time, the other takes the launches; same results as alone."""
    import threading

    from pdac_b200 import configs
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    case = Case(configs.plume_3d(nx=40, ny=37, nz=33))
    alone = Engine(case)
    nit = [alone.step(s) for s in (1, 2, 3)]
    want = alone.download()
    alone.close()
    engines, got = [Engine(case), Engine(case)], [None, None]

    def work(q):
        got[q] = [engines[q].step(s) for s in (1, 2, 3)]

    th = [threading.Thread(target=work, args=(q,)) for q in (0, 1)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for q in (0, 1):
        assert got[q] == nit
        out = engines[q].download()
        for name in want:
            assert np.array_equal(out[name], want[name]), name
        engines[q].close()
