"""Host threads that step explicit contexts of their own: one cooperative grid
at a time is in flight, a thread that finds it taken does not wait but runs its
wavefront in separate launches; same results as alone.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_step_their_own_explicit_contexts():
    from pdac_b200 import configs
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    steps = 6
    case = Case(configs.plume_3d_rk3(nx=40, ny=37, nz=33))
    alone = Engine(case)
    for s in range(1, steps + 1):
        alone.step(s)
    want, tiled = alone.download(), alone.stats()["launches"]
    alone.close()
    engines = [Engine(case) for _ in range(4)]
    start = threading.Barrier(len(engines))

    def work(e):
        start.wait()
        for s in range(1, steps + 1):
            e.step(s)

    th = [threading.Thread(target=work, args=(e,)) for e in engines]
    for t in th:
        t.start()
    for t in th:
        t.join()
    # some step of some thread found the grid of another in flight
    assert max(e.stats()["launches"] for e in engines) > tiled
    for e in engines:
        got = e.download()
        for name in want:
            assert np.array_equal(got[name], want[name]), name
        e.close()
