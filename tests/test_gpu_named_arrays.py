"""The arrays that pdac_gpu_get_array reads by name keep what the call they
belong to left in them.

tilde writes the momentum fluxes ("mf" in 3D, "ugfe" ... "wsft" in 2D), the
stresses ("vis", 3D) and the interphase terms; the calls after it in a time
step only read them.  So after iter, ygas, htilde and ftem, and after a whole
step, they hold the same bits as after tilde, and zero in the cells tilde does
not visit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TILDE_2D = ("ugfe", "ugft", "wgfe", "wgft", "usfe", "usft", "wsfe", "wsft", "appu", "appw", "rug", "rwg", "rus", "rws")
TILDE_3D = ("mf", "vis", "appu", "appv", "appw", "rug", "rvg", "rwg", "rus", "rvs", "rws")


def _case(kind, ns):
    from pdac_b200 import configs
    from pdac_b200.setup_state import Case
    kw = dict(diameters=tuple(np.geomspace(30.0, 1000.0, ns)), ep_solid=tuple([0.02 / ns] * ns))
    return Case(configs.small_2d(**kw) if kind == "2d" else configs.small_3d(**kw))


@pytest.mark.parametrize("kind,ns", [("2d", 2), ("2d", 5), ("3d", 1), ("3d", 2), ("3d", 3), ("3d", 4), ("3d", 5)])
def test_tilde_arrays_outlive_the_corrector(kind, ns):
    from pdac_b200.engine import Engine
    case = _case(kind, ns)
    names = TILDE_2D if kind == "2d" else TILDE_3D
    e, whole = Engine(case), Engine(case)
    dt = case.deck["dt"]
    fluid = (case.flag & 1) == 1
    for sweep in (1, 2):
        whole.step(sweep)
        e.boundary(sweep)
        e.fieldn()
        e.tilde(dt)
        want = {n: e.get(n) for n in names}
        if kind == "3d":
            assert not want["vis"].reshape(-1, case.ncell)[:, ~fluid].any()
        for call in (lambda: e.iter(dt), lambda: e.ygas(dt), lambda: e.htilde(dt), lambda: e.ftem(dt)):
            call()
            for n in names:
                assert np.array_equal(e.get(n), want[n]), f"step {sweep}: {n}"
        for n in names:
            assert np.array_equal(whole.get(n), want[n]), f"step {sweep}: {n} after a whole step"
    e.close()
    whole.close()
