"""pdac_gpu_stats counts the kernels that ran: tilde of a 3D mesh is the stress
and the momentum-flux pass, each in a launch for the simple cells and one for
the others where there are both, and k_tilde3d."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("muscl,nx,launches", [(1, 12, 5), (0, 12, 3), (1, 5, 5)])
def test_tilde_counts_its_launches(muscl, nx, launches):
    from pdac_b200 import configs
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    case = Case(configs.small_3d(nx=nx, muscl=muscl))
    e = Engine(case)
    e.boundary(1)
    e.fieldn()
    e.reset_stats()
    e.tilde(case.deck["dt"])
    assert e.stats()["launches"] == launches
    e.close()
