"""The bounded waits of the gas-enthalpy wavefront: with a limit of one look, a
tile far from the first gives up on its neighbours' pressures, the kernel
returns, the call reports PDAC_ERR_TIMEOUT, and the context is good for the
next call.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [(12, 130, 70), (9, 35, 23), (30, 700)])
def test_a_wait_that_runs_out_is_reported(mesh):
    from pdac_b200 import abi, configs
    from pdac_b200.engine import Engine, PdacError
    from pdac_b200.setup_state import Case
    if len(mesh) == 3:
        case = Case(configs.plume_3d_rk3(nx=mesh[0], ny=mesh[1], nz=mesh[2], vent_cells=2))
    else:
        case = Case(configs.plume_2d_rk3(nx=mesh[0], nz=mesh[1], irand=0))
    e, fresh = Engine(case), Engine(case)
    assert e.forms()["wave_tiles"] > 1
    for _ in range(2):  # the flag is cleared for the next call
        e.set_forms(wave_looks=1)
        e.upload(case.state)
        with pytest.raises(PdacError) as err:
            e.step(1)
        assert err.value.status == abi.PDAC_ERR_TIMEOUT and "wavefront" in str(err.value)
        e.set_forms()
        e.upload(case.state)
        assert e.step(1) == fresh.step(1)
        got, want = e.download(), fresh.download()
        for name in want:
            assert np.array_equal(got[name], want[name]), name
        fresh.upload(case.state)
    e.close()
    fresh.close()
