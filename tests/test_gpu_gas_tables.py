"""The gas tables of a run: seven gases, the three specific-heat modes, and a
restart that brings other gases.

The specific heats (hcapgs.f:33-85), molar weights and viscosity factors
(visc.f:37-148) of the run's gases are tables by their order in the run, made
at create and again when a restart file names other gases.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _restart(tmp_path, nx, nz, gas):
    """A restart file of a plume whose vent gas is `gas`, three steps in."""
    from pdac_b200 import configs
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    d = configs.small_2d(nx=nx, nz=nz)
    d.set("inlet", vent_H2O=0.0, **{f"vent_{gas}": 1.0})
    e = Engine(Case(d))
    for sweep in (1, 2, 3):
        e.step(sweep)
    path = str(tmp_path / f"pdac_{gas}.res")
    e.write_restart(path, 0.03, 1)
    e.close()
    return path


def test_a_batch_member_reads_a_restart_with_other_gases(tmp_path):
    """The member's steps are in the batch's captured graph; after the restart
    they give the bits of a context stepped alone."""
    from pdac_b200 import configs
    from pdac_b200.engine import Engine
    from pdac_b200.ensemble import Batch
    from pdac_b200.setup_state import Case
    path = _restart(tmp_path, 14, 19, "CO2")
    case, other = Case(configs.small_2d(nx=14, nz=19)), Case(configs.small_2d())
    alone, member, rest = Engine(case), Engine(case), Engine(other)
    batch = Batch([member, rest])
    for sweep in (1, 2):
        assert batch.step(sweep)[0] == alone.step(sweep)
    for e in (alone, member):
        assert e.read_restart(path) == (0.03, 1)
    for sweep in (4, 5):
        assert batch.step(sweep)[0] == alone.step(sweep)
        got, want = member.download(), alone.download()
        for name in want:
            assert np.array_equal(got[name], want[name]), f"step {sweep}: {name}"
    # and alone again, in the launches of iter's graph
    batch.close()
    member.reset_stats(False)
    assert member.step(6) == alone.step(6)
    for e in (alone, member, rest):
        e.close()
