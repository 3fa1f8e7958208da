"""The gas tables of a run: seven gases, the three specific-heat modes, and a
restart that brings other gases.

The specific heats (hcapgs.f:33-85), molar weights and viscosity factors
(visc.f:37-148) of the run's gases are tables by their order in the run, made
at create and again when a restart file names other gases.
"""
import numpy as np
import pytest

from helpers import STEP_FIELDS, compare_state

pytestmark = pytest.mark.gpu

GAS = ("O2", "N2", "CO2", "H2", "H2O", "Air", "SO2")
AIR = dict(O2=0.2, N2=0.7, Air=0.1)
VENTS = {2: dict(Air=0.3, SO2=0.7), 3: dict(CO2=0.6, H2=0.05, Air=0.35), 7: dict(H2O=0.5, CO2=0.3, SO2=0.1, H2=0.1)}


def _deck(kind, solver, icpc, ngas, compute_mixture=False):
    """A small plume of air (of one, or of three gases for seven) and a vent of
    VENTS; icpc = 0, 1 take specific heats of fixed temperature, 0 fixed values
    for water vapour and air."""
    from pdac_b200 import configs
    d = getattr(configs, f"small_{kind}" + ("_rk3" if solver == "rk3" else ""))()
    atm = AIR if ngas == 7 else dict(Air=1.0)
    vent = VENTS[ngas]
    d.set("model", ngas=ngas, icpc=icpc, compute_mixture=compute_mixture)
    d.set("atmosphere", **{f"atm_{g}": atm.get(g, 0.0) for g in GAS})
    if d["ivent"]:
        d.set("inlet", **{f"vent_{g}": vent.get(g, 0.0) for g in GAS})
    for b in d.blocks:
        b["ygc"] = [vent.get(g, 0.0) for g in GAS]
    return d


@pytest.mark.parametrize("icpc", [0, 1, 2])
@pytest.mark.parametrize("ngas", [2, 3, 7])
@pytest.mark.parametrize("kind,solver", [("2d", "semi"), ("3d", "semi"), ("2d", "rk3"), ("3d", "rk3")])
def test_mixtures_match_the_oracle(kind, solver, ngas, icpc, tmp_path):
    """Steps of every gas at 1e-9 of the oracle (the bound of the path's other
    parity tests); the specific heat a restart derives is the step's own."""
    import pyoracle
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    case = Case(_deck(kind, solver, icpc, ngas))
    assert case.ngas == ngas
    e, ora = Engine(case), pyoracle.Oracle(case)
    fields = STEP_FIELDS + (("vg", "vs") if case.is3d else ())
    for sweep in (1, 2, 3):
        assert e.step(sweep) == ora.step(sweep)
        errs, bad = compare_state(e.download(), ora.get_state(), fields, 1e-9, case.nsolid, case.ncell)
        assert not bad, (sweep, bad)
    for name in ("mug", "kapg"):
        assert np.max(np.abs(e.get(name) - ora.get(name))) <= 1e-9 * np.max(np.abs(ora.get(name))), name
    path = str(tmp_path / "pdac.res")
    e.write_restart(path, 0.03, 1)
    again = Engine(case)
    again.read_restart(path)
    # sum of specific heat by mass fraction, in plain FP64 from the file's own state
    st = again.download()
    n = case.ncell
    want = sum(_hcapg(icpc, case.deck["tref"], st["tg"])[g - 1] * st["ygc"][q * n:(q + 1) * n]
               for q, g in enumerate(case.gas_type))
    assert np.max(np.abs(st["cg"] - want)) <= 1e-13 * np.max(want)
    e.close()
    again.close()


def _hcapg(icpc, tref, tg):
    """hcapgs.f:33-85 for the seven gases."""
    t = np.full_like(tg, tref) if icpc <= 1 else tg
    cp = [2.811e1 - 3.68e-6 * t + 1.746e-5 * t**2 - 1.065e-8 * t**3, 3.115e1 - 1.357e-2 * t + 2.680e-5 * t**2 - 1.168e-8 * t**3,
          1.980e1 + 7.344e-2 * t - 5.602e-5 * t**2 + 1.715e-8 * t**3, 2.714e1 + 9.274e-3 * t - 1.381e-5 * t**2 + 7.645e-9 * t**3,
          3.224e1 + 1.924e-3 * t + 1.055e-5 * t**2 - 3.596e-9 * t**3, 3.0413e1 - 1.059e-2 * t + 2.458e-5 * t**2 - 1.135e-8 * t**3,
          2.385e1 + 6.699e-2 * t - 4.961e-5 * t**2 + 1.328e-8 * t**3]
    cp = [c / (1e-3 * m) for c, m in zip(cp, (32.0, 28.0, 44.0, 2.0, 18.0, 28.96442, 64.0))]
    if icpc == 0:
        cp[4], cp[5] = np.full_like(t, 1810.0), np.full_like(t, 1004.0)
    return cp


@pytest.mark.parametrize("kind", ["2d", "3d"])
@pytest.mark.parametrize("icpc", [0, 2])
def test_mixture_temperature_of_seven_gases(kind, icpc):
    """tm of compute_mixture (derived.f:269-296) from the state, in plain FP64."""
    from pdac_b200.engine import Engine
    from pdac_b200.setup_state import Case
    case = Case(_deck(kind, "semi", icpc, 7, compute_mixture=True))
    e = Engine(case)
    e.step(1)
    e.step(2)
    st, n, tm = e.download(), case.ncell, e.get("tm")
    cg = sum(c[1] * st["ygc"][q * n:(q + 1) * n]
             for q, c in enumerate((g, _hcapg(icpc, case.deck["tref"], st["tg"])[g - 1]) for g in case.gas_type))
    num, den = st["rgp"] * cg * st["tg"], st["rgp"] * cg
    for s in range(case.nsolid):
        w = st["rlk"][s * n:(s + 1) * n] * case.deck["specific_heat"][s]
        num, den = num + w * st["ts"][s * n:(s + 1) * n], den + w
    assert np.max(np.abs(tm - num / den)) <= 1e-12 * np.max(tm)
    e.close()


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
