"""The corrector's face records: a context without them gathers the same terms,
bit for bit, and no allocation of the library fails because of them.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _case(kind, ns, **mesh):
    from pdac_b200 import configs
    from pdac_b200.setup_state import Case
    kw = dict(diameters=tuple(np.geomspace(30.0, 1000.0, ns)) if ns > 1 else (100.0,), ep_solid=tuple([0.02 / ns] * ns))
    if kind == "2d":
        return Case(configs.plume_2d(**{"nx": 37, "nz": 45, **mesh}, **kw))
    return Case(configs.plume_3d(**{"nx": 21, "ny": 18, "nz": 17, **mesh}, **kw))


def _same(a, b, what=""):
    got, want = a.download(), b.download()
    for name in want:
        assert np.array_equal(got[name], want[name]), f"{what} {name}"


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("kind,ns", [("2d", 1), ("2d", 2), ("2d", 3), ("2d", 5), ("3d", 1), ("3d", 2), ("3d", 3), ("3d", 5)])
def test_same_bits_without_records(kind, ns, batch):
    from pdac_b200.engine import Engine
    from pdac_b200.ensemble import Batch
    case = _case(kind, ns)
    recs, none = Engine(case), Engine(case)
    none.set_forms(no_records=1)
    assert recs.forms()["records"] == 1 and none.forms()["records"] == 0
    b = Batch([none]) if batch else None
    for sweep in (1, 2, 3):
        nit = b.step(sweep)[0] if batch else none.step(sweep)
        assert recs.step(sweep) == nit
        _same(none, recs, f"step {sweep}")
        if sweep == 2:  # taken and given back between two steps: graphs are built again
            none.set_forms(no_records=0)
            recs.set_forms(no_records=1)
            assert none.forms()["records"] == 1 and recs.forms()["records"] == 0
    if batch:
        b.close()
    recs.close()
    none.close()


def test_a_context_that_fits_without_records_is_created(tmp_path):
    """With the device filled up to half the records' size below what a second
    context takes without them, the second context is created, the first one's
    records make room for it, and both go on with the same results; neither
    has room for records then.  The autotuner's copy of the state likewise."""
    import torch
    from pdac_b200.engine import Engine
    case = _case("3d", 5, nx=64, ny=60, nz=56)
    # 84 doubles a cell: 21 interphase terms and 6 momenta, padded to pairs, per axis
    rec_bytes = 84 * 8 * case.ncell
    free = lambda: torch.cuda.mem_get_info()[0]
    ref = Engine(case)
    nit = [ref.step(s) for s in (1, 2)]
    first = Engine(case)  # once for the kernels' own memory on the device
    first.step(1)
    before = free()
    second = Engine(case)
    takes = before - free() - rec_bytes  # what a context takes without records
    assert second.forms()["records"] == 1 and takes > rec_bytes
    second.close()
    ref.set_forms(no_records=1)
    fill = torch.empty(free() - (takes - rec_bytes // 2), dtype=torch.uint8, device="cuda")
    try:
        second = Engine(case)
        assert first.forms()["records"] == second.forms()["records"] == 0
        assert [first.step(2), second.step(1), second.step(2)] == [nit[1], nit[0], nit[1]]
        _same(first, ref)
        _same(second, ref)
        second.close()
    finally:
        del fill
        torch.cuda.empty_cache()
    # the autotuner's copy takes the fields' size again
    first.set_forms(no_records=0)
    assert first.forms()["records"] == 1
    arena = sum(8 * first.get(n).size for n in ARENA_SAMPLE)
    assert arena < takes
    fill = torch.empty(free() - (takes - rec_bytes // 2), dtype=torch.uint8, device="cuda")
    try:
        cache = str(tmp_path / "tune.txt")
        shapes = first.autotune(cache)
        assert shapes["coop_cells_per_block"] in (64, 256, 1024, 4096)
        _same(first, ref)
    finally:
        del fill
        torch.cuda.empty_cache()
    assert first.step(3) == ref.step(3)
    _same(first, ref)
    first.close()
    ref.close()


def test_records_are_taken_back_from_a_context_that_another_thread_steps():
    """The allocation waits for the running iter; the steps around it have the
    bits of a context stepped alone."""
    import threading

    import torch
    from pdac_b200.engine import Engine
    case = _case("3d", 5, nx=64, ny=60, nz=56)
    steps = 12
    alone = Engine(case)
    nit = [alone.step(s) for s in range(1, steps + 1)]
    rec_bytes = 84 * 8 * case.ncell
    free = lambda: torch.cuda.mem_get_info()[0]
    first = Engine(case)
    first.step(1)
    before = free()
    second = Engine(case)
    takes = before - free() - rec_bytes
    second.close()
    alone.set_forms(no_records=1)
    fill = torch.empty(free() - (takes - rec_bytes // 2), dtype=torch.uint8, device="cuda")
    got, go = [], threading.Event()

    def work():
        for s in range(2, steps + 1):
            got.append(first.step(s))
            go.set()

    t = threading.Thread(target=work)
    try:
        assert first.forms()["records"] == 1
        t.start()
        go.wait()
        second = Engine(case)
        t.join()
        assert first.forms()["records"] == 0 and second.step(1) == nit[0]
        second.close()
    finally:
        t.join()
        del fill
        torch.cuda.empty_cache()
    assert got == nit[1:]
    _same(first, alone)
    first.close()
    alone.close()


ARENA_SAMPLE = ("p", "mf", "vis", "appu", "appv", "appw")
