"""find_connected_dets with every unit of work (one slot of a det, some, 32, all), in one pass and in
several where a budget leaves no room for one, and for systems with no or one electron."""
import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def c_case(oracle_mod):
    o = oracle_mod.Oracle(C_ATOM, 4, 2, "d2h")
    o.run_all_variations([2e-4], [2e-3, 1e-3, 5e-4], 5e-5)
    up, dn, co = o.dets()
    rng = np.random.default_rng(17)
    lo = 10.0 ** rng.uniform(-6, -1.5, len(up))
    hi = np.where(rng.random(len(up)) < 0.5, 1e100, lo * 10.0 ** rng.uniform(-1, 2, len(up)))
    return o, up, dn, lo, hi


def _ctx(budget=0):
    import shci_gb300
    c = shci_gb300.Context(hbm_budget=budget)
    c.load_fcidump(C_ATOM, 4, 2, "d2h")
    c.build_queues()
    return c


@pytest.mark.parametrize("per", [1, 2, 7, 20, 21, 32, 33, 1000])
def test_units_match_oracle(monkeypatch, c_case, per):
    """6 electrons: 21 slots a det."""
    o, up, dn, lo, hi = c_case
    monkeypatch.setenv("SHCI_CONNECTED_SLOTS", str(per))
    idx = np.random.default_rng(per).choice(len(up), 150, replace=False)
    c = _ctx()
    off, cu, cd, nx = c.find_connected(up[idx], dn[idx], hi[idx], lo[idx])
    c.close()
    for k, i in enumerate(idx):
        ou, od, onx = o.find_connected((int(up[i]), int(dn[i])), hi[i], lo[i])
        a, b = int(off[k]), int(off[k + 1])
        assert np.array_equal(cu[a:b], ou) and np.array_equal(cd[a:b], od), k
        assert np.array_equal(nx[a:b], onx.astype(np.uint8)), k


@pytest.mark.parametrize("per", ["1", "32", "64"])
def test_units_of_many_electrons(monkeypatch, per):
    """13 electrons: 91 slots, so that a det has several units of 32 and the last is not full.  All
    slots of a det in one unit are the reference."""
    import shci_gb300
    from shci_gb300 import synthetic
    h, g = synthetic.integrals(22, 5)
    rng = np.random.default_rng(2)
    up = np.array([sum(1 << int(k) for k in rng.choice(22, 7, replace=False)) for _ in range(300)], np.uint64)
    dn = np.array([sum(1 << int(k) for k in rng.choice(22, 6, replace=False)) for _ in range(300)], np.uint64)
    lo = 10.0 ** rng.uniform(-4, 0, 300)
    c = shci_gb300.Context()
    c.set_integrals(h, g, 7, 6, 0x7f, 0x3f)
    c.build_queues()
    monkeypatch.setenv("SHCI_CONNECTED_SLOTS", "1000")
    want = c.find_connected(up, dn, 1e100, lo)
    monkeypatch.setenv("SHCI_CONNECTED_SLOTS", per)
    got = c.find_connected(up, dn, 1e100, lo)
    c.close()
    assert want[0][-1] > 100000
    assert all(np.array_equal(a, b) for a, b in zip(want, got))


def test_passes_within_a_budget(c_case):
    """Inputs and offsets of all dets need about 12 MB with a unit per slot, the lists more; from 16 MB
    of room down to half a megabyte the results are the same."""
    _, up, dn, lo, hi = c_case
    c = _ctx()
    live = c.memory_stats()[0] - c.memory_cached()[0]
    k = np.arange(24000) % len(up)
    args = up[k], dn[k], hi[k], lo[k]
    want = c.find_connected(*args)
    c.close()
    assert len(want[1]) * 17 > 1 << 24
    for room in (1 << 24, 1 << 22, 1 << 20, 1 << 19):
        c = _ctx(live + room)
        got = c.find_connected(*args)
        assert c.memory_stats()[0] <= live + room
        c.close()
        assert all(np.array_equal(a, b) for a, b in zip(want, got)), room


@pytest.mark.parametrize("nu", [0, 1])
def test_no_or_one_electron(monkeypatch, nu):
    """No electron has no slot and no pair, one electron a single slot: its targets are the other
    orbitals with a matrix element."""
    import shci_gb300
    from shci_gb300 import synthetic
    h, g = synthetic.integrals(5, 3)
    for per in ("1", "32"):
        monkeypatch.setenv("SHCI_CONNECTED_SLOTS", per)
        c = shci_gb300.Context()
        c.set_integrals(h, g, nu, 0, nu, 0)
        c.build_queues()
        off, cu, cd, nx = c.find_connected(np.array([nu], np.uint64), np.zeros(1, np.uint64), 1e100, 1e-9)
        c.close()
        assert sorted(int(u) for u in cu) == ([2, 4, 8, 16] if nu else [])
        assert int(off[1]) == len(cu) and np.all(cd == 0) and np.all(nx == 1)
