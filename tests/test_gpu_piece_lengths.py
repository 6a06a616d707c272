"""PT2 and selection with windows cut into pieces of every kind of length: shorter than a warp's
rounds, around the shortest and the longest that the library takes by itself (256 and 16,384 entries)
and in between, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def system(oracle_mod, tmp_path_factory):
    from shci_gb300 import synthetic
    path = str(tmp_path_factory.mktemp("pieces") / "FCIDUMP")
    h, g = synthetic.integrals(30, 41)
    synthetic.write_fcidump(path, h, g, 11)
    o = oracle_mod.Oracle(path, 6, 5)
    o.run_all_variations([4e-3], [], 5e-5)
    ref = {"dets": o.dets(), "e": o.energy_var}
    for nb in (1, 13):
        ref["dtm", nb] = o.pt_dtm(3e-7, nb)
    ref["psto"] = o.pt_psto(3e-6, 3e-7, 4, 0.0, 0.0)
    o.run_variation_step(1e-3, False, 5e-5)
    ref["selected"] = o.dets()[:2]
    return path, ref


@pytest.mark.parametrize("piece", [33, 255, 257, 1000, 16383, 16384, 1 << 20])
def test_piece_lengths(monkeypatch, system, piece):
    """Counts are equal and sums of fewer than 1e6 terms below 1e-3 within 1e-13; the selected list is
    the same, in order."""
    import shci_gb300
    path, ref = system
    monkeypatch.setenv("SHCI_WALK_PIECE", str(piece))
    c = shci_gb300.Context()
    c.load_fcidump(path, 6, 5)
    c.build_queues()
    c.set_dets(*ref["dets"])
    up, dn, co = ref["dets"]
    off = c.find_connected(up[:1], dn[:1], 1e100, 3e-7 / abs(co[0]))[0]
    assert off[-1] > 16384  # the first det's window has several pieces of up to that length
    for nb in (1, 13):
        v, _, m = c.pt2_dtm(ref["e"], 3e-7, nb)
        vo, _, mo = ref["dtm", nb]
        assert m == mo and abs(v - vo) < 1e-13
    v, _, m, b = c.pt2_psto(ref["e"], 3e-6, 3e-7, 4, 0.0, 0.0)
    vo, _, mo, bo = ref["psto"]
    assert (m, b) == (mo, bo) and abs(v - vo) < 1e-13
    # a walk over all of a det's window, second rejection off and on
    c.set_dets(up, dn, co)
    c.select(1e-3)
    got = c.dets()[:2]
    assert np.array_equal(got[0], ref["selected"][0]) and np.array_equal(got[1], ref["selected"][1])
    c.set_dets(up, dn, co)
    c.set_second_rejection(True)
    c.select(1e-3)
    some = c.n_dets(), c.eps_tried()
    monkeypatch.delenv("SHCI_WALK_PIECE")
    c.set_dets(up, dn, co)
    c.select(1e-3)
    assert c.n_dets() == some[0] and np.array_equal(c.eps_tried(), some[1])
    c.close()
