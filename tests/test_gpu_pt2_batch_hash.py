"""Batch membership from the low bits of the hash (powers of two up to 128) and from all of it: each
batch of the pseudo-stochastic and deterministic stages against the oracle's."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nu,nd", [(12, 3, 2), (34, 2, 2), (64, 2, 1)])
@pytest.mark.parametrize("nb", [2, 3, 16, 64, 96, 128, 256])
def test_batches_match_oracle(oracle_mod, tmp_path, n, nu, nd, nb):
    """Equal numbers of dets over the batches; sums to 1e-13 (fewer than 1e6 terms below 1e-3)."""
    import shci_gb300
    from shci_gb300 import synthetic
    path = str(tmp_path / "FCIDUMP")
    h, g = synthetic.integrals(n, 3 + n)
    synthetic.write_fcidump(path, h, g, nu + nd)
    o = oracle_mod.Oracle(path, nu, nd)
    o.run_all_variations([1e-2], [], 5e-5)
    up, dn, coefs = o.dets()
    c = shci_gb300.Context()
    c.load_fcidump(path, nu, nd)
    c.build_queues()
    c.set_dets(up, dn, coefs)
    v, _, m = c.pt2_dtm(o.energy_var, 1e-6, nb)
    vo, _, mo = o.pt_dtm(1e-6, nb)
    assert m == mo and abs(v - vo) < 1e-13
    v, _, m, b = c.pt2_psto(o.energy_var, 1e-5, 1e-6, nb, -1.0, 0.0)
    vo, _, mo, bo = o.pt_psto(1e-5, 1e-6, nb, -1.0, 0.0)
    c.close()
    assert (m, b) == (mo, bo) and abs(v - vo) < 1e-13
