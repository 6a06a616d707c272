"""Grouping of the PT2 records: determinants reached from hundreds of others (runs of records longer
than a warp's 32), few records, and determinants that share a key (the keys are short for few records,
so that some do in every case)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nu,nd,eps_var,eps", [(4, 1, 1, 2e-1, 1e-9), (6, 2, 2, 1e-2, 1e-10),
                                                 (9, 4, 4, 3e-4, 1e-12), (10, 5, 4, 1e-3, 1e-12),
                                                 (16, 2, 2, 1e-4, 1e-12)])
def test_long_runs(oracle_mod, tmp_path, n, nu, nd, eps_var, eps):
    """Counts equal the oracle's and the deterministic sums agree to 1e-13 (fewer than 1e5 terms below
    1e-3 in FP64).  A target error below 0 runs every batch: in an exhausted space the uncertainty that
    stops a stage is rounding noise around 0."""
    import shci_gb300
    from shci_gb300 import synthetic
    path = str(tmp_path / "FCIDUMP")
    h, g = synthetic.integrals(n, 5 + n)
    synthetic.write_fcidump(path, h, g, nu + nd)
    o = oracle_mod.Oracle(path, nu, nd)
    o.run_all_variations([eps_var], [], 5e-5)
    up, dn, coefs = o.dets()
    c = shci_gb300.Context()
    c.load_fcidump(path, nu, nd)
    c.build_queues()
    c.set_dets(up, dn, coefs)
    for nb in (1, 3):
        v, _, m = c.pt2_dtm(o.energy_var, eps, nb)
        vo, _, mo = o.pt_dtm(eps, nb)
        assert m == mo and abs(v - vo) < 1e-13
        v, _, m, b = c.pt2_psto(o.energy_var, 10 * eps, eps, nb, -1.0, 0.0)
        vo, _, mo, bo = o.pt_psto(10 * eps, eps, nb, -1.0, 0.0)
        assert (m, b) == (mo, bo) and abs(v - vo) < 1e-13
    c.close()
