"""PT2 emission in pieces of a source's window: windows of several pieces (more than 4,096 entries),
more than 32 orbitals, one and several batches, an empty beta string."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nu,nd,eps_var,eps", [(34, 4, 3, 3e-3, 1e-7), (21, 3, 0, 1e-3, 1e-8),
                                                 (18, 6, 5, 3e-3, 1e-7)])
def test_pt2_matches_oracle(oracle_mod, tmp_path, n, nu, nd, eps_var, eps):
    """Same dets, batches and thresholds as the oracle: counts equal, sums to 1e-13 (sums of fewer
    than 1e6 terms below 1e-3 in FP64)."""
    import shci_gb300
    from shci_gb300 import synthetic
    path = str(tmp_path / "FCIDUMP")
    h, g = synthetic.integrals(n, 11 + n)
    synthetic.write_fcidump(path, h, g, nu + nd)
    o = oracle_mod.Oracle(path, nu, nd)
    o.run_all_variations([eps_var], [], 5e-5)
    up, dn, coefs = o.dets()
    c = shci_gb300.Context()
    c.load_fcidump(path, nu, nd)
    c.build_queues()
    c.set_dets(up, dn, coefs)
    # the first det's window is longer than a piece where the system is large enough for it
    off = c.find_connected(up[:1], dn[:1], 1e100, eps / abs(coefs[0]))[0]
    assert nd == 0 or off[-1] > 4096
    for nb in (1, 2, 13):
        v, _, m = c.pt2_dtm(o.energy_var, eps, nb)
        vo, _, mo = o.pt_dtm(eps, nb)
        assert m == mo and abs(v - vo) < 1e-13
        v, _, m, b = c.pt2_psto(o.energy_var, 10 * eps, eps, nb, 0.0, 0.0)
        vo, _, mo, bo = o.pt_psto(10 * eps, eps, nb, 0.0, 0.0)
        assert (m, b) == (mo, bo) and abs(v - vo) < 1e-13
    c.close()
