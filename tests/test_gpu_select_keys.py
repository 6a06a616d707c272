"""Selection's candidate order: ranked keys against the sort by strings, and both against the oracle's
list, over several sources' passes, unequal and empty spins, more than 32 orbitals, with second rejection."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nu,nd,eps", [(4, 1, 1, 1e-4), (9, 3, 0, 1e-4), (12, 5, 2, 1e-4),
                                          (33, 2, 2, 5e-4), (36, 4, 3, 2e-3)])
def test_selection_orders_agree(monkeypatch, oracle_mod, tmp_path, n, nu, nd, eps):
    import shci_gb300
    from shci_gb300 import synthetic
    path = str(tmp_path / "FCIDUMP")
    h, g = synthetic.integrals(n, 23 + n)
    synthetic.write_fcidump(path, h, g, nu + nd)
    for rej in (False, True):
        lists = []
        for keys in ("", "strings"):
            monkeypatch.setenv("SHCI_SELECT_KEYS", keys)
            c = shci_gb300.Context()
            c.load_fcidump(path, nu, nd)
            c.build_queues()
            c.set_second_rejection(rej, 0.2)
            c.run_variation([eps], [10 * eps, 3 * eps], 5e-5)
            lists.append(c.dets()[:2])
            c.close()
        assert np.array_equal(lists[0][0], lists[1][0]) and np.array_equal(lists[0][1], lists[1][1])
        if not rej:
            o = oracle_mod.Oracle(path, nu, nd)
            o.run_all_variations([eps], [10 * eps, 3 * eps], 5e-5)
            ou, od, _ = o.dets()
            assert np.array_equal(lists[0][0], ou) and np.array_equal(lists[0][1], od)
