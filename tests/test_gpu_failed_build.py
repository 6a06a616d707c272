"""A build that fails gives the join's index back."""
import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


def test_index_is_given_back(oracle_mod):
    """15 entries a det.  31 bytes of room an entry hold the index (26 with 15 % to spare), not the
    stored elements; what is left after the error is within 64 bytes a det of row arrays, where the
    index is 180.  The context then builds a short list."""
    import shci_gb300
    o = oracle_mod.Oracle(C_ATOM, 4, 2, "d2h")
    o.run_all_variations([1e-4], [2e-3, 1e-3, 5e-4, 2e-4], 5e-5)
    up, dn, co = o.dets()
    n = len(up)

    def ctx(budget):
        c = shci_gb300.Context(hbm_budget=budget)
        c.load_fcidump(C_ATOM, 4, 2, "d2h")
        c.set_dets(up, dn, co)
        return c

    def live(c):
        return c.memory_stats()[0] - c.memory_cached()[0]

    c = ctx(0)
    base = live(c)
    nnz, _ = c.update_hamiltonian(shci_gb300.PREC_MIXED)
    assert nnz * 4 > 31 * 15 * n - 12 * 15 * n  # (the columns do not fit beside the index)
    want = c.hamiltonian_rows(np.arange(50, dtype=np.uint64))
    c.close()
    c = ctx(base + 31 * 15 * n)
    with pytest.raises(shci_gb300.ShciError) as e:
        c.update_hamiltonian(shci_gb300.PREC_MIXED)
    assert e.value.status == 1
    assert live(c) - base < 64 * n
    c.set_dets(up[:50], dn[:50], co[:50])
    nnz, _ = c.update_hamiltonian(shci_gb300.PREC_MIXED)
    rp, cols, vals, _ = c.hamiltonian(nnz)
    for i in range(50):
        a, b = int(want[0][i]), int(want[0][i + 1])
        keep = want[1][a:b] < 50
        p, q = int(rp[i]), int(rp[i + 1])
        o = np.argsort(cols[p:q])
        assert np.array_equal(cols[p:q][o], want[1][a:b][keep])
        assert np.array_equal(vals[p:q][o], want[2][a:b][keep])
    c.close()
