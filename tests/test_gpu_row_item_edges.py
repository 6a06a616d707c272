"""Rows cut into work items of 512 elements (csrc/items.cuh): rows of 511, 512, 513 and three times 512
elements, and whole rows where there is no list of items."""
import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("items", ["1", "0"])
@pytest.mark.parametrize("n", [512, 513, 514, 1025, 1026, 1537, 1538])
def test_davidson_csr_rows_around_an_item(monkeypatch, n, items):
    """Arrow matrices: row 0 holds n - 1 elements, a middle row some, the rest none.  The lowest
    eigenpair of the dense matrix is the reference; couplings of 1e-3 and a gap of 1 leave Davidson's
    tolerance of 1e-14 on the eigenvalue."""
    import shci_gb300
    monkeypatch.setenv("SHCI_ROW_ITEMS", items)
    rng = np.random.default_rng(n)
    diag = np.concatenate([[-1.0], np.linspace(0.0, 1.0, n - 1)])
    cols = [np.arange(1, n)] + [np.arange(i + 1, n)[::7] if i == n // 2 else np.zeros(0, int)
                                for i in range(1, n)]
    cnt = np.array([len(c) for c in cols])
    row_ptr = np.concatenate([[0], np.cumsum(cnt)]).astype(np.uint64)
    col = np.concatenate(cols).astype(np.uint32)
    val = 1e-3 * rng.standard_normal(len(col))
    dense = np.diag(diag)
    r = np.repeat(np.arange(n), cnt)
    dense[r, col] = val
    dense[col, r] = val
    w, v = np.linalg.eigh(dense)
    init = np.zeros(n)
    init[0] = 1.0
    c = shci_gb300.Context(0)
    e, vec, _ = c.davidson_csr(row_ptr, col, val, diag, init, 1e-14)
    c.close()
    assert abs(e - w[0]) < 1e-11
    assert abs(abs(vec @ v[:, 0]) - 1.0) < 1e-9


def test_whole_rows_without_a_list(monkeypatch):
    """Products, the energy correction and the RDMs of two segments, both with items, the older one
    without and both without.  Mixed products add integers: the same bits.  The others' sums are in
    another order: 1e-12 of values of order one (thousands of terms below 1e-3 in FP64)."""
    import shci_gb300
    got = []
    for first, second in (("1", "1"), ("0", "1"), ("0", "0")):
        c = shci_gb300.Context(0)
        c.load_fcidump(C_ATOM, 4, 2, "d2h")
        c.build_queues()
        monkeypatch.setenv("SHCI_ROW_ITEMS", "1")
        for eps in (2e-3, 5e-4):
            c.select(eps)
            c.update_hamiltonian(shci_gb300.PREC_FP64)
            c.davidson(1e-8)
        up, dn, co = c.dets()
        out = []
        for prec in (shci_gb300.PREC_FP64, shci_gb300.PREC_MIXED):
            c.set_dets(up, dn, got[0][0] if got else co)
            monkeypatch.setenv("SHCI_ROW_ITEMS", first)
            c.update_hamiltonian(prec)
            c.select(2e-4)
            monkeypatch.setenv("SHCI_ROW_ITEMS", second)
            c.update_hamiltonian(prec)
            n = c.n_dets()
            x = np.random.default_rng(1).standard_normal(n) / np.sqrt(n)
            c.set_coefs(x)
            out += [c.hv(x), c.rdm2_half(), c.energy_fp64()]
            if prec == shci_gb300.PREC_MIXED:
                c.davidson(1e-10)
                out.append(c.energy_fp64())
        c.close()
        got.append([co] + out)
    assert len(got[0][1]) > 3000
    for g in got[1:]:
        for k in (1, 2, 3, 5, 6, 7):
            assert np.max(np.abs(np.asarray(g[k]) - got[0][k])) < 1e-12
        assert np.array_equal(g[4], got[0][4])
