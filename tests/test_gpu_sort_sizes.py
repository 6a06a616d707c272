"""Radix sorts around the edges of a tile (4,096 items) and of the sorts whose tiles form their own
offsets (64 tiles), as the core join uses them (15 entries a det): the join's matrix against the scan's,
which sorts the list by other keys."""
import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 273, 274, 546, 17475, 17476, 17477, 17749])
def test_join_at_sort_sizes(monkeypatch, count):
    """count x 15 entries: 15, 4,095, 4,110, 8,190, 262,125, 262,140, 262,155 and 266,235; an element is
    formed by the same device functions on both paths, so that the values agree bit for bit."""
    import shci_gb300
    rng = np.random.default_rng(count)
    strings = {}
    for ne in (4, 2):
        s = set()
        while len(s) < 140:
            s.add(tuple(sorted(rng.choice(12 if ne == 4 else 20, ne, replace=False).tolist())))
        strings[ne] = np.array([sum(1 << o for o in t) for t in sorted(s)], dtype=np.uint64)
    pick = rng.permutation(140 * 140)[:count]
    up, dn = strings[4][pick // 140], strings[2][pick % 140]
    got = []
    for path in ("join", "scan"):
        monkeypatch.setenv("SHCI_HBUILD", path)
        c = shci_gb300.Context(0)
        c.load_fcidump(C_ATOM, 4, 2, "d2h")
        c.set_dets(up, dn, np.ones(count))
        nnz, _ = c.update_hamiltonian(shci_gb300.PREC_FP64)
        rp, cols, vals, diag = c.hamiltonian(nnz)
        c.close()
        rows = np.repeat(np.arange(count), np.diff(rp.astype(np.int64)))
        o = np.lexsort((cols, rows))
        got.append((nnz, rows[o], cols[o], vals[o], diag))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
