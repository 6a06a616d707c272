"""Exclusive scans by one block (up to 16,384 values) and by tiles (more), in both widths: the row
starts and the row pieces of det lists around the edges of a thread's four values, of a chunk and of
the one-block range."""
import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 3, 4, 5, 127, 129, 4095, 4096, 4097, 16383, 16384, 16385, 20000])
def test_rows_and_pieces(count):
    """y = H x against the stored rows in numpy: FP64 sums of at most a few thousand terms of order
    1, 1e-11."""
    import shci_gb300
    rng = np.random.default_rng(count)
    strings = {}
    for ne in (4, 2):
        s = set()
        while len(s) < 150:
            s.add(tuple(sorted(rng.choice(22, ne, replace=False).tolist())))
        strings[ne] = np.array([sum(1 << o for o in t) for t in sorted(s)], dtype=np.uint64)
    pick = rng.permutation(150 * 150)[:count]
    up, dn = strings[4][pick // 150], strings[2][pick % 150]
    c = shci_gb300.Context(0)
    c.load_fcidump(C_ATOM, 4, 2, "d2h")
    c.set_dets(up, dn, np.ones(count))
    nnz, _ = c.update_hamiltonian(shci_gb300.PREC_FP64)
    rp, cols, vals, diag = c.hamiltonian(nnz)
    x = rng.standard_normal(count)
    y = c.hv(x)
    c.close()
    rows = np.repeat(np.arange(count), np.diff(rp.astype(np.int64)))
    want = diag * x
    np.add.at(want, rows, vals * x[cols])
    np.add.at(want, cols, vals * x[rows])
    np.testing.assert_allclose(y, want, rtol=0, atol=1e-11 * max(1.0, np.abs(want).max()))
