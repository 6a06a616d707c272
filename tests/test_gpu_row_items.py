"""Rows cut into work items (csrc/items.cuh): lengths around the piece length, several pieces per
row, empty rows, and whole-matrix products against numpy in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 1024, 1025, 1026, 2049, 2051, 3333])
def test_davidson_csr_rows_longer_than_a_piece(n):
    """Arrow matrices: row 0 holds n - 1 elements (1023, 1024, 1025, 2048 ... around one and two
    pieces), a middle row holds some and the rest are empty.  The lowest eigenpair of the dense
    matrix is the reference; a coupling of 1e-3 and a gap of 1 leave Davidson's tolerance of 1e-12
    on the eigenvalue."""
    import shci_gb300
    rng = np.random.default_rng(n)
    diag = np.concatenate([[-1.0], np.linspace(0.0, 1.0, n - 1)])
    mid = n // 2
    cols = [np.arange(1, n)] + [np.arange(i + 1, n)[:: 7] if i == mid and mid > 0 else np.zeros(0, int)
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
