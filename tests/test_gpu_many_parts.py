"""Rows of the Hamiltonian join in more parts than the CTA that closes their gaps reads at a time
(256)."""
import numpy as np
import pytest

from conftest import C_ATOM
from test_gpu_long_rows import _doubles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["FP64", "MIXED"])
@pytest.mark.parametrize("cand,part", [(3988, 8), (3988, 15), (3988, 16), (2048, 8), (2049, 8), (3988, 1)])
def test_more_parts_than_one_read(monkeypatch, cand, part, prec):
    """250 to 3,988 parts: row 0 has `cand` candidates.  The scan path builds the same rows without
    the join; its elements are evaluated by the same device functions, so that values agree bit for
    bit."""
    import shci_gb300
    dets = _doubles()[:cand + 1]
    up = np.array([d[0] for d in dets], dtype=np.uint64)
    dn = np.array([d[1] for d in dets], dtype=np.uint64)
    got = []
    for path in ("join", "scan"):
        monkeypatch.setenv("SHCI_HBUILD", path)
        monkeypatch.setenv("SHCI_JOIN_PART", str(part))
        c = shci_gb300.Context(0)
        c.load_fcidump(C_ATOM, 4, 2, "d2h")
        c.set_dets(up, dn, np.ones(len(up)))
        nnz, _ = c.update_hamiltonian(getattr(shci_gb300, "PREC_" + prec))
        rp, cols, vals, diag = c.hamiltonian(nnz)
        c.close()
        rows = np.repeat(np.arange(len(up)), np.diff(rp.astype(np.int64)))
        o = np.lexsort((cols, rows))
        got.append((nnz, rows[o], cols[o], np.asarray(vals)[o], diag))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
