"""Ends of the core join's buckets (runs of equal hash bits): runs inside a group of 32 positions
and runs of hundreds of positions, the spans written straight to their entries or by way of the
entries' leading bits, give the same matrix."""
import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 3, 43, 64, 700])
def test_bucket_lengths(monkeypatch, count):
    """15 entries a det: from fewer entries than one warp reads to runs of all 10,500 with 4 hash
    bits (about 650 positions a run).  Same columns and bit-equal values for every width."""
    import shci_gb300
    rng = np.random.default_rng(count)
    occ = sorted({(tuple(sorted(rng.choice(9, 4, replace=False))),
                   tuple(sorted(rng.choice(9, 2, replace=False)))) for _ in range(4 * count)})
    occ = [occ[k] for k in rng.permutation(len(occ))[:count]]
    up = np.array([sum(1 << int(o) for o in a) for a, _ in occ], dtype=np.uint64)
    dn = np.array([sum(1 << int(o) for o in b) for _, b in occ], dtype=np.uint64)
    got = []
    for env in ({}, {"SHCI_JOIN_BITS": "4"}, {"SHCI_JOIN_BITS": "9"}, {"SHCI_JOIN_BITS": "40"},
                {"SHCI_JOIN_SPLIT": "1"}, {"SHCI_JOIN_SPLIT": "1", "SHCI_JOIN_BITS": "4"},
                {"SHCI_JOIN_SPLIT": "1", "SHCI_JOIN_BITS": "40"}, {"SHCI_HBUILD": "scan"}):
        for k in ("SHCI_HBUILD", "SHCI_JOIN_BITS", "SHCI_JOIN_SPLIT"):
            monkeypatch.delenv(k, raising=False)
        for k, v in env.items():
            monkeypatch.setenv(k, v)
        c = shci_gb300.Context(0)
        c.load_fcidump(C_ATOM, 4, 2, "d2h")
        c.set_dets(up, dn, np.ones(len(up)))
        nnz, _ = c.update_hamiltonian(shci_gb300.PREC_FP64)
        rp, cols, vals, diag = c.hamiltonian(nnz)
        c.close()
        rows = np.repeat(np.arange(len(up)), np.diff(rp).astype(int))
        o = np.lexsort((cols, rows))
        got.append((rows[o], cols[o], vals[o], diag))
    for g in got[:-1]:
        for a, b in zip(g, got[-1]):
            assert np.array_equal(a, b)
