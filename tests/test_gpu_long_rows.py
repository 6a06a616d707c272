"""Rows of the Hamiltonian join that are cut into parts over warps: candidate counts around the line
(two parts), whole and broken last parts, several stretches a part, and no gaps left between them."""
import itertools

import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


def _doubles():
    """The reference det (4 alpha, 2 beta electrons in 22 orbitals) and its 3,988 double excitations:
    each shares one two-hole core with the reference, one candidate of its row."""
    def moves(ne, k):
        out = []
        for holes in itertools.combinations(range(ne), k):
            for parts in itertools.combinations(range(ne, 22), k):
                out.append(sum(1 << o for o in set(range(ne)) - set(holes) | set(parts)))
        return out
    ref = (0b1111, 0b11)
    d = [(u, ref[1]) for u in moves(4, 2)] + [(ref[0], x) for x in moves(2, 2)]
    d += [(u, x) for u in moves(4, 1) for x in moves(2, 1)]
    rng = np.random.default_rng(3)
    return [ref] + [d[k] for k in rng.permutation(len(d))]


@pytest.mark.parametrize("prec", ["FP64", "MIXED"])
@pytest.mark.parametrize("cand", [1024, 2047, 2048, 2049, 3071, 3072, 3073, 3988])
def test_parts_of_long_rows(monkeypatch, cand, prec):
    """The scan path builds the same rows without the join; its elements are evaluated by the same
    device functions, so that the values agree bit for bit."""
    import shci_gb300
    dets = _doubles()[:cand + 1]
    assert len(dets) == cand + 1
    up = np.array([d[0] for d in dets], dtype=np.uint64)
    dn = np.array([d[1] for d in dets], dtype=np.uint64)
    got = []
    for path, part in (("join", None), ("join", "0"), ("join", "64"), ("join", "1024"),
                       ("join", "1500"), ("scan", None)):
        monkeypatch.setenv("SHCI_HBUILD", path)
        if part is None:
            monkeypatch.delenv("SHCI_JOIN_PART", raising=False)
        else:
            monkeypatch.setenv("SHCI_JOIN_PART", part)
        c = shci_gb300.Context(0)
        c.load_fcidump(C_ATOM, 4, 2, "d2h")
        c.set_dets(up, dn, np.ones(len(up)))
        nnz, _ = c.update_hamiltonian(getattr(shci_gb300, "PREC_" + prec))
        rp, cols, vals, diag = c.hamiltonian(nnz)
        c.close()
        rows = np.repeat(np.arange(len(up)), np.diff(rp.astype(np.int64)))
        o = np.lexsort((cols, rows))
        got.append((nnz, rows[o], cols[o], np.asarray(vals)[o], diag))
    for g in got[:-1]:
        for a, b in zip(g, got[-1]):
            assert np.array_equal(a, b)
