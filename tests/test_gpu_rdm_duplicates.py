"""The 1-RDM of a list with equal dets: a det's partners, itself among them, are the first of their
kind."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [0, 1, 40])
def test_rdm1_with_equal_dets(copies):
    """Brute force over all pairs in FP64; sums of fewer than 1e4 terms of at most 1."""
    import shci_gb300
    from shci_gb300 import synthetic
    n, nu, nd = 7, 3, 2
    h, g = synthetic.integrals(n, 8)
    up = [sum(1 << o for o in t) for t in itertools.combinations(range(n), nu)][:12]
    dn = [sum(1 << o for o in t) for t in itertools.combinations(range(n), nd)][:8]
    rng = np.random.default_rng(copies)
    dets = [p for p in itertools.product(up, dn)]
    dets += [dets[k] for k in rng.integers(0, len(dets), copies)]
    dets = [dets[k] for k in rng.permutation(len(dets))]
    co = rng.standard_normal(len(dets)) / np.sqrt(len(dets))
    first = {}
    for k, d in enumerate(dets):
        first.setdefault(d, k)
    want = np.zeros((n, n))
    for (u, d), c in zip(dets, co):
        for spin, s in enumerate((u, d)):
            for p in range(n):
                for r in range(n):
                    if not s >> p & 1 or (r != p and s >> r & 1):
                        continue
                    t = s & ~(1 << p) | 1 << r
                    j = first.get((u, t) if spin else (t, d))
                    if j is None:
                        continue
                    lo, hi = min(p, r), max(p, r)
                    odd = bin(s >> (lo + 1) & ((1 << max(hi - lo - 1, 0)) - 1)).count("1") & 1 if p != r else 0
                    want[p, r] += c * co[j] * (-1) ** odd
    ctx = shci_gb300.Context()
    ctx.set_integrals(h, g, nu, nd, 0b111, 0b11)
    ctx.set_dets(np.array([d[0] for d in dets], np.uint64), np.array([d[1] for d in dets], np.uint64), co)
    for _ in range(3):
        assert np.max(np.abs(np.asarray(ctx.rdm1()).reshape(n, n) - want)) < 1e-13
    ctx.close()
