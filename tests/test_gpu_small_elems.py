"""Matrix elements of few pairs (passed as kernel arguments) against the same pairs in one large call,
at the edges of the argument sizes (64, 256, 1,000 pairs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 63, 64, 65, 255, 256, 257, 999, 1000, 1001])
def test_small_calls_equal_a_large_one(w1_fcidump, n):
    import shci_gb300
    c = shci_gb300.Context()
    c.load_fcidump(w1_fcidump, 5, 5)
    c.build_queues()
    c.run_variation([5e-4], [], 5e-5)
    up, dn, _ = c.dets()
    rng = np.random.default_rng(n)
    i, j = rng.integers(0, len(up), (2, 4096))
    j[::3] = i[::3]
    pairs = up[i], dn[i], up[j], dn[j]
    big = c.h_elems(*pairs)
    assert np.count_nonzero(big) > 1000
    assert np.array_equal(c.h_elems(*(p[:n] for p in pairs)), big[:n])
    c.close()
