"""The cache of released device blocks keeps those released last."""
import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


def test_old_blocks_make_room(monkeypatch):
    """The cache has room for 16 MB.  A call leaves two string arrays of 6 MB each in it, later calls,
    whose arrays take no block of more than twice their size, two of 2 MB: one of 6 MB has to go (what
    else the calls leave is below 1.2 MB), so that less than the two remains."""
    import shci_gb300
    monkeypatch.setenv("SHCI_CACHE_MB", "16")
    c = shci_gb300.Context()
    c.load_fcidump(C_ATOM, 4, 2, "d2h")
    c.build_queues()
    up, dn = np.array([0b1111], np.uint64), np.array([0b11], np.uint64)
    one = 8 * int(c.find_connected(up, dn, 1e100, 0.0)[0][1])
    big = np.zeros((6 << 20) // one, int)
    want = c.find_connected(up[big], dn[big], 1e100, 0.0)
    both = 2 * 8 * len(want[1])
    assert c.memory_cached()[0] > both
    small = big[: len(big) // 3]
    for _ in range(3):
        got = c.find_connected(up[small], dn[small], 1e100, 0.0)
        assert np.array_equal(got[1], want[1][: len(got[1])])
        assert c.memory_cached()[0] <= 16 << 20
    assert c.memory_cached()[0] < both
    c.close()
