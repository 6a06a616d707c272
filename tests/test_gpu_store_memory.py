"""Device memory of the element store: its arrays live as long as the matrix and take no cached block
that is much too large for them."""
import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


def _step(shci, fill):
    """A build, a selection and an incremental build.  fill: bytes of the blocks that are in the cache
    when the second build begins (the two string arrays of find_connected_dets).  Returns what the
    second build added to the live blocks, its candidates and the number of dets."""
    c = shci.Context()
    c.load_fcidump(C_ATOM, 4, 2, "d2h")
    c.build_queues()
    for eps in (2e-3, 5e-4):
        c.select(eps)
        c.update_hamiltonian(shci.PREC_MIXED)
        c.davidson(1e-8)
    c.select(1e-4)
    if fill:
        up, dn, _ = c.dets()
        off = c.find_connected(up[:1], dn[:1], 1e100, 0.0)[0]
        k = np.zeros(fill // (8 * int(off[1])), int)
        c.find_connected(up[k], dn[k], 1e100, 0.0)
    live = c.memory_stats()[0] - c.memory_cached()[0]
    c.update_hamiltonian(shci.PREC_MIXED)
    st = c.hamiltonian_stats()
    live = c.memory_stats()[0] - c.memory_cached()[0] - live
    c.close()
    return live, st["candidates"], st["n"]


def test_store_takes_no_much_larger_block():
    """The store asks for 12 bytes a candidate and a tenth more and may take a quarter above that; 64
    bytes a det for the arrays of the rows.  With cached blocks of 1.9 times its arrays' size it took
    two of these."""
    import shci_gb300
    _, cand, n = _step(shci_gb300, 0)
    live, _, _ = _step(shci_gb300, int(1.9 * 4.4 * cand))
    assert cand > 20 * n
    assert live < 12 * 1.1 * 1.25 * cand + 64 * n
