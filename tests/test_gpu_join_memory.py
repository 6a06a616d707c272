"""Device memory of the core join's index."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", ["0", "1"])
@pytest.mark.parametrize("bits", ["32", "40"])
def test_index_within_its_estimate(monkeypatch, split, bits):
    """16,000 random dets of 20 electrons in 40 orbitals: 3 million entries and next to no elements, so
    that the build's peak is the index.  It may hold the 26 bytes an entry (28 with 64-bit keys, whose
    sort keeps two copies of 12 bytes and a quarter) that the choice of the join allows for, and 64
    bytes a det of row arrays."""
    import shci_gb300
    from shci_gb300 import synthetic
    h, g = synthetic.integrals(40, 9)
    rng = np.random.default_rng(1)
    up, dn = (np.array([sum(1 << int(o) for o in rng.choice(40, 10, replace=False)) for _ in range(16000)],
                       np.uint64) for _ in range(2))
    monkeypatch.setenv("SHCI_JOIN_SPLIT", split)
    monkeypatch.setenv("SHCI_JOIN_BITS", bits)
    c = shci_gb300.Context()
    c.set_integrals(h, g, 10, 10, 0x3ff, 0x3ff)
    c.set_dets(up, dn)
    live = c.memory_stats()[0] - c.memory_cached()[0]
    c.update_hamiltonian(shci_gb300.PREC_MIXED)
    assert c.hamiltonian_stats()["path"] == "core_join"
    peak = c.memory_cached()[1]
    c.close()
    entries = 16000 * 190
    assert peak - live < entries * (26 if bits == "32" else 28) + 16000 * 64
