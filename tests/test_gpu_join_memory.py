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


@pytest.mark.parametrize("bits", ["9", "40"])
def test_without_room_to_split(monkeypatch, bits):
    """Without storage to place spans by their entries' leading bits they go straight: the join
    still builds the matrix, with the same columns and bit-equal values."""
    import shci_gb300
    from conftest import C_ATOM
    rng = np.random.default_rng(4)
    occ = {(tuple(sorted(rng.choice(9, 4, replace=False))), tuple(sorted(rng.choice(9, 2, replace=False))))
           for _ in range(900)}
    up = np.array([sum(1 << int(o) for o in a) for a, _ in sorted(occ)], np.uint64)
    dn = np.array([sum(1 << int(o) for o in b) for _, b in sorted(occ)], np.uint64)
    monkeypatch.setenv("SHCI_JOIN_BITS", bits)
    got = []
    for split in ("0", "1", "2"):
        monkeypatch.setenv("SHCI_JOIN_SPLIT", split)
        c = shci_gb300.Context()
        c.load_fcidump(C_ATOM, 4, 2, "d2h")
        c.set_dets(up, dn)
        nnz, _ = c.update_hamiltonian(shci_gb300.PREC_FP64)
        assert c.hamiltonian_stats()["path"] == "core_join"
        rp, cols, vals, diag = c.hamiltonian(nnz)
        c.close()
        o = np.lexsort((cols, np.repeat(np.arange(len(up)), np.diff(rp).astype(int))))
        got.append((rp, cols[o], vals[o], diag))
    for g in got[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(g, got[0]))


def test_scratch_is_given_back():
    """After the build of next to no elements the context holds row arrays and items, 64 bytes a det,
    and not the digit counts of the entries' sorts (0.3 bytes an entry, 60 a det)."""
    import shci_gb300
    from shci_gb300 import synthetic
    h, g = synthetic.integrals(40, 9)
    rng = np.random.default_rng(1)
    n = 16000
    up, dn = (np.array([sum(1 << int(o) for o in rng.choice(40, 10, replace=False)) for _ in range(n)],
                       np.uint64) for _ in range(2))
    c = shci_gb300.Context()
    c.set_integrals(h, g, 10, 10, 0x3ff, 0x3ff)
    c.set_dets(up, dn)
    live = c.memory_stats()[0] - c.memory_cached()[0]
    c.update_hamiltonian(shci_gb300.PREC_FP64)
    assert c.memory_stats()[0] - c.memory_cached()[0] - live < 64 * n
    c.close()
