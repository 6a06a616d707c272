"""The core join with the electrons of a det held by the lanes of a warp (up to 32) and looked up
in the strings (more): every stored element against the pairwise kernel, and no pair missing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fcidump(path, n, n_up, n_dn, rng):
    with open(path, "w") as f:
        f.write(f"&FCI NORB={n},NELEC={n_up + n_dn},MS2={n_up - n_dn},\n ORBSYM={'1,' * n}\n"
                " ISYM=1,\n&END\n")
        for p in range(1, n + 1):
            for q in range(1, p + 1):
                for r in range(1, p + 1):
                    for s in range(1, r + 1):
                        if r == p and s > q:
                            continue
                        if (p + q + r + s) % 3 == 0 or (p == q and r == s):
                            f.write(f"{0.1 * rng.standard_normal():.12f} {p} {q} {r} {s}\n")
        for p in range(1, n + 1):
            for q in range(1, p + 1):
                f.write(f"{rng.standard_normal():.12f} {p} {q} 0 0\n")
        f.write("0.0 0 0 0 0\n")


def _dets(n, n_up, n_dn, count, rng):
    """Distinct dets a few excitations away from the lowest one."""
    out = {((1 << n_up) - 1, (1 << n_dn) - 1)}
    while len(out) < count:
        strings = []
        for ne in (n_up, n_dn):
            occ = list(range(ne))
            for _ in range(int(rng.integers(0, 3))):
                if ne and ne < n:
                    occ[int(rng.integers(0, ne))] = int(rng.integers(ne, n))
            strings.append(sum(1 << o for o in set(occ)) if len(set(occ)) == ne else None)
        if None not in strings:
            out.add(tuple(strings))
    return [np.array(x, dtype=np.uint64) for x in zip(*sorted(out))]


@pytest.mark.parametrize("n,n_up,n_dn", [(6, 1, 1), (6, 2, 0), (18, 16, 15), (18, 16, 16),
                                         (18, 17, 16), (24, 20, 20)])
def test_join_elements_at_electron_counts(tmp_path, n, n_up, n_dn):
    """The element of a stored pair is formed from the same integrals as the pairwise kernel's in
    the same order but for the sum over common electrons, at most 40 terms of order 1: 1e-12."""
    import shci_gb300
    rng = np.random.default_rng(n + n_up)
    _fcidump(tmp_path / "FCIDUMP", n, n_up, n_dn, rng)
    count = 30 if n == 6 and n_dn else 12 if n == 6 else 150
    up, dn = _dets(n, n_up, n_dn, count, rng)
    c = shci_gb300.Context(0)
    c.load_fcidump(str(tmp_path / "FCIDUMP"), n_up, n_dn, "c1")
    c.set_dets(up, dn, np.ones(len(up)))
    nnz, _ = c.update_hamiltonian(shci_gb300.PREC_FP64)
    assert c.hamiltonian_stats()["path"] == "core_join"
    rp, cols, vals, _ = c.hamiltonian(nnz)
    i, j = np.triu_indices(len(up), 1)
    want = np.zeros((len(up), len(up)))
    want[i, j] = c.h_elems(up[i], dn[i], up[j], dn[j])
    c.close()
    got = np.zeros_like(want)
    for r in range(len(up)):
        a, b = int(rp[r]), int(rp[r + 1])
        assert len(set(cols[a:b].tolist())) == b - a
        got[r, cols[a:b]] = vals[a:b]
    scale = max(1.0, np.abs(want).max())
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-12 * scale)
