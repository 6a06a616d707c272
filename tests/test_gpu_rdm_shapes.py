"""RDM kernels at the sizes where they can go wrong: more than 32 orbitals (a second orbital per
lane), an empty spin string, fewer dets than a warp, lists of a few hundred random dets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random_dets(rng, n, nu, nd, count):
    """Distinct dets within a few moves of the lowest one (most pairs connected), it first."""
    seen = {((1 << nu) - 1, (1 << nd) - 1): None}
    for _ in range(50 * count):
        if len(seen) == count:
            break
        u, d = list(seen)[rng.integers(0, len(seen))]
        for _ in range(int(rng.integers(1, 3))):
            s, ne = (u, nu) if (rng.random() < 0.5 and nu) or not nd else (d, nd)
            occ = [o for o in range(n) if s >> o & 1]
            vir = [o for o in range(n) if not s >> o & 1]
            t = s ^ (1 << occ[rng.integers(0, ne)]) ^ (1 << vir[rng.integers(0, len(vir))])
            if s == u and ne == nu and (nd == 0 or rng.random() < 0.5):
                u = t
            elif bin(t).count("1") == nd:
                d = t
            else:
                u = t
        seen[(u, d)] = None
    up = np.array([k[0] for k in seen], np.uint64)
    dn = np.array([k[1] for k in seen], np.uint64)
    return up, dn


@pytest.mark.parametrize("n,nu,nd,count", [(5, 2, 0, 7), (9, 1, 1, 40), (32, 3, 2, 150), (33, 2, 2, 200),
                                            (40, 4, 3, 300)])
def test_rdms_match_oracle(oracle_mod, tmp_path, n, nu, nd, count):
    """Sums of fewer than 1e5 terms of magnitude <= 1 in FP64: 1e-12 absolute."""
    import shci_gb300
    from shci_gb300 import synthetic
    rng = np.random.default_rng(n)
    path = str(tmp_path / "FCIDUMP")
    h, g = synthetic.integrals(n, 5 + n)
    synthetic.write_fcidump(path, h, g, nu + nd)
    up, dn = _random_dets(rng, n, nu, nd, count)
    coefs = rng.standard_normal(len(up))
    coefs /= np.linalg.norm(coefs)
    o = oracle_mod.Oracle(path, nu, nd)
    o.set_dets(up, dn, coefs)
    o.update_hamiltonian()
    for prec in (shci_gb300.PREC_FP64, shci_gb300.PREC_MIXED):
        c = shci_gb300.Context()
        c.load_fcidump(path, nu, nd)
        c.set_dets(up, dn, coefs)
        c.update_hamiltonian(prec)
        assert np.max(np.abs(c.rdm1() - o.rdm1())) < 1e-12
        assert np.max(np.abs(c.rdm2_half() - o.rdm2_half())) < 1e-12
        c.close()
