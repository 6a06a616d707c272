"""find_connected_dets of systems without electrons (no slots, no pairs) and with one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu", [0, 1])
def test_no_or_one_electron(nu):
    """No electron has no slot and no pair, one electron a single slot: its targets are the other
    orbitals with a matrix element."""
    import shci_gb300
    from shci_gb300 import synthetic
    h, g = synthetic.integrals(5, 3)
    c = shci_gb300.Context()
    c.set_integrals(h, g, nu, 0, nu, 0)
    c.build_queues()
    off, cu, cd, nx = c.find_connected(np.array([nu], np.uint64), np.zeros(1, np.uint64), 1e100, 1e-9)
    c.close()
    assert sorted(int(u) for u in cu) == ([2, 4, 8, 16] if nu else [])
    assert int(off[1]) == len(cu) and np.all(cd == 0) and np.all(nx == 1)
