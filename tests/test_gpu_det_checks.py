"""A det list with equal dets is refused by the selection, whose check shares a wait with its counts."""
import numpy as np
import pytest

from conftest import C_ATOM

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [1, 2, 40])
def test_select_refuses_duplicates(at):
    import itertools
    import shci_gb300
    up = [sum(1 << o for o in t) for t in itertools.combinations(range(8), 4)][:at]
    up = np.array(up + up[:1], dtype=np.uint64)
    dn = np.full(len(up), 3, dtype=np.uint64)
    c = shci_gb300.Context(0)
    c.load_fcidump(C_ATOM, 4, 2, "d2h")
    c.build_queues()
    c.set_dets(up, dn, np.ones(len(up)))
    with pytest.raises(Exception, match="duplicates"):
        c.select(1e-3)
    c.set_dets(up[:-1], dn[:-1], np.ones(len(up) - 1))
    assert c.select(1e-3) > 0
    c.close()
