"""PT2 within a budget that does not hold a batch's records: the batch is taken in parts, with the same
dets and the same values up to the order of the sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wave():
    import shci_gb300
    from shci_gb300 import synthetic
    h, g = synthetic.integrals(26, 77)
    c = shci_gb300.Context()
    c.set_integrals(h, g, 7, 6, 0x7f, 0x3f)
    c.build_queues()
    c.run_variation([2e-3], [], 5e-5)
    e, dets = c.energy_fp64(), c.dets()
    c.close()
    return h, g, e, dets


CALLS = {
    "dtm": lambda c, e: c.pt2_dtm(e, 1e-8, 1)[::2],
    "dtm13": lambda c, e: c.pt2_dtm(e, 1e-8, 13)[::2],
    "psto": lambda c, e: [c.pt2_psto(e, 1e-6, 1e-8, 16, -1.0, 0.0)[k] for k in (0, 2, 3)],
    "sto": lambda c, e: c.pt2_sto(e, 1e-6, 1e-8, 16, 300, 5, 8, 0.0, 0.0)[2],
    "sto_pilot": lambda c, e: c.pt2_sto(e, 1e-6, 1e-8, 16, 0, 5, 8, 0.0, 0.0, pt_mem_avail=1e9)[2],
}


@pytest.mark.parametrize("call", list(CALLS))
@pytest.mark.parametrize("share", [0.7, 0.3])
def test_parts_of_a_batch(wave, call, share):
    """Room for a share of what the call's live blocks take at their peak.  Counts are equal, sums of
    about 1e6 terms below 1e-3 within 1e-13."""
    import shci_gb300
    h, g, e, dets = wave

    def ctx(budget):
        c = shci_gb300.Context(hbm_budget=budget)
        c.set_integrals(h, g, 7, 6, 0x7f, 0x3f)
        c.build_queues()
        c.set_dets(*dets)
        return c

    c = ctx(0)
    base = c.memory_stats()[0] - c.memory_cached()[0]
    want = CALLS[call](c, e)
    peak = c.memory_cached()[1]
    c.close()
    assert peak - base > 2e7
    c = ctx(int(base + share * (peak - base)))
    got = CALLS[call](c, e)
    assert c.memory_stats()[0] <= base + share * (peak - base)
    c.close()
    assert len(want) == len(got)
    for a, b in zip(want, got):
        if isinstance(a, int):
            assert a == b
        else:
            assert abs(a - b) < 1e-13
