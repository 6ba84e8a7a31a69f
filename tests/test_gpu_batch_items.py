"""Batch passes with fewer work items than CTAs, as many, and more, at every number of CTAs per SM,
in batches without and with rates that need the general decision: every replica equals the
oracle.  The deepest pass that a lattice row fits in a CTA's shared memory, and the one beyond it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cps", [1, 2, 3])
@pytest.mark.parametrize("lxs,general", [([8], False), ([8] * 5, True), ([12], False), ([11, 12, 8], True),
                                         ([8] * 460, False), ([8] * 460, True)])
def test_items_and_modes(kpzb, oracle, lxs, general, cps):
    rates = [(1.0, 0.0), (0.5, 0.5), (0.75, 0.25), (0.875, 0.0)] + ([(0.95, 0.05), (0.75, 0.1), (0.9375, 0.0)] if general else [])
    pq = [rates[(i + len(lxs)) % len(rates)] for i in range(len(lxs))]
    b = kpzb.Batch(lxs, [r[0] for r in pq], [r[1] for r in pq], [40 + i for i in range(len(lxs))])
    b.setFusion(3, 2)
    b.setCtasPerSm(cps)
    n = 11
    b.mcs(n)
    for i in range(0, len(lxs), 1 if len(lxs) < 10 else 23):
        ref = oracle.homogeneous(lxs[i], lxs[i], oracle.ENC_CBBIT)
        oracle.sca_mcs_words(ref, lxs[i], lxs[i], 40 + i, 0, 0, n, *pq[i])
        assert np.array_equal(b.pop(i), ref), (i, lxs[i], pq[i])
    b.close()


@pytest.mark.parametrize("lx,cps,k", [(12, 2, 28), (13, 2, 13), (12, 3, 18), (13, 3, 9), (14, 3, 4)])
def test_deepest_pass(kpzb, oracle, lx, cps, k):
    b = kpzb.Batch([lx, 8], [1.0, 0.5], [0.0, 0.5], [3, 4])
    b.setFusion(k)  # the default depth of 8 does not fit every row below
    b.setCtasPerSm(cps)
    with pytest.raises(kpzb.KpzbError) as e:
        b.setFusion(k + 1)
    assert e.value.status == 1
    b.setFusion(k)
    b.mcs(k)
    for i, (l, p, q) in enumerate([(lx, 1.0, 0.0), (8, 0.5, 0.5)]):
        ref = oracle.homogeneous(l, l, oracle.ENC_CBBIT)
        oracle.sca_mcs_words(ref, l, l, 3 + i, 0, 0, k, p, q)
        assert np.array_equal(b.pop(i), ref)
    b.close()
