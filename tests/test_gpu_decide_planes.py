"""The decision of general rates at every number of random planes around the line between its two
forms, and at pairs of a coarse and a fine threshold, whose sites drop out of the comparison at
different planes: half-steps, band passes (three choices of CTAs per SM) and stream passes, with
counters, and with disorder over the same rates: word for word against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RATES = [(0.75, 0.25), (0.875, 0.0), (0.875, 0.125), (0.9375, 0.0), (0.9375, 0.0625), (0.96875, 0.0), (0.75, 0.1),
         (0.5, 0.3), (0.3, 0.5), (0.0, 0.7), (1.0, 0.7), (0.7, 1.0), (0.875, 0.95), (2.0**-32, 1.0 - 2.0**-32)]


@pytest.mark.parametrize("p,q", RATES)
@pytest.mark.parametrize("kernel,k,lx,ly", [("half", 1, 8, 7), ("half", 1, 12, 5), ("band1", 3, 9, 7), ("band2", 4, 12, 6),
                                            ("band3", 3, 8, 9), ("stream", 3, 10, 9)])
def test_plane_counts(kpzb, oracle, monkeypatch, kernel, k, lx, ly, p, q):
    monkeypatch.setenv("KPZB_PASS_KERNEL", kernel)
    s = kpzb.Scheduler(lx, ly)
    start = oracle.homogeneous(lx, ly, oracle.ENC_CBBIT)
    oracle.sca_mcs_words(start, lx, ly, 3, 0, 0, 8, 0.5, 0.5)
    s.pushSystem(start)
    s.setPQ(p, q)
    s.setFusion(k)
    s.supplySeed(21, 5)
    s.enableCounters(True)
    n = 3 * k + 2
    s.mcsPQSyncRng(n)
    cnt = oracle.sca_mcs_words(start, lx, ly, 21, 5, 0, n, p, q)
    assert np.array_equal(s.popSystem(), start)
    assert s.counters() == tuple(cnt)
    s.close()


@pytest.mark.parametrize("rates", [[(0.75, 0.25), (0.9375, 0.1)], [(1.0, 0.0), (0.5, 0.3), (0.875, 0.0), (0.95, 0.05)]])
def test_disorder_of_few_and_many_planes(kpzb, oracle, rates):
    lx, ly = 10, 7
    s = kpzb.Scheduler(lx, ly, scheduler="sca")
    s.supplySeed(8, 1)
    words = np.random.RandomState(4).randint(0, 1 << 32, s.size_words(), dtype=np.uint32)
    if len(rates) == 2:
        words &= np.uint32(0x55555555)
    for c, (p, q) in enumerate(rates):
        s.setPQ(p, q, c)
    s.setDisorder(words)
    s.mcsDisorder2SyncRng(9)
    ref = oracle.homogeneous(lx, ly, oracle.ENC_LOCAL)
    oracle.sca_mcs_dis(ref, lx, ly, oracle.ENC_LOCAL, 8, 1, 0, 9, [r[0] for r in rates], [r[1] for r in rates], words)
    assert np.array_equal(s.popSystem(), ref)
    s.close()
