"""MCS left over from whole passes: every count from 1 to two passes, for each pass kernel that
takes shallower passes, split over calls in different ways, word for word against the oracle,
with the counters."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p,q", [(1.0, 0.0), (0.5, 0.5), (0.75, 0.25)])
@pytest.mark.parametrize("kernel,k,lx,ly", [("strip32", 8, 11, 7), ("strip8", 8, 12, 5), ("strip64", 6, 12, 7),
                                            ("strip44", 4, 13, 6), ("band1", 7, 8, 8), ("band2", 5, 10, 6), ("band", 8, 8, 6)])
def test_left_over_mcs(kpzb, oracle, monkeypatch, kernel, k, lx, ly, p, q):
    monkeypatch.setenv("KPZB_PASS_KERNEL", kernel)
    s = kpzb.Scheduler(lx, ly)
    s.setPQ(p, q)
    s.setFusion(k)
    s.enableCounters(True)
    for n in list(range(1, k)) + [k + 3, 2 * k - 1]:
        for split in ([n], [n // 2, n - n // 2]):
            s.initHomogeneous()
            s.supplySeed(9, 1)
            s.counters(reset=True)
            for m in split:
                s.mcsPQSyncRng(m)
            ref = oracle.homogeneous(lx, ly, oracle.ENC_CBBIT)
            cnt = oracle.sca_mcs_words(ref, lx, ly, 9, 1, 0, n, p, q)
            assert np.array_equal(s.popSystem(), ref), (n, split)
            assert s.counters() == tuple(cnt), (n, split)
    s.close()
