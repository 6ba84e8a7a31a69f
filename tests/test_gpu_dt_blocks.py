"""The random-sequential schemes that scatter their sites, at lattices on both sides of the number
of blocks at which the warps per block change (512 and 128 blocks a launch, and one), from a grown
surface, with counters and with disorder: word for word against the CPU emulations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inner", ["dbsh", "db", "dtdbsh", "dbshrep"])
@pytest.mark.parametrize("lx,ly,dis", [(14, 12, False), (14, 12, True), (12, 12, False), (9, 8, True)])
def test_scattered_schemes(kpzb, oracle, inner, lx, ly, dis):
    n = 2
    w = oracle.homogeneous(lx, ly, oracle.ENC_CBBIT)
    oracle.sca_mcs_words(w, lx, ly, 5, 0, 0, 12, 0.5, 0.5)
    ref = oracle.cbbit_to_local(w, lx, ly)
    s = kpzb.Scheduler(lx, ly, scheduler="dt")
    s.setDtInner(inner)
    s.pushSystem(ref)
    s.setPQ(0.9, 0.2)
    s.supplySeed(77, 3)
    s.enableCounters(True)
    words = None
    p, q = 0.9, 0.2
    if dis:
        words = np.random.RandomState(1).randint(0, 1 << 32, ref.size, dtype=np.uint32) & np.uint32(0x55555555)
        p, q = [0.9, 1.0], [0.2, 0.5]
        s.setPQ(1.0, 0.5, 1)
        s.setDisorder(words)
        s.mcsDisorder2SyncRng(n)
    else:
        s.mcsPQSyncRng(n)
    if inner in ("dbsh", "db"):
        if dis:
            cnt = oracle.dt_mcs_dbsh(ref, lx, ly, 77, 3, 0, n, p, q, words, shift=inner == "dbsh")
        else:
            cnt = oracle.dt_mcs_dbsh(ref, lx, ly, 77, 3, 0, n, p, q, shift=inner == "dbsh")
    else:
        cnt = oracle.dt_mcs_inner(ref, lx, ly, 77, 3, 0, n, p, q, inner, words) if dis else \
            oracle.dt_mcs_inner(ref, lx, ly, 77, 3, 0, n, p, q, inner)
    assert np.array_equal(s.popSystem(), ref)
    assert s.counters() == cnt
    s.close()
