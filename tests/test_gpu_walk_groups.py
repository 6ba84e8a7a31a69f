"""The roughness / correlator walk by groups of eight sites against the oracle, at every row
width at which the split of rows over lanes, warps and parts changes, on surfaces inside and far
outside the height bins a CTA keeps, and on words whose rows do not close.  Power sums, extremes
and slope agreement are whole numbers and must be equal; the higher moments are FP64 sums of
terms of one sign pattern per height, each rounded a few times: relative error below 1e-12, as
for the other roughness tests."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def triangle(n, amp):
    """A closed walk of +-1 steps over n sites between -amp/2 and amp/2."""
    ph = (np.arange(n) + amp // 2) % (2 * amp)
    return np.where(ph < amp, ph, 2 * amp - ph) - amp // 2


def cbbit(h):
    """ENC_CBBIT words of the slopes of the heights h[y, x]."""
    rows, L = h.shape
    quads = []
    for sub in (0, 1):
        for axis in (1, 0):
            s = (h > np.roll(h, 1, axis)).astype(np.uint8)
            bits = np.stack([s[y, (sub ^ (y & 1))::2] for y in range(rows)])
            quads.append(np.packbits(bits, axis=1, bitorder="little").view(np.uint32).ravel())
    return np.concatenate(quads)


def surface(oracle, kind, lx, ly):
    if kind == "grown":
        w = oracle.homogeneous(lx, ly, oracle.ENC_CBBIT)
        oracle.sca_mcs_words(w, lx, ly, 5, 0, 0, 20, 0.5, 0.5)
        return w
    if kind == "words":
        return np.random.RandomState(lx * 32 + ly).randint(0, 1 << 32, 1 << (lx + ly - 4), dtype=np.uint32)
    amp = 1 << (lx - 2)  # steep: heights from one end of the bins to far outside them
    return cbbit(triangle(1 << lx, amp)[None, :] + triangle(1 << ly, max(1, 1 << (ly - 2)))[:, None])


@pytest.mark.parametrize("kind", ["grown", "steep", "words"])
@pytest.mark.parametrize("lx,ly", [(8, 6), (8, 9), (9, 5), (10, 4), (11, 3), (11, 8), (12, 2), (12, 7), (13, 2), (13, 6), (14, 5)])
def test_walk_matches_oracle(kpzb, oracle, kind, lx, ly):
    w = surface(oracle, kind, lx, ly)
    s = kpzb.Scheduler(lx, ly)
    s.pushSystem(w)
    ps = oracle.power_sums(oracle.heights(w, lx, ly, oracle.ENC_CBBIT))
    h = oracle.heights(w, lx, ly, oracle.ENC_CBBIT)
    for _ in range(2):  # the second call finds the tickets as the first left them
        assert s.heightSums() == ((ps[0], ps[1]), (int(h.min()), int(h.max())))
    tag = s.correlateTag()
    np.testing.assert_allclose([tag.w2] + tag.h, oracle.roughness(w, lx, ly, oracle.ENC_CBBIT), rtol=1e-12, atol=1e-12)
    cur = surface(oracle, "grown" if kind == "steep" else kind, lx, ly)
    if kind == "words":
        cur = cur ^ np.where(np.arange(cur.size) % 7 == 0, np.uint32(0x10204080), np.uint32(0))
    s.pushSystem(cur)
    r, ch, cs = s.correlate()
    s.close()
    ref = oracle.correlate(cur, w, lx, ly, oracle.ENC_CBBIT, tag.h[0])
    np.testing.assert_allclose([r.w2] + r.h, ref[:8], rtol=1e-12, atol=1e-12)
    np.testing.assert_allclose(ch, ref[8], rtol=1e-10, atol=1e-12 * max(1.0, abs(tag.h[0] * r.h[0])))
    assert cs == ref[9]


def exact_sums(h, g):
    """Whole-number sums of h^k, |h|^k (k = 1..7) and of h g over all sites."""
    lo = int(h.min())
    n = np.bincount((h - lo).ravel())
    at = [(int(i) + lo, int(n[i])) for i in np.flatnonzero(n)]
    cross = h.astype(np.int64).ravel() * g.astype(np.int64).ravel()
    cross = (int((cross >> 20).sum()) << 20) + int((cross & ((1 << 20) - 1)).sum())
    return [sum(c * x**k for x, c in at) for k in range(1, 8)], [sum(c * abs(x) ** k for x, c in at) for k in range(1, 8)], cross


@pytest.mark.parametrize("kind", ["grown", "steep", "words"])
@pytest.mark.parametrize("lx,ly", [(8, 13), (8, 17), (15, 4), (16, 3), (20, 3)])
def test_tall_and_wide_lattices(kpzb, oracle, kind, lx, ly):
    """Blocks of 32 and of 512 rows (several steps of a block's row loop), and rows whose quarters
    take several steps of a warp, against whole-number sums of the oracle's heights: the oracle's own
    sums in FP64 lose digits to heights of thousands that cancel.  The higher moments are off by at
    most 1e-12 of their terms' size, the covariance by that of its two terms."""
    N = 1 << (lx + ly)
    w = surface(oracle, kind, lx, ly)
    cur = w ^ np.where(np.arange(w.size) % 5 == 0, np.uint32(0x01020810), np.uint32(0))  # open rows
    h, g = oracle.heights(w, lx, ly, oracle.ENC_CBBIT), oracle.heights(cur, lx, ly, oracle.ENC_CBBIT)
    s = kpzb.Scheduler(lx, ly)
    s.pushSystem(w)
    sums, size, _ = exact_sums(h, h)
    assert s.heightSums() == ((sums[0], sums[1]), (int(h.min()), int(h.max())))
    tag = s.correlateTag()
    for k in range(7):
        assert abs(tag.h[k] - sums[k] / N) <= 1e-12 * size[k] / N, k
    s.pushSystem(cur)
    r, ch, cs = s.correlate()
    s.close()
    sums_g, size, cross = exact_sums(g, h)
    for k in range(7):
        assert abs(r.h[k] - sums_g[k] / N) <= 1e-12 * size[k] / N, k
    exact = (cross * N - sums[0] * sums_g[0]) / N**2
    assert abs(ch - exact) <= 1e-12 * (abs(cross) / N + abs(sums[0] * sums_g[0]) / N**2)
    assert cs == oracle.correlate(cur, w, lx, ly, oracle.ENC_CBBIT, tag.h[0])[9]
