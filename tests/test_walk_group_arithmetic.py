"""CPU restatement of the roughness walk's arithmetic (analysis.cu: walk_kernel, add_chunk): the bins
of a chunk's eight groups formed as bytes of two words, the moments from counts of (height, pattern),
the correlator's heights as biased bytes, and the power sums of a chunk outside the bins.  Checked:
no carry between bytes and no bin outside the table at the ends of the accepted ranges, and the
moments against exact integer sums, with the tolerance of the GPU roughness tests (rtol 1e-12)."""
from math import comb

import numpy as np
import pytest

RTOL = 1e-12
M32 = 0xFFFFFFFF
BINS, REACH = 192, 128  # height bins of a CTA; chunks start within REACH of the middle


def words(bits):
    """Even-x and odd-x slope words of 64 slope bits."""
    e = sum(int(b) << i for i, b in enumerate(bits[0::2]))
    o = sum(int(b) << i for i, b in enumerate(bits[1::2]))
    return e, o


def walks():
    rng = np.random.default_rng(1)
    yield np.zeros(64, dtype=int)
    yield np.ones(64, dtype=int)
    yield np.arange(64) & 1
    yield (np.arange(64) // 8) & 1
    for p in (0.1, 0.5, 0.5, 0.5, 0.9):
        for _ in range(8):
            yield (rng.random(64) < p).astype(int)


def byte_popc(v):
    return sum(bin((v >> (8 * i)) & 255).count("1") << (8 * i) for i in range(4))


def patterns(e, o):
    return (e & 0x0F0F0F0F) | ((o & 0x0F0F0F0F) << 4), ((e >> 4) & 0x0F0F0F0F) | (o & 0xF0F0F0F0)


@pytest.mark.parametrize("rel", [-REACH, -REACH + 1, -1, 0, 1, REACH - 2, REACH - 1])
@pytest.mark.parametrize("parity", [0, 1])
def test_bins_of_groups(rel, parity):
    h0_rel = BINS - parity  # the middle, counted from the first bin's height
    s0 = (rel + h0_rel) >> 1
    for bits in walks():
        A, B = patterns(*words(bits))
        pa, pb = byte_popc(A), byte_popc(B)
        sa = ((pa + pb) * 0x01010100 + s0 * 0x01010101 - 0x18100800) & M32
        sb = (sa + pa - 0x04040404) & M32
        for g in range(8):
            before = int(bits[:8 * g].sum())
            s = ((sb if g & 1 else sa) >> (8 * (g >> 1))) & 255
            assert s == s0 + before - 4 * g and 0 <= s < BINS
            p = ((B if g & 1 else A) >> (8 * (g >> 1))) & 255
            site = bits[8 * g:8 * g + 8]
            assert [(p >> ((j & 1) * 4 + (j >> 1))) & 1 for j in range(8)] == list(site)


@pytest.mark.parametrize("H0", [-192, -5, 0, 1000, -250_001, 3_000_000])
def test_moments_from_counts(H0):
    """sum over sites of h^k, k = 1..7, from the power sums of the groups' heights per pattern (in FP64
    from k = 3 on) and the patterns' own offsets'."""
    rng = np.random.default_rng(abs(H0))
    counts = {}
    for _ in range(300):
        counts.setdefault(int(rng.integers(0, 256)), []).append((int(rng.integers(0, BINS)), int(rng.integers(1, 1 << 20))))
    got, exact = [0, 0] + [0.0] * 5, [0] * 7
    for p, hits in counts.items():
        d, off = 0, []
        for j in range(8):
            d += 2 * ((p >> ((j & 1) * 4 + (j >> 1))) & 1) - 1
            off.append(d)
        t = [sum(x ** k for x in off) for k in range(8)]
        n0, n1, n2 = (sum(n * s ** k for s, n in hits) for k in range(3))
        m = [n0, H0 * n0 + 2 * n1, H0 * H0 * n0 + 4 * H0 * n1 + 4 * n2] + [0.0] * 5
        for s, n in hits:
            h = float(H0 + 2 * s)
            for k in range(3, 8):
                m[k] += float(n) * h ** k
        got[0] += 8 * m[1] + t[1] * m[0]
        got[1] += 8 * m[2] + 2 * t[1] * m[1] + t[2] * m[0]
        for k in range(3, 8):
            got[k - 1] += sum(comb(k, j) * float(t[j]) * float(m[k - j]) for j in range(k + 1))
        for s, n in hits:
            for k in range(7):
                exact[k] += n * sum((H0 + 2 * s + x) ** (k + 1) for x in off)
    scale = [abs(e) for e in exact]
    assert got[:2] == exact[:2]
    for k in range(2, 7):
        # odd moments may cancel: against the size of their terms
        size = sum(n * 8 * (abs(H0) + 2 * BINS) ** (k + 1) for hits in counts.values() for _, n in hits)
        assert abs(got[k] - exact[k]) <= RTOL * max(scale[k], 1e-3 * size), k


@pytest.mark.parametrize("rel", [-63, -1, 0, 63])
def test_correlator_bytes(rel):
    """u = h - mid + 128 stays in [1, 255] over a chunk that starts within 63 of the middle, and no
    intermediate byte (the value before a group, less the table's bias of 8) borrows."""
    for bits in walks():
        b, h = rel + 120, rel
        for g in range(8):
            assert 0 <= b <= 239
            cum = 8
            for j in range(8):
                step = 2 * int(bits[8 * g + j]) - 1
                cum += step
                h += step
                assert 0 <= cum <= 16 and b + cum == h + 128 and 1 <= b + cum <= 255
            b = b + cum - 8


@pytest.mark.parametrize("b", [0, 7, -13, 64, -100, 1_000, -250_000, 3_000_000])
@pytest.mark.parametrize("is_open", [False, True])
def test_far_chunk(b, is_open):
    """Offsets as bytes d + 128 four at a time, power sums exact in FP64, the binomial expansion about
    the height before the chunk; the first site of an open row left out."""
    for bits in walks():
        e, o = words(bits)
        A = (e & 0x33333333) | ((o & 0x33333333) << 2)
        B = ((e >> 2) & 0x33333333) | (o & 0xCCCCCCCC)
        base, d = 0x7C, []
        for g in range(16):
            n = ((B if g & 1 else A) >> (4 * (g >> 1))) & 15
            cum = 4
            for j in range(4):
                cum += 2 * ((n >> ((j & 1) * 2 + (j >> 1))) & 1) - 1
                assert 0 <= cum <= 8 and 64 <= base + cum <= 192
                d.append(base + cum - 128)
            base = base + cum - 4
        assert d == list(np.cumsum(2 * np.asarray(bits) - 1))
        use = d[1:] if is_open else d
        a = [sum(x ** k for x in use) for k in range(8)]
        assert all(abs(v) < 1 << 53 and sum(abs(x) ** k for x in use) < 1 << 53 for k, v in enumerate(a))
        n, exact = len(use), [sum((b + x) ** k for x in use) for k in range(8)]
        assert n * b + a[1] == exact[1]
        assert n * b * b + 2 * b * a[1] + a[2] == exact[2]
        for k in range(3, 8):
            got = sum(comb(k, j) * float(b) ** (k - j) * float(a[j]) for j in range(k + 1))
            assert got == pytest.approx(exact[k], rel=RTOL, abs=1e-9), (k, b)
