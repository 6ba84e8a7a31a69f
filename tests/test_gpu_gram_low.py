"""The one-limb tensor Gram against the int64 Gram, equal in every word: triangle waves of up to 132
from their integer mean (the larger ones go to the three-limb kernel) for few, 33 and 64 snapshots
and at the smallest and odd-shaped lattices; surfaces whose largest height is exactly 125, 126 and 127
from it, with those heights inside rows and at their starts; and a lattice large enough that a warp
pair's int32 accumulators are added up and started anew in the middle of its run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ridges(lx, ly, ax, ay, shift):
    """ENC_CBBIT words of h(x, y) = t(x) + u(y), triangle waves of ax and ay steps up and down,
    the first moved by `shift` sites."""
    def slopes(n, a, s):
        return (((np.arange(n) + s) % (2 * a)) < a).astype(np.uint8) if a > 1 else (np.arange(n) + s) & 1
    L, rows = 1 << lx, 1 << ly
    sx, sy = slopes(L, ax, shift).astype(np.uint8), slopes(rows, ay, 0).astype(np.uint8)
    pat = [np.packbits(sx[a::2], bitorder="little").view(np.uint32) for a in (0, 1)]
    y = np.arange(rows)
    quads = []
    for sub in (0, 1):
        quads.append(np.where(((y ^ sub) & 1)[:, None] == 1, pat[1][None, :], pat[0][None, :]).ravel())
        quads.append(np.repeat(np.where(sy == 1, np.uint32(0xFFFFFFFF), np.uint32(0)), L // 64))
    return np.concatenate(quads).astype(np.uint32)


@pytest.mark.parametrize("lx,ly,ax,n", [(8, 6, 1, 1), (8, 6, 64, 5), (9, 5, 128, 33), (10, 8, 256, 64), (10, 8, 128, 64),
                                        (11, 7, 32, 64), (14, 13, 128, 3)])
def test_low_range_gram_equals_int64(kpzb, lx, ly, ax, n):
    g = kpzb.Gram(lx, ly, n)
    for i in range(n):
        g.add_host(ridges(lx, ly, ax, [1, 2, 8][i % 3], 7 * i))
    G, S1 = g.compute(g.TENSOR)
    R, S = g.compute(g.INT64)
    again, _ = g.compute(g.TENSOR)
    g.close()
    assert np.array_equal(S1, S)
    assert np.array_equal(G, R)
    assert np.array_equal(again, R)


def profile(lx, ly, up, down, shift):
    """ENC_CBBIT words of rows that climb `up`, fall `up + down`, climb `down` and zigzag from there,
    moved by `shift` sites, over a zigzag in y."""
    L, rows = 1 << lx, 1 << ly
    sx = np.tile(np.array([1, 0], np.uint8), L // 2)
    sx[:up], sx[up:2 * up + down], sx[2 * up + down:2 * up + 2 * down] = 1, 0, 1
    sx = np.roll(sx, shift)
    pat = [np.packbits(sx[a::2], bitorder="little").view(np.uint32) for a in (0, 1)]
    y = np.arange(rows)
    quads = []
    for sub in (0, 1):
        quads.append(np.where(((y ^ sub) & 1)[:, None] == 1, pat[1][None, :], pat[0][None, :]).ravel())
        quads.append(np.repeat(np.where(y & 1, np.uint32(0xFFFFFFFF), np.uint32(0)), L // 64))
    return np.concatenate(quads).astype(np.uint32)


@pytest.mark.parametrize("lx,ly", [(9, 5), (10, 6)])
@pytest.mark.parametrize("r,up,down", [(125, 124, 124), (126, 124, 125), (127, 125, 126)])
def test_edges_of_the_range(kpzb, oracle, lx, ly, r, up, down):
    shifts = [0, 1 - up, -up, 1 - 2 * up - down, -2 * up - down, 37]
    g = kpzb.Gram(lx, ly, 2 * len(shifts))
    far = []
    for sh in shifts:
        w = profile(lx, ly, up, down, sh)
        for words in (w, ~w):
            h = oracle.heights(words, lx, ly, oracle.ENC_CBBIT)
            c = int(np.floor(h.mean()))
            far.append(max(c - int(h.min()), int(h.max()) - c))
            g.add_host(words)
    assert max(far) == r
    G, S1 = g.compute(g.TENSOR)
    R, S = g.compute(g.INT64)
    g.close()
    assert np.array_equal(S1, S)
    assert np.array_equal(G, R)


def test_accumulators_started_anew(kpzb, oracle):
    """2^28 sites in 148 x 8 runs of 1771 or 1772 tiles of 128; int32 holds 2^31 / (126^2 * 128) = 1056
    tiles of heights up to 126 (the range, not the heights themselves, sets the length of a window)."""
    lx = ly = 14
    g = kpzb.Gram(lx, ly, 3)
    for sh in (0, -124, 5000):
        # rows are alike but for the zigzag in y, so 16 of them tell the range of all
        h = oracle.heights(profile(lx, 4, 125, 125, sh), lx, 4, oracle.ENC_CBBIT)
        c = int(np.floor(h.mean()))
        assert 125 <= max(c - int(h.min()), int(h.max()) - c) <= 126
        g.add_host(profile(lx, ly, 125, 125, sh))
    G, S1 = g.compute(g.TENSOR)
    R, S = g.compute(g.INT64)
    g.close()
    assert np.array_equal(S1, S)
    assert np.array_equal(G, R)
