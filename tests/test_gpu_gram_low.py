"""The one-limb tensor Gram at the edges of its range (heights up to 126 from the snapshot's integer
mean), one beyond (the three-limb kernel), with and without full accumulation windows, for few,
33 and 64 snapshots and at the smallest and odd-shaped lattices, against the int64 Gram: equal."""
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
