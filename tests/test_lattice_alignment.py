"""Entry points that read a caller's own device lattice take one that starts at any 32-bit word
of a buffer (a view, a slice of an arena) and give the results of the aligned lattice, at every
row width at which the row counts are loaded differently; a pointer off a word boundary is
refused before anything is launched."""
import ctypes as C

import numpy as np
import pytest

EINVAL = 1


def noalloc(lib, ptr, lx, ly):
    out = (C.c_double * 8)()
    return lib.kpzb_roughness_noalloc(C.c_void_p(ptr), lx, ly, out, None), np.array(out[:])


@pytest.mark.parametrize("off", [1, 2, 3])
def test_off_word_pointer_is_refused(kpzb, off):
    from cudakpz_b200._lib import lib
    st, _ = noalloc(lib, 0x10000 + off, 10, 10)
    assert st == EINVAL and b"word boundary" in lib.kpzb_last_error()


@pytest.mark.gpu
@pytest.mark.parametrize("lx,ly", [(8, 6), (10, 9), (12, 4), (13, 4), (14, 5), (16, 2)])
def test_lattice_at_any_word(kpzb, lx, ly):
    import torch
    from cudakpz_b200._lib import lib
    s = kpzb.Scheduler(lx, ly)
    s.supplySeed(3)
    s.setPQ(0.6, 0.3)
    s.mcsPQSyncRng(9)
    words = s.popSystem()
    s.close()
    buf = torch.zeros(words.size + 4, dtype=torch.int32, device="cuda")
    g = kpzb.Gram(lx, ly, 4)
    rough = []
    for off in range(4):
        view = buf[off:off + words.size]
        view.copy_(torch.from_numpy(words.view(np.int32)))
        torch.cuda.synchronize()
        st, got = noalloc(lib, view.data_ptr(), lx, ly)
        assert st == 0, lib.kpzb_last_error()
        rough.append(got)
        g.add_device(view.data_ptr())
    for off in range(1, 4):
        assert np.array_equal(rough[off], rough[0])
    for method in (g.TENSOR, g.INT64):
        G, S1 = g.compute(method)
        assert (G == G[0, 0]).all() and (S1 == S1[0]).all()
    ref = kpzb.Gram(lx, ly, 1)
    ref.add_host(words)
    R, S = ref.compute(ref.INT64)
    assert R[0, 0] == G[0, 0] and S[0] == S1[0]
    with pytest.raises(kpzb.KpzbError) as e:
        g2 = kpzb.Gram(lx, ly, 1)
        g2.add_device(buf.data_ptr() + 2)
    assert e.value.status == EINVAL
    g.close()
    ref.close()
