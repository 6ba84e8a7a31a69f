"""Device memory that a handle of a tall, narrow lattice holds beside its lattice: the row tables of
the measurements take at most 32 bytes a row (system and snapshot together), so that the tallest
lattices the library accepts still fit with their second buffer."""
import pytest

pytestmark = pytest.mark.gpu


def test_row_tables_of_a_tall_lattice(kpzb):
    import torch
    lx, ly = 8, 22
    kpzb.Scheduler(lx, 6).close()  # the context and the module are there
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    s = kpzb.Scheduler(lx, ly)
    r = s.roughness()
    held = before - torch.cuda.mem_get_info()[0]
    assert abs(r.w2 - 0.25) < 1e-12  # flat: heights 0 and 1 in turn
    s.close()
    assert held <= (1 << (lx + ly - 2)) + 32 * (1 << ly) + (8 << 20)
