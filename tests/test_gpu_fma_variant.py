"""The FP64_FMA path's shifting variant follows from a rule, not from a timing: a context
that was not told a variant does what one pinned to it does, launch for launch and bit
for bit, and can still be given another."""
import pytest

from tests.gpu_helpers import cells_bitwise_equal, particles_bitwise_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cid,grid", [(1, (37, 17)), (4, (64, 61)), (5, (33, 15)), (3, (40, 10, 10)), (2, (33, 8, 9))])
def test_no_timed_choice(gpu_mod, cid, grid):
    M = gpu_mod
    cs, p, c = M.make_case(cid, grid)
    out = []
    for pinned in (False, True):
        g = M.MPM(cs, 2)
        if pinned:
            g.tune("pst", 8)
        g.upload_particles(p)
        g.upload_cells(c)
        n = []
        for steps in (1, 1, 4):
            g.advance(steps)
            g.sync()
            n.append(g.launch_count())
        assert g.tune() == 8
        g.tune("pst", -1)
        g.advance(1)
        g.sync()
        assert g.tune() == 8
        n.append(g.launch_count())
        out.append((g.download_particles(), g.download_cells(), n))
        assert g.tune("pst", 2) == 2
        g.advance(1)
        g.sync()
        g.close()
    (pa, ca, na), (pb, cb, nb) = out
    assert na == nb
    assert particles_bitwise_equal(pa, pb) == [] and cells_bitwise_equal(ca, cb) == []
