"""The FP64 residual on either side of the grid size from which a cell is one thread instead of
eight lanes: the exact path bit for bit the oracle, from the queue and (with room for one problem)
inline."""
import pytest

from tests.gpu_helpers import cells_bitwise_equal, particles_bitwise_equal

pytestmark = pytest.mark.gpu
GRIDS = [(1, (184, 79)), (1, (186, 79)), (5, (186, 79)), (3, (78, 20, 20)), (2, (80, 20, 20))]


@pytest.mark.parametrize("iface_cap", [-1, 1])
@pytest.mark.parametrize("cid,grid", GRIDS)
def test_either_side_of_the_line(gpu_mod, oracle_mod, cid, grid, iface_cap):
    M, O = gpu_mod, oracle_mod
    cs, p, c = M.make_case(cid, grid)
    g, o = M.MPM(cs, 0), O.Oracle(cs)
    for x in (g, o):
        x.upload_particles(p)
        x.upload_cells(c)
    if iface_cap > 0:
        g.tune("iface_cap", iface_cap)
    g.advance(1)
    o.advance(1)
    g.sync()
    assert o.stats()["mgfm_calls"] > 0 and g.stats()["mgfm_calls"] == o.stats()["mgfm_calls"]
    assert cells_bitwise_equal(g.download_cells(), o.download_cells()) == []
    assert particles_bitwise_equal(g.download_particles(), o.download_particles()) == []
    g.close()
