"""Split and merge passes whose slots end at, before and after a tile of 2048 of the
rank prefix, with events in every tile: bit for bit the oracle."""
import numpy as np
import pytest

from tests.gpu_helpers import particles_bitwise_equal
from tests.test_gpu_split_merge import _event_state, _lists_match

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cid,grid,inlet,outlet", [(1, (9, 7), 0, 0), (4, (32, 16), 0, 0), (4, (33, 31), 0, 0),
                                                   (3, (16, 4, 4), 9, 7), (2, (25, 5, 5), 11, 5)])
def test_events_at_tile_edges(gpu_mod, oracle_mod, cid, grid, inlet, outlet):
    M, O = gpu_mod, oracle_mod
    cs, po, co, off, ent = _event_state(M, O, cid, grid, 2, seed=7, frac=0.04, outlet=outlet, inlet=inlet)
    g, o = M.MPM(cs, 0), O.Oracle(cs)
    for x in (g, o):
        x.upload_particles(po)
        x.upload_cells(co)
        x.upload_lists(off, ent)
        x.Map_the_particle_to_tree()
    for call in ("Split_particle_fast",) + ("Merge_particle_fast",) * 3:
        getattr(g, call)()
        getattr(o, call)()
        g.sync()
        assert particles_bitwise_equal(g.download_particles(), o.download_particles()) == [], call
        gl, ol = g.download_cell_lists(), o.download_cell_lists()
        assert np.array_equal(gl[0], ol[0]) and np.array_equal(gl[1], ol[1]), call
    sg, so = g.stats(), o.stats()
    assert sg["n_split"] > 0 and sg["n_merge"] > 0
    for k in ("n_split", "n_merge", "n_inlet", "n_outlet", "n_affected"):
        assert sg[k] == so[k], k
    assert _lists_match(g, o) == 0
