"""Exact path with particles far outside the box: binning clamps them into the edge
cells, and the shifting sum takes the neighbours within 2h of them as the oracle does,
pairs a little on either side of 2h among them."""
import numpy as np
import pytest

from tests.gpu_helpers import particles_bitwise_equal

pytestmark = pytest.mark.gpu


def far_pairs(cs, p, grid, shift, seed=3):
    """Pairs from the last column of cells, moved out by `shift` cells, one partner
    2h (1 + e) from the other, |e| from 1e-6 to 1e-2, mostly along x."""
    rng = np.random.default_rng(seed)
    dim = cs.dim
    ps = np.array([(cs.box_r[d] - cs.box_l[d]) / grid[d] for d in range(dim)])
    last = np.flatnonzero(p.coord[:, 0] >= cs.box_r[0] - ps[0])
    idx = rng.permutation(last)[:len(last) // 4 * 2]  # half of them stay
    a, b = idx[::2], idx[1::2]
    p.coord[a, 0] += shift * ps[0] + rng.uniform(0, 40, len(a)) * ps[0]
    e = rng.choice([-1.0, 1.0], len(a)) * 10.0 ** rng.uniform(-6, -2, len(a))
    t = rng.uniform(-0.3, 0.3, (len(a), dim - 1))
    r = 2.0 * p.h[a] * (1.0 + e)
    p.coord[b, 1:dim] = np.clip(p.coord[a, 1:dim] + r[:, None] * t, np.array(cs.box_l[1:dim]) + 1e-3 * ps[1:],
                                np.array(cs.box_r[1:dim]) - 1e-3 * ps[1:])
    dy = ((p.coord[b, 1:dim] - p.coord[a, 1:dim]) ** 2).sum(1)
    p.coord[b, 0] = p.coord[a, 0] + np.sqrt(r * r - dy)
    return a, b


@pytest.mark.parametrize("shift", [3.0, 1e3, 1e5])
@pytest.mark.parametrize("cid,grid", [(1, (20, 9)), (3, (16, 5, 4)), (3, (9, 6, 3))])
def test_far_pairs_bitwise(gpu_mod, oracle_mod, cid, grid, shift):
    M, O = gpu_mod, oracle_mod
    cs, p, c = M.make_case(cid, grid)
    a, _ = far_pairs(cs, p, grid, shift)
    assert len(a) > 8
    g, o = M.MPM(cs, 0), O.Oracle(cs)
    for x in (g, o):
        x.upload_particles(p)
        x.upload_cells(c)
        x.Set_timestep()
        x.set_iterate(1)
        x.Used_state_update()
        x.Map_the_particle_to_tree()
        x.Refresh_membership()
        x.Refresh_neighbors()
        x.MLS_P2G()
        x.Calculate_limiter()
        x.Grid_acceleration()
        x.Update_grid(0)
        x.Update_particle(0)
    g.sync()
    q = o.download_particles()
    assert np.isfinite(q.tv[:, :cs.dim]).all()
    assert particles_bitwise_equal(g.download_particles(), q) == []
