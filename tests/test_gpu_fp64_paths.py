"""The FP64 paths' shifting kernel and residual at the sizes where their bricks,
groups of lanes and queues end: the exact path against the oracle bit for bit,
the FMA path's cell-scanning variant against its row-scanning one."""
import numpy as np
import pytest

from tests.gpu_helpers import cells_bitwise_equal, particles_bitwise_equal

pytestmark = pytest.mark.gpu


def _pair(M, O, cs, p, c, prec=0, **kw):
    g, o = M.MPM(cs, prec, **kw), O.Oracle(cs)
    for x in (g, o):
        x.upload_particles(p)
        x.upload_cells(c)
    return g, o


@pytest.mark.parametrize("iface_cap", [-1, 1])
@pytest.mark.parametrize("cid,grid", [(3, (9, 3, 5)), (2, (13, 4, 3)), (3, (26, 7, 6)), (1, (19, 9)), (4, (13, 11))])
def test_exact_steps_bitwise(gpu_mod, oracle_mod, cid, grid, iface_cap):
    """Whole steps; with room for one problem every stage is solved inline."""
    cs, p, c = gpu_mod.make_case(cid, grid)
    g, o = _pair(gpu_mod, oracle_mod, cs, p, c)
    if iface_cap > 0:
        g.tune("iface_cap", iface_cap)
    for n in (1, 4):
        g.advance(n)
        o.advance(n)
        g.sync()
        assert particles_bitwise_equal(g.download_particles(), o.download_particles()) == []
        assert cells_bitwise_equal(g.download_cells(), o.download_cells()) == []
    sg, so = g.stats(), o.stats()
    assert sg["mgfm_calls"] == so["mgfm_calls"] and sg["mgfm_iters"] == so["mgfm_iters"]


def _crowd(cs, p, k):
    """Each particle of the left half of the box as k thinner ones side by side."""
    from pgdg_p2_gb300.abi import Particles
    left = np.flatnonzero(p.coord[:, 0] < 0.5 * (cs.box_l[0] + cs.box_r[0]))
    n = p.n + (k - 1) * len(left)
    src = np.concatenate([np.arange(p.n)] + [left] * (k - 1))
    q = Particles(n, cs.dim)
    for name in Particles.NAMES:
        getattr(q, name)[...] = getattr(p, name)[src]
    q.seq[...] = np.arange(n)
    part, thin = np.zeros(n, np.int64), np.zeros(n, bool)
    part[p.n:] = np.repeat(np.arange(1, k), len(left))
    thin[left] = True
    thin[p.n:] = True
    q.coord[thin, 0] += (part[thin] - 0.5 * (k - 1)) * cs.p_sz / k
    for name in ("vol", "mass"):
        getattr(q, name)[thin] /= k
    q.h[thin] /= k ** (1.0 / cs.dim)
    return q


@pytest.mark.parametrize("cid,grid,k", [(3, (16, 5, 4), 2), (3, (16, 4, 4), 7), (1, (20, 9), 3), (1, (20, 9), 5)])
def test_exact_crowded_cells_bitwise(gpu_mod, oracle_mod, cid, grid, k):
    """One stage with cells beyond the staging room and queues that fill: 16 and 56
    particles per cell in 3D, 12 and 20 in 2D."""
    cs, p, c = gpu_mod.make_case(cid, grid)
    p = _crowd(cs, p, k)
    g, o = _pair(gpu_mod, oracle_mod, cs, p, c, capacity=2 * p.n)
    for x in (g, o):
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
    assert particles_bitwise_equal(g.download_particles(), o.download_particles()) == []


@pytest.mark.parametrize("cid,grid", [(3, (26, 7, 6)), (2, (17, 5, 4)), (1, (37, 17)), (4, (33, 31))])
def test_fma_cell_scan_sums_the_same_members(gpu_mod, cid, grid):
    """Variant 8 (cells) against variant 0 (sorted rows): FP64 sums of at most 150
    terms in another order, which cancel to about 1/20 of the terms."""
    M = gpu_mod
    cs, p, c = M.make_case(cid, grid)
    out = []
    for variant in (0, 8):
        g = M.MPM(cs, 2)
        g.upload_particles(p)
        g.upload_cells(c)
        g.tune("pst", variant)
        g.Set_timestep()
        g.set_iterate(1)
        g.MPM_run_simulation(1)
        g.sync()
        q = g.download_particles()
        out.append((q.tv - q.v)[np.argsort(q.seq)])
        g.close()
    a, b = out
    assert a.shape == b.shape
    # tv - v is a difference of stored values: their rounding enters too
    tol = 2 * 150 * 2.0 ** -53 * 20 + 4 * 2.0 ** -53 * float(np.abs(q.v).max()) * a.size / float(np.abs(a).sum())
    assert float(np.abs(a - b).sum()) / float(np.abs(a).sum()) <= tol
