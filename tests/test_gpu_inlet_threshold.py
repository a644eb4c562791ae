"""The inlet's test x - box_l.x >= vol^(1/DIM) of marked particles, decided in FP32 away from
the threshold: on it and from one unit in the last place to a per cent to either side of it,
over volumes from below the FP32 range's use to the nominal one, bit for bit the oracle on the
exact path and the oracle's count on FP32 values on the mixed path."""
import numpy as np
import pytest

from tests.gpu_helpers import particles_bitwise_equal
from tests.test_gpu_split_merge import _event_state

pytestmark = pytest.mark.gpu
OFFSETS = np.array([0.0] + [s * e for e in (2.0 ** -52, 1e-12, 1e-8, 1e-6, 2.0 ** -23, 9e-5, 1.1e-4, 9.9e-4, 1.01e-3, 1e-2)
                            for s in (-1.0, 1.0)])


@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("cid,grid", [(1, (30, 14)), (4, (24, 25)), (3, (16, 5, 4)), (2, (18, 4, 5))])
def test_inlet_threshold(gpu_mod, oracle_mod, cid, grid, prec):
    M, O = gpu_mod, oracle_mod
    cs, po, co, off, ent = _event_state(M, O, cid, grid, 2, seed=5, frac=0.0)
    rng = np.random.default_rng(cid)
    scale = np.array([1.0, 0.3, 1.4, 1e-3, 1e-12, 1e-27, 1e-34])
    k = len(OFFSETS) * len(scale)
    near = np.argsort(po.coord[:, 0], kind="stable")[:k]
    assert len(near) == k
    e, s = np.tile(OFFSETS, len(scale)), np.repeat(scale, len(OFFSETS))
    vol = cs.p_sz ** cs.dim * s * rng.uniform(0.9, 1.1, k)
    if prec == 1:
        vol = vol.astype(np.float32).astype(np.float64)
    root = vol ** (1.0 / cs.dim)
    po.mark_in[near] = 1
    po.vol[near] = vol
    po.coord[near, 0] = cs.box_l[0] + root * (1.0 + e)
    if prec == 1:
        po.coord[:] = po.coord.astype(np.float32)
        po.vol[:] = po.vol.astype(np.float32)
    g, o = M.MPM(cs, prec), O.Oracle(cs)
    for x in (g, o):
        x.upload_particles(po)
        x.upload_cells(co)
        x.upload_lists(off, ent)
        x.Map_the_particle_to_tree()
        x.Split_particle_fast()
    g.sync()
    so = o.stats()
    assert 0 < so["n_inlet"] < k
    assert g.stats()["n_inlet"] == so["n_inlet"]
    if prec == 0:
        assert particles_bitwise_equal(g.download_particles(), o.download_particles()) == []
