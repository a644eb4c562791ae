"""The mixed path without a surrogate solves a stage's interface problems as a
batch: bit for bit the inline solve (a queue for one problem), with a queue that
holds some of them and with one that holds all, eager and from graphs."""
import pytest

from tests.gpu_helpers import cells_bitwise_equal, particles_bitwise_equal
from tests.test_gpu_graphs import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cid,grid", [(1, (45, 19, 1)), (5, (45, 19, 1)), (4, (33, 31, 1)), (2, (49, 11, 13)),
                                      (3, (48, 12, 12))])
def test_batched_interface_problems_equal_the_inline_solve(gpu_mod, cid, grid):
    M = gpu_mod
    from pgdg_p2_gb300 import surrogate as S
    from pgdg_p2_gb300.abi import PREC_MIXED
    cs, p, c = M.make_case(cid, grid)
    pa, ca, sa, chosen = _run(M, S, cs, p, c, PREC_MIXED, False, -1, False, iface_cap=1)
    assert sa["mgfm_calls"] > 0
    for graphs, cap in ((False, 101), (False, -1), (True, 101), (True, -1)):
        pb, cb, sb, _ = _run(M, S, cs, p, c, PREC_MIXED, graphs, chosen, False, iface_cap=cap)
        assert particles_bitwise_equal(pb, pa) == [], (graphs, cap)
        assert cells_bitwise_equal(cb, ca) == [], (graphs, cap)
        assert sb["mgfm_calls"] == sa["mgfm_calls"] and sb["mgfm_iters"] == sa["mgfm_iters"], (graphs, cap)
