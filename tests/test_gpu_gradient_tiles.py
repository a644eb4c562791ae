"""The gradient kernel's tiles of 32 samples: ragged last tiles, one block, every
resident block and several tiles per block, against the NumPy FP64 restatement."""
import ctypes as C

import numpy as np
import pytest
from tests import mlp_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n", [1, 31, 32, 33, 64, 304 * 32 - 1, 304 * 32 + 1, 3 * 304 * 32 + 17])
def test_gradient_at_tile_edges(gpu_mod, n, bf16):
    import torch
    from pgdg_p2_gb300 import surrogate as S
    p = S.load_default()
    rng = np.random.default_rng(n)
    norm = p[S.NPARAM:]
    mx, sx, my, sy = norm[:12], norm[12:24], norm[24:26], norm[26:28]
    X = (mx + sx * rng.standard_normal((n, 12))).astype(np.float32)
    T = (my + sy * rng.standard_normal((n, 2))).astype(np.float32)
    net = S.Surrogate(p, bf16=bf16)
    # one sample more than the batch, with values that would show in the sums
    Xd = torch.from_numpy(np.vstack([X, np.full((1, 12), np.nan, np.float32)])).cuda()
    Td = torch.from_numpy(np.vstack([T, np.full((1, 2), np.nan, np.float32)])).cuda()
    loss, runs = C.c_double(), []
    torch.cuda.synchronize()
    for _ in range(2):
        g = np.zeros(S.NPARAM, np.float32)
        assert gpu_mod.lib().pgdg_surrogate_gradients(net.h, Xd.data_ptr(), Td.data_ptr(), n,
                                                      g.ctypes.data_as(C.POINTER(C.c_float)), C.byref(loss)) == 0
        runs.append((g, loss.value))
    net.close()
    assert np.array_equal(runs[0][0], runs[1][0]) and runs[0][1] == runs[1][1]  # a fixed order of summation
    lr, gr = R.loss_grad(p, X, T, bf16)
    assert abs(runs[0][1] - lr) <= 1e-5 * lr
    # a term passes at most 3 products of 64 terms each way, relative error about 400 u = 2.4e-5 of the
    # sum of its absolute values; random data cancels in the sums over the batch by about sqrt(n):
    # 1e-4 of the layer's norm, the bound of the plain comparison, holds up to n = 300, sqrt(n) above
    tol = 1e-4 * max(1.0, (n / 300) ** 0.5)
    o = 0
    for a, b in R.SHAPES:
        for size in (a * b, a):
            sl = slice(o, o + size)
            assert np.linalg.norm(runs[0][0][sl] - gr[sl]) <= tol * np.linalg.norm(gr[sl]) + 1e-9, (a, b, size)
            o += size
