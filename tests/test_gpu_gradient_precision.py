"""The gradient kernel keeps FP32's precision over the batch: against the NumPy FP64
restatement within a bound that does not grow with the batch.

A sample's term dz a of a weight's gradient comes through at most 400 rounded operations (three
products of 64 terms each way), whose errors add as a random walk: sqrt(400) u = 20 u of the term,
u = 2^-24, independent from sample to sample.  So a layer's error is about 20 u of Q, the root of
the sum of its squared terms; four times that is allowed."""
import ctypes as C

import numpy as np
import pytest
from tests import mlp_ref as R

pytestmark = pytest.mark.gpu


def _terms(p, X, T, bf16):
    """Root of the summed squares of the samples' terms, laid out as the parameters."""
    layers, (_, _, my, sy) = R.unpack(p, bf16)
    Y, acts = R.forward(p, X, bf16)
    dz = 2.0 * (Y - (T.astype(np.float64) - my) / sy) / Y.size
    out = []
    for li in range(len(layers) - 1, -1, -1):
        out = [np.sqrt((dz * dz).T @ (acts[li] * acts[li])).ravel(), np.sqrt((dz * dz).sum(0))] + out
        if li:
            dz = (dz @ layers[li][0]) * (1.0 - acts[li] * acts[li])
    return np.concatenate(out)


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n", [33, 500, 304 * 32 + 1, 32768])
def test_gradient_precision(gpu_mod, n, bf16):
    import torch
    from pgdg_p2_gb300 import surrogate as S
    p = S.load_default()
    rng = np.random.default_rng(n + 1)
    norm = p[S.NPARAM:]
    X = (norm[:12] + norm[12:24] * rng.standard_normal((n, 12))).astype(np.float32)
    T = (norm[24:26] + norm[26:28] * rng.standard_normal((n, 2))).astype(np.float32)
    net = S.Surrogate(p, bf16=bf16)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    torch.cuda.synchronize()
    loss, g = C.c_double(), np.zeros(S.NPARAM, np.float32)
    assert gpu_mod.lib().pgdg_surrogate_gradients(net.h, Xd.data_ptr(), Td.data_ptr(), n,
                                                  g.ctypes.data_as(C.POINTER(C.c_float)), C.byref(loss)) == 0
    net.close()
    _, gr = R.loss_grad(p, X, T, bf16)
    q, o = _terms(p, X, T, bf16), 0
    for a, b in R.SHAPES:
        for size in (a * b, a):
            sl = slice(o, o + size)
            assert np.linalg.norm(g[sl] - gr[sl]) <= 80 * 2.0 ** -24 * np.linalg.norm(q[sl]), (a, b, size)
            o += size
