"""The features p_inf / P0 (quotients formed from a shared reciprocal) against plain
division rounded to FP32, bit for bit: signed zeros, subnormal, tiny and huge numerators
and pressures on either side of the reciprocal's range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_pinf_quotients_bitwise(gpu_mod):
    import torch
    pinf = np.array([0.0, -0.0, 5e-324, 1e-310, 1e-200, 1e-188, 1e-187, 1e-30, 3.0, 3.309e8, 1e100, 1e172, 1e173, 1e300])
    gam = np.full(len(pinf), 1.4)
    rng = np.random.default_rng(11)
    m = np.array([(a, b) for a in range(len(pinf)) for b in range(len(pinf))], np.int8)
    mat = np.repeat(m, 16, 0)
    n = len(mat)
    in6 = np.zeros((n, 6))
    in6[:, 2:4] = 10.0 ** rng.uniform(-10, 12, (n, 2))
    in6[::16, 2] = 1e200
    in6[1::16, 2:4] = 0.0
    in6[:, 4:6] = 10.0 ** rng.uniform(-3, 3, (n, 2))
    d = [torch.from_numpy(a).cuda() for a in (in6, mat, gam, pinf)]
    X = torch.zeros(n, 12, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert gpu_mod.lib().pgdg_surrogate_features(*[t.data_ptr() for t in d], X.data_ptr(), n) == 0
    torch.cuda.synchronize()
    got = X.cpu().numpy()
    il, ir = pinf[mat[:, 0]], pinf[mat[:, 1]]
    P0 = np.maximum(np.maximum(in6[:, 2], 1e-10) + il, np.maximum(in6[:, 3], 1e-10) + ir)
    with np.errstate(over="ignore", under="ignore"):
        for k, inf in ((7, il), (8, ir)):
            want = (inf / P0).astype(np.float32)
            assert np.array_equal(got[:, k].view(np.uint32), want.view(np.uint32)), k
