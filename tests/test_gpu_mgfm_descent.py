"""The MGFM solve's replayed descent and shared reciprocals against the oracle's
plain 50-iteration loop, bit for bit: problems without a positive root from
every starting pressure, f(1e-8) on either side of the tolerance, the iteration
cap reached on the way down, zero and tiny pressures and densities, and batch
sizes around the sorted path's limit."""
import numpy as np
import pytest

from tests.test_gpu_mgfm import _run_gpu

pytestmark = pytest.mark.gpu
GAM = np.array([1.4, 1.648, 7.15, 2.0])
PINF = np.array([0.0, 0.0, 3.309e8, 0.0])


def _f0(in6, mat):
    """f(1e-8) of the two-shock relation."""
    ul, ur, pl, pr, rl, rr = (in6[:, k] for k in range(6))
    out = ul - ur
    for p, r, m in ((pl, rl, mat[:, 0]), (pr, rr, mat[:, 1])):
        g, i = GAM[m], PINF[m]
        out = out - (1e-8 - p) / np.sqrt(0.5 * r * ((g + 1) * 1e-8 + (g - 1) * p + 2 * g * i))
    return out


def _problems(kind, n, seed):
    rng = np.random.default_rng(seed)
    mat = rng.integers(0, 4, (n, 2)).astype(np.int8)
    lo, hi = {"ordinary": (2, 7), "high": (7, 14), "low": (-12, 0), "cap": (11, 18)}.get(kind, (2, 7))
    p = 10.0 ** rng.uniform(lo, hi, (n, 2))
    r = 10.0 ** rng.uniform(-3, 3, (n, 2))
    if kind == "low":
        r = 10.0 ** rng.uniform(-12, 0, (n, 2))
        p[::7, 0] = 0.0
        p[::5, 1] = 0.0
    u = rng.uniform(-500, 500, (n, 2))
    in6 = np.stack([u[:, 0], u[:, 1], p[:, 0], p[:, 1], r[:, 0], r[:, 1]], 1)
    if kind != "ordinary":
        # separating fast enough to have no root, by a margin from far beyond to
        # a millionth of the tolerance on either side
        in6[:, 0] = in6[:, 1] = 0.0
        gap = _f0(in6, mat)
        frac = rng.choice([1.5, 1.1, 1.002, 1.001, 1.000999, 1.0 + 1e-9, 1.0, 0.999], n)
        in6[:, 1] = gap * frac
    return in6, mat


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("kind", ["ordinary", "edge", "high", "low", "cap"])
def test_descent_bitwise(gpu_mod, oracle_mod, kind, variant):
    in6, mat = _problems(kind, 1 << 14, 3 + variant)
    og, ig = _run_gpu(gpu_mod, in6, mat, GAM, PINF, variant)
    oo, io = oracle_mod.mgfm_batched(in6, mat, GAM, PINF, variant)
    assert np.array_equal(ig, io)
    # the bits of every number; a NaN's own sign and payload differ between processors
    assert np.array_equal(np.isnan(og), np.isnan(oo))
    assert og[~np.isnan(og)].tobytes() == oo[~np.isnan(oo)].tobytes()
    if kind in ("edge", "high"):
        assert (io == 50).mean() > 0.1  # the descent is what this is about


@pytest.mark.parametrize("n", [1, 31, 63, 64, 65, 16384, 16385])
@pytest.mark.parametrize("tc", [False, True])
def test_seeded_batch_sizes(gpu_mod, n, tc):
    """A problem's seeded result does not depend on the batch it is in."""
    from pgdg_p2_gb300 import surrogate as S
    in6, mat = S.c5_problems(20000, seed=9)
    net = S.Surrogate(S.load_default(), tc=tc)
    ref, it = S.mgfm_gpu(in6, mat, GAM, PINF, net)
    out, jt = S.mgfm_gpu(in6[:n], mat[:n], GAM, PINF, net)
    net.close()
    assert np.array_equal(jt, it[:n])
    assert out.tobytes() == np.ascontiguousarray(ref[:n]).tobytes()
