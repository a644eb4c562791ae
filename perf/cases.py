"""The work this library is used for, as cases that can be timed.

A program that uses the library keeps a context, uploads a start state, advances
it by some steps and reads fields back; beside that it solves batches of
two-material Riemann problems and trains the network that seeds them.  Each case
below is one such piece of work, called through the public entry points
(`pgdg_p2_gb300.mpm`, `pgdg_p2_gb300.surrogate` and the C ABI they load).

  kind "steps"      a run from the program's start state: upload it, advance by
                    `steps` steps, read the solution (DG coefficients, volume
                    fractions, pressure, phase flags) and the particles
                    (position, velocity, volume, density, phase) back into
                    page-locked host memory
  kind "exchange"   the same with few steps and the whole state read back: a
                    driver that keeps its state on the host
  kind "riemann"    a batch of two-material Riemann problems on device buffers,
                    from the plain or the learned seed
  kind "gradient"   loss and weight gradients of the seed network on one batch

Workloads (`config`): 1 triple point, 2 shock and helium cylinder, 3 shock and
helium sphere, 4 underwater explosion, 5 triple point with three materials.
The simulations start from developed states, not from the lattice at rest: the
shock of workloads 2 and 3 is about to reach the bubble and the fluid behind it
is compressed, particles are disordered, and every field carries small smooth
waves drawn from the seed.  Every pass starts from the same state, so a pass is
the same work however often it is repeated (the method itself, and so the amount
of splitting and merging, changes along a run).

The mixed path keeps its state in FP32 and the host arrays are FP64, so a
program that goes on in FP32 narrows what it reads: the outputs of the mixed
cases come back as FP32.  The FP64 paths' outputs come back as FP64.
"""
import ctypes as C
import math

import numpy as np
import torch

from pgdg_p2_gb300 import mpm as M
from pgdg_p2_gb300 import surrogate as S
from pgdg_p2_gb300.abi import PREC_FP64, PREC_FP64_FMA, PREC_MIXED, Cells, Particles, check, pgdg_cells, pgdg_particles

PRECISIONS = {"mixed": PREC_MIXED, "fp64": PREC_FP64, "fp64_fma": PREC_FP64_FMA}
DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _steps(name, config, grid, precision="mixed", learned=False, steps=12):
    return {"name": name, "kind": "steps", "config": config, "nx": grid[0], "ny": grid[1],
            "nz": grid[2] if len(grid) > 2 else 1, "precision": precision, "learned": learned, "steps": steps}


def listed():
    return [
        # the triple point at its own size: a small run, bound by latency and launches
        _steps("triple_point_112x48", 1, (112, 48)),
        # the same box with three materials (the second library)
        _steps("three_materials_112x48", 5, (112, 48)),
        # the underwater explosion at its own size, stiffened gas, learned seed: the large 2D run
        _steps("underwater_1024x1024_learned", 4, (1024, 1024), learned=True),
        # the spherical bubble on the sample grid that accuracy runs use
        _steps("sphere_96x24x24_learned", 3, (96, 24, 24), learned=True),
        # the cylindrical bubble on a grid that divides nothing, plain seed, problems solved inline
        _steps("cylinder_171x45x39", 2, (171, 45, 39)),
        # the spherical bubble at full size: the library's headline workload
        _steps("sphere_384x96x96_learned", 3, (384, 96, 96), learned=True),
        # the plain FP64 path that the mixed one is judged against
        _steps("sphere_64x16x16_fp64_fma", 3, (64, 16, 16), precision="fp64_fma", steps=3),
        # the exact-order FP64 path that a port is verified with, bit for bit
        _steps("cylinder_48x12x12_fp64", 2, (48, 12, 12), precision="fp64", steps=3),
        # a driver that holds its state on the host: up, three steps, down
        {"name": "exchange_128x32x32_learned", "kind": "exchange", "config": 3, "nx": 128, "ny": 32, "nz": 32,
         "precision": "mixed", "learned": True, "steps": 3},
        # batched Riemann problems: a stage's worth from the plain seed, and a large batch from the learned one
        {"name": "riemann_65537_plain", "kind": "riemann", "n": 65537, "learned": False, "variant": 1},
        {"name": "riemann_4194304_learned", "kind": "riemann", "n": 1 << 22, "learned": True, "variant": 0},
        # one batch of the seed network's training
        {"name": "gradient_8192", "kind": "gradient", "n": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps"] * 7 + ["exchange", "riemann", "riemann", "gradient"])
    if kind == "riemann":
        return {"kind": kind, "n": _log_int(rng, 1000, 1 << 22), "learned": rng.random() < 0.5,
                "variant": rng.randrange(2)}
    if kind == "gradient":
        return {"kind": kind, "n": _log_int(rng, 500, 32768)}
    if kind == "exchange":
        m = _log_int(rng, 8, 32)
        return {"kind": kind, "config": rng.choice([2, 3]), "nx": 4 * m + rng.randrange(-2, 3), "ny": m, "nz": m,
                "precision": "mixed", "learned": rng.random() < 0.5, "steps": 3}
    config = rng.choice([1, 2, 2, 3, 3, 3, 4, 5])
    precision = rng.choice(["mixed"] * 4 + ["fp64_fma", "fp64"])
    learned = precision == "mixed" and config != 5 and rng.random() < 0.5
    case = {"kind": kind, "config": config, "precision": precision, "learned": learned,
            "steps": 12 if precision == "mixed" else 3}
    if config in (2, 3):
        m = _log_int(rng, 10, 80 if precision == "mixed" else 16)
        return dict(case, nx=4 * m + rng.randrange(-2, 3), ny=m + rng.randrange(2), nz=m + rng.randrange(2))
    if config == 4:
        m = _log_int(rng, 64, 1000 if precision == "mixed" else 256)
        return dict(case, nx=m, ny=m + rng.randrange(2), nz=1)
    m = _log_int(rng, 24, 200 if precision == "mixed" else 100)
    return dict(case, nx=int(m * 7 / 3) + rng.randrange(2), ny=m, nz=1)


# ---------------------------------------------------------------------------
# a developed state of each workload
# ---------------------------------------------------------------------------
SHOCK_X = 1.2  # workloads 2 and 3: the bubble (centre 1.5, radius 0.25) begins at 1.25


def _post_shock():
    """(density, velocity, pressure) behind a Mach 1.22 shock into air (gamma 1.4, rho 1, p 1)."""
    g, m2 = 1.4, 1.22 * 1.22
    p = 1.0 + 2.0 * g / (g + 1.0) * (m2 - 1.0)
    rho = (g + 1.0) * m2 / ((g - 1.0) * m2 + 2.0)
    return rho, 1.22 * math.sqrt(g) * (1.0 - 1.0 / rho), p


def _regions(config, x):
    """phase (1-based), density, pressure and x velocity at positions x [n, 3]."""
    n = x.shape[0]
    one = torch.ones(n, dtype=torch.float64, device=x.device)
    phase = torch.ones(n, dtype=torch.int32, device=x.device)
    rho, p, u = one.clone(), one.clone(), torch.zeros_like(one)
    if config in (2, 3):
        r2, u2, p2 = _post_shock()
        d2 = (x[:, 0] - 1.5) ** 2 + x[:, 1] ** 2 + (x[:, 2] ** 2 if config == 3 else 0.0)
        bubble, behind = d2 < 0.0625, x[:, 0] < SHOCK_X
        rho = torch.where(behind, r2, 1.0).double()
        p, u = torch.where(behind, p2, 1.0).double(), torch.where(behind, u2, 0.0).double()
        phase[bubble] = 2
        rho[bubble], p[bubble], u[bubble] = 0.138, 1.0, 0.0
    elif config == 4:
        bubble = x[:, 0] ** 2 + x[:, 1] ** 2 < 0.09
        rho, p = 1000.0 * one, 1e5 * one
        phase[bubble] = 2
        rho[bubble], p[bubble] = 1270.0, 8.29e8
    else:
        left, low = x[:, 0] < 1.0, x[:, 1] < 1.5
        p = torch.where(left, 1.0, 0.1).double()
        rho = torch.where(~left & ~low, 0.125, 1.0).double()
        phase[~left & ~low] = 2
        if config == 5:
            phase[left] = 3
    return phase, rho, p, u


def _state(cs, config, seed):
    """Particles of a developed state on the device: a dict of FP64 tensors and the phase."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    dim = cs.dim

    def axis(lo, hi, dp):
        n = max(1, round((hi - lo) / dp))
        return lo + (torch.arange(n, dtype=torch.float64, device=DEV) + 0.5) * ((hi - lo) / n), (hi - lo) / n

    dp = cs.p_sz
    if config in (2, 3):
        # behind the shock the lattice is compressed along x as the fluid is
        xa, da = axis(cs.box_l[0], SHOCK_X, dp / _post_shock()[0])
        xb, db = axis(SHOCK_X, cs.box_r[0], dp)
        gx = torch.cat([xa, xb])
        wx = torch.cat([torch.full_like(xa, da), torch.full_like(xb, db)])
    else:
        gx, da = axis(cs.box_l[0], cs.box_r[0], dp)
        wx = torch.full_like(gx, da)
    gy, wy = axis(cs.box_l[1], cs.box_r[1], dp)
    gz, wz = axis(cs.box_l[2], cs.box_r[2], dp) if dim == 3 else (torch.zeros(1, dtype=torch.float64, device=DEV), 1.0)
    n = gx.numel() * gy.numel() * gz.numel()
    x = torch.stack(torch.meshgrid(gx, gy, gz, indexing="ij"), -1).reshape(n, 3)
    vol = (wx * (wy * wz))[:, None, None].expand(-1, gy.numel(), gz.numel()).reshape(n).clone()
    x[:, :dim] += (0.06 * dp) * (torch.rand((n, dim), generator=gen, dtype=torch.float64, device=DEV) - 0.5)
    phase, rho, p, u = _regions(config, x)
    lut = lambda a: torch.tensor(list(a), dtype=torch.float64, device=DEV)[(phase - 1).long()]  # noqa: E731
    gam, pinf = lut(cs.gamma), lut(cs.pinf)
    span = torch.tensor([cs.box_r[d] - cs.box_l[d] if d < dim else 1.0 for d in range(3)], dtype=torch.float64, device=DEV)

    def wave():
        s = torch.zeros(n, dtype=torch.float64, device=DEV)
        for _ in range(3):
            k = torch.randint(1, 4, (3,), generator=gen, device=DEV).double() / span
            k[dim:] = 0
            ph = 2 * math.pi * torch.rand(1, generator=gen, dtype=torch.float64, device=DEV)
            s += torch.cos(2 * math.pi * (x @ k) + ph) / 3
        return s

    c = torch.sqrt(gam * (p + pinf) / rho)
    amp = 0.02 * p / (rho * c)  # acoustic: velocity waves of the size that 2% of the pressure drives
    v = torch.zeros((n, 3), dtype=torch.float64, device=DEV)
    v[:, 0] = u
    for d in range(dim):
        v[:, d] += amp * wave()
    s = 0.02 * wave()
    rho = rho * (1.0 + s * p / (gam * (p + pinf)))
    p = p * (1.0 + s)
    E = (p + gam * pinf) / (gam - 1.0) + 0.5 * rho * (v * v).sum(1)
    h = 1.6 * (vol.sqrt() if dim == 2 else vol.pow(1.0 / 3.0))
    return {"coord": x, "v": v, "tv": v.clone(), "rhov": rho[:, None] * v, "vol": vol, "mass": vol * rho, "h": h,
            "P": p, "rho": rho, "E": E, "c": torch.sqrt(gam * (p + pinf) / rho), "phase": phase}


# ---------------------------------------------------------------------------
# host arrays of the C ABI
# ---------------------------------------------------------------------------
def _pinned(shape, dtype):
    n = max(1, int(np.prod(shape)) * np.dtype(dtype).itemsize)
    return torch.empty(n, dtype=torch.uint8, pin_memory=True).numpy()[:n].view(dtype).reshape(shape)


def _pointers(struct, arrays):
    ctype = {np.dtype(np.float64): C.c_double, np.dtype(np.int32): C.c_int32, np.dtype(np.uint64): C.c_uint64}
    for k, a in arrays.items():
        setattr(struct, k, a.ctypes.data_as(C.POINTER(ctype[a.dtype])))
    return struct


def _to_host(state):
    out = {}
    for k, t in state.items():
        a = _pinned(tuple(t.shape), np.int32 if k == "phase" else np.float64)
        torch.from_numpy(a).copy_(t)
        out[k] = a
    return out


def _as_read(arrays, mixed):
    """What the program goes on with: FP32 on the device (mixed path) or the FP64 host arrays."""
    out = {}
    for k, a in arrays.items():
        t = torch.from_numpy(a)
        out[k] = t.to(DEV, non_blocking=True).float() if mixed and t.is_floating_point() else t
    return out


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
class _Run:
    """A simulation's context, with what its program keeps."""

    def start(self):
        """Back to the start state."""
        check(self.lib.pgdg_upload_particles(self.g.h, C.byref(self.p_start)), "upload_particles")
        check(self.lib.pgdg_upload_cells(self.g.h, C.byref(self.c_start)), "upload_cells")
        self.g.set_iterate(0)


def _simulation(case, seed):
    r = _Run()
    grid = (case["nx"], case["ny"], case["nz"])
    r.cs = cs = M.case_setup(case["config"], grid)
    state = _state(cs, case["config"], seed)
    n = state["phase"].numel()
    r.g = M.MPM(cs, PRECISIONS[case["precision"]], capacity=n * 3 // 2 + 4096)
    r.lib = M.lib(cs.nfld)
    r.keep = _to_host(state)
    del state
    r.p_start = _pointers(pgdg_particles(), r.keep)
    r.p_start.n = n
    # the cells as the case starts them (the projection fills them on the first step)
    cells = _default_cells(cs)
    r.keep_cells = cells
    r.c_start = _pointers(pgdg_cells(), cells)
    r.c_start.n = cs.ncells
    if case["learned"]:
        r.net = S.Surrogate(S.load_default(), tc=True)
        r.g.set_surrogate(r.net)
    r.mixed, r.steps, r.room = case["precision"] == "mixed", case["steps"], n + n // 4 + 4096
    # a first short run on this context: the library chooses its kernels here
    r.start()
    r.g.advance(3)
    r.g.sync()
    return r


def _default_cells(cs):
    nc, nf, dim = cs.ncells, cs.nfld, cs.dim
    ini, c0 = np.array(list(cs.ini_rho)[:nf]), np.array(list(cs.c_ini)[:nf])
    shape = {"rho": (nf,), "rhov": (nf, 3), "E": (nf,), "c": (nf,), "alph": (nf,), "coef": (nf, dim + 2, dim + 1),
             "v": (3,), "P": (), "ph_state": (nf,), "ph_state_b": (nf,)}
    out = {k: _pinned((nc, *sh), np.int32 if k.startswith("ph") else np.float64) for k, sh in shape.items()}
    for k, a in out.items():
        a[...] = {"rho": ini, "c": c0, "ph_state": 1}.get(k, 0)
    return out


def prepare(case, seed):
    if case["kind"] == "riemann":
        return _riemann(case, seed)
    if case["kind"] == "gradient":
        return _gradient(case, seed)
    r = _simulation(case, seed)
    dim, nf, nc = r.cs.dim, r.cs.nfld, r.cs.ncells
    if case["kind"] == "exchange":
        r.p_out, r.c_out = Particles(r.room, dim, _pinned), Cells(nc, dim, _pinned, nf)
        return r
    r.cells = {"coef": _pinned((nc, nf, dim + 2, dim + 1), np.float64), "alph": _pinned((nc, nf), np.float64),
               "P": _pinned((nc,), np.float64), "ph_state": _pinned((nc, nf), np.int32)}
    r.parts = {"coord": _pinned((r.room, 3), np.float64), "v": _pinned((r.room, 3), np.float64),
               "vol": _pinned((r.room,), np.float64), "rho": _pinned((r.room,), np.float64),
               "phase": _pinned((r.room,), np.int32)}
    r.c_read, r.p_read = _pointers(pgdg_cells(), r.cells), _pointers(pgdg_particles(), r.parts)
    r.c_read.n = nc
    return r


def run(s):
    if isinstance(s, dict):
        return _run_riemann(s) if s["kind"] == "riemann" else _run_gradient(s)
    s.start()
    s.g.advance(s.steps)
    if hasattr(s, "p_out"):
        s.p_out.n = s.room
        p, c = s.g.download_particles(s.p_out), s.g.download_cells(s.c_out)
        particles = {k: getattr(p, k)[:p.n] for k in ("coord", "v", "rhov", "vol", "mass", "h", "P", "rho", "E", "c",
                                                      "phase", "mark_in")}
        cells = {k: getattr(c, k) for k in ("rho", "rhov", "E", "c", "alph", "coef", "v", "P", "ph_state", "used")}
    else:
        s.p_read.n = s.room
        check(s.lib.pgdg_download_particles(s.g.h, C.byref(s.p_read)), "download_particles")
        check(s.lib.pgdg_download_cells(s.g.h, C.byref(s.c_read)), "download_cells")
        particles = {k: a[:int(s.p_read.n)] for k, a in s.parts.items()}
        cells = s.cells
    return {"cells": _as_read(cells, s.mixed), "particles": _as_read(particles, s.mixed)}


def _log_uniform(gen, n, lo, hi):
    return 10.0 ** (lo + (hi - lo) * torch.rand(n, generator=gen, dtype=torch.float64, device=DEV))


def _riemann(case, seed):
    """Problems of the batched micro-benchmark's distribution: densities over five decades, a
    pressure ratio over seven around 1e5, all pairs of four materials."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    n = case["n"]
    rl, rr = _log_uniform(gen, n, -2, 3), _log_uniform(gen, n, -2, 3)
    high = 1e5 * _log_uniform(gen, n, -3, 4)
    swap = torch.rand(n, generator=gen, device=DEV) < 0.5
    base = torch.full_like(high, 1e5)
    u = 1000.0 * torch.rand((2, n), generator=gen, dtype=torch.float64, device=DEV) - 500.0
    s = {"kind": "riemann", "n": n, "variant": case["variant"],
         "in6": torch.stack([u[0], u[1], torch.where(swap, high, base), torch.where(swap, base, high), rl, rr], 1).contiguous(),
         "mat": torch.randint(0, 4, (n, 2), generator=gen, device=DEV).to(torch.int8).contiguous(),
         "gam": torch.tensor(S.C5_GAMMA, device=DEV), "pinf": torch.tensor(S.C5_PINF, device=DEV),
         "out": torch.empty((n, 3), dtype=torch.float64, device=DEV),
         "iters": torch.empty(n, dtype=torch.int32, device=DEV),
         "net": S.Surrogate(S.load_default(), tc=True) if case["learned"] else None}
    return s


def _run_riemann(s):
    check(M.lib().pgdg_mgfm_batched(s["net"].h if s["net"] else None, s["in6"].data_ptr(), s["mat"].data_ptr(),
                                    s["gam"].data_ptr(), s["pinf"].data_ptr(), 4, s["variant"], s["out"].data_ptr(),
                                    s["iters"].data_ptr(), s["n"]), "mgfm_batched")
    return {"star": s["out"], "iterations": s["iters"]}


def _gradient(case, seed):
    """A training batch: the network's own feature and target ranges."""
    gen = torch.Generator(device=DEV).manual_seed(int(seed))
    params = S.load_default()
    norm = torch.tensor(params[S.NPARAM:], device=DEV)
    n = case["n"]
    mx, sx = norm[:S.NI], norm[S.NI:2 * S.NI]
    my, sy = norm[2 * S.NI:2 * S.NI + S.NO], norm[2 * S.NI + S.NO:]
    return {"kind": "gradient", "n": n, "net": S.Surrogate(params), "grad": np.zeros(S.NPARAM, np.float32),
            "X": (mx + sx * torch.randn((n, S.NI), generator=gen, device=DEV)).contiguous(),
            "T": (my + sy * torch.randn((n, S.NO), generator=gen, device=DEV)).contiguous()}


def _run_gradient(s):
    loss = C.c_double()
    check(M.lib().pgdg_surrogate_gradients(s["net"].h, s["X"].data_ptr(), s["T"].data_ptr(), s["n"],
                                           s["grad"].ctypes.data_as(C.POINTER(C.c_float)), C.byref(loss)), "gradients")
    return {"gradients": s["grad"], "loss": np.float32(loss.value)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    if case["kind"] == "riemann":
        # six inputs and two materials in, three states and the count out; five
        # Newton iterations of two shock speeds, their Jacobians and the density
        return {"bytes": case["n"] * (48 + 2 + 24 + 4), "flops": case["n"] * 5 * 60}
    if case["kind"] == "gradient":
        return {"bytes": case["n"] * 4 * (S.NI + S.NO) + 8 * S.NPARAM, "flops": case["n"] * 6 * S.NPARAM}
    d3 = case["config"] in (2, 3)
    real = 4 if case["precision"] == "mixed" else 8
    cells = case["nx"] * case["ny"] * case["nz"]
    parts = cells * (8 if d3 else 4)
    dim = 3 if d3 else 2
    nf = 3 if case["config"] == 5 else 2
    # per step: each particle's and each cell's state read once and written once
    pvals = 4 * dim + 8 + (dim + 2) * dim
    cvals = nf * ((dim + 2) * (dim + 1) + dim + 4) + dim + 1
    nbytes = case["steps"] * 2 * real * (parts * pvals + cells * cvals)
    # two stages; per cell and stage about 70 kflop in 3D and 11 kflop in 2D,
    # most of it in the neighbour sums (147 and 32 members a particle)
    flops = case["steps"] * 2 * cells * (70e3 if d3 else 11e3)
    # the start state in, the fields out
    start = 8 * (parts * 19 + cells * nf * ((dim + 2) * (dim + 1) + 8))
    read = 8 * (parts * 8 + cells * (nf * ((dim + 2) * (dim + 1) + 1) + 1))
    if case["kind"] == "exchange":
        read = start + 8 * (parts * (dim + 2) * dim + cells * nf * (dim + 2) * (dim + 2))
    return {"bytes": nbytes + start + read, "flops": flops}


# ---------------------------------------------------------------------------
# what the outputs are in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed)
    if case["kind"] == "riemann" and not case["learned"]:
        return {"star": _exact_newton(_riemann(case, seed)), "iterations": None}
    return None  # whole steps of the method have no short restatement


def _exact_newton(s):
    """The plain two-shock Newton solve of every problem, FP64, all problems at once."""
    ul, ur, pl, pr, rl, rr = (s["in6"][:, k] for k in range(6))
    m = s["mat"].long()
    gl, gr, il, ir = s["gam"][m[:, 0]], s["gam"][m[:, 1]], s["pinf"][m[:, 0]], s["pinf"][m[:, 1]]
    if s["variant"] == 0:
        pl, pr, rl, rr = (t.clamp_min(1e-10) for t in (pl, pr, rl, rr))
        p = torch.maximum(pl, pr)
    else:
        pl, pr = pl.clamp_min(0.0), pr.clamp_min(0.0)
        p = 0.5 * (pl + pr)
    tol = (1e-3 * (ul - ur).abs()).clamp_min(1e-8)
    rho_s, u_s = torch.zeros_like(p), torch.zeros_like(p)
    live = torch.ones_like(p, dtype=torch.bool)

    def speed(r, q, g, i):
        return torch.sqrt(0.5 * r * ((g + 1.0) * p + (g - 1.0) * q + 2.0 * g * i))

    def slope(w, q, r, g):
        return 1.0 / w - (p - q) / (w * w) * r * (g + 1.0) / 4.0 / w

    for _ in range(50):
        wl, wr = speed(rl, pl, gl, il), speed(rr, pr, gr, ir)
        num = (gl + 1) * p + (gl - 1) * pl + 2 * gl * il
        den = (gl - 1) * p + (gl + 1) * pl + 2 * gl * il
        rho_s = torch.where(live, rl * num / den, rho_s)
        u_s = torch.where(live, ul - (p - pl) / wl, u_s)
        f = ul - ur - (p - pl) / wl - (p - pr) / wr
        dp = f / (slope(wl, pl, rl, gl) + slope(wr, pr, rr, gr))
        cap = 0.6 * p
        dp = torch.where(dp.abs() > cap, torch.copysign(cap, dp), dp)
        p = torch.where(live, (p + dp).clamp_min(1e-8), p)
        live = live & (f.abs() > tol)
        if not bool(live.any()):
            break
    if s["variant"] == 1:
        wl = speed(rl, pl, gl, il)
        u_s = ul - (p - pl) / wl
    return torch.stack([rho_s, p, u_s], 1)


def _exact_gradient(case, seed):
    s = _gradient(case, seed)
    params = torch.tensor(S.load_default(), device=DEV)
    sizes = [(S.NH, S.NI), (S.NH, S.NH), (S.NH, S.NH), (S.NO, S.NH)]
    w, b, o = [], [], 0
    for j, k in sizes:
        # weights are held in BF16 on the forward and backward passes, biases in FP32
        w.append(params[o:o + j * k].bfloat16().double().reshape(j, k).requires_grad_())
        b.append(params[o + j * k:o + j * k + j].double().requires_grad_())
        o += j * k + j
    norm = params[S.NPARAM:].double()
    a = (s["X"].double() - norm[:S.NI]) / norm[S.NI:2 * S.NI]
    t = (s["T"].double() - norm[2 * S.NI:2 * S.NI + S.NO]) / norm[2 * S.NI + S.NO:]
    for k in range(4):
        a = a @ w[k].T + b[k]
        a = torch.tanh(a) if k < 3 else a
    loss = ((a - t) ** 2).mean()
    loss.backward()
    grad = torch.cat([g for k in range(4) for g in (w[k].grad.reshape(-1), b[k].grad)])
    return {"gradients": grad, "loss": loss.detach()}
