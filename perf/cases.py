"""Performance cases: the calls a flow solver makes through this package.

Each case is one pass through the public Python entry points -- a pressure
solve, a two-phase projection step, a time step of the turbulence or channel
example, a learned guess, a training gradient -- on inputs made on the GPU
from a seed.  ``exact`` restates each of them in plain float64 torch.

Arrays follow NGA2's layout [k, j, i] with ``ghost`` overlap layers.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from nga2_b200 import bbmg as B
from nga2_b200.incomp import HIT, Channel, Incomp
from nga2_b200.learned import LearnedGuess, UNet
from nga2_b200.problems import STC7
from nga2_b200.projection import Projection

DEV = "cuda"
F64 = torch.float64
PERIODIC = (True, True, True)
WALLS_Y = (True, False, True)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest solve a program makes: a coarse two-phase run, all of it latency
        {"name": "drops_32_mixed", "kind": "solve", "problem": "drops", "nx": 32, "ny": 32, "nz": 32, "ghost": 1,
         "mixed": True},
        # the turbulence example's pressure solve at its default size
        {"name": "periodic_64_fp64", "kind": "solve", "problem": "periodic", "nx": 64, "ny": 64, "nz": 64, "ghost": 1,
         "mixed": False},
        # a domain cut to its geometry: odd sizes on several levels, also in a periodic direction
        {"name": "drops_ragged_mixed", "kind": "solve", "problem": "drops", "nx": 150, "ny": 108, "nz": 75,
         "ghost": 2, "mixed": True},
        # the two-phase pressure solve at production size, in the reference's arithmetic and in mixed precision
        {"name": "drops_256_fp64", "kind": "solve", "problem": "drops", "nx": 256, "ny": 256, "nz": 256, "ghost": 1,
         "mixed": False},
        {"name": "drops_256_mixed", "kind": "solve", "problem": "drops", "nx": 256, "ny": 256, "nz": 256, "ghost": 1,
         "mixed": True},
        # a wall-bounded channel on a stretched grid: many iterations
        {"name": "channel_256_fp64", "kind": "solve", "problem": "channel", "nx": 256, "ny": 128, "nz": 128,
         "ghost": 1, "mixed": False},
        # a host (Fortran-side) caller of the linear-solver object: new operator and solve from host arrays
        {"name": "helmholtz_host_128", "kind": "host", "nx": 128, "ny": 128, "nz": 128, "ghost": 1, "mixed": True},
        # a two-phase time step's projection: the density has moved, so the operator is rebuilt
        {"name": "two_phase_128_mixed", "kind": "projection", "nx": 128, "ny": 128, "nz": 128, "ghost": 1,
         "mixed": True},
        # one time step of the forced turbulence example at its default size
        {"name": "hit_step_64", "kind": "hit", "n": 64, "mixed": False},
        # one time step of the channel example (implicit viscous solves) with a spanwise extent
        {"name": "channel_step_128x40x32", "kind": "channel", "nx": 128, "ny": 40, "nz": 32, "mixed": False},
        # the learned initial guess of a 128^3 solve
        {"name": "guess_128", "kind": "guess", "nx": 128, "ny": 128, "nz": 128, "rho": False, "coarse": False},
        # the gradient of one training sample
        {"name": "train_64", "kind": "train", "nx": 64, "ny": 64, "nz": 64, "rho": True},
    ]


def draw(rng):
    def size(lo, hi, mult=1):
        return max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / mult)) * mult)

    def box(lo, hi, most, mult=1):
        while True:
            nx, ny, nz = (size(lo, hi, mult) for _ in range(3))
            if nx * ny * nz <= most and max(nx, ny, nz) <= 6 * min(nx, ny, nz):
                return {"nx": nx, "ny": ny, "nz": nz}

    kind = rng.choice(("solve", "solve", "solve", "solve", "host", "projection", "projection", "hit", "channel",
                       "guess", "train"))
    mixed = rng.random() < 0.5
    if kind == "solve":
        problem = rng.choice(("drops", "drops", "periodic", "helmholtz", "channel"))
        mult = rng.choice((1, 2, 8, 16))
        c = box(24, 200, 90 ** 3 if problem == "channel" else 160 ** 3, mult)
        # the stretched channel runs in FP64: FP32 cannot resolve its smoothest modes
        return {"kind": kind, "problem": problem, **c, "ghost": rng.choice((1, 2, 3)),
                "mixed": mixed and problem != "channel"}
    if kind == "host":
        return {"kind": kind, **box(32, 144, 112 ** 3, rng.choice((1, 2, 8))), "ghost": rng.choice((1, 2, 3)),
                "mixed": mixed}
    if kind == "projection":
        return {"kind": kind, **box(32, 192, 144 ** 3, rng.choice((1, 2, 8, 16))), "ghost": rng.choice((1, 2)),
                "mixed": mixed}
    if kind == "hit":
        n = size(32, 128, rng.choice((1, 2, 8)))
        return {"kind": kind, "n": n if n != 64 else 68, "mixed": mixed}
    if kind == "channel":
        while True:
            nx, ny, nz = size(48, 160, 2), size(24, 64, 2), size(8, 48, 2)
            if nx * ny * nz <= 128 * 40 * 32:
                return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "mixed": False}
    if kind == "guess":
        coarse = rng.random() < 0.5
        return {"kind": kind, **box(64 if coarse else 32, 256 if coarse else 128, 256 ** 3 if coarse else 128 ** 3,
                                    16 if coarse else 8), "rho": rng.random() < 0.5, "coarse": coarse}
    return {"kind": kind, **box(24, 96, 80 ** 3, 8), "rho": rng.random() < 0.5}


def work(case):
    """Floors: each input read once, each output written once.  A 7-point
    operator that is symmetric holds four values per cell."""
    kind = case["kind"]
    if kind == "hit":
        n = case["n"] ** 3
        # U, V, W, P in and out, the viscosity in; two sub-iterations of explicit terms and projection
        return {"bytes": 9 * 8 * n, "flops": 2 * (400 + 60) * n}
    n = case["nx"] * case["ny"] * case["nz"]
    if kind == "solve":
        return {"bytes": (4 + 2) * 8 * n, "flops": 14 * n}
    if kind == "host":
        return {"bytes": (7 + 2) * 8 * n, "flops": 14 * n}
    if kind == "projection":
        # face densities and U, V, W, P in; the solution and U, V, W, P out
        return {"bytes": (3 + 4 + 5) * 8 * n, "flops": 60 * n}
    if kind == "channel":
        return {"bytes": 9 * 8 * n, "flops": 2 * (600 + 60) * n}
    v = n // 8 if case.get("coarse") else n
    conv = sum(2 * 27 * ci * co * (v >> (3 * lv)) for ci, co, lv in _layers())
    nf = 3 if case["rho"] else 2
    if kind == "guess":
        return {"bytes": 8 * nf * n + 8 * n + 4 * v, "flops": conv}
    return {"bytes": 8 * (nf + 1) * n + 4 * v + 2 * 4 * _nparam(), "flops": 3 * conv}


def tolerance(case):
    """About four times the largest error against ``exact`` seen over the ranges."""
    kind = case["kind"]
    if kind in ("solve", "host", "projection"):
        # stopped at max|r| <= 1e-10 max|r0|: up to 2e-11 off the exact solution
        return {"rel": 1e-10, "max": 4e-9}
    if kind == "hit":
        return {"rel": 1e-11, "max": 4e-10}
    if kind == "channel":
        # the implicit velocity solves stop at 1e-6 of their residual: up to 3e-10 off
        return {"rel": 2e-9, "max": 8e-8}
    if kind == "guess":
        # bf16 activations and weights through 14 layers: up to 1.2e-2 off the float64 network
        return {"rel": 2e-2, "max": 0.5}
    return {"rel": 2.5e-2, "max": 0.9}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


# ----------------------------------------------------------- fields from seeds
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _bc(v, d):
    """A 1-D array along x (0), y (1) or z (2)."""
    return v[None, None, :] if d == 0 else (v[None, :, None] if d == 1 else v[:, None, None])


def _nodes(case):
    """Node coordinates and periodicity."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    if case["kind"] == "channel" or case.get("problem") == "channel":
        s, ly = (2.1, 1.0) if case["kind"] == "channel" else (2.0, 2.0)
        lx, lz = (5.0, 0.04 * nz) if case["kind"] == "channel" else (2.0 * math.pi, math.pi)
        y = 0.5 * ly * np.tanh(s * (2.0 * np.arange(ny + 1) / ny - 1.0)) / np.tanh(s)
        z = np.arange(nz + 1) / nz * lz
        return np.arange(nx + 1) / nx * lx, y, z - 0.5 * lz if case["kind"] == "channel" else z, WALLS_Y
    length = 1e-2 if case["kind"] == "host" or case.get("problem") == "helmholtz" else 1.0
    h = length / max(nx, ny, nz)
    per = PERIODIC if case.get("problem") == "periodic" else WALLS_Y
    return h * np.arange(nx + 1), h * np.arange(ny + 1), h * np.arange(nz + 1), per


def _drops(case, per, g):
    """Density 1 in the gas, 1000 in seeded drops, smeared over 1.5 cells."""
    ns = (case["nx"], case["ny"], case["nz"])
    big = max(ns)
    count = max(3, round(48 * ns[0] * ns[1] * ns[2] / big ** 3))
    c = torch.rand((count, 3), generator=g, device=DEV, dtype=F64).cpu().numpy()
    r = (6.0 + 14.0 * torch.rand(count, generator=g, device=DEV, dtype=F64).cpu().numpy()) * big / 256.0
    x = [torch.arange(n, device=DEV, dtype=F64) + 0.5 for n in ns]
    H = torch.full((ns[2], ns[1], ns[0]), -1e30, dtype=F64, device=DEV)
    for m in range(count):
        d2 = []
        for d in range(3):
            t = x[d] - c[m, d] * ns[d]
            d2.append(_bc((t - ns[d] * torch.round(t / ns[d]) if per[d] else t) ** 2, d))
        H = torch.maximum(H, r[m] - torch.sqrt(d2[0] + d2[1] + d2[2]))
    return 1.0 + 999.0 * 0.5 * (1.0 + torch.tanh(H / 1.5))


def _velocity(case, per, g, noise=0.01):
    """Face velocities on faces 0..n-1: a few large modes and noise, zero on walls."""
    ns = (case["nx"], case["ny"], case["nz"])
    out = []
    for comp in range(3):
        a = noise * torch.randn((ns[2], ns[1], ns[0]), generator=g, device=DEV, dtype=F64)
        p = torch.rand((6, 7), generator=g, device=DEV, dtype=F64).cpu().numpy()
        for m in range(6):
            w = [torch.cos(2.0 * math.pi * (torch.arange(ns[d], device=DEV, dtype=F64) / ns[d]
                                            * (1 + int(4 * p[m, d])) + p[m, 3 + d])) for d in range(3)]
            a = a + (p[m, 6] - 0.5) * (_bc(w[0], 0) * _bc(w[1], 1) * _bc(w[2], 2))
        if not per[comp]:
            a.select(2 - comp, 0).zero_()
        out.append(a)
    return out


def _pad(a, g, per, edge=False):
    """Interior array -> padded array: periodic images; in wall directions zero, or the edge value."""
    out = torch.nn.functional.pad(a, (g,) * 6)
    for ax, p in ((2, per[0]), (1, per[1]), (0, per[2])):
        n = a.shape[ax]
        if p:
            out.narrow(ax, 0, g).copy_(out.narrow(ax, n, g))
            out.narrow(ax, n + g, g).copy_(out.narrow(ax, g, g))
        elif edge:
            out.narrow(ax, 0, g).copy_(out.narrow(ax, g, 1))
            out.narrow(ax, n + g, g).copy_(out.narrow(ax, n + g - 1, 1))
    return out.contiguous()


def _lo(a, d, per, fill="edge"):
    """The value at the lower neighbour along d; at a wall the cell's own (edge) or 0."""
    r = torch.roll(a, 1, 2 - d)
    if not per[d]:
        r.select(2 - d, 0).copy_(a.select(2 - d, 0) if fill == "edge" else torch.zeros_like(a.select(2 - d, 0)))
    return r


def _hi(a, d, per, fill="edge"):
    r = torch.roll(a, -1, 2 - d)
    if not per[d]:
        e = a.select(2 - d, a.shape[2 - d] - 1)
        r.select(2 - d, a.shape[2 - d] - 1).copy_(e if fill == "edge" else torch.zeros_like(e))
    return r


def _face_rho(rho, per):
    return [0.5 * (_lo(rho, d, per) + rho) for d in range(3)]


# ------------------------------------------------------------- pressure solves
DT = 1e-3
RHO_L, RHO_G, C_L, C_G = 1000.0, 1.0, 1500.0, 340.0  # water drops in air


def _helmholtz(case, seed):
    """The compressible solver's pressure system: 1 / (rho c^2), face densities, dt and rhs (interior)."""
    x, y, z, per = _nodes(case)
    g = _gen(seed)
    rho = _drops(case, per, g)
    vf = (rho - 1.0) / 999.0
    k = vf / (RHO_L * C_L ** 2) + (1.0 - vf) / (RHO_G * C_G ** 2)
    h = float(x[1] - x[0])
    dt = 0.5 * h
    u = _velocity(case, per, g)
    div = sum(_hi(u[d], d, per, "zero") - u[d] for d in range(3)) / h
    pa = 1e5 + 20.0 * vf + 100.0 * torch.randn(rho.shape, generator=g, device=DEV, dtype=F64)
    return per, h, dt, k, [RHO_G * f for f in _face_rho(rho, per)], pa * k - dt * div


def _helmholtz_operator(case, seed):
    per, h, dt, k, rf, rhs = _helmholtz(case, seed)
    opr = torch.zeros(rhs.shape + (7,), dtype=F64, device=DEV)
    opr[..., 0] = k
    for d in range(3):
        lo = (dt / h) ** 2 / rf[d]
        if not per[d]:
            lo.select(2 - d, 0).zero_()
        hi = _hi(lo, d, per, "zero")
        opr[..., 0] += lo + hi
        opr[..., 1 + 2 * d] = -hi
        opr[..., 2 + 2 * d] = -lo
    return per, opr, rhs


def _pad_opr(opr, g):
    return torch.nn.functional.pad(opr, (0, 0) + (g,) * 6).contiguous()


def _solver(case, per, method=B.PCG_BBOX):
    return B.BBMG(case["nx"], case["ny"], case["nz"], *per, ghost=case["ghost"], method=method,
                  precision=B.MIXED if case["mixed"] else B.FP64, maxit=300)


def _flow(case, seed):
    """Density (None if constant) and face velocities of a Poisson problem."""
    _, _, _, per = _nodes(case)
    g = _gen(seed)
    rho = _drops(case, per, g) if case.get("problem", "drops") == "drops" else None
    return per, rho, _velocity(case, per, g)


def _prep_solve(case, seed):
    g = case["ghost"]
    x, y, z, per = _nodes(case)
    proj = Projection(x, y, z, *per, ghost=g)
    h = _solver(case, per)
    if case["problem"] == "helmholtz":
        _, opr, rhs = _helmholtz_operator(case, seed)
        h.setup(STC7, _pad_opr(opr, g))
        rhs = _pad(rhs, g, per)
    else:
        _, rho, u = _flow(case, seed)
        rf = [_pad(f, g, per, edge=True) for f in _face_rho(rho, per)] if rho is not None else (None, None, None)
        h.setup(STC7, proj.update_laplacian(*rf))
        _, rhs = proj.get_div(*[_pad(a, g, per) for a in u], rho=1.0, dt=DT, want_div=False)
    return {"run": _run_solve, "proj": proj, "h": h, "rhs": rhs, "sol": torch.zeros_like(rhs),
            "shift": case["problem"] != "helmholtz"}


def _run_solve(s):
    s["sol"].zero_()
    s["h"].solve(s["rhs"], s["sol"])
    if s["shift"]:
        s["proj"].shift_p(s["sol"])
    return s["sol"]


def _prep_host(case, seed):
    g = case["ghost"]
    per, opr, rhs = _helmholtz_operator(case, seed)
    s = B.ILS(case["nx"], case["ny"], case["nz"], *per, ghost=g, nst=7, maxit=300,
              precision=B.MIXED if case["mixed"] else B.FP64)
    s.stc[:] = STC7
    s.opr[...] = _pad_opr(opr, g).cpu().numpy()
    s.rhs[...] = _pad(rhs, g, per).cpu().numpy()
    s.init(B.PCG_BBOX)
    return {"run": _run_host, "ils": s}


def _run_host(s):
    ils = s["ils"]
    ils.setup()
    ils.sol[...] = 0.0
    ils.solve()
    return ils.sol


def _prep_projection(case, seed):
    g = case["ghost"]
    x, y, z, per = _nodes(case)
    _, rho, u = _flow(case, seed)
    proj = Projection(x, y, z, *per, ghost=g)
    st = {"run": _run_projection, "proj": proj, "h": _solver(case, per),
          "rf": [_pad(f, g, per, edge=True) for f in _face_rho(rho, per)], "star": [_pad(a, g, per) for a in u]}
    z0 = torch.zeros(proj.shape, dtype=F64, device=DEV)
    st.update(opr=torch.zeros(proj.shape + (7,), dtype=F64, device=DEV), u=[z0.clone() for _ in range(3)],
              p=z0.clone(), rhs=z0.clone(), sol=z0.clone())
    return st


def _run_projection(s):
    for a, b in zip(s["u"], s["star"]):
        a.copy_(b)  # the predicted velocity
    s["p"].zero_()
    s["proj"].update_laplacian(*s["rf"], opr=s["opr"])
    s["h"].setup(STC7, s["opr"])
    s["proj"].get_div(*s["u"], rho=1.0, dt=DT, rhs=s["rhs"], want_div=False)
    s["sol"].zero_()
    s["h"].solve(s["rhs"], s["sol"])
    s["proj"].shift_p(s["sol"])
    s["proj"].correct(s["sol"], DT, *s["u"], s["p"], *s["rf"])
    return [s["sol"], *s["u"], s["p"]]


# ---------------------------------------------------------------- exact solves
def _pcg(apply, diag, b, singular, tol=1e-13, maxit=20000):
    """Jacobi-preconditioned conjugate gradients."""
    x = torch.zeros_like(b)
    r = b - b.mean() if singular else b.clone()
    stop = tol * float(r.abs().max())
    z = r / diag
    p = z.clone()
    rz = (r * z).sum()
    for it in range(maxit):
        q = apply(p)
        alpha = rz / (p * q).sum()
        x += alpha * p
        r -= alpha * q
        if it % 20 == 19 and float(r.abs().max()) <= stop:
            break
        z = r / diag
        new = (r * z).sum()
        p = z + (new / rz) * p
        rz = new
    return x


def _metrics(x):
    """Cell sizes, their inverses and the inverse centre distances on faces 0..n (one layer of extension)."""
    xe = np.concatenate([[x[0] - (x[1] - x[0])], x, [x[-1] + (x[-1] - x[-2])]])
    xm = 0.5 * (xe[:-1] + xe[1:])
    d = np.diff(x)
    return d, 1.0 / d, 1.0 / np.diff(xm)


def _const_solve(case, rhs):
    """-vol div(grad p) = rhs with constant density, zero mean: Fourier in x and z, a dense solve along y."""
    x, y, z, per = _nodes(case)
    dx, dz = x[1] - x[0], z[1] - z[0]
    dy, dyi, dmi = _metrics(y)
    nz, ny, nx = rhs.shape
    lo, hi = dyi * dmi[:-1], dyi * dmi[1:]
    if not per[1]:
        lo[0] = hi[-1] = 0.0
    T = np.diag(-(lo + hi))
    for j in range(ny):
        T[j, (j - 1) % ny] += lo[j]
        T[j, (j + 1) % ny] += hi[j]
    T = torch.from_numpy(T).to(DEV)
    kx = (2.0 * torch.sin(math.pi * torch.arange(nx // 2 + 1, device=DEV, dtype=F64) / nx) / dx) ** 2
    kz = (2.0 * torch.sin(math.pi * torch.arange(nz, device=DEV, dtype=F64) / nz) / dz) ** 2
    vol = torch.from_numpy(dx * dy * dz).to(DEV)
    r = torch.fft.rfft2(-rhs / _bc(vol, 1), dim=(0, 2))  # [kz, j, kx]
    out = torch.empty_like(r)
    eye = torch.eye(ny, dtype=F64, device=DEV)
    for m in range(nz):
        A = T[None] - (kz[m] + kx)[:, None, None] * eye[None]
        b = torch.view_as_real(r[m].T.contiguous())
        if m == 0:
            A[0, 0] = 0.0
            A[0, 0, 0] = 1.0
            b[0, 0] = 0.0
        out[m] = torch.view_as_complex(torch.linalg.solve(A, b).contiguous()).T
    p = torch.fft.irfft2(out, s=(nz, nx), dim=(0, 2))
    return p - (p * _bc(vol, 1)).sum() / (vol.sum() * nx * nz)


def _drops_solve(case, per, rho, u):
    """Solution of -vol div(grad p / rho) = -vol div(u) / dt on a uniform grid, zero mean; the face densities."""
    x, _, _, _ = _nodes(case)
    h = float(x[1] - x[0])
    rf = _face_rho(rho, per)
    c = [h / f for f in rf]
    for d in range(3):
        if not per[d]:
            c[d].select(2 - d, 0).zero_()
    ch = [_hi(c[d], d, per, "zero") for d in range(3)]
    diag = sum(c) + sum(ch)

    def apply(p):
        q = diag * p
        for d in range(3):
            q -= c[d] * torch.roll(p, 1, 2 - d)
            q -= ch[d] * torch.roll(p, -1, 2 - d)
        return q

    div = sum(_hi(u[d], d, per, "zero") - u[d] for d in range(3)) / h
    p = _pcg(apply, diag, -h ** 3 * div / DT, True)
    return p - p.mean(), rf, h


def _exact_solve(case, seed):
    g = case["ghost"]
    if case["problem"] == "helmholtz":
        return _exact_host(case, seed, as_numpy=False)
    per, rho, u = _flow(case, seed)
    if rho is not None:
        return _pad(_drops_solve(case, per, rho, u)[0], g, per)
    x, y, z, _ = _nodes(case)
    rhs = sum((_hi(u[d], d, per, "zero") - u[d]) * _bc(torch.from_numpy(1.0 / np.diff(a)).to(DEV), d)
              for d, a in enumerate((x, y, z)))
    vol = torch.from_numpy((x[1] - x[0]) * (z[1] - z[0]) * np.diff(y)).to(DEV)
    return _pad(_const_solve(case, -_bc(vol, 1) * rhs / DT), g, per)


def _exact_host(case, seed, as_numpy=True):
    g = case["ghost"]
    per, opr, rhs = _helmholtz_operator(case, seed)

    def apply(p):
        q = opr[..., 0] * p
        for d in range(3):
            q += opr[..., 1 + 2 * d] * torch.roll(p, -1, 2 - d)
            q += opr[..., 2 + 2 * d] * torch.roll(p, 1, 2 - d)
        return q

    p = _pcg(apply, opr[..., 0].contiguous(), rhs, False)
    # the solver writes the interior only
    p = torch.nn.functional.pad(p, (g,) * 6)
    return p.cpu().numpy() if as_numpy else p


def _exact_projection(case, seed):
    g = case["ghost"]
    per, rho, u = _flow(case, seed)
    p, rf, h = _drops_solve(case, per, rho, u)
    out = []
    for d in range(3):
        grad = (p - _lo(p, d, per)) / h  # zero on the wall faces
        out.append(_pad(u[d] - DT * grad / rf[d], g, per))
    return [_pad(p, g, per), *out, _pad(p, g, per)]


# ------------------------------------------------------------------ time steps
def _turbulence(n, seed, urms=5.0):
    """Solenoidal random velocity with spectrum k^4 exp(-2 (k/4)^2), rms ``urms``."""
    g = _gen(seed)
    k = torch.fft.fftfreq(n, 1.0 / n, dtype=F64, device=DEV)
    kk = [_bc(k, d) for d in range(3)]
    k2 = kk[0] ** 2 + kk[1] ** 2 + kk[2] ** 2
    amp = k2 * torch.exp(-k2 / 16.0) / torch.sqrt(k2.clamp(min=1.0))
    f = [torch.fft.fftn(torch.randn((n, n, n), generator=g, device=DEV, dtype=F64)) * amp for _ in range(3)]
    kdot = sum(a * b for a, b in zip(kk, f)) / k2.clamp(min=1.0)
    u = [torch.fft.ifftn(f[d] - kk[d] * kdot).real for d in range(3)]
    rms = torch.sqrt(sum((a ** 2).mean() for a in u) / 3.0)
    return [(a * (urms / rms)).contiguous() for a in u]


def _energy(u, per):
    c = [0.5 * (u[d] + _hi(u[d], d, per, "zero")) for d in range(3)]
    return 0.5 * (c[0] ** 2 + c[1] ** 2 + c[2] ** 2).sum()


def _channel_velocity(case, seed):
    """A parabolic profile of bulk velocity 1 with 5 % noise."""
    x, y, z, per = _nodes(case)
    g = _gen(seed)
    ns = (case["nx"], case["ny"], case["nz"])
    u = [0.05 * torch.randn((ns[2], ns[1], ns[0]), generator=g, device=DEV, dtype=F64) for _ in range(3)]
    ym = torch.from_numpy(0.5 * (y[:-1] + y[1:])).to(DEV)
    u[0] += _bc(1.5 * (1.0 - (2.0 * ym) ** 2), 1)
    u[1].select(1, 0).zero_()
    return u


def _keep_start(fs: Incomp, u):
    """Put the velocities into the flow solver and keep them for the next pass."""
    start = [_pad(a, fs.g, fs.per) for a in u] + [torch.zeros(fs.shape, dtype=F64, device=DEV)]
    for a, b in zip((fs.U, fs.V, fs.W, fs.P), start):
        a.copy_(b)
    return start


def _prep_hit(case, seed):
    hit = HIT(n=case["n"], seed=0, precision=B.MIXED if case["mixed"] else B.FP64)
    u = _turbulence(case["n"], seed)
    hit.KE0 = float(_energy(u, PERIODIC))
    return {"run": _run_step, "loop": hit, "start": _keep_start(hit.fs, u)}


def _prep_channel(case, seed):
    ch = Channel(nx=case["nx"], ny=case["ny"], nz=case["nz"], Lz=0.04 * case["nz"],
                 precision=B.MIXED if case["mixed"] else B.FP64)
    return {"run": _run_step, "loop": ch, "start": _keep_start(ch.fs, _channel_velocity(case, seed))}


def _run_step(s):
    """One time step from the start (the loop's clock and fields set back to it)."""
    fs, time = s["loop"].fs, s["loop"].time
    for a, b in zip((fs.U, fs.V, fs.W, fs.P), s["start"]):
        a.copy_(b)
    time.dt, time.t, time.n = time.dtmax, 0.0, 0
    s["loop"].step()
    return [fs.U, fs.V, fs.W, fs.P]


class _Staggered:
    """The staggered momentum terms with constant viscosity, x and z uniform
    and periodic, y periodic or between walls (rho = 1)."""

    def __init__(self, x, y, z, per, visc):
        self.per, self.visc = per, visc
        self.di, self.dmi = [], []
        for a in (x, y, z):
            _, di, dmi = _metrics(np.asarray(a))
            self.di.append(torch.from_numpy(di).to(DEV))
            self.dmi.append(torch.from_numpy(dmi).to(DEV))
        xe = np.concatenate([[y[0] - (y[1] - y[0])], y, [y[-1] + (y[-1] - y[-2])]])
        ym = 0.5 * (xe[:-1] + xe[1:])
        wm = (ym[1:] - y) / np.diff(ym)  # weight of the cell below each y-face 0..n
        gd = 1.0 / np.diff(ym)
        if not per[1]:  # a tangential velocity is 0 at the wall, its gradient over half a cell
            wm[0], wm[-1] = 1.0, 0.0
            gd[0], gd[-1] = 1.0 / (ym[1] - y[0]), 1.0 / (y[-1] - ym[-2])
        self.wm, self.gd = torch.from_numpy(wm).to(DEV), torch.from_numpy(gd).to(DEV)

    def cells(self, q, d):
        """Mean and gradient at the cells of a component along its own direction d."""
        hi = _hi(q, d, self.per, "zero")
        return 0.5 * (q + hi), (hi - q) * _bc(self.di[d], d)

    def edges(self, q, d, own):
        """Value and gradient on the faces along d of a component of direction ``own`` != d."""
        if own == 1 and not self.per[1]:  # the upper wall face carries 0
            q = torch.nn.functional.pad(q, (0, 0, 0, 1))
        if d != 1:
            lo = torch.roll(q, 1, 2 - d)
            return 0.5 * (lo + q), (q - lo) * _bc(self.dmi[d][:q.shape[2 - d]], d)
        if self.per[1]:
            lo, w, gd = torch.roll(q, 1, 1), self.wm[:-1], self.gd[:-1]
        else:
            q = torch.nn.functional.pad(q, (0, 0, 1, 1))
            lo, q, w, gd = q[:, :-1], q[:, 1:], self.wm, self.gd
        return _bc(w, 1) * lo + _bc(1.0 - w, 1) * q, (q - lo) * _bc(gd, 1)

    def gather(self, fl, own):
        """The divergence at the faces of component ``own`` of its fluxes fl (cells along own, edges along the others)."""
        out = 0.0
        for d in range(3):
            f = fl[d]
            if d == own:
                out = out + (f - torch.roll(f, 1, 2 - d)) * _bc(self.dmi[d][:f.shape[2 - d]], d)
                continue
            if own == 1 and not self.per[1]:
                f = f[:, :-1]
            n = self.di[d].numel()
            hi = torch.roll(f, -1, 2 - d) if f.shape[2 - d] == n else f.narrow(2 - d, 1, n)
            out = out + (hi - f.narrow(2 - d, 0, n)) * _bc(self.di[d], d)
        if not self.per[own]:
            out.select(2 - own, 0).zero_()
        return out

    def dmomdt(self, u, P):
        mu, c = self.visc, [self.cells(u[d], d) for d in range(3)]
        div = c[0][1] + c[1][1] + c[2][1]
        res = []
        for o in range(3):
            fl = [None] * 3
            for d in range(3):
                if d == o:
                    fl[d] = -c[o][0] ** 2 + mu * (2.0 * c[o][1] - 2.0 / 3.0 * div) - P
                else:
                    a, ga = self.edges(u[o], d, o)
                    b, gb = self.edges(u[d], o, d)
                    fl[d] = -a * b + mu * (ga + gb)
            res.append(self.gather(fl, o))
        return res

    def implicit(self, u, o, dt):
        """x -> x - dt/2 (the linearised terms of component o in itself)."""
        base = self.cells(u[o], o)[0]
        adv = [None if d == o else self.edges(u[d], o, d)[0] for d in range(3)]

        def apply(x):
            fl = [None] * 3
            for d in range(3):
                if d == o:
                    m, gr = self.cells(x, o)
                    fl[d] = -2.0 * base * m + 4.0 / 3.0 * self.visc * gr
                else:
                    a, ga = self.edges(x, d, o)
                    fl[d] = -a * adv[d] + self.visc * ga
            return x - 0.5 * dt * self.gather(fl, o)
        return apply


def _bicgstab(apply, b, tol=1e-13):
    x, r = torch.zeros_like(b), b.clone()
    r0, p = r.clone(), r.clone()
    rho, stop = (r0 * r).sum(), tol * float(b.norm())
    for _ in range(400):
        v = apply(p)
        alpha = rho / (r0 * v).sum()
        s = r - alpha * v
        t = apply(s)
        tt = (t * t).sum()
        om = (t * s).sum() / tt if float(tt) > 0.0 else tt
        x += alpha * p + om * s
        r = s - om * t
        if float(r.norm()) <= stop:
            break
        new = (r0 * r).sum()
        p = r + (new / rho) * (alpha / om) * (p - om * v)
        rho = new
    return x


def _exact_step(case, seed):
    """One time step: dt from the CFL, two mid-point sub-iterations, each closed by a pressure projection."""
    channel = case["kind"] == "channel"
    if channel:
        x, y, z, per = _nodes(case)
        box, u = case, _channel_velocity(case, seed)
        dt0 = 2e-2
    else:
        n = case["n"]
        x = y = z = np.arange(n + 1) / n
        per, u = PERIODIC, _turbulence(n, seed)
        box = {"kind": "solve", "problem": "periodic", "nx": n, "ny": n, "nz": n}
        dt0, ke0 = 1e-3, _energy(u, PERIODIC)
    visc, S = 0.01, _Staggered(x, y, z, per, 0.01)
    cfl = 0.0
    for d in range(3):
        cfl = max(cfl, float((u[d].abs() * _bc(S.dmi[d][:u[d].shape[2 - d]], d)).max()) * dt0,
                  float((4.0 * visc * S.di[d] ** 2).max()) * dt0)
    dt = min(dt0 * 0.9 / cfl, dt0) if cfl > 0.0 else dt0
    vol = torch.from_numpy((x[1] - x[0]) * (z[1] - z[0]) * np.diff(y)).to(DEV)
    nx, ny, nz = len(x) - 1, len(y) - 1, len(z) - 1
    P, old = torch.zeros_like(u[0]), [a.clone() for a in u]
    for _ in range(2):
        u = [0.5 * (a + b) for a, b in zip(u, old)]
        dm = S.dmomdt(u, P)
        res = [-2.0 * (a - b) + dt * m for a, b, m in zip(u, old, dm)]
        if channel:
            w = _bc(vol, 1)
            for o, bulk in ((0, 1.0), (2, 0.0)):
                res[o] = res[o] + bulk - ((2.0 * u[o] - old[o]) * w).sum() / (vol.sum() * nx * nz)
            res = [_bicgstab(S.implicit(u, o, dt), res[o]) for o in range(3)]
        else:
            f = dt * ke0 / _energy(u, per) / 0.2
            res = [r + f * (a - a.mean()) for r, a in zip(res, u)]
        u = [2.0 * a - b + r for a, b, r in zip(u, old, res)]
        div = sum((_hi(u[d], d, per, "zero") - u[d]) * _bc(S.di[d], d) for d in range(3))
        p = _const_solve(box, -_bc(vol, 1) * div / dt)
        P = P + p
        u = [u[d] - dt * (p - _lo(p, d, per)) * _bc(S.dmi[d][:u[d].shape[2 - d]], d) for d in range(3)]
    return [_pad(a, 1, per) for a in (*u, P)]


# --------------------------------------------------------------------- network
CH = (16, 32, 64, 128)
KAPPA = 0.05


def _layers():
    """(input channels, output channels, level) of the network's convolutions."""
    c1, c2, c3, c4 = CH
    return [(16, c1, 0), (c1, c1, 0), (c1, c2, 1), (c2, c2, 1), (c2, c3, 2), (c3, c3, 2), (c3, c4, 3), (c4, c4, 3),
            (c4 + c3, c3, 2), (c3, c3, 2), (c3 + c2, c2, 1), (c2, c2, 1), (c2 + c1, c1, 0), (c1, c1, 0)]


def _nparam():
    return sum(27 * ci * co + co for ci, co, _ in _layers()) + CH[0] + 1


def _params(nf, seed):
    """He-normal weights, small biases and a head of order one, as a trained network has."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, (ci, co, _) in enumerate(_layers()):
        w = rng.standard_normal((27, ci, co)) * math.sqrt(2.0 / (27 * (nf if i == 0 else ci)))
        if i == 0:
            w[:, nf:] = 0.0
        parts += [w.ravel(), 0.05 * rng.standard_normal(co)]
    parts += [rng.standard_normal(CH[0]) / 4.0, np.zeros(1)]
    return np.concatenate(parts).astype(np.float32)


def _record(case, seed):
    """A solve's right-hand side, previous increment, density and increment (dense, FP64)."""
    g = _gen(seed)
    shape = (case["nz"], case["ny"], case["nx"])
    ns = shape[::-1]

    def smooth():
        a = 0.05 * torch.randn(shape, generator=g, device=DEV, dtype=F64)
        p = torch.rand((8, 7), generator=g, device=DEV, dtype=F64).cpu().numpy()
        for m in range(8):
            w = [torch.cos(2.0 * math.pi * (torch.arange(ns[d], device=DEV, dtype=F64) / ns[d]
                                            * (1 + int(6 * p[m, d])) + p[m, 3 + d])) for d in range(3)]
            a = a + (p[m, 6] - 0.5) * (_bc(w[0], 0) * _bc(w[1], 1) * _bc(w[2], 2))
        return a

    rec = {"rhs": smooth(), "p_prev": smooth()}
    rec["dp"] = rec["p_prev"] + 0.2 * smooth()
    if case["rho"]:
        rec["rho"] = _drops(case, PERIODIC, g)
    return rec


def _prep_net(case, seed):
    nf = 3 if case["rho"] else 2
    net = UNet(nf=nf, ch=CH, params=_params(nf, seed))
    guess = LearnedGuess(net, kappa=KAPPA, use_rho=case["rho"], ratio=1000.0, coarse=case.get("coarse", False))
    rec = _record(case, seed)
    if case["kind"] == "guess":
        return {"run": _run_guess, "guess": guess, "rec": rec, "out": torch.zeros_like(rec["rhs"])}
    return {"run": _run_train, "guess": guess, "rec": rec, "target": (rec["dp"] - rec["p_prev"]).contiguous()}


def _run_guess(s):
    guess, rec = s["guess"], s["rec"]
    guess.guess(rec, s["out"])
    k = 2 if guess.coarse else 1
    nz, ny, nx = rec["rhs"].shape
    return [s["out"], guess.net.buffers((1, nz // k, ny // k, nx // k), False)["out"]]


def _run_train(s):
    """Forward, loss and backward of one sample: the gradients an optimiser step takes."""
    net, rec = s["guess"].net, s["rec"]
    f, sc, bmax = s["guess"].fields(rec)
    b = net.buffers((1,) + tuple(rec["rhs"].shape), True)
    net.embed(b, f, sc)
    net.forward(b)
    loss = net.loss_grad(b, s["target"], 1.0 / (KAPPA * bmax))
    net.grads.zero_()
    net.backward(b)
    return [b["out"], loss, net.grads]


class _Conv(torch.autograd.Function):
    """Periodic 3x3x3 convolution in float64: x [d, h, w, ci], w [27, ci, co]."""

    @staticmethod
    def forward(ctx, x, w):
        ctx.save_for_backward(x, w)
        y = 0.0
        for t in range(27):
            y = y + torch.roll(x, (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3), (0, 1, 2)) @ w[t]
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w = ctx.saved_tensors
        dx, dw = 0.0, torch.empty_like(w)
        for t in range(27):
            s = (1 - t // 9, 1 - t // 3 % 3, 1 - t % 3)
            dw[t] = torch.roll(x, s, (0, 1, 2)).reshape(-1, x.shape[3]).T @ dy.reshape(-1, dy.shape[3])
            dx = dx + torch.roll(dy @ w[t].T, tuple(-a for a in s), (0, 1, 2))
        return dx, dw


def _net64(theta, x):
    """The network in float64 from the flat parameter vector; x [d, h, w, 16]."""
    off, it = 0, iter(_layers())

    def conv(a):
        nonlocal off
        ci, co, _ = next(it)
        w = theta[off:off + 27 * ci * co].reshape(27, ci, co)
        b = theta[off + 27 * ci * co:off + 27 * ci * co + co]
        off += 27 * ci * co + co
        return torch.relu(_Conv.apply(a, w) + b)

    def pool(a):
        d, h, w, c = a.shape
        return a.reshape(d // 2, 2, h // 2, 2, w // 2, 2, c).mean(dim=(1, 3, 5))

    def up(a):
        return a.repeat_interleave(2, 0).repeat_interleave(2, 1).repeat_interleave(2, 2)

    skips = []
    for lv in range(3):
        x = conv(conv(x))
        skips.append(x)
        x = pool(x)
    x = conv(conv(x))
    for lv in (2, 1, 0):
        x = conv(conv(torch.cat([up(x), skips[lv]], -1)))
    return (x @ theta[off:off + CH[0]] + theta[off + CH[0]]).reshape(-1)


def _exact_net(case, seed):
    nf = 3 if case["rho"] else 2
    theta = torch.from_numpy(_params(nf, seed)).to(DEV).double()
    rec = _record(case, seed)
    coarse = case.get("coarse", False)
    bmax = float(rec["rhs"].abs().max())
    f = [rec["rhs"] / bmax, rec["p_prev"] / float(rec["p_prev"].abs().max())]
    if case["rho"]:
        f.append(rec["rho"] / 1000.0)
    if coarse:
        f = [torch.nn.functional.avg_pool3d(a[None, None], 2)[0, 0] for a in f]
    x = torch.stack(f + [torch.zeros_like(f[0])] * (16 - nf), -1)
    if case["kind"] == "guess":
        with torch.no_grad():
            out = _net64(theta, x)
        e = out.reshape(x.shape[:3])
        if coarse:  # trilinear between cell centres, periodic
            for d in range(3):
                lo, hi = 0.25 * torch.roll(e, 1, d) + 0.75 * e, 0.75 * e + 0.25 * torch.roll(e, -1, d)
                e = torch.stack([lo, hi], d + 1).flatten(d, d + 1)
        return [rec["p_prev"] + KAPPA * bmax * e, out]
    theta.requires_grad_(True)
    out = _net64(theta, x)
    diff = out - ((rec["dp"] - rec["p_prev"]) / (KAPPA * bmax)).reshape(-1)
    (diff ** 2).mean().backward()
    return [out.detach(), (diff.detach() ** 2).sum().reshape(1), theta.grad]


_PREPARE = {"solve": _prep_solve, "host": _prep_host, "projection": _prep_projection, "hit": _prep_hit,
            "channel": _prep_channel, "guess": _prep_net, "train": _prep_net}
_EXACT = {"solve": _exact_solve, "host": _exact_host, "projection": _exact_projection, "hit": _exact_step,
          "channel": _exact_step, "guess": _exact_net, "train": _exact_net}
