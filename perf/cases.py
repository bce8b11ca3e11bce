"""The work a user of this framework has it do, as cases to be timed.

Each case is one call, or one short sequence of calls, of the public API (hymor_gb300.solver
and the C ABI of include/hymor.h) on inputs made from a seed:

  march        ADVECT_FLOW of a host-resident solution in page-locked arrays (advect_host):
               upload, `steps` RK4 steps, download; each pass marches on from the last
  residual     PDE on a channel flow: one residual of the solution, returned to the host
  linearize    LINEARIZE_L of a shock-fitted flow, then the operator on `k` device vectors;
               with `shock` the shock-position blocks too (perturb_shock)
  matvec       the linearised operator on `k` device vectors in one call
  propagate    the Taylor propagator exp(L dt)^steps of the eigen and transient-growth
               solvers on `k` device vectors, forward or adjoint; with `shock` the operator
               carries the shock-position unknowns
  receptivity  the Taylor propagator of the freestream-receptivity operator on one complex
               device vector, `nw` disturbance frequencies

The operators of matvec, propagate and receptivity are made here: the Jacobian blocks of the
compressible Euler equations with second-order diffusion on a stretched grid under a shock
(rows above the shocked row are zero, as in the linearised shock-fitted residual), set through
set_blocks / set_shock_blocks / hymor_b_set.
"""
import ctypes
import math

import numpy as np
import torch

from hymor_gb300 import case as C
from hymor_gb300 import solver as S
from hymor_gb300._lib import dp, ip
from hymor_gb300.mesh import Mapping

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # the small end: one residual of the channel tutorial's grid, bound by its launches
        dict(name="residual_channel_180x60", kind="residual", nchi=180, neta=60),
        # a parameter study marches many small grids; the reference's own cylinder size
        dict(name="march_cylinder_100x80", kind="march", flow="cylinder", nchi=100, neta=80, steps=10,
             viscosity="constant"),
        # the headline benchmark: one step of the 800 x 400 cylinder end to end
        dict(name="march_cylinder_800x400", kind="march", flow="cylinder", nchi=800, neta=400, steps=1,
             viscosity="constant"),
        # the axisymmetric sphere-cone of the modal analysis, Sutherland viscosity
        dict(name="march_cone_1200x400", kind="march", flow="cone", nchi=1200, neta=400, steps=5,
             viscosity="sutherland"),
        # linearisation about a base flow: the transient-growth grid
        dict(name="linearize_cylinder_600x300", kind="linearize", nchi=600, neta=300, k=4, shock=False),
        # and with the shock-position unknowns
        dict(name="linearize_shock_200x100", kind="linearize", nchi=200, neta=100, k=1, shock=True),
        # the operator on a block of vectors (the benchmark's matvec)
        dict(name="matvec_800x400_k64", kind="matvec", nchi=800, neta=400, k=64, adjoint=False),
        # one Krylov vector of a small modal analysis
        dict(name="propagate_100x80_k1", kind="propagate", nchi=100, neta=80, k=1, steps=50, order=5, adjoint=False,
             shock=False),
        # one Krylov vector of the sphere-cone's modal analysis: 50 steps of degree 4
        dict(name="propagate_1200x400_k1", kind="propagate", nchi=1200, neta=400, k=1, steps=50, order=4,
             adjoint=False, shock=False),
        # a block of adjoint vectors of the transient-growth grid
        dict(name="adjoint_600x300_k8", kind="propagate", nchi=600, neta=300, k=8, steps=10, order=5, adjoint=True,
             shock=False),
        # transient growth with the shock-position unknowns: the adjoint propagation
        dict(name="adjoint_shock_160x97_k1", kind="propagate", nchi=160, neta=97, k=1, steps=50, order=5, adjoint=True,
             shock=True),
        # freestream receptivity: one grid of the uneven batch, 24 frequencies
        dict(name="receptivity_98x73_w24", kind="receptivity", nchi=98, neta=73, nw=24, steps=50, order=5,
             adjoint=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["march", "march", "residual", "linearize", "matvec", "propagate", "propagate", "receptivity"])
    nchi = _log(rng, 48, 900)
    neta = max(40, int(nchi * rng.uniform(0.35, 0.8)))
    if kind == "residual":
        return dict(kind=kind, nchi=_log(rng, 24, 720), neta=_log(rng, 16, 240))
    if kind == "march":
        steps = rng.randint(1, 10)
        return dict(kind=kind, flow=rng.choice(["cylinder", "cylinder", "cone"]), nchi=nchi, neta=min(neta, 400),
                    steps=steps, viscosity=rng.choice(["constant", "constant", "sutherland"]))
    if kind == "linearize":
        shock = rng.random() < 0.4
        nchi = _log(rng, 64, 320 if shock else 640)
        return dict(kind=kind, nchi=nchi, neta=max(48, int(nchi * rng.uniform(0.4, 0.8))), k=rng.randint(1, 6),
                    shock=shock)
    if kind == "matvec":
        k = _log(rng, 1, 64)
        return dict(kind=kind, nchi=nchi, neta=min(neta, 400), k=k, adjoint=rng.random() < 0.5)
    if kind == "propagate":
        shock = rng.random() < 0.35
        nchi = _log(rng, 48, 400 if shock else 800)
        neta = max(40, int(nchi * rng.uniform(0.35, 0.8)))
        k = rng.choice([1, 1, 2, 3, 4, 6, 8, 13])
        steps = max(4, min(60, int(2.4e7 / (nchi * neta * k))))
        return dict(kind=kind, nchi=nchi, neta=neta, k=k, steps=steps, order=rng.choice([3, 4, 5, 5]),
                    adjoint=rng.random() < 0.5, shock=shock)
    nchi = _log(rng, 48, 240)
    return dict(kind=kind, nchi=nchi, neta=max(40, int(nchi * rng.uniform(0.35, 0.8))), nw=rng.randint(1, 24),
                steps=rng.randint(10, 60), order=rng.choice([4, 5]), adjoint=rng.random() < 0.5)


# ---------------------------------------------------------------------------
# inputs


def _flow_config(c):
    """The marched flows: the domains and the first-order extrapolation of the base-flow
    marches, which reach a steady state."""
    kw = dict(shock_interp="1st", viscosity=c["viscosity"])
    if c["flow"] == "cone":
        return C.blunt_cone_config(c["nchi"], c["neta"], **kw)
    return C.cylinder_config(c["nchi"], c["neta"], mapping=Mapping(dRs=0.75, dRe=2.2), **kw)


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.float64 if a.dtype == np.float64 else torch.int32, pin_memory=True)
    v = t.numpy()
    v[...] = a
    return v


def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, device=DEV, dtype=F64) * 2 - 1


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 17)


def _rows(nchi, neta, seed):
    """The shocked row (1-based) of every column: a smooth line at about 3/4 of the rows."""
    r = np.random.default_rng(seed)
    x = np.linspace(0, 1, nchi)
    f = 0.74 + 0.03 * np.cos(math.pi * x + r.uniform(0, 1)) + 0.02 * np.sin(5 * x + r.uniform(0, 6))
    return np.clip(np.round(f * neta), 5, neta - 2).astype(np.int32)


def _blocks(nchi, neta, seed):
    """Stencil blocks (9, 4, 4, neta, nchi) of -d(F_x)/dx - d(F_y)/dy + diffusion at a smooth
    shock-layer state on a wall-stretched grid, and the time step at CFL 0.5."""
    gen = _gen(seed)
    g = 1.4
    eta = (torch.arange(neta, device=DEV, dtype=F64) + 0.5) / neta
    chi = (torch.arange(nchi, device=DEV, dtype=F64) + 0.5) / nchi
    E, X = torch.meshgrid(eta, chi, indexing="ij")
    ph = _uniform(gen, 6)

    def wave(k):
        return torch.sin(3 * X + ph[k] * 3) * torch.cos(4 * E + ph[k])
    rho = 5 + 0.8 * wave(0) + 2 * torch.exp(-6 * E)
    u = -0.15 * (1 - X) * E + 0.02 * wave(1)
    v = 0.8 * X * (1 - torch.exp(-8 * E)) + 0.02 * wave(2)
    p = 0.75 - 0.3 * X * X + 0.02 * wave(3)
    H = (p * g / (g - 1) + 0.5 * rho * (u * u + v * v)) / rho
    q2, gm = 0.5 * (u * u + v * v), g - 1
    zero, one = torch.zeros_like(u), torch.ones_like(u)
    a_x = torch.stack([zero, one, zero, zero,
                       gm * q2 - u * u, (3 - g) * u, -gm * v, gm * one,
                       -u * v, v, u, zero,
                       u * (gm * q2 - H), H - gm * u * u, -gm * u * v, g * u]).reshape(4, 4, neta, nchi)
    a_y = torch.stack([zero, zero, one, zero,
                       -u * v, v, u, zero,
                       gm * q2 - v * v, -gm * u, (3 - g) * v, gm * one,
                       v * (gm * q2 - H), -gm * u * v, H - gm * v * v, g * v]).reshape(4, 4, neta, nchi)
    dx = (1.6 / nchi) * (1 + 0.5 * E)                             # along the wall
    ratio = 1.05 ** (80.0 / neta)
    w = ratio ** torch.arange(neta, device=DEV, dtype=F64)
    dy = (0.6 * w / w.sum())[:, None] * one                       # wall-normal
    c = torch.sqrt(g * p / rho)
    lx, ly = (u.abs() + c) / dx, (v.abs() + c) / dy
    nu = 1.4e-4 / rho
    ex, ey = 0.1 * lx + nu / dx**2, 0.1 * ly + nu / dy**2
    cross = 0.25 * nu / (dx * dy)
    eye = torch.eye(4, device=DEV, dtype=F64)[:, :, None, None]
    vel = torch.zeros(4, 4, device=DEV, dtype=F64)
    vel[1, 2], vel[2, 1], vel[1, 0], vel[2, 0] = 1 / 3, 1 / 3, -0.1, -0.1
    vel = vel[:, :, None, None]

    def shifted(m, a, b):
        return torch.roll(m, (-b, -a), dims=(-2, -1))
    B = torch.zeros(9, 4, 4, neta, nchi, device=DEV, dtype=F64)
    B[5] = -shifted(a_x, 1, 0) / (2 * dx) + ex * eye
    B[3] = shifted(a_x, -1, 0) / (2 * dx) + ex * eye
    B[7] = -shifted(a_y, 0, 1) / (2 * dy) + ey * eye
    B[1] = shifted(a_y, 0, -1) / (2 * dy) + ey * eye
    B[4] = -2 * (ex + ey) * eye + 0.01 * (lx + ly) * (a_x - a_y)
    B[8], B[0], B[6], B[2] = cross * vel, cross * vel, -cross * vel, -cross * vel
    # no entries across the grid's edges, nor at or above the shocked row
    for q in range(9):
        a, b = q % 3 - 1, q // 3 - 1
        if a:
            B[q, ..., 0 if a < 0 else nchi - 1] = 0
        if b:
            B[q, :, :, 0 if b < 0 else neta - 1] = 0
    rows = torch.as_tensor(_rows(nchi, neta, seed), device=DEV)
    flow = (torch.arange(1, neta + 1, device=DEV)[:, None] < rows[None, :]).to(F64)
    B *= flow
    dt = 0.5 / float((lx + ly + 4 * nu / dy**2).max())
    return B, dt


def _shock_blocks(nchi, seed, dt):
    """A21, A12, A22 of the shock-position unknowns: local couplings, spread over a few
    columns by the smoothing spline."""
    r = np.random.default_rng(seed + 5)
    d = np.abs(np.arange(nchi)[:, None] - np.arange(nchi)[None, :])
    spread = np.exp(-d / 2.5) * np.cos(1.3 * d)
    sc = 0.1 / dt
    a21 = sc * r.uniform(-1, 1, (nchi, 8))
    a12 = np.ascontiguousarray((sc * r.uniform(-1, 1, (4, nchi, 1)) * spread[None]).reshape(4 * nchi, nchi))
    a22 = np.ascontiguousarray(-2 * sc * spread * (1 + 0.1 * r.uniform(-1, 1, (nchi, 1))))
    return a21, a12, a22


def _upstream_blocks(nchi, seed, dt):
    r = np.random.default_rng(seed + 9)
    bq = 0.05 / dt * r.uniform(-1, 1, (nchi, 3, 4, 4))
    bs = 0.05 / dt * r.uniform(-1, 1, (nchi, 3, 4))
    bq[0, 0], bq[-1, 2], bs[0, 0], bs[-1, 2] = 0, 0, 0, 0
    return bq, bs


def _vectors(c, n, m, seed):
    """m unit-norm vectors of n entries, smooth modes with noise as Krylov vectors carry."""
    x = torch.randn(m, n, generator=_gen(seed + 3), device=DEV, dtype=F64)
    t = torch.arange(n, device=DEV, dtype=F64) / n
    k = torch.arange(1, m + 1, device=DEV, dtype=F64)[:, None]
    x = 0.3 * x + torch.sin(40 * k * t + k)
    return (x / x.norm(dim=1, keepdim=True)).contiguous()


def _operator(c, seed):
    sol = S.Solution(C.initial_state(C.cylinder_config(c["nchi"], c["neta"]), seed=1))
    L = S.LinearOperatorGPU(sol)
    B, dt = _blocks(c["nchi"], c["neta"], seed)
    L.set_blocks(B.permute(3, 4, 0, 1, 2).reshape(-1).cpu().numpy())
    return sol, L, dt


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "march":
        cs = C.initial_state(_flow_config(c), seed=seed + 1)
        sol = S.Solution(cs)
        host = [_pinned(np.ascontiguousarray(v)) for v in (cs.q_flat(), cs.pts_x, cs.pts_y, cs.pts_chi, cs.pts_eta,
                                                          cs.cell_idx)]
        return dict(c=c, sol=sol, host=host, t=float(cs.t))
    if kind == "residual":
        cs = C.initial_state(C.channel_config(c["nchi"], c["neta"]), seed=1, noise=0.0)
        sol = S.Solution(cs)
        q = _channel_state(c, seed)
        full = np.zeros((4, c["neta"] + 2, c["nchi"] + 2))
        full[:, 1:-1, 1:-1] = q
        full[:, 0], full[:, -1] = full[:, 1], full[:, -2]
        full[:, :, 0], full[:, :, -1] = full[:, :, -2], full[:, :, 1]
        sol.set_state(full.reshape(-1), cs.pts_x, cs.pts_y, cs.pts_chi, cs.pts_eta, cs.cell_idx, 0.0)
        return dict(c=c, sol=sol)
    if kind == "linearize":
        cfg = C.cylinder_config(c["nchi"], c["neta"], perturb_shock=bool(c["shock"]))
        sol = S.Solution(C.initial_state(cfg, seed=seed + 1, noise=1e-4))
        n = 4 * sol.N + (sol.nchi if c["shock"] else 0)
        X = _vectors(c, n, c["k"], seed)
        return dict(c=c, sol=sol, X=X, Y=torch.empty_like(X))
    sol, L, dt = _operator(c, seed)
    st = dict(c=c, sol=sol, L=L, dt=dt)
    nchi, neta = c["nchi"], c["neta"]
    rows = _rows(nchi, neta, seed)
    if kind == "propagate" and c["shock"]:
        L.set_shock_blocks((rows,) + _shock_blocks(nchi, seed, dt))
    if kind == "receptivity":
        bq, bs = _upstream_blocks(nchi, seed, dt)
        sol.ctx.check(sol.ctx.L.hymor_b_set(sol.ctx.h, ip(rows), dp(np.ascontiguousarray(bq.ravel())),
                                            dp(np.ascontiguousarray(bs.ravel()))))
        st["w"] = np.linspace(0.0, 0.2 / dt / c["steps"], c["nw"])
        n = ctypes.c_int64()
        sol.ctx.check(sol.ctx.L.hymor_recept_size(sol.ctx.h, c["nw"], ctypes.byref(n)))
        st["X"] = _vectors(c, n.value, 2, seed)          # real and imaginary part
    else:
        st["X"] = _vectors(c, L.n, c["k"], seed)
    st["Y"] = torch.empty_like(st["X"])
    return st


# ---------------------------------------------------------------------------
# one pass


def run(state):
    c, sol = state["c"], state["sol"]
    kind = c["kind"]
    if kind == "march":
        q, px, py, pc, pe, ci = state["host"]
        state["t"] = sol.advect_host(q, px, py, pc, pe, ci, state["t"], c["steps"])
        return dict(q=q, pts_x=px, pts_y=py, pts_chi=pc, pts_eta=pe, cell_idx=ci, t=state["t"])
    if kind == "residual":
        return S.PDE(sol)
    X, Y = state["X"], state["Y"]
    lib, h = sol.ctx.L, sol.ctx.h
    if kind == "linearize":
        _, L = S.LINEARIZE_L(sol)
        sol.ctx.check(lib.hymor_matvec_dev(h, c["k"], X.data_ptr(), Y.data_ptr(), 0))
        if c["shock"]:
            return [Y, *L.shock_blocks()]
        return Y
    if kind == "matvec":
        sol.ctx.check(lib.hymor_matvec_dev(h, c["k"], X.data_ptr(), Y.data_ptr(), int(c["adjoint"])))
    elif kind == "propagate":
        sol.ctx.check(lib.hymor_expm_apply_dev(h, c["k"], state["dt"], c["steps"], c["order"], X.data_ptr(),
                                               Y.data_ptr(), int(c["adjoint"])))
    else:
        sol.ctx.check(lib.hymor_recept_expm_dev(h, 1, c["nw"], dp(state["w"]), state["dt"], c["steps"], c["order"],
                                                X.data_ptr(), Y.data_ptr(), int(c["adjoint"])))
    return Y


def work(case):
    """Bytes: each input read once and each output written once per pass, the operator once per
    application (a propagation applies it steps x order times). Flops: the residual's ~600 per
    cell of face fluxes, gradients and sums, 288 per cell and vector of the stencil blocks."""
    c = dict(case)
    N = c["nchi"] * c["neta"]
    kind = c["kind"]
    if kind == "march":
        # per stage: 4 variables read and written, 4 geometry planes of either face family
        return dict(bytes=c["steps"] * 4 * N * 8 * (4 + 4 + 9 + 9) + 2 * 32 * N, flops=c["steps"] * 4 * N * 640)
    if kind == "residual":
        return dict(bytes=N * 8 * (4 + 4 + 18), flops=N * 600)
    op = 144 * 8 * N
    if kind == "linearize":
        shock = 8 * 10 * c["nchi"] ** 2 if c["shock"] else 0
        return dict(bytes=N * 8 * (4 + 18) + 2 * op + 64 * N * c["k"] + shock, flops=36 * N * 600 + 288 * N * c["k"])
    if kind == "matvec":
        return dict(bytes=op + 64 * N * c["k"], flops=288 * N * c["k"])
    m = c["steps"] * c["order"]
    if kind == "propagate":
        shock = 10 * c["nchi"] ** 2 if c["shock"] else 0
        return dict(bytes=m * (op + 4 * shock) + 64 * N * c["k"], flops=m * (288 * N + shock) * c["k"])
    return dict(bytes=m * op + 2 * 16 * (4 * N + 4 * c["nchi"] * c["nw"]),
                flops=m * 2 * (288 * N + 16 * c["nchi"] * c["nw"]))


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits


def _channel_state(c, seed):
    """(4, neta, nchi): a plane Poiseuille profile with smooth perturbations and noise."""
    r = np.random.default_rng(seed + 21)
    nchi, neta = c["nchi"], c["neta"]
    x = (np.arange(nchi) + 0.5)[None, :] / nchi * 2 * math.pi
    y = ((np.arange(neta) + 0.5) / neta)[:, None]
    f = 4 * y * (1 - y)
    ph = r.uniform(0, 6, 4)
    rho = 1 + 1e-3 * np.sin(x + ph[0]) * f + 1e-5 * r.standard_normal((neta, nchi))
    u = f * (1 + 0.02 * np.sin(2 * x + ph[1])) + 1e-4 * r.standard_normal((neta, nchi))
    v = 0.02 * np.cos(x + ph[2]) * f + 1e-4 * r.standard_normal((neta, nchi))
    p = 1 / 1.4 / 0.05**2 * (1 + 2e-4 * np.cos(x + ph[3]) * f)
    return np.stack([rho, rho * u, rho * v, p / 0.4 + 0.5 * rho * (u * u + v * v)])


def _channel_residual(c, seed):
    """The finite-volume residual on the channel's rectangular cells: central face averages,
    viscous gradients from the cells across a face and the corner averages along it (whose
    sign along the face is the reference's, VISCOUS_FLUX.jl:98-127)."""
    nchi, neta, g, Pr, Re = c["nchi"], c["neta"], 1.4, 0.73, 7500.0
    q = torch.as_tensor(_channel_state(c, seed))
    e = torch.linspace(0, 1, neta + 1, dtype=F64)
    s = 1.6
    yl = 2.0 * torch.where(e <= 0.5, 2 ** (s - 1) * e.abs() ** s, 1 - 2 ** (s - 1) * (1 - e).abs() ** s)
    dy = (yl[1:] - yl[:-1])[:, None]
    yc = (yl[1:] + yl[:-1]) / 2
    yg = torch.cat([2 * yl[:1] - yc[:1], yc, 2 * yl[-1:] - yc[-1:]])
    dyf = (yg[1:] - yg[:-1])[:, None]
    dx = 2 * math.pi / nchi

    def wrap(a):
        return torch.cat([a[..., -1:], a, a[..., :1]], dim=-1)
    r, ru, rv, rE = (wrap(a) for a in q)
    ei = rE - 0.5 * (ru * ru + rv * rv) / r
    p, T = ei * (g - 1), ei / r

    def walls(a, lo, hi):
        return torch.cat([lo[None], a, hi[None]])
    R, U, V = walls(r, r[0], r[-1]), walls(ru, -ru[0], -ru[-1]), walls(rv, -rv[0], -rv[-1])
    E, P = walls(rE, 2 * rE[0] - rE[1], 2 * rE[-1] - rE[-2]), walls(p, 2 * p[0] - p[1], 2 * p[-1] - p[-2])
    T = walls(T, T[0], T[-1])
    u, v = U / R, V / R

    def corner(a):
        return (a[:-1, :-1] + a[1:, :-1] + a[:-1, 1:] + a[1:, 1:]) / 4

    def flux(A, nx, ny, d, along):
        # A: (first, second) of each variable across the face; d: the gradients' distances
        (ra, rb), (ua, ub), (va, vb), (ea, eb), (pa, pb) = A[:5]
        sr, su, sv, se, sp = ra + rb, ua + ub, va + vb, ea + eb, pa + pb
        vn = (su * nx + sv * ny) / sr
        dn = [(b - a) / d for a, b in A[5:]]                    # u, v, T across
        ux, uy = (dn[0], along[0]) if nx else (along[0], dn[0])
        vx, vy = (dn[1], along[1]) if nx else (along[1], dn[1])
        div = ux + vy
        if nx:
            tx, ty = (2 * ux - 2 / 3 * div) / Re, (uy + vx) / Re
        else:
            tx, ty = (uy + vx) / Re, (2 * vy - 2 / 3 * div) / Re
        qn = g / (Re * Pr) * dn[2]
        w = (su * tx + sv * ty) / sr
        return [(su * nx + sv * ny) / 2, su * vn / 2 + sp * nx / 2 - tx, sv * vn / 2 + sp * ny / 2 - ty,
                (se + sp) * vn / 2 - w - qn]
    uc, vc = corner(u), corner(v)
    lr = [(a[1:-1, :-1], a[1:-1, 1:]) for a in (R, U, V, E, P, u, v, T)]
    fx = flux(lr, 1.0, 0.0, dx, [(a[:-1] - a[1:]) / dy for a in (uc, vc)])
    bt = [(a[:-1, 1:-1], a[1:, 1:-1]) for a in (R, U, V, E, P, u, v, T)]
    fy = flux(bt, 0.0, 1.0, dyf, [(a[:, :-1] - a[:, 1:]) / dx for a in (uc, vc)])
    out = [(a[:, :-1] - a[:, 1:]) / dx + (b[:-1] - b[1:]) / dy for a, b in zip(fx, fy)]
    return torch.stack(out).reshape(-1).numpy()


def _apply(B, x, adjoint):
    """The stencil operator on x (m, 4, neta, nchi)."""
    m, _, neta, nchi = x.shape
    y = torch.zeros_like(x)
    pad = torch.nn.functional.pad
    for q in range(9):
        a, b = q % 3 - 1, q // 3 - 1
        if not adjoint:
            xs = pad(x, (1, 1, 1, 1))[:, :, 1 + b:1 + b + neta, 1 + a:1 + a + nchi]
            for o in range(4):
                for i in range(4):
                    y[:, o] += B[q, o, i] * xs[:, i]
        else:
            z = torch.zeros_like(x)
            for i in range(4):
                for o in range(4):
                    z[:, i] += B[q, o, i] * x[:, o]
            y += pad(z, (1, 1, 1, 1))[:, :, 1 - b:1 - b + neta, 1 - a:1 - a + nchi]
    return y


def exact(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "residual":
        return _channel_residual(c, seed)
    if kind in ("march", "linearize"):
        return None
    nchi, neta = c["nchi"], c["neta"]
    N = nchi * neta
    B, dt = _blocks(nchi, neta, seed)
    adj = bool(c["adjoint"])
    col = torch.arange(nchi, device=DEV)
    rows = torch.as_tensor(_rows(nchi, neta, seed), device=DEV).long()

    def stencil(x):
        return _apply(B, x[:, :4 * N].reshape(-1, 4, neta, nchi), adj).reshape(x.shape[0], 4 * N)
    if kind == "matvec":
        X = _vectors(c, 4 * N, c["k"], seed)
        return torch.cat([stencil(X[i:i + 8]) for i in range(0, c["k"], 8)])
    if kind == "propagate" and not c["shock"]:
        op, n, m = stencil, 4 * N, c["k"]
    elif kind == "propagate":
        a21, a12, a22 = (torch.as_tensor(a, device=DEV) for a in _shock_blocks(nchi, seed, dt))
        n, m = 4 * N + nchi, c["k"]
        # cells (i, sc_i - 1) and (i, sc_i - 2) of every variable, ordered (j, v, i)
        cells = torch.stack([torch.stack([v * N + col + (rows - 1 - j) * nchi for v in range(4)]) for j in (1, 2)])
        a21 = a21.T.reshape(2, 4, nchi)

        def op(x):
            y, r = stencil(x), x[:, 4 * N:]
            near = cells[0].reshape(-1)
            if not adj:
                y[:, near] += r @ a12.T
                return torch.cat([y, (a21 * x[:, cells]).sum(dim=(1, 2)) + r @ a22.T], dim=1)
            tail = x[:, near] @ a12 + r @ a22
            for j in range(2):
                y[:, cells[j]] += a21[j] * r[:, None, :]
            return torch.cat([y, tail], dim=1)
    else:
        bq = torch.as_tensor(_upstream_blocks(nchi, seed, dt)[0], device=DEV)
        nw = c["nw"]
        w = torch.as_tensor(np.linspace(0.0, 0.2 / dt / c["steps"], nw), device=DEV)[None, :, None, None]
        n, m = 4 * N + 4 * nchi * nw, 2
        near = torch.stack([v * N + col + (rows - 2) * nchi for v in range(4)])           # (4, nchi)

        def op(x):
            y, u = stencil(x), x[:, 4 * N:].reshape(2, nw, 4, nchi)
            rot = torch.stack([w[0] * u[1], -w[0] * u[0]])       # -i w u
            if adj:
                rot = -rot
                up = torch.nn.functional.pad(torch.zeros_like(x[:, near]), (1, 1))
                for d in range(3):
                    t = torch.einsum("noi,ron->rin", bq[:, d], x[:, near])
                    up[:, :, d:d + nchi] += t
                rot = rot + up[:, None, :, 1:-1]
            else:
                s = torch.nn.functional.pad(u.sum(dim=1), (1, 1))
                for d in range(3):
                    y[:, near] += torch.einsum("noi,rin->ron", bq[:, d], s[:, :, d:d + nchi])
            return torch.cat([y, rot.reshape(2, -1)], dim=1)
    x = _vectors(c, n, m, seed)
    for _ in range(c["steps"]):
        term, out = x, x.clone()
        for j in range(1, c["order"] + 1):
            term = op(term) * (dt / j)
            out += term
        x = out
    return x
