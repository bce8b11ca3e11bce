"""The float-float propagation of a small grid resident on chip: tilings of one tile in a
direction, periodic wraps onto the tile itself and onto a single neighbour, ragged last tiles,
repeated calls (the flags start anew), and several contexts at once."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S
from hymor_gb300.krylov import DeviceBuffer

from helpers import rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-11   # float-float rounding ~2^-44 per product sum over 40 matvecs


def _solution(make, nchi, neta, seed=1):
    sol = S.Solution(C.initial_state(make(nchi, neta), seed=seed))
    if sol.cfg.shock_enabled:
        S.ADVECT_FLOW(sol, 2)
    _, L = S.LINEARIZE_L(sol)
    return sol, L, S.CFL_TIMESTEP(sol)


@pytest.mark.parametrize("make,nchi,neta,k", [
    (C.channel_config, 4, 5, 2),       # one tile, its own periodic neighbour
    (C.channel_config, 8, 300, 1),     # two tiles in chi, each the other's neighbour twice
    (C.channel_config, 64, 4, 3),
    (C.channel_config, 101, 79, 1),
    (C.cylinder_config, 100, 80, 1),
    (C.cylinder_config, 53, 29, 7),
    (C.cylinder_config, 160, 121, 2),  # nearly all of the shared memory
    (C.blunt_cone_config, 31, 23, 4),
])
@pytest.mark.parametrize("order,steps", [(2, 20), (5, 8)])
def test_against_fp64(require_gpu, make, nchi, neta, k, order, steps):
    sol, L, dt = _solution(make, nchi, neta)
    X = np.random.Generator(np.random.PCG64(7)).standard_normal((L.n, k))
    for A in (L, L.T):
        sol.set_expm_arith(1)
        yf = A.expm(X, dt, steps, order=order)
        assert np.array_equal(yf, A.expm(X, dt, steps, order=order))
        sol.set_expm_arith(0)
        assert rel_err(yf, A.expm(X, dt, steps, order=order)) < TOL
    sol.close()


def test_contexts_at_once(require_gpu):
    """Propagations of several contexts in flight together give what each gives alone."""
    sets = [_solution(C.cylinder_config, 60 + 20 * c, 45, seed=c) for c in range(3)]
    rng = np.random.Generator(np.random.PCG64(8))
    xs = [rng.standard_normal(L.n) for _, L, _ in sets]
    alone = [L.expm(x, dt, 30) for (_, L, dt), x in zip(sets, xs)]
    bufs = [(DeviceBuffer(s.ctx, 8 * L.n), DeviceBuffer(s.ctx, 8 * L.n)) for s, L, _ in sets]
    for (bx, _), x in zip(bufs, xs):
        bx.upload(x)
    for _ in range(4):
        for (s, L, dt), (bx, by) in zip(sets, bufs):
            s.ctx.check(s.ctx.L.hymor_expm_apply_dev(s.ctx.h, 1, dt, 30, 5, bx.ptr, by.ptr, 0))
    for (s, L, _), (_, by), ref in zip(sets, bufs, alone):
        s.ctx.check(s.ctx.L.hymor_synchronize(s.ctx.h))
        assert np.array_equal(by.download(L.n), ref)
    for pair in bufs:
        for b in pair:
            b.free()
    for s, _, _ in sets:
        s.close()
