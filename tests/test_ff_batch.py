"""The float-float propagation's batch tiles and one-cell-per-thread path: sizes at the edges of
the tiles and of their chunks, periodic wraps, per-vector step counts, and cells without entries,
against the FP64 propagation."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S
from hymor_gb300._lib import dp, ip
from hymor_gb300.krylov import DeviceBuffer

from helpers import rel_err

pytestmark = pytest.mark.gpu

# float-float rounding ~2^-44 per product sum, 20 matvecs of an operator of norm ~1 per step
TOL = 1e-11


def _solution(make, nchi, neta):
    sol = S.Solution(C.initial_state(make(nchi, neta)))
    if sol.cfg.shock_enabled:
        S.ADVECT_FLOW(sol, 2)
    _, L = S.LINEARIZE_L(sol)
    return sol, L, S.CFL_TIMESTEP(sol)


@pytest.mark.parametrize("make,nchi,neta,k", [
    (C.cylinder_config, 97, 45, 11),    # chunks of 4, 4, 3; a tile column of one cell
    (C.cylinder_config, 64, 160, 5),    # whole tiles, chunks of 3 and 2
    (C.channel_config, 33, 35, 36),     # periodic; rows and columns past the last tile
    (C.channel_config, 128, 100, 4),
    (C.blunt_cone_config, 201, 101, 2),
    (C.cylinder_config, 230, 180, 1),   # one vector, a cell per thread
    (C.channel_config, 209, 193, 1),
    (C.cylinder_config, 60, 40, 13),    # below the tiles: a thread per output
])
def test_against_fp64(require_gpu, make, nchi, neta, k):
    sol, L, dt = _solution(make, nchi, neta)
    X = np.random.Generator(np.random.PCG64(5)).standard_normal((L.n, k))
    for A in (L, L.T):
        sol.set_expm_arith(1)
        yf = A.expm(X, dt, 5, order=4)
        sol.set_expm_arith(0)
        assert rel_err(yf, A.expm(X, dt, 5, order=4)) < TOL
    sol.close()


def test_step_counts_shrink_the_batch(require_gpu):
    """Vectors that finish early leave the batch: each equals its own propagation bit for bit
    (the tiles, the cell-per-thread and the thread-per-output path form the same pairs)."""
    sol, L, dt = _solution(C.cylinder_config, 110, 90)
    k, n = 6, L.n
    X = np.random.Generator(np.random.PCG64(6)).standard_normal((k, n))
    steps = np.array([9, 7, 7, 6, 4, 4], dtype=np.int32)
    dts = dt * np.linspace(1.0, 0.5, k)
    bx, by = DeviceBuffer(sol.ctx, 8 * n * k), DeviceBuffer(sol.ctx, 8 * n * k)
    bx.upload(X.ravel())
    sol.ctx.check(sol.ctx.L.hymor_expm_apply_multi_dev(sol.ctx.h, k, dp(dts), ip(steps), 5, bx.ptr, by.ptr, 0))
    Y = by.download(n * k).reshape(k, n)
    for c in range(k):
        assert np.array_equal(Y[c], L.expm(X[c], dts[c], int(steps[c])))
    bx.free()
    by.free()
    sol.close()
