"""Storage in several parts of which only the first fits: the entry point fails each time it is
called, and works once there is room (a part alone must not pass for the whole)."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import receptivity as R
from hymor_gb300 import solver as S
from hymor_gb300._lib import HymorError

pytestmark = pytest.mark.gpu

NCHI, NETA = 64, 33
N = NCHI * NETA
BLOCKS = 8 * 152 * N + 5 * N          # the stencil blocks with their masks and workspace


def _refused(call):
    with pytest.raises(HymorError) as e:
        call()
    assert e.value.code == -2


@pytest.mark.parametrize("limit", [8 * 144 * N, 8 * 144 * N + 5 * N])
def test_jacobian(require_gpu, limit):
    sol = S.Solution(C.initial_state(C.cylinder_config(NCHI, NETA)))
    B = np.random.Generator(np.random.PCG64(1)).standard_normal(144 * N)
    L = S.LinearOperatorGPU(sol)
    x = np.ones(L.n)
    sol.ctx.check(sol.ctx.L.hymor_set_workspace_limit(sol.ctx.h, limit))
    for _ in range(3):
        _refused(lambda: L.set_blocks(B))
    sol.ctx.check(sol.ctx.L.hymor_set_workspace_limit(sol.ctx.h, BLOCKS))   # nothing was kept
    L.set_blocks(B)
    assert np.isfinite(L @ x).all()
    sol.close()


def test_shock_blocks(require_gpu):
    sol = S.Solution(C.initial_state(C.cylinder_config(NCHI, NETA)))
    L = S.LinearOperatorGPU(sol)
    L.set_blocks(np.zeros(144 * N))
    r = np.random.Generator(np.random.PCG64(2))
    blocks = (np.full(NCHI, 12, np.int32), r.standard_normal((NCHI, 8)), r.standard_normal((4, NCHI, NCHI)),
              r.standard_normal((NCHI, NCHI)))
    sol.ctx.check(sol.ctx.L.hymor_set_workspace_limit(sol.ctx.h, BLOCKS + 8 * (10 * NCHI * NCHI + 11 * NCHI)))
    for _ in range(3):
        _refused(lambda: L.set_shock_blocks(blocks))
    sol.ctx.check(sol.ctx.L.hymor_set_workspace_limit(sol.ctx.h, 0))
    L.set_shock_blocks(blocks)
    assert np.array_equal(L.shock_blocks()[0], blocks[0])
    sol.close()


def test_upstream_operator(require_gpu):
    sol = S.Solution(C.initial_state(C.cylinder_config(NCHI, NETA)))
    S.LinearOperatorGPU(sol).set_blocks(np.zeros(144 * N))
    sol.ctx.check(sol.ctx.L.hymor_set_workspace_limit(sol.ctx.h, BLOCKS + 8 * 65 * NCHI))
    for _ in range(3):
        _refused(lambda: R.LINEARIZE_B(sol))
    sol.ctx.check(sol.ctx.L.hymor_set_workspace_limit(sol.ctx.h, 0))
    rows, bq, bs = R.LINEARIZE_B(sol)
    assert (rows >= 2).all() and np.isfinite(bq).all()
    sol.close()
