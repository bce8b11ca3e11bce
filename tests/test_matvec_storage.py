"""The storage of the fixed-point matvec: FP64 instructions in hymor_set_expm_arith(0), and in the
direction whose integer parts do not fit; the parts give way to what the context needs beside
them, and come back with room and a write of the blocks."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S

pytestmark = pytest.mark.gpu

NCHI, NETA, K = 203, 141, 42    # a batch that takes the fixed point
N = NCHI * NETA
BLOCKS, PARTS = 1221 * N, 1184 * N


def test_storage(require_gpu):
    sol = S.Solution(C.initial_state(C.cylinder_config(NCHI, NETA)))
    L = S.LinearOperatorGPU(sol)
    r = np.random.Generator(np.random.PCG64(1))
    B, X = r.standard_normal(144 * N) / 12, r.standard_normal((L.n, K))
    limit = lambda b: sol.ctx.check(sol.ctx.L.hymor_set_workspace_limit(sol.ctx.h, b))
    L.set_blocks(B)
    fx, fx_t = L @ X, L.T @ X
    sol.set_expm_arith(0)
    fp, fp_t = L @ X, L.T @ X
    assert not np.array_equal(fx, fp) and not np.array_equal(fx_t, fp_t)
    assert np.allclose(fx, fp, rtol=0, atol=1e-13)
    propagated = L.expm(X[:, 0], 1e-3, 10)
    sol.close()

    sol = S.Solution(C.initial_state(C.cylinder_config(NCHI, NETA)))
    L = S.LinearOperatorGPU(sol)
    L.set_blocks(B)
    limit(BLOCKS + PARTS + 1000)
    for _ in range(2):                       # room for one direction's parts
        assert np.array_equal(L @ X, fx) and np.array_equal(L.T @ X, fp_t)
    # the propagator's copy of the blocks needs their room, and keeps it
    limit(BLOCKS + PARTS + 200 * N)
    assert np.allclose(L.expm(X[:, 0], 1e-3, 10), propagated, rtol=0, atol=1e-11)
    for _ in range(2):
        assert np.array_equal(L @ X, fp)
    limit(0)
    assert np.array_equal(L @ X, fx) and np.array_equal(L.T @ X, fx_t)
    # a mode of FP64 gives them back: what fits beside the blocks alone fits now
    sol.set_expm_arith(0)
    assert np.array_equal(L @ X, fp)
    sol.set_expm_arith(1)
    assert np.array_equal(L @ X, fx)
    L.set_blocks(2 * B)
    assert np.array_equal(L @ X, 2 * fx)
    sol.close()


def test_linearisation_beside_the_parts(require_gpu):
    """Parts that fill the limit do not cost the linearisation its lanes."""
    cs = C.initial_state(C.cylinder_config(NCHI, NETA))
    ref = S.Solution(cs)
    _, L0 = S.LINEARIZE_L(ref)
    sol = S.Solution(cs)
    L = S.LinearOperatorGPU(sol)
    L.set_blocks(L0.blocks())
    sol.ctx.check(sol.ctx.L.hymor_set_workspace_limit(sol.ctx.h, BLOCKS + PARTS + 1000))
    X = np.ones((L.n, K))
    fx = L @ X
    _, L1 = S.LINEARIZE_L(sol)
    assert np.array_equal(L1.blocks(), L0.blocks())
    assert np.allclose(L1 @ X, fx, rtol=1e-10, atol=1e-10 * np.abs(fx).max())
    for s in (ref, sol):
        s.close()
