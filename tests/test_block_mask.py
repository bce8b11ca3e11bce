"""The matvecs that leave out cells without entries: the same products as the ones that read
every block, and the same NaN where a zero block meets an infinity or a NaN."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S
from oracle import oracle as O

from helpers import rel_err

pytestmark = pytest.mark.gpu


def _blocks(nchi, neta, seed):
    """Random blocks (zero across the grid's edges) with empty cells: a band at the top, scattered
    single cells, and cells with entries of one input variable only."""
    r = np.random.Generator(np.random.PCG64(seed))
    B = r.standard_normal((neta, nchi, 9, 4, 4))
    for q in range(9):
        a, b = q % 3 - 1, q // 3 - 1
        if a:
            B[:, 0 if a < 0 else nchi - 1, q] = 0
        if b:
            B[0 if b < 0 else neta - 1, :, q] = 0
    empty = r.random((neta, nchi)) < 0.2
    empty[2 * neta // 3:] = True
    B[empty] = 0
    B[neta // 4, ::3, :, :, 1:] = 0
    return np.ascontiguousarray(B.reshape(-1))


def _operator(nchi, neta, seed=1):
    cs = C.initial_state(C.cylinder_config(nchi, neta))
    sol = S.Solution(cs)
    L = S.LinearOperatorGPU(sol)
    co = _blocks(nchi, neta, seed)
    L.set_blocks(co)
    return cs, sol, L, co


@pytest.mark.parametrize("nchi,neta", [(83, 59), (230, 131)])
def test_batched_matvec(require_gpu, nchi, neta):
    """Past the thread-per-output path with an odd last chunk: in FP64, and in fixed point."""
    k = 41
    cs, sol, L, co = _operator(nchi, neta)
    orc = O.Oracle(cs)
    X = np.random.Generator(np.random.PCG64(2)).standard_normal((L.n, k))
    N = nchi * neta
    # non-finite inputs in and below the empty band, in the middle and in the last vectors
    for vec, v, m, val in ((0, 2, N - 5, np.inf), (17, 0, N // 2, np.nan), (40, 3, (2 * neta // 3) * nchi + 7, -np.inf)):
        X[v * N + m, vec] = val
    for A in (L, L.T):
        Y = A @ X
        for vec in (0, 17, 40):           # one vector: every block is read
            one = A @ np.ascontiguousarray(X[:, vec])
            assert np.array_equal(np.isnan(Y[:, vec]), np.isnan(one)) and np.isnan(one).any()
            ok = np.isfinite(one)
            assert rel_err(Y[ok, vec], one[ok]) < 1e-14
        for vec in (1, 39):
            ref = orc.matvec(co, X[:, vec], transpose=A is not L)
            assert rel_err(Y[:, vec], ref) < 1e-13
    sol.close()


@pytest.mark.parametrize("nan", [False, True])
def test_one_vector_on_a_large_grid(require_gpu, nan):
    """FP64 matvec and float-float propagation of one vector past the thread-per-output path,
    against the FP64 propagation in steps too few for the cooperative kernel (no mask there up
    to its FP64 matvecs, whose own masks the test above covers)."""
    nchi, neta = 410, 381
    cs, sol, L, co = _operator(nchi, neta)
    x = np.random.Generator(np.random.PCG64(3)).standard_normal(L.n)
    if nan:
        x[3 * nchi * neta - 9] = np.inf
    for A in (L, L.T):
        got = A.expm(x, 1e-3, 4, order=4)
        ref = x
        for _ in range(4):
            ref = A.expm(ref, 1e-3, 1, order=4)
        assert np.array_equal(np.isfinite(got), np.isfinite(ref))
        ok = np.isfinite(ref)
        assert ok.all() != nan and rel_err(got[ok], ref[ok]) < 1e-11
    sol.close()
