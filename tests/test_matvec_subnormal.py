"""The batched matvec on factors below the normal range: a vector, or a patch of blocks, whose
values are subnormal is not zero, and its products with large factors are ordinary numbers. Held
against sums in extended precision to the bound of a dot product in FP64 (36 products)."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S

pytestmark = pytest.mark.gpu

NCHI, NETA, K = 203, 141, 42    # a batch that takes the fixed point
PATCH = (slice(60, 67), slice(40, 80))    # cells (eta, chi) of the subnormal blocks


def _apply(B, X, transpose, absolute=False):
    B, X = B.astype(np.longdouble), X.astype(np.longdouble)
    if absolute:
        B, X = np.abs(B), np.abs(X)
    Y = np.zeros_like(X)
    for q in range(9):
        a, b = q % 3 - 1, q // 3 - 1
        jo = slice(max(0, -b), NETA - max(0, b))
        io = slice(max(0, -a), NCHI - max(0, a))
        ji = slice(max(0, b), NETA - max(0, -b))
        ii = slice(max(0, a), NCHI - max(0, -a))
        if transpose:
            Y[:, ji, ii] += np.einsum("jioe,oji->eji", B[jo, io, q], X[:, jo, io])
        else:
            Y[:, jo, io] += np.einsum("jioe,eji->oji", B[jo, io, q], X[:, ji, ii])
    return Y


@pytest.mark.parametrize("where", ["vector", "component", "blocks"])
def test_subnormal_factors(require_gpu, where):
    sol = S.Solution(C.initial_state(C.cylinder_config(NCHI, NETA)))
    L = S.LinearOperatorGPU(sol)
    r = np.random.Generator(np.random.PCG64(11))
    B = r.standard_normal((NETA, NCHI, 9, 4, 4)) * 1e5
    X = r.standard_normal((L.n, K))
    if where == "vector":
        X[:, 1] *= 1e-310
    elif where == "component":       # one component alone, in a patch of its vector
        x = np.zeros((4, NETA, NCHI))
        x[2][PATCH] = 1e-310 * r.standard_normal(x[2][PATCH].shape)
        X[:, 1] = x.reshape(-1)
    else:
        B[PATCH] *= 1e-315
        X[:, 1] *= 1e5
    L.set_blocks(np.ascontiguousarray(B.reshape(-1)))
    for A, tr in ((L, False), (L.T, True)):
        Y = A @ X
        for v in (0, 1):
            x = X[:, v].reshape(4, NETA, NCHI)
            err = np.abs(Y[:, v].reshape(x.shape) - _apply(B, x, tr))
            assert (err <= 36 * 2.0**-53 * _apply(B, x, tr, True) + 36 * 5e-324).all()
    sol.close()
