"""The batched matvec in fixed point against sums in extended precision: never further off than
the bound of an FP64 dot product, in the norm no further than the FP64 one-vector path, exact for
unit vectors, and in FP64 where its parts could not hold the factors."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S

pytestmark = pytest.mark.gpu

NCHI, NETA, K = 203, 141, 42    # a batch that takes the fixed point; no multiples of tiles or chunks


def _operator(make=C.cylinder_config, scale=lambda r, s: 1.0, seed=1):
    sol = S.Solution(C.initial_state(make(NCHI, NETA)))
    L = S.LinearOperatorGPU(sol)
    r = np.random.Generator(np.random.PCG64(seed))
    B = r.standard_normal((NETA, NCHI, 9, 4, 4)) * scale(r, (NETA, NCHI, 9, 4, 4))
    L.set_blocks(np.ascontiguousarray(B.reshape(-1)))
    return sol, L, B, make is C.channel_config


def _apply(B, X, transpose, periodic, absolute=False):
    """Σ a x (or Σ |a| |x|) in extended precision; X (4, NETA, NCHI)."""
    B, X = B.astype(np.longdouble), X.astype(np.longdouble)
    if absolute:
        B, X = np.abs(B), np.abs(X)
    Y = np.zeros_like(X)
    for q in range(9):
        a, b = q % 3 - 1, q // 3 - 1
        for j in range(NETA):
            if not 0 <= j + b < NETA:
                continue
            i = np.arange(NCHI)
            ii = i + a
            ok = np.ones(NCHI, bool) if periodic else (ii >= 0) & (ii < NCHI)
            i, ii = i[ok], ii[ok] % NCHI
            if transpose:
                np.add.at(Y[:, j + b], (slice(None), ii), np.einsum("noi,on->in", B[j, i, q], X[:, j, i]))
            else:
                Y[:, j, i] += np.einsum("noi,in->on", B[j, i, q], X[:, j + b, ii])
    return Y


def _check(L, B, X, periodic, vecs=(0, K - 1)):
    for A, tr in ((L, False), (L.T, True)):
        Y = A @ X
        for v in vecs:
            x = X[:, v].reshape(4, NETA, NCHI)
            ref = _apply(B, x, tr, periodic)
            err = np.abs(Y[:, v].reshape(ref.shape) - ref)
            assert (err <= 36 * 2.0**-53 * _apply(B, x, tr, periodic, True)).all()
            one = np.abs((A @ np.ascontiguousarray(X[:, v])).reshape(ref.shape) - ref)
            assert np.sqrt((err**2).sum()) <= np.sqrt((one**2).sum())


@pytest.mark.parametrize("make", [C.cylinder_config, C.channel_config])
def test_random(require_gpu, make):
    sol, L, B, per = _operator(make, lambda r, s: np.where(r.random(s) < 0.3, 10.0 ** r.integers(-6, 1, s), 1.0))
    X = np.random.Generator(np.random.PCG64(2)).standard_normal((L.n, K))
    X[:NCHI * NETA] *= 1e-3      # components of different magnitudes
    _check(L, B, X, per)
    sol.close()


def test_wide_ranges(require_gpu):
    """Vectors that fall by ten orders within a tile, sparse ones, and blocks whose rows do."""
    sol, L, B, per = _operator(scale=lambda r, s: 10.0 ** (-12 * r.random(s)))
    r = np.random.Generator(np.random.PCG64(3))
    X = r.standard_normal((L.n, K))
    X[:, 0] *= 10.0 ** (-10 * r.random(L.n))
    X[:, K - 1] *= r.random(L.n) < 0.05
    X[:, 5] = 0.0
    for A, tr in ((L, False), (L.T, True)):
        Y = A @ X
        assert not Y[:, 5].any()
        for v in (0, K - 1):
            x = X[:, v].reshape(4, NETA, NCHI)
            err = np.abs(Y[:, v].reshape(x.shape) - _apply(B, x, tr, per))
            assert (err <= 36 * 2.0**-53 * _apply(B, x, tr, per, True)).all()
    sol.close()


def test_unit_vectors_and_extremes(require_gpu):
    """L e_i is the operator's column bit for bit; magnitudes whose products leave the exponents
    of the parts go through FP64."""
    sol, L, B, per = _operator(scale=lambda r, s: 10.0 ** (-8 * r.random(s)))
    n, N = L.n, NCHI * NETA
    cells = np.random.Generator(np.random.PCG64(4)).choice(N, K, replace=False)
    X = np.zeros((n, K))
    for v, c in enumerate(cells):
        X[(v % 4) * N + c, v] = 1.0
    for A, tr in ((L, False), (L.T, True)):
        Y = A @ X
        for v in range(K):
            assert np.array_equal(Y[:, v], _apply(B, X[:, v].reshape(4, NETA, NCHI), tr, per).reshape(-1).astype(float))
    X = np.random.Generator(np.random.PCG64(5)).standard_normal((n, K))
    X[:, 1] *= 1e-290
    X[:, 2] *= 1e290
    for A in (L, L.T):
        Y = A @ X
        for v in (1, 2):
            one = A @ np.ascontiguousarray(X[:, v])
            assert np.allclose(Y[:, v], one, rtol=1e-11, atol=0 if v == 2 else 5e-324 * 100)
    sol.close()
