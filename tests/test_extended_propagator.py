"""The one-launch propagation of the extended operators against the Taylor recurrence over
single operator applications: degrees with and without the late first term, the shock-position
unknowns and the receptivity operator alone and together, B's rows on and off the A12 rows."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import receptivity as R
from hymor_gb300 import solver as S
from hymor_gb300._lib import dp, ip

pytestmark = pytest.mark.gpu

# both sides apply the same blocks in FP64, in different orders: ~sqrt(row length) 2^-53 per
# term, over at most 24 x 5 terms of a propagation that neither grows nor decays by more than e
TOL = 1e-13


def _setup(nchi, neta, shock):
    cs = C.initial_state(C.cylinder_config(nchi, neta, perturb_shock=shock))
    sol = S.Solution(cs)
    S.ADVECT_FLOW(sol, 3)
    _, L = S.LINEARIZE_L(sol)
    return sol, L, S.CFL_TIMESTEP(sol) * 0.3


@pytest.mark.parametrize("nchi,neta", [(35, 21), (96, 40)])
@pytest.mark.parametrize("order", [1, 2, 5])
def test_shock_propagation(require_gpu, nchi, neta, order):
    sol, L, dt = _setup(nchi, neta, True)
    X = np.random.Generator(np.random.PCG64(3)).standard_normal((L.n, 3))
    steps = 24 // order
    for A in (L, L.T):
        got = A.expm(X, dt, steps, order=order)
        ref = X
        for _ in range(steps):
            term, out = ref, ref.copy()
            for j in range(1, order + 1):
                term = (A @ term) * (dt / j)
                out = out + term
            ref = out
        assert np.max(np.abs(got - ref)) <= TOL * np.max(np.abs(ref))
    sol.close()


@pytest.mark.parametrize("shock,shift", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("order", [1, 4])
def test_receptivity_propagation(require_gpu, shock, shift, order):
    sol, L, dt = _setup(37, 22, shock)
    rows, bq, bs = R.LINEARIZE_B(sol)
    _, Lr = R.LINEARIZE_L_(L, sol, np.linspace(0, 3, 35))   # more frequencies than lanes
    if shift:  # B of another linearisation: some of its rows are not the A12 rows
        rows = rows.copy()
        rows[::3] -= 1
        c = sol.ctx
        c.check(c.L.hymor_b_set(c.h, ip(rows), dp(np.ascontiguousarray(bq.ravel())),
                                dp(np.ascontiguousarray(bs.ravel()))))
    rng = np.random.Generator(np.random.PCG64(4))
    x = rng.standard_normal(Lr.n) + 1j * rng.standard_normal(Lr.n)
    for adj in (False, True):
        got = Lr.expm(x, dt, 24 // order, adjoint=adj, order=order)
        ref = x
        for _ in range(24 // order):
            term, out = ref, ref.copy()
            for j in range(1, order + 1):
                term = Lr.apply(term, adjoint=adj) * (dt / j)
                out = out + term
            ref = out
        assert np.max(np.abs(got - ref)) <= TOL * np.max(np.abs(ref))
    sol.close()
