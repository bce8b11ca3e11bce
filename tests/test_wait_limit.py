"""A resident propagation whose wait for a neighbour's value runs out: NaN in its results and
HYMOR_ERR_TIMEOUT, once, from the call that returns or synchronises; the context goes on. The wait
is made to run out on purpose by a limit of no polls: the kernel returns at once."""
import ctypes

import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S
from hymor_gb300._lib import HymorError, dp
from hymor_gb300.krylov import DeviceBuffer

pytestmark = pytest.mark.gpu


@pytest.fixture
def linear(require_gpu):
    sol = S.Solution(C.initial_state(C.cylinder_config(60, 45), seed=1))
    _, L = S.LINEARIZE_L(sol)
    yield sol, L, S.CFL_TIMESTEP(sol)
    sol.close()


def test_host_call(linear):
    sol, L, dt = linear
    X = np.random.Generator(np.random.PCG64(1)).standard_normal((L.n, 2))
    y = L.expm(X, dt, 10)
    sol.ctx.check(sol.ctx.L.hymor_set_wait_limit(sol.ctx.h, 0))
    Y = np.zeros((2, L.n))
    x = np.ascontiguousarray(X.T)
    rc = sol.ctx.L.hymor_expm_apply(sol.ctx.h, 2, dt, 10, 5, dp(x), dp(Y), 0)
    assert rc == -5 and b"propagation" in sol.ctx.L.hymor_last_error(sol.ctx.h)
    assert np.isnan(Y).all()
    S.PDE(sol)                        # reported once, and not by calls that did not wait
    sol.ctx.check(sol.ctx.L.hymor_synchronize(sol.ctx.h))
    sol.ctx.check(sol.ctx.L.hymor_set_wait_limit(sol.ctx.h, 1 << 20))
    assert np.array_equal(L.expm(X, dt, 10), y)
    assert sol.ctx.L.hymor_set_wait_limit(sol.ctx.h, -1) == -1


@pytest.mark.parametrize("sync", ["synchronize", "download", "dot"])
def test_device_call_reports_when_waited_for(linear, sync):
    sol, L, dt = linear
    n = L.n
    sol.ctx.check(sol.ctx.L.hymor_set_wait_limit(sol.ctx.h, 0))
    bx, by = DeviceBuffer(sol.ctx, 8 * n), DeviceBuffer(sol.ctx, 8 * n)
    bx.upload(np.ones(n))
    sol.ctx.check(sol.ctx.L.hymor_expm_apply_dev(sol.ctx.h, 1, dt, 10, 5, bx.ptr, by.ptr, 0))
    out = ctypes.c_double()
    with pytest.raises(HymorError) as e:
        if sync == "synchronize":
            sol.ctx.check(sol.ctx.L.hymor_synchronize(sol.ctx.h))
        elif sync == "download":
            by.download(n)
        else:
            sol.ctx.check(sol.ctx.L.hymor_dot_dev(sol.ctx.h, n, 1, by.ptr, n, by.ptr, ctypes.byref(out)))
    assert e.value.code == -5
    assert np.isnan(by.download(n)).all()
    for b in (bx, by):
        b.free()


def test_solvers(linear):
    sol, L, dt = linear
    sol.ctx.check(sol.ctx.L.hymor_set_wait_limit(sol.ctx.h, 0))
    for solve in (lambda: S.EIGENVALUES(L, sol, 2, T_ref=10 * dt), lambda: S.TRANSIENT_GROWTH_DOWNSTREAM(L, sol, 1, 20 * dt)):
        with pytest.raises(HymorError) as e:
            solve()
        assert e.value.code == -5
