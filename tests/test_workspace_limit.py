"""The linearisation with less device memory than its lanes would take (hymor_set_workspace_limit):
two groups of nine lanes, one of nine, one of three, and the same bits from all; an error, and a
context that goes on, where three do not fit either."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import receptivity as R
from hymor_gb300 import solver as S
from hymor_gb300._lib import HymorError

pytestmark = pytest.mark.gpu


def _bytes(cfg):
    """(kept beside the lanes, one lane), of the arrays' sizes, each lane array rounded up"""
    n, N, G = cfg.nchi, cfg.nchi * cfg.neta, (cfg.nchi + 2) * (cfg.neta + 2)
    kept = 1221 * N + 8 * ((10 * n * n if cfg.perturb_shock else 0) + 77 * n)
    return kept, 8 * (7 * G + 4 * N + 28 * n + 21 * 32)


def _blocks(sol):
    _, L = S.LINEARIZE_L(sol)
    out = [L.blocks()]
    if sol.cfg.perturb_shock:
        out += list(L.shock_blocks())
    if sol.cfg.shock_enabled:
        out += list(R.LINEARIZE_B(sol))
    return out


@pytest.mark.parametrize("make,nchi,neta,kw", [
    (C.cylinder_config, 100, 80, dict(perturb_shock=True)),
    (C.blunt_cone_config, 65, 33, dict(perturb_shock=True)),
    (C.channel_config, 31, 17, {}),          # periodic in chi, nchi = 1 (mod 3)
    (C.channel_config, 32, 12, {}),
    (C.cylinder_config, 450, 300, {}),       # 9 lanes a group to begin with
])
def test_fewer_lanes_same_bits(require_gpu, make, nchi, neta, kw):
    cs = C.initial_state(make(nchi, neta, **kw))
    kept, lane = _bytes(cs.cfg)
    ref = None
    for lanes in (0, 18, 9, 3):       # of the plan that fits, and no larger one
        sol = S.Solution(cs)
        sol.ctx.check(sol.ctx.L.hymor_set_workspace_limit(sol.ctx.h, int(kept + (lanes + 1) * lane) if lanes else 0))
        got = _blocks(sol)
        sol.close()
        if ref is None:
            ref = got
        for a, b in zip(ref, got):
            assert np.array_equal(a, b)


def test_nothing_fits(require_gpu):
    cs = C.initial_state(C.cylinder_config(100, 80))
    kept, lane = _bytes(cs.cfg)
    sol = S.Solution(cs)
    h, lib = sol.ctx.h, sol.ctx.L
    for limit in (1, int(kept + 2 * lane)):
        sol.ctx.check(lib.hymor_set_workspace_limit(h, limit))
        with pytest.raises(HymorError) as e:
            S.LINEARIZE_L(sol)
        assert e.value.code == -2
    sol.ctx.check(lib.hymor_set_workspace_limit(h, 0))
    S.PDE(sol)
    _, L = S.LINEARIZE_L(sol)
    other = S.Solution(cs)
    S.PDE(other)
    _, M = S.LINEARIZE_L(other)
    assert np.array_equal(L.blocks(), M.blocks())
    for s in (sol, other):
        s.close()
