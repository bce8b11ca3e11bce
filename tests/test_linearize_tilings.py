"""The linearisation under every tiling of the flux. The base flux of a small grid and the fluxes
of the perturbed states may come from different instances of the flux kernel; an entry whose two
fluxes are equal is an exact zero only where the instances round alike, so the blocks have to be
the same bits whichever instance gave the base flux, and zero outside what a perturbation reaches."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S

pytestmark = pytest.mark.gpu


def _suth(nchi, neta):
    return C.cylinder_config(nchi, neta, viscosity="sutherland")


@pytest.mark.parametrize("make,nchi,neta", [
    (C.cylinder_config, 100, 80), (C.cylinder_config, 30, 21), (_suth, 33, 27), (C.channel_config, 36, 20),
    (C.channel_config, 180, 60), (C.blunt_cone_config, 96, 40), (C.cylinder_config, 186, 200),
])
def test_blocks_of_every_tiling(require_gpu, make, nchi, neta):
    cs = C.initial_state(make(nchi, neta), seed=1, noise=1e-6)
    got = []
    for rows in (8, 4, 16):
        sol = S.Solution(cs)
        sol.ctx.check(sol.ctx.L.hymor_set_flux_tiling(sol.ctx.h, rows, 1, 0))
        _, L = S.LINEARIZE_L(sol)
        got.append(L.blocks())
        if sol.cfg.shock_enabled:
            rows_now = sol.get_state()["cell_idx"]
        sol.close()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
    if make is not C.channel_config:
        # rows at and above the shocked row have no residual: exact zeros
        B = got[0].reshape(neta, nchi, -1)
        for i in range(nchi):
            assert not B[int(rows_now[i]) - 1:, i].any()
