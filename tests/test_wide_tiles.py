"""Blocks of a warp per face row (grids of few half-height tiles) against blocks of a warp per
tile row (31 x 8 tiles, which never take them): every face flux has the same arithmetic, so the
marched state and the residual are equal bit for bit."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S

pytestmark = pytest.mark.gpu


def _suth(nchi, neta):
    return C.cylinder_config(nchi, neta, viscosity="sutherland")


@pytest.mark.parametrize("make,nchi,neta", [
    (C.cylinder_config, 30, 21), (C.cylinder_config, 31, 24), (_suth, 33, 27), (C.channel_config, 36, 20),
    (C.blunt_cone_config, 96, 40), (C.cylinder_config, 126, 61),  # ragged last tiles
    (C.cylinder_config, 186, 200), (C.cylinder_config, 187, 200),  # 300 and 350 half tiles
])
def test_march_and_residual(require_gpu, make, nchi, neta):
    cs = C.initial_state(make(nchi, neta), seed=1, noise=1e-6)
    got = []
    for rows in (8, 4):
        sol = S.Solution(cs)
        sol.ctx.check(sol.ctx.L.hymor_set_flux_tiling(sol.ctx.h, rows, 1, 0))
        S.ADVECT_FLOW(sol, 3)
        st = sol.get_state()
        got.append((st["q"], st["pts_x"], S.PDE(sol)))
        sol.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
