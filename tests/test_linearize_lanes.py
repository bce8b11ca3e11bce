"""The linearisation's batched residuals (a group of perturbations per launch): every group
size, grids whose sizes are no multiples of the three colours or of the tiles, periodic
wraps, both forms of the finite-difference quotient, and the tilings of the shock band."""
import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S
from oracle import oracle as O

from helpers import rel_err

pytestmark = pytest.mark.gpu

# entries are quotients by eps of residual differences that agree with the oracle's to ~1e-13
# of the flux: 1e-13 / 1e-8
FD_TOL = 1e-5


@pytest.mark.parametrize("make,nchi,neta", [
    (C.cylinder_config, 37, 19),       # 32 residuals per group at most, 18 of the colours
    (C.channel_config, 31, 17),        # periodic in chi, no shock; nchi = 1 (mod 3)
    (C.channel_config, 32, 12),
    (C.blunt_cone_config, 64, 33),
    (C.cylinder_config, 300, 240),     # 72 000 cells: 18 per group
    (C.cylinder_config, 450, 300),     # 135 000 cells: 9 per group
])
def test_jacobian_blocks(require_gpu, make, nchi, neta):
    cs = C.initial_state(make(nchi, neta))
    sol, orc = S.Solution(cs), O.Oracle(cs)
    _, L = S.LINEARIZE_L(sol)
    assert rel_err(L.blocks(), orc.linearize()) < FD_TOL
    sol.close()


@pytest.mark.parametrize("eps", [2.0**-27, 1e-8, (1 - 2.0**-53) * 2.0**-26])
def test_quotient(require_gpu, eps):
    """Exact power of two, an ordinary eps, and one whose significand is all ones (divided)."""
    cs = C.initial_state(C.cylinder_config(24, 18, perturbation_magnitude=eps))
    sol, orc = S.Solution(cs), O.Oracle(cs)
    _, L = S.LINEARIZE_L(sol)
    assert rel_err(L.blocks(), orc.linearize()) < 2 * FD_TOL
    sol.close()


@pytest.mark.parametrize("nchi,neta", [(70, 41), (33, 26)])
def test_shock_band_tilings(require_gpu, nchi, neta):
    """The shock-position blocks are the same bit for bit whichever tiles cover the band."""
    cs = C.initial_state(C.blunt_cone_config(nchi, neta, perturb_shock=True))
    got = []
    for rows in (4, 8, 16):
        sol = S.Solution(cs)
        sol.ctx.check(sol.ctx.L.hymor_set_flux_tiling(sol.ctx.h, rows, 0, 0))
        _, L = S.LINEARIZE_L(sol)
        got.append(L.shock_blocks())
        sol.close()
    for other in got[1:]:
        for a, b in zip(got[0], other):
            assert np.array_equal(a, b)
