"""The spline's fitted values from the fit or from the columns, by the rule on the grid's columns and
half tiles: grids on either side of its lines, against the oracle (as the other marches and
residuals), and the linearisation's lanes, which read the base residual's fit."""
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S
from oracle import oracle as O

from helpers import rel_err, residual_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make,nchi,neta", [
    (C.cylinder_config, 310, 120),       # 300 half tiles: the columns
    (C.cylinder_config, 311, 120),       # 330: the fit
    (C.blunt_cone_config, 512, 148), (C.blunt_cone_config, 513, 148),   # 629 half tiles; 512 columns are the last
    (C.cylinder_config, 300, 252), (C.cylinder_config, 300, 260),       # 630 and 650 half tiles
])
def test_either_side(require_gpu, make, nchi, neta):
    cs = C.initial_state(make(nchi, neta))
    sol, orc = S.Solution(cs), O.Oracle(cs)
    assert max(residual_rel(S.PDE(sol), orc.residual(), cs)) < 1e-11
    sol.close()
    sol, orc = S.Solution(cs), O.Oracle(cs)
    S.ADVECT_FLOW(sol, 3)
    orc.advect(3)
    a, b = sol.get_state(), orc.get_state()
    assert rel_err(a["q"], b["q"]) < 1e-11
    for k in ("pts_x", "pts_y"):
        assert rel_err(a[k], b[k]) < 1e-11
    sol.close()


def test_linearised_lanes(require_gpu):
    cs = C.initial_state(C.cylinder_config(311, 120))
    sol, orc = S.Solution(cs), O.Oracle(cs)
    _, L = S.LINEARIZE_L(sol)
    assert rel_err(L.blocks(), orc.linearize()) < 1e-5   # differences of 1e-13 over 1e-8
    sol.close()
