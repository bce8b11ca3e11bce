"""The residual's small-grid paths: both boundary phases in one block (up to 512 points a phase),
half-height tiles while there are no more of them than SMs, and its flux through the staging
buffer, straight into page-locked memory, or straight into pageable memory (above 128 KB)."""
import numpy as np
import pytest
import torch

from hymor_gb300 import case as C
from hymor_gb300 import solver as S
from oracle import oracle as O

from helpers import residual_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make,nchi,neta", [
    (C.channel_config, 3, 4), (C.channel_config, 31, 8), (C.cylinder_config, 33, 17),
    (C.cylinder_config, 126, 40), (C.cylinder_config, 127, 40),      # 256 and 258 points a phase
    (C.blunt_cone_config, 254, 96), (C.cylinder_config, 255, 97),    # 512 and 514
    (C.cylinder_config, 270, 243),                                   # 2.1 MB of flux
])
def test_residual(require_gpu, make, nchi, neta):
    cs = C.initial_state(make(nchi, neta))
    orc = O.Oracle(cs)
    fo = orc.residual()
    sol = S.Solution(cs)
    fg = S.PDE(sol)
    assert max(residual_rel(fg, fo, cs)) < 1e-12
    sol.close()
    pinned = torch.empty(4 * nchi * neta, dtype=torch.float64, pin_memory=True).numpy()
    sol = S.Solution(cs)
    S.PDE(sol, pinned)
    assert np.array_equal(pinned, fg)
    sol.close()
