"""The exchange of the resident propagation: a published half and its term's number travel in one
64-bit element, the unit that the memory model keeps whole (the elements of a vector access have no
order), and a long propagation, every value of which goes through the exchange, repeats its bits."""
import os
import re

import numpy as np
import pytest

from hymor_gb300 import case as C
from hymor_gb300 import solver as S

from helpers import rel_err

SRC = os.path.join(os.path.dirname(__file__), "..", "hymor_gb300", "csrc", "linear.cu")


def test_accesses_of_whole_elements():
    text = open(SRC).read()
    start = text.index("k_expm_res_ff(MvFf")
    kernel = text[start:text.index("\n}\n", start)]
    ops = re.findall(r'"((?:ld|st)\.[\w.]+)', kernel)
    assert sorted(ops) == ["ld.relaxed.gpu.global.v2.b64", "st.relaxed.gpu.global.v2.b64"]


@pytest.mark.gpu
@pytest.mark.parametrize("make,nchi,neta,k", [(C.cylinder_config, 100, 80, 1), (C.channel_config, 64, 48, 5)])
def test_long_propagation_repeats(require_gpu, make, nchi, neta, k):
    sol = S.Solution(C.initial_state(make(nchi, neta), seed=1))
    _, L = S.LINEARIZE_L(sol)
    dt = 0.2 * S.CFL_TIMESTEP(sol)
    X = np.random.Generator(np.random.PCG64(9)).standard_normal((L.n, k))
    y = L.expm(X, dt, 1000, order=4)
    for _ in range(4):
        assert np.array_equal(y, L.expm(X, dt, 1000, order=4))
    sol.set_expm_arith(0)
    assert rel_err(y, L.expm(X, dt, 1000, order=4)) < 1e-9   # 4000 matvecs of ~2^-44, grown by the flow's modes
    sol.close()
