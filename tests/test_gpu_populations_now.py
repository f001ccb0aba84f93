"""Populations read right behind queued steps are those after the last of them."""
import numpy as np
import pytest

import tmixer_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("form", ["fp64", "fp32", "fp16"])
def test_populations_wait(gpu, form):
    spec = T.w_layout(32, u_max=0.05, tau_f=0.6, tau_c=0.6, k=1e-3, rho=1.0, precision=T.PRECISIONS[form])
    with T.Solver(spec) as s:
        s.init()
        s.populations(0, 0)
        s.step(1500)  # about 0.1 s on the GPU, queued in a few milliseconds
        now = s.populations(0, 0)
        s.sync()
        assert np.array_equal(now, s.populations(0, 0))
