"""Krylov form: vector updates made by the first application that reads them
(degree above 1) against updates of their own (degree 1)."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


# Remainders of the launch tiles, one plane, walls and wrapped x.  Both solves
# stop at 1e-12 of the right-hand side; the operator's smallest mode on these
# boxes (40 cells at most, relaxation 1 / tau of order 1) is above 1e-5, so the
# pressures agree to better than 1e-6 of their size.
@pytest.mark.parametrize("shape", [(33, 9, 5), (17, 40, 3), (6, 5, 1), (32, 16, 24)])
@pytest.mark.parametrize("degree", [2, 5])
@pytest.mark.parametrize("periodic", [0, 1])
def test_updates_in_the_first_application(shape, degree, periodic):
    p, f = wavy_box(shape, periodic)
    got = []
    for m in (1, degree):
        g = L.InamuroCUDA(p, f)
        g.set_poisson_form("krylov")
        g.set_poisson_accel(krylov_degree=m)
        g.set_poisson(tolerance=1e-12, max_sweeps=100000)
        st = g.step(1)
        assert st[0]["converged"] == 1
        got.append(g.download("p"))
        g.close()
    assert np.max(np.abs(got[1] - got[0])) <= 1e-6 * np.max(np.abs(got[0]))
