"""The transposed sweeps' check intervals (one graph each): an odd interval
alternates between the two iterate buffers and must converge to the same
gradient as an even one, on both x boundaries."""
import numpy as np
import pytest

import lbm_b200 as L
from tests.test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("periodic", [0, 1])
def test_odd_and_even_check_intervals_give_one_gradient(periodic):
    p, f = wavy_box((20, 12, 10), periodic)
    rng = np.random.default_rng(3)
    lam = {k: rng.standard_normal(f["phi"].shape) for k in ("phi", "u")}
    got = []
    for interval in (40, 25, 1):
        a = L.Adjoint(p, checkpoint_interval=2, check_interval=interval, tolerance=1e-11 * interval,
                      max_sweeps=400_000 // interval * interval)
        a.set_poisson(check_interval=100, tolerance=1e-6, max_sweeps=200_000)
        a.forward(f, 3, [800, 800, 800])
        for _ in range(2):     # the second pass updates the graphs of the first
            g, st = a.backward(lam)
        got.append((g, st))
        a.close()
    for g, st in got[1:]:
        # (dJ/dp is the mean of a sum of differences: zero, so nothing but rounding)
        for k in ("phi", "rho", "u", "v", "w"):
            scale = np.max(np.abs(got[0][0][k]))
            assert np.max(np.abs(g[k] - got[0][0][k])) <= 1e-6 * max(scale, 1e-30), k
        assert abs(st["grad_kappa_f"] - got[0][1]["grad_kappa_f"]) <= 1e-6 * abs(got[0][1]["grad_kappa_f"])
