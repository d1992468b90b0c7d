"""Check intervals of transposed sweeps longer than one graph."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


def resident_mb():
    with open("/proc/self/statm") as f:
        return int(f.read().split()[1]) * 4096 / 1e6


def gradients(interval, tolerance, steps=2):
    p, f = wavy_box((20, 12, 10), 0)
    rng = np.random.default_rng(3)
    lam = {k: rng.standard_normal(f["phi"].shape) for k in ("phi", "u")}
    a = L.Adjoint(p, checkpoint_interval=2, check_interval=interval, tolerance=tolerance)
    a.set_poisson(check_interval=100, tolerance=1e-6, max_sweeps=200_000)
    a.forward(f, steps, [800] * steps)
    for _ in range(2):     # the second pass updates the graphs of the first
        g, st = a.backward(lam)
    return a, g, st


# just within one graph of 512, one sweep more, two whole graphs, odd and even
# remainders.  The change per sweep that ends a solve is 1e-11 of the iterate on
# each (the test divides by the norm after the interval), and its smallest mode
# decays within some hundred sweeps, so the gradients agree to 1e-6.
@pytest.mark.parametrize("interval", [511, 512, 513, 1024, 1025])
def test_long_intervals_give_the_same_gradient(interval):
    got = []
    for ci in (40, interval):
        a, g, st = gradients(ci, 1e-11 * ci)
        a.close()
        got.append((g, st["grad_kappa_f"]))
    for k in ("phi", "rho", "u", "v", "w"):
        scale = np.max(np.abs(got[0][0][k]))
        assert np.max(np.abs(got[1][0][k] - got[0][0][k])) <= 1e-6 * max(scale, 1e-30), k
    assert abs(got[1][1] - got[0][1]) <= 1e-6 * abs(got[0][1])


# (as one graph an interval of 40 000 sweeps held 230 MB)
def test_a_long_interval_takes_no_memory():
    a, _, _ = gradients(40, 1e-3, 1)
    a.close()
    before = resident_mb()
    a, _, _ = gradients(40_000, 1e-3, 1)
    grown = resident_mb() - before
    a.close()
    assert grown < 60, grown
