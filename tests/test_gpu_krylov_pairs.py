"""Krylov form: the polynomial's applications two per pass give bitwise the
single applications' solve (small boxes run single applications, so the pairs
are compared on a box above their threshold, cut so that no tile divides it)."""
import numpy as np
import pytest

import lbm_b200 as L
from tests.test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("degree", [3, 4, 8])
@pytest.mark.parametrize("periodic", [0, 1])
def test_pairs_of_applications_are_single_applications(degree, periodic, monkeypatch):
    p, f = wavy_box((91, 83, 77), periodic)
    got = []
    for pairs in ("0", "1"):
        monkeypatch.setenv("LBM_KRYLOV_PAIRS", pairs)
        g = L.InamuroCUDA(p, f)
        g.set_poisson_form("krylov")
        g.set_poisson_accel(krylov_degree=degree)
        g.set_poisson(tolerance=1e-9, max_sweeps=200)
        st = g.step(2)
        got.append((g.download_fields(), [s["iterations"] for s in st]))
        g.close()
    assert got[0][1] == got[1][1]
    for k in L.FIELDS:
        assert np.array_equal(got[0][0][k], got[1][0][k]), k
