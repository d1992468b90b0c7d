"""Checks of small boxes, a plane per CTA: bitwise the checks that take a run's
planes in turn, which the dual residual's always do."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


# runs of 8 planes: whole, one plane over, one short, less than one; several
# tiles with and without a remainder; the last box is the smallest in y.  A mixed
# box is compared after one check: the dual residual's sweep C takes the next
# sweep's place and rounds to FP32 elsewhere than it.
@pytest.mark.parametrize("precision,sweeps", [("fp64", [8, 12]), ("mixed", [4])])
@pytest.mark.parametrize("shape", [(32, 8, 8), (33, 9, 9), (40, 20, 23), (5, 3, 3), (64, 24, 40), (70, 1, 17)])
@pytest.mark.parametrize("periodic", [0, 1])
def test_plane_per_cta_checks(precision, sweeps, shape, periodic):
    p, f = wavy_box(shape, periodic)
    got = []
    for dual in (True, False):
        g = L.InamuroCUDA(p, f, precision=precision)
        g.set_poisson(check_interval=4, dual=dual)
        stats = g.step_replay(sweeps)
        got.append((g.download_fields(), stats))
        g.close()
    for k in L.FIELDS:
        assert np.array_equal(got[0][0][k], got[1][0][k]), k
    for a, b in zip(got[0][1], got[1][1]):
        for k in ("relative_error", "pressure_l1_delta", "pressure_l1_norm", "pressure_gauge_target",
                  "pressure_gauge_max_shift"):
            assert a[k] == b[k], k
