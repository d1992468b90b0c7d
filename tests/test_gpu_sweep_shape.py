"""Plain sweeps take smaller CTAs than the kernels with partial sums: bitwise
the two-sweep passes, which have a launch shape of their own."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


# tiles wider and narrower than a sweep's CTA, remainders in x and y, both sides
# of the 2^16 cells at which FP32 sweeps change their CTAs, and a box whose rows
# are more than a grid's y extent in rows of small CTAs
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,tile", [((33, 9, 5), "16"), ((130, 7, 4), "128"), ((40, 40, 40), "32"),
                                        ((41, 40, 40), "64"), ((2, 140001, 1), "16")])
def test_sweep_shapes(precision, shape, tile, monkeypatch):
    p, f = wavy_box(shape, 0)
    monkeypatch.setenv("LBM_TILE_BX", tile)
    got = []
    for z in ("0", "4"):
        monkeypatch.setenv("LBM_SWEEP2_ZLEN", z)
        g = L.InamuroCUDA(p, f, precision=precision)
        g.set_poisson(check_interval=10)
        g.step_replay([20, 30])
        got.append(g.download_fields())
        g.close()
    for k in L.FIELDS:
        assert np.array_equal(got[0][k], got[1][k]), k
