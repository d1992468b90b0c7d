"""Boxes with more tile rows than a grid's y extent run single sweeps, also
where the z run length of the two-sweep passes is set from outside."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


# (rows of 6 for FP64, of 8 for FP32; the first extent is the last that fits)
@pytest.mark.parametrize("precision,ly,passes", [("fp64", 393210, True), ("fp64", 393211, False),
                                                 ("mixed", 524280, True), ("mixed", 524281, False)])
def test_tile_rows_beyond_the_grid(precision, ly, passes, monkeypatch):
    p, f = wavy_box((2, ly, 1), 0)
    got = []
    for z in ("0", "4"):
        monkeypatch.setenv("LBM_SWEEP2_ZLEN", z)
        g = L.InamuroCUDA(p, f, precision=precision)
        g.set_poisson(check_interval=10)
        g.step_replay([20, 30])
        got.append((g.download_fields(), g.timing()["fused_sweeps"]))
        g.close()
    assert got[0][1] == 0 and (got[1][1] > 0) == passes
    for k in L.FIELDS:
        assert np.array_equal(got[0][0][k], got[1][0][k]), k
