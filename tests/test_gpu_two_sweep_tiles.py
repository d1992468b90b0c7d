"""The two-sweep passes that boxes take by default, and the mixed box's tall
tile: bitwise the single sweeps."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


def run(monkeypatch, zlen, shape, periodic, precision="mixed", form="kinetic"):
    p, f = wavy_box(shape, periodic)
    if zlen is None:
        monkeypatch.delenv("LBM_SWEEP2_ZLEN", raising=False)
    else:
        monkeypatch.setenv("LBM_SWEEP2_ZLEN", zlen)
    g = L.InamuroCUDA(p, f, precision=precision)
    g.set_poisson(check_interval=20)
    g.set_poisson_form(form)
    g.step_replay([40, 60])
    got = g.download_fields(), g.timing()["fused_sweeps"]
    g.close()
    return got


# one 32 x 16 tile with and without a remainder, several with one, extents below
# the tile, one plane, z runs that do not divide the box
@pytest.mark.parametrize("shape,zlen", [((32, 16, 9), 4), ((33, 17, 5), 5), ((65, 35, 12), 5), ((31, 15, 3), 2),
                                        ((2, 1, 1), 1), ((5, 40, 2), 8), ((90, 3, 7), 3), ((64, 48, 34), 32)])
@pytest.mark.parametrize("periodic", [0, 1])
def test_tall_tile_on_ragged_boxes(shape, zlen, periodic, monkeypatch):
    single, tall = (run(monkeypatch, z, shape, periodic) for z in ("0", f"{zlen}x16"))
    assert single[1] == 0 and tall[1] > 0
    for k in L.FIELDS:
        assert np.array_equal(single[0][k], tall[0][k]), k


# boxes on which the rules choose passes: the tall tile (96^3, 90 x 75 x 131), the
# low one (95 x 67 x 96), FP64's, the refinement form's
@pytest.mark.parametrize("precision,form,shape", [("mixed", "kinetic", (96, 96, 96)), ("mixed", "kinetic", (90, 75, 131)),
                                                  ("mixed", "kinetic", (95, 67, 96)), ("fp64", "kinetic", (96, 96, 96)),
                                                  ("fp64", "kinetic", (90, 75, 131)), ("mixed", "refine", (96, 96, 96)),
                                                  ("mixed", "refine", (91, 98, 73))])
def test_passes_that_the_rules_choose(precision, form, shape, monkeypatch):
    single, default = (run(monkeypatch, z, shape, 0, precision, form) for z in ("0", None))
    assert single[1] == 0 and default[1] > 0
    for k in L.FIELDS:
        assert np.array_equal(single[0][k], default[0][k]), k
