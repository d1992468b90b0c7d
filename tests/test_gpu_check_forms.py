"""Checks of small boxes: a plane per CTA against a run's planes in turn, bitwise
over several checks and steps, for FP64, mixed and refinement boxes."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu

KEYS = ("relative_error", "pressure_l1_delta", "pressure_l1_norm", "pressure_gauge_target", "pressure_gauge_max_shift")


def run(monkeypatch, planes, shape, form, periodic):
    p, f = wavy_box(shape, periodic)
    if planes is None:
        monkeypatch.delenv("LBM_CHECK_PLANES", raising=False)
    else:
        monkeypatch.setenv("LBM_CHECK_PLANES", planes)
    g = L.InamuroCUDA(p, f, precision="fp64" if form == "fp64" else "mixed")
    g.set_poisson(check_interval=4)
    if form == "refine":
        g.set_poisson_form("refine")
    stats = g.step_replay([8, 12])
    got = g.download_fields(), [{k: s[k] for k in KEYS} for s in stats]
    g.close()
    return got


# runs of 8 planes: whole, one plane over, one short, less than one; tiles with
# and without a remainder; one plane; more runs than SMs (90 x 40 x 130: 255), more
# than five an SM (40 x 56 x 600: 900), which the default rule takes in turn
@pytest.mark.parametrize("form", ["fp64", "mixed", "refine"])
@pytest.mark.parametrize("shape", [(32, 8, 8), (33, 9, 9), (40, 20, 23), (5, 3, 3), (64, 24, 40), (70, 1, 17), (16, 16, 1),
                                   (90, 40, 130), (40, 56, 600)])
def test_a_plane_per_cta_is_planes_in_turn(form, shape, monkeypatch):
    turn = run(monkeypatch, "0", shape, form, 0)
    for planes in ("1", None):
        got = run(monkeypatch, planes, shape, form, 0)
        for k in L.FIELDS:
            assert np.array_equal(turn[0][k], got[0][k]), (planes, k)
        assert turn[1] == got[1], planes


@pytest.mark.parametrize("form", ["fp64", "mixed", "refine"])
def test_a_plane_per_cta_with_wrapped_x(form, monkeypatch):
    turn, got = (run(monkeypatch, planes, (33, 9, 20), form, 1) for planes in ("0", "1"))
    for k in L.FIELDS:
        assert np.array_equal(turn[0][k], got[0][k]), k
    assert turn[1] == got[1]
