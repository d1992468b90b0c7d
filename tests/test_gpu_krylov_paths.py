"""Krylov form: pairs of applications on boxes of any remainder, and vector
updates within the first application, bitwise against launches of their own."""
import numpy as np
import pytest

import lbm_b200 as L
from test_gpu_two_sweep import wavy_box

pytestmark = pytest.mark.gpu


def solve(monkeypatch, shape, periodic, degree, pairs=None, updates=None, sweeps=200):
    for name, value in (("LBM_KRYLOV_PAIRS", pairs), ("LBM_KRYLOV_UPDATES", updates)):
        if value is None:
            monkeypatch.delenv(name, raising=False)
        else:
            monkeypatch.setenv(name, value)
    p, f = wavy_box(shape, periodic)
    g = L.InamuroCUDA(p, f)
    g.set_poisson_form("krylov")
    g.set_poisson_accel(krylov_degree=degree)
    g.set_poisson(tolerance=1e-9, max_sweeps=sweeps)
    st = g.step(2)
    got = g.download_fields(), [s["iterations"] for s in st], g.timing()["fused_sweeps"]
    g.close()
    return got


def same(a, b):
    assert a[1] == b[1]
    for k in L.FIELDS:
        assert np.array_equal(a[0][k], b[0][k]), k


# remainders of the 30 x 6 tile, extents below it, one plane, z runs that do not
# divide the box; degrees that leave a single application between (5, 7) and none
@pytest.mark.parametrize("shape,zlen", [((31, 7, 9), 4), ((60, 12, 10), 5), ((17, 40, 3), 2), ((6, 5, 1), 1), ((33, 13, 20), 32)])
@pytest.mark.parametrize("degree", [4, 5, 7, 8])
@pytest.mark.parametrize("periodic", [0, 1])
def test_pairs_on_ragged_boxes(shape, zlen, degree, periodic, monkeypatch):
    single, pairs = (solve(monkeypatch, shape, periodic, degree, pairs=v) for v in ("0", f"z{zlen}"))
    assert single[2] == 0 and pairs[2] > 0
    same(single, pairs)


# the degrees that have no application to pair, and a box on which the rule pairs
@pytest.mark.parametrize("shape,degree,paired", [((33, 13, 20), 3, False), ((33, 13, 20), 1, False), ((91, 83, 77), 8, True)])
def test_where_pairs_run(shape, degree, paired, monkeypatch):
    assert (solve(monkeypatch, shape, 0, degree, pairs=None if paired else "z4")[2] > 0) == paired


@pytest.mark.parametrize("shape", [(33, 9, 5), (17, 40, 3), (6, 5, 1), (32, 16, 24), (64, 40, 33)])
@pytest.mark.parametrize("degree", [2, 5, 8])
@pytest.mark.parametrize("periodic", [0, 1])
def test_updates_in_the_first_application(shape, degree, periodic, monkeypatch):
    own, within = (solve(monkeypatch, shape, periodic, degree, updates=v) for v in ("0", None))
    same(own, within)
