"""The two-sweep Poisson passes on boxes that no tile divides: bitwise the
single sweeps."""
import numpy as np
import pytest

import lbm_b200 as L

pytestmark = pytest.mark.gpu


def wavy_box(shape, periodic):
    lx, ly, lz = shape
    p = L.make_params(lx=lx, ly=ly, lz=lz, rho_L=50.0, rho_G=1.0, mu_L=5.0, mu_G=0.1, k_f=0.06, k_g=6e-6,
                      periodic_x=periodic)
    rng = np.random.default_rng(7)
    z, y, x = np.meshgrid(*[np.arange(n) / n for n in (lz, ly, lx)], indexing="ij")
    wave = np.cos(2 * np.pi * x) + np.cos(2 * np.pi * y) + np.cos(2 * np.pi * z)
    frac = 0.5 + 0.5 * np.tanh(wave)
    f = {"phi": p.fei_min + frac * (p.fei_max - p.fei_min) + rng.uniform(-1e-4, 1e-4, frac.shape),
         "rho": p.rho_G + frac * (p.rho_L - p.rho_G), "p": np.zeros_like(frac)}
    for k, a in zip("uvw", (x, y, z)):
        f[k] = 0.01 * np.sin(2 * np.pi * a)
    return p, f


# one tile with and without a remainder, several with one, extents below the
# tile, one plane, z runs that do not divide the box
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("shape,zlen", [((30, 6, 9), "4"), ((31, 7, 5), "5"), ((61, 13, 12), "5"), ((33, 9, 3), "2"),
                                        ((65, 17, 10), "32"), ((2, 1, 1), "1"), ((5, 40, 2), "8"), ((90, 3, 7), "3")])
@pytest.mark.parametrize("periodic", [0, 1])
def test_two_sweep_pass_on_ragged_boxes(precision, shape, zlen, periodic, monkeypatch):
    p, f = wavy_box(shape, periodic)
    got = []
    for z in ("0", zlen):
        monkeypatch.setenv("LBM_SWEEP2_ZLEN", z)
        g = L.InamuroCUDA(p, f, precision=precision)
        g.set_poisson(check_interval=20)
        g.step_replay([40, 60])
        got.append((g.download_fields(), g.timing()["fused_sweeps"]))
        g.close()
    assert got[0][1] == 0 and got[1][1] > 0
    for k in L.FIELDS:
        assert np.array_equal(got[0][0][k], got[1][0][k]), k


@pytest.mark.parametrize("shape", [(45, 20, 14), (31, 9, 8)])
def test_two_sweep_corrections_on_ragged_boxes(shape, monkeypatch):
    p, f = wavy_box(shape, 0)
    got = []
    for z in ("0", "5"):
        monkeypatch.setenv("LBM_SWEEP2_ZLEN", z)
        g = L.InamuroCUDA(p, f, precision="mixed")
        g.set_poisson(check_interval=20)
        g.set_poisson_form("refine")
        g.step_replay([40, 60])
        got.append(g.download_fields())
        g.close()
    for k in L.FIELDS:
        assert np.array_equal(got[0][k], got[1][k]), k
