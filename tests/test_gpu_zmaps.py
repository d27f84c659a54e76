"""Y-maps with a Z term against the FP64 oracle: the column walks that cross
detector rows, in both directions of x and y, at every depth and lane layout,
with windows inside the detector and clamped at its edges."""
import numpy as np
import pytest

import mtr
import oracle
import phantom
from conftest import rel_l2

pytestmark = pytest.mark.gpu

# FP32 positions (~4e-6 px over a column) and fixed-point sums (2^-17 of the
# brick's largest value per addition): the bound of the windowed kernels' tests.
TOL = 1e-4


def _case(vol, px, py, phi, slopes, steep=False, seed=3):
    v = mtr.VolumeSize.make(*vol)
    c = phantom.make_case(v, px, np.arange(-60.0, 61.0, 15.0), [phi], 5, "gaussian", 0.02, seed, axis_cls=mtr.AxisData,
                          py=py)
    a = c.axes[0]
    x, y = a.x_coef.copy(), a.y_coef.copy()
    n = len(x) // 4
    b3 = np.resize(slopes, n)
    y[3::4] += b3
    y[0::4] -= b3 * (v.Zstart + 0.5 * (v.Z - 1))
    if steep:
        x[3::4] = np.resize([0.99, -0.99, 0.0, 1.2], n)
    return v, [mtr.AxisData(x, y, a.data)]


@pytest.mark.parametrize("depths", ["4,8,0,0,0", "16,16,1,1,0", "8,32,2,2,0", "16,8,2,1,1", "8,16,0,2,1", "32,32,1,0,0"])
@pytest.mark.parametrize("slopes", [(0.04,), (-0.31, 0.0, 0.31), (0.97, -0.97, 1.1), (1e-7, -1e-7)])
def test_z_maps_match_oracle(ctx, monkeypatch, depths, slopes):
    monkeypatch.setenv("MTR_FORCE_DEPTHS", depths)
    v, axes = _case((2, 47, -3, 36, 0, 35), 96, 104, 30.0, slopes)
    p = mtr.params(iter_times=1, sirt_inner=2, sirt_step=0.5, mace_step=0.7)
    got = ctx.reconstruct(axes, v, p)
    assert rel_l2(got, oracle.reconstruct(oracle.FP64, axes, v, 1, 2, 0.5, 0.7)) < TOL


@pytest.mark.parametrize("prec,tol", [(mtr.PREC_FP32, TOL), (mtr.PREC_MIXED_FP16, 1e-3)])
@pytest.mark.parametrize("vol,px,py,phi,steep", [((0, 64, 0, 60, 0, 20), 56, 52, 135.0, False),
                                                 ((0, 33, 0, 9, 0, 1), 48, 48, 80.0, False),
                                                 ((0, 40, 0, 40, 0, 24), 96, 96, 10.0, True)])
def test_z_maps_at_the_detector_edge(ctx, vol, px, py, phi, steep, prec, tol):
    v, axes = _case(vol, px, py, phi, (0.07, -0.2), steep)
    got = ctx.reconstruct(axes, v, mtr.params(1, 2, 0.5, 0.7, prec))
    assert rel_l2(got, oracle.reconstruct(oracle.FP64, axes, v, 1, 2, 0.5, 0.7)) < tol
