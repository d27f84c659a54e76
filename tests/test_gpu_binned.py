"""Reconstructions with several detector pixels per voxel (binned volumes) against
the FP64 oracle."""
import numpy as np
import pytest

import mtr
import oracle
import phantom
from conftest import rel_l2

pytestmark = pytest.mark.gpu

# positions to ~4e-6 px, sums in fixed point at 2^-17 of a brick's largest value
# or finer: the bounds of the windowed kernels' tests
TOL = {mtr.PREC_FP32: 1e-4, mtr.PREC_MIXED_FP16: 1e-3}


def binned(mag, phi, vol=(2, 47, -3, 36, 0, 21), lean=0.0, cover=1.1, shift=0.0, seed=4):
    """One axis whose detector has `mag` pixels to a voxel and covers the volume `cover` times."""
    v = mtr.VolumeSize.make(*vol)
    px = int(mag * cover * max(v.X, v.Y)) + 8
    c = phantom.make_case(v, px, np.arange(-60.0, 61.0, 15.0), [phi], 5, "gaussian", 0.02, seed, axis_cls=mtr.AxisData,
                          py=px + 3)
    a = c.axes[0]
    mid = np.array([(v.Xstart + v.Xend - 1) / 2, (v.Ystart + v.Yend - 1) / 2, (v.Zstart + v.Zend - 1) / 2])
    maps = []
    for q, n in ((a.x_coef, px), (a.y_coef, px + 3)):
        m = q.reshape(-1, 4).copy()
        m[:, 1:] *= mag
        if q is a.y_coef:
            m[:, 3] += lean
        m[:, 0] = (n + 1) / 2 + shift - m[:, 1:] @ mid
        maps.append(m.ravel())
    return v, [mtr.AxisData(maps[0], maps[1], a.data)]


def check(ctx, v, axes, prec=mtr.PREC_FP32, **kw):
    r = mtr.Recon(ctx, axes, v, mtr.params(1, 2, 0.5, 0.7, prec, **kw))
    r.run()
    got, plan = r.download(), r.describe()[0]
    r.close()
    assert rel_l2(got, oracle.reconstruct(oracle.FP64, axes, v, 1, 2, 0.5, 0.7)) < TOL[prec]
    return plan


@pytest.mark.parametrize("depths", ["8,8,0,0,0", "8,16,1,1,0", "8,32,2,2,0", "8,5,0,2,0"])
@pytest.mark.parametrize("mag,cover", [(1.7, 1.1), (2.5, 0.7), (4.0, 1.1)])
@pytest.mark.parametrize("phi", [30.0, 135.0])
def test_steep_columns_match_oracle(ctx, monkeypatch, depths, phi, mag, cover):
    """Slopes from zero to 3.5 pixels per voxel of both signs, windows inside and at the detector's edges."""
    monkeypatch.setenv("MTR_FORCE_DEPTHS", depths)
    check(ctx, *binned(mag, phi, cover=cover))


@pytest.mark.parametrize("depths", ["8,8,0,0,0", "8,16,0,1,0", "8,32,0,0,0", "8,32,0,1,0", "8,5,0,0,0"])
@pytest.mark.parametrize("mag,cover", [(1.4, 1.1), (2.5, 0.7), (4.0, 1.1)])
@pytest.mark.parametrize("phi", [0.0, 90.0, 180.0])
def test_rows_summed_per_warp_match_oracle(ctx, monkeypatch, depths, phi, mag, cover):
    """Binned axes along a volume axis, in the layout whose lanes share their rows and in the other."""
    monkeypatch.setenv("MTR_FORCE_DEPTHS", depths)
    # (off whole pixels: no voxel whose only tap on the detector has a weight of rounding error)
    check(ctx, *binned(mag, phi, cover=cover, shift=0.3))


def test_rows_summed_per_warp_of_many_columns_on_one_pixel(ctx, monkeypatch):
    """All 32 columns of a warp on a few pixels: the largest sums of a row."""
    monkeypatch.setenv("MTR_FORCE_DEPTHS", "8,32,0,0,0")
    v, axes = binned(2.0, 0.0)
    x = axes[0].x_coef.copy()
    x[1::4] *= 0.05
    check(ctx, v, [mtr.AxisData(x, axes[0].y_coef, axes[0].data)])


@pytest.mark.parametrize("prec", [mtr.PREC_FP32, mtr.PREC_MIXED_FP16])
@pytest.mark.parametrize("phi,lean", [(0.0, 0.0), (30.0, 0.0), (45.0, 0.05), (90.0, -0.3)])
@pytest.mark.parametrize("mag", [2.0, 3.0, 4.0])
def test_tuned_tiles_are_windowed_and_match_oracle(ctx, mag, phi, lean, prec):
    plan = check(ctx, *binned(mag, phi, lean=lean, shift=0.3), prec)
    assert plan["back_projection"]["tma"] and plan["forward"]["tma"]


@pytest.mark.parametrize("depths", ["4,8,0,2,0", "8,16,1,2,0", "16,16,2,2,0", "32,8,2,2,0", "8,8,0,0,0"])
@pytest.mark.parametrize("phi,lean,cover", [(45.0, 0.0, 1.1), (30.0, 0.07, 0.7), (135.0, -0.6, 1.1), (0.0, 0.0, 1.1)])
@pytest.mark.parametrize("mag", [2.5, 4.0])
def test_plain_row_windows_match_oracle(ctx, monkeypatch, depths, phi, lean, cover, mag):
    """Windows of plain rows in every lane layout and depth, inside the detector and over its edges."""
    monkeypatch.setenv("MTR_FORCE_DEPTHS", depths)
    check(ctx, *binned(mag, phi, vol=(0, 47, 0, 39, 0, 37), lean=lean, cover=cover, shift=0.3))


def test_untuned_tiles_are_windowed(ctx, monkeypatch):
    monkeypatch.setenv("MTR_AUTOTUNE", "0")
    for mag, phi in ((3.0, 45.0), (4.0, 30.0)):
        v, axes = binned(mag, phi, vol=(1, 46, 0, 37, 0, 22), shift=0.3)
        assert check(ctx, v, axes)["back_projection"]["tma"]


@pytest.mark.parametrize("forced,phi,lean", [("32,16,2,2,3", 0.0, 0.05), ("4,16,1,2,0", 15.0, 0.0)])
def test_wbp_takes_a_window_that_fits(ctx, monkeypatch, forced, phi, lean):
    """An update whose tile leaves the WBP no window of its own depth and layout."""
    monkeypatch.setenv("MTR_FORCE_DEPTHS", forced)
    v, axes = binned(5.0, phi, vol=(0, 40, 0, 33, 0, 40), lean=lean, shift=0.3)
    r = mtr.Recon(ctx, axes, v, mtr.params(1, 0, 0.5, 0.7, mtr.PREC_MIXED_FP16))
    assert r.describe()[0]["back_projection"]["depth"] == int(forced.split(",")[0])
    n = ctx.windowed_launch_count()
    r.run()
    got, launched = r.download(), ctx.windowed_launch_count() - n
    r.close()
    assert launched == 1  # the WBP: no SIRT iteration runs
    assert rel_l2(got, oracle.wbp(oracle.FP64, axes[0], v)) < TOL[mtr.PREC_MIXED_FP16]
