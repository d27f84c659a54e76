"""Line kernels (axes whose maps separate) against the FP64 oracle, over line
directions, ragged sizes, row spacings, per-view shifts and slabs, and against
the windowed kernels on the same inputs."""
import numpy as np
import pytest

import cases
import mtr
import oracle
import phantom
from conftest import rel_l2

pytestmark = pytest.mark.gpu

# FP32 arithmetic on both sides: tap positions to ~4e-6 px and a few hundred
# FP32 roundings per ray leave the volumes within 1e-5 (the run-to-run bound).
TOL = 1e-5


def _case(vol, px, py, tilts, phi, seed, change=None):
    c = phantom.make_case(mtr.VolumeSize.make(*vol), px, np.asarray(tilts, np.float64), [phi], 5, "gaussian", 0.02, seed,
                          axis_cls=mtr.AxisData, py=py)
    a = c.axes[0]
    x, y = a.x_coef.copy(), a.y_coef.copy()
    if change:
        change(x, y, np.random.default_rng(seed))
        c.axes[0] = mtr.AxisData(x, y, a.data)
    return c


def _shift_views(x, y, rng):  # every view its own row offset: one row table per angle
    y[0::4] += rng.uniform(-1.5, 1.5, len(y) // 4)


def _spread_rows(x, y, rng):  # detector rows 0.8 voxels apart
    y[1::4] *= 1.25
    y[2::4] *= 1.25
    y[0::4] -= 0.25 * 20


def _steep(x, y, rng):  # nearly one pixel per plane, both signs, and exact halves
    n = len(x) // 4
    x[3::4] = np.resize([0.998, -0.998, 0.5, -0.5, 0.0], n)


CASES = {
    # lines along Y and X; widths below, at and above the brick's; one plane to several bricks
    "y_small": ((0, 12, 0, 40, 0, 1), 24, 44, range(-60, 61, 20), 0.0, None),
    "y_ragged": ((-3, 30, 5, 70, 2, 19), 48, 72, range(-60, 61, 10), 0.0, None),
    "x_ragged": ((4, 133, -6, 31, 0, 33), 56, 140, range(-60, 61, 12), 90.0, None),
    "y_wide": ((0, 17, 0, 129, 0, 9), 40, 150, range(-50, 51, 25), 180.0, None),
    "x_long": ((0, 260, 0, 24, 0, 16), 40, 272, range(-60, 61, 30), 270.0, None),
    # columns that leave the detector on both sides of x
    "y_off": ((0, 60, 0, 40, 0, 24), 38, 48, range(-60, 61, 15), 0.0, None),
    "x_off": ((0, 40, 0, 64, 0, 20), 44, 50, range(-60, 61, 15), 90.0, None),
    "views_shifted": ((0, 30, 0, 40, 0, 12), 40, 52, range(-60, 61, 10), 0.0, _shift_views),
    "rows_spread": ((0, 30, 0, 40, 0, 12), 40, 64, range(-60, 61, 10), 0.0, _spread_rows),
    "steep": ((0, 25, 0, 40, 0, 37), 64, 48, range(-60, 61, 15), 0.0, _steep),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_lines_match_fp64_oracle(ctx, name):
    vol, px, py, tilts, phi, change = CASES[name]
    c = _case(vol, px, py, tilts, phi, 31 + len(name), change)
    p = mtr.params(iter_times=1, sirt_inner=3, sirt_step=0.5, mace_step=0.7)
    r = mtr.Recon(ctx, c.axes, c.vol, p)
    assert r.describe()[0]["back_projection"]["window_format"] == "line image"
    r.run()
    got = r.download()
    want = oracle.reconstruct(oracle.FP64, c.axes, c.vol, 1, 3, 0.5, 0.7)
    assert rel_l2(got, want) < TOL


@pytest.mark.parametrize("prec", [mtr.PREC_FP32, mtr.PREC_MIXED_FP16, mtr.PREC_MIXED_BF16])
@pytest.mark.parametrize("flags,slab", [(0, 0), (mtr.FLAG_STREAM_SLABS, 5), (mtr.FLAG_GRAPH, 0)])
def test_lines_equal_windows(ctx, monkeypatch, prec, flags, slab):
    """The same inputs on line kernels and on the windowed kernels, with residual norms."""
    c = cases.get("mid")
    p = mtr.params(2, 3, 0.5, 0.7, prec, flags | mtr.FLAG_RECORD_NORMS, slab)

    def once():
        r = mtr.Recon(ctx, c.axes, c.vol, p)
        r.run()
        return r.describe()[0]["back_projection"]["window_format"], r.download(), r.norms()

    fmt, got, norms = once()
    monkeypatch.setenv("MTR_FORCE_DEPTHS", "8,16")
    fmt_w, want, norms_w = once()
    assert fmt == "line image" and fmt_w == "fp32"
    # mixed precision: an FP32 rounding flips an FP16/BF16 rounding now and then (run_to_run_tol)
    tol = TOL if prec == mtr.PREC_FP32 else 1e-4
    assert rel_l2(got, want) < tol and rel_l2(norms, norms_w) < tol


@pytest.mark.parametrize("views", [None, _shift_views], ids=["shared", "shifted"])
@pytest.mark.parametrize("phi", [0.0, 90.0])
@pytest.mark.parametrize("shape", ["128x8", "64x16", "64x8"])
def test_wbp_brick_shapes_match_fp64_oracle(ctx, shape, phi, views):
    """WBP in every brick shape (the small one: above), one row table or one per
    angle, with columns that leave the detector on both sides."""
    w, m, z = {"128x8": (250, 190, 56), "64x16": (190, 208, 64), "64x8": (60, 490, 40)}[shape]
    vol = (0, m, 0, w, 0, z) if phi == 0.0 else (0, w, 0, m, 0, z)
    c = _case(vol, int(0.8 * m), w + 8, (-52, -17, 0, 31), phi, 11, views)
    got = ctx.wbp(c.axes[0], c.vol)
    assert rel_l2(got, oracle.wbp(oracle.FP64, c.axes[0], c.vol)) < TOL


@pytest.mark.parametrize("change", ["lean", "turn", "squeeze", "narrow"])
def test_axes_that_do_not_separate_keep_the_windows(ctx, change):
    c = _case((0, 40, 0, 48, 0, 12), 56, 56, range(-60, 61, 20), 0.0, 5)
    a = c.axes[0]
    x, y, d = a.x_coef.copy(), a.y_coef.copy(), a.data
    if change == "lean":
        y[3::4] = 1e-4
    elif change == "turn":
        x[2::4] = 1e-6
    elif change == "squeeze":
        y[2::4] *= 0.3
    else:  # fewer detector rows than line positions: the line image does not fit
        d = np.ascontiguousarray(d[:, 8:48])
        y[0::4] -= 8
    p = mtr.params(iter_times=1, sirt_inner=2, sirt_step=0.5, mace_step=0.7)
    r = mtr.Recon(ctx, [mtr.AxisData(x, y, d)], c.vol, p)
    assert r.describe()[0]["back_projection"]["window_format"] != "line image"
    r.run()
    want = oracle.reconstruct(oracle.FP64, [mtr.AxisData(x, y, d)], c.vol, 1, 2, 0.5, 0.7)
    assert rel_l2(r.download(), want) < 1e-4


@pytest.mark.parametrize("phi", [0.0, 90.0])
def test_volumes_in_host_memory_keep_the_windows(ctx, phi):
    c = _case((0, 40, 0, 48, 0, 12), 56, 56, range(-60, 61, 20), phi, 6)
    p = mtr.params(1, 2, 0.5, 0.7, mtr.PREC_FP32, mtr.FLAG_HOST_VOLUMES)
    r = mtr.Recon(ctx, c.axes, c.vol, p)
    assert r.describe()[0]["back_projection"]["window_format"] != "line image"
    r.run()
    assert rel_l2(r.download(), oracle.reconstruct(oracle.FP64, c.axes, c.vol, 1, 2, 0.5, 0.7)) < TOL
