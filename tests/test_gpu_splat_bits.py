"""Fixed-point bits of the forward splats at untilted views: a pixel receives at
most 2^lw = depth times the largest voxel from one column, and the values keep
21 - lw bits (16 at depth 32, 17 at the line kernels' 16).

One plane of values k 2^-bits (k odd, below 2^bits, so that the least bit
counts), every other plane zero, whole-pixel maps: each ray sum is one value
exactly, and one SIRT iteration of step 1 against projections of zero subtracts
s / rows.  A bit less rounds every value by 2^-bits: 2^-bits / planes = 4.8e-7 in
the result.  Kept bits leave the rounding of the row sums (2e-6 relative at the
slope 1e-7 px per voxel that stands for zero: 6e-8 of s / rows <= 1 / 16 is below
1.3e-7) and of the result (2^-25 = 3e-8)."""
import numpy as np
import pytest

import mtr
import phantom

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lines,planes,bits", [(False, 32, 16), (True, 16, 17)])
def test_untilted_views_keep_their_bits(ctx, monkeypatch, lines, planes, bits):
    if not lines:  # prefix sums at depth 32
        monkeypatch.setenv("MTR_FORCE_DEPTHS", "8,32,0,0")
    n = 128 if lines else 64
    vol = mtr.VolumeSize.make(0, n, 0, n, 0, planes)
    xc, yc = phantom.axis_maps(n + 8, n + 8, [0.0], 0.0, vol)
    xc, yc = np.round(xc), np.round(yc)  # whole pixels
    start = np.zeros(vol.shape, np.float32)
    k = np.random.default_rng(1).integers(0, 2 ** (bits - 1), (n, n)) * 2 + 1
    start[0] = k * 2.0 ** -bits
    axis = mtr.AxisData(xc, yc, np.zeros((1, n + 8, n + 8), np.float32))
    got = ctx.sirt(axis, vol, start, 1, 1.0)
    want = start.astype(np.float64) - start[0].astype(np.float64) / planes
    assert np.abs(got - want).max() < 2.5e-7
