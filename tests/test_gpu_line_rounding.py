"""Rounding of the line kernels' sums over the angles: a tilt's value is
interpolated first and added once, so 61 positive values leave one rounding each
at the size of the partial sum: 0.42 x 2^-24 x sqrt(61 / 3) = 1.1e-7 of the
result (a rounding of a value of any mantissa is 0.42 x 2^-24 of it in the mean
square).  A second rounding per tilt, as when the two taps are added one by one,
makes it 1.6e-7."""
import numpy as np
import pytest

import mtr
import phantom

pytestmark = pytest.mark.gpu

N = 61


@pytest.mark.parametrize("phi", [0.0, 90.0])
def test_wbp_rounds_once_per_view(ctx, phi):
    vol = mtr.VolumeSize.make(0, 96, 0, 128, 0, 16)
    px, py = 160, 144
    xc, yc = phantom.axis_maps(px, py, np.linspace(-60.0, 60.0, N), phi, vol)
    xc, yc = xc.reshape(-1, 4), yc.reshape(-1, 4)
    yc[:, 0] += 0.3
    swapped = abs(np.sin(np.deg2rad(phi))) > 0.5  # lines along X
    m, w = (2, 1) if swapped else (1, 2)
    xc[:, w] = 0.0
    yc[:, m] = 0.0
    data = (1.0 + 0.1 * np.random.default_rng(2).random((N, py, px))).astype(np.float32)
    got = ctx.wbp(mtr.AxisData(xc.reshape(-1), yc.reshape(-1), data), vol)  # [Z][Y][X]
    if swapped:
        got = got.transpose(0, 2, 1)
    got = got.transpose(0, 2, 1)  # [Z][m][w]
    zs, ms, ws = (np.arange(n, dtype=np.float64) for n in got.shape)
    want = np.zeros(got.shape)
    for a in range(N):
        x = xc[a, 0] - 1.0 + xc[a, m] * ms[None, :] + xc[a, 3] * zs[:, None]
        y = yc[a, 0] - 1.0 + yc[a, w] * ws
        ix, iy = np.floor(x).astype(int), np.floor(y).astype(int)
        assert ix.min() >= 0 and ix.max() + 1 < px and iy.min() >= 0 and iy.max() + 1 < py
        fx, fy = (x - ix)[..., None], (y - iy)[:, None]
        image = data[a, iy] * (1.0 - fy) + data[a, iy + 1] * fy  # [w][px]
        want += image.T[ix] * (1.0 - fx) + image.T[ix + 1] * fx
    want /= N
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 1.35e-7
