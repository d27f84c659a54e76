"""Row-pair windows whose y extent is a whole number of pixels: the brick's rows
stay in the window whatever the fraction of the first one, where the FP32 sums of
the ends round up to the next row just below one."""
import numpy as np
import pytest

import mtr
import oracle
import phantom
from conftest import rel_l2

pytestmark = pytest.mark.gpu

BELOW = (6e-8, 2e-7, 5e-7, 9e-7, 1e-6, 0.25)  # the first row's fraction is one less this


def _axis(phi, below):
    v = mtr.VolumeSize.make(0, 70, 0, 66, 0, 18)
    c = phantom.make_case(v, 84, np.arange(-60.0, 61.0, 20.0), [phi], 5, "gaussian", 0.02, 3, axis_cls=mtr.AxisData, py=80)
    a = c.axes[0]
    x, y = a.x_coef.copy(), a.y_coef.copy()
    for q in (1, 2, 3):
        y[q::4] = np.round(y[q::4])
    lo = min(float(y[0] + sum(y[q] * e for q, e in ((1, ex), (2, ey)))) for ex in (0, 69) for ey in (0, 65))
    y[0::4] += np.floor(5.0 - lo) - y[0] + np.floor(y[0]) + 1.0 - below
    return v, [mtr.AxisData(x, y, a.data)]


@pytest.mark.parametrize("below", BELOW)
@pytest.mark.parametrize("phi", [0.0, 90.0, 180.0])
@pytest.mark.parametrize("flags,forced", [(mtr.FLAG_HOST_VOLUMES, None), (0, "16,16,0,0,0"), (0, "8,8,1,1,0"),
                                          (0, "32,32,2,2,0")])
def test_whole_extents_match_oracle(ctx, monkeypatch, phi, below, flags, forced):
    if forced:
        monkeypatch.setenv("MTR_FORCE_DEPTHS", forced)
    v, axes = _axis(phi, below)
    r = mtr.Recon(ctx, axes, v, mtr.params(1, 2, 0.5, 0.7, mtr.PREC_FP32, flags))
    assert r.describe()[0]["back_projection"]["tma"]
    r.run()
    # FP32 positions and fixed-point sums: the bound of the windowed kernels' tests
    assert rel_l2(r.download(), oracle.reconstruct(oracle.FP64, axes, v, 1, 2, 0.5, 0.7)) < 1e-4
