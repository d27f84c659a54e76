"""Forward splat over prefix sums (y-maps without a Z term) against the FP64
oracle: depths that divide the volume and that do not, every lane layout,
slopes of both signs from zero past one pixel per voxel, exact pixel
boundaries, and windows clamped at the detector's edges."""
import numpy as np
import pytest

import mtr
import oracle
import phantom
from conftest import rel_l2

pytestmark = pytest.mark.gpu

# positions to ~4e-6 px, sums in fixed point at 2^-17 of a brick's largest
# value or finer: the bound of the windowed kernels' tests
TOL = 1e-4
SLOPES = {"tilts": None, "flat": (0.0, 1e-9, -1e-9, 1e-6), "steep": (0.999, -0.999, 1.0, -1.0, 1.3), "halves": (0.5, -0.5, 0.25, -0.25)}


@pytest.mark.parametrize("depths", ["8,8,0,0,0", "8,16,1,1,0", "8,32,2,2,0", "8,5,0,0,0", "8,1,0,2,0"])
@pytest.mark.parametrize("kind", sorted(SLOPES))
@pytest.mark.parametrize("phi,px,py", [(30.0, 96, 104), (135.0, 52, 48)])
def test_prefix_splat_matches_oracle(ctx, monkeypatch, depths, kind, phi, px, py):
    monkeypatch.setenv("MTR_FORCE_DEPTHS", depths)
    v = mtr.VolumeSize.make(2, 47, -3, 36, 0, 21)
    c = phantom.make_case(v, px, np.arange(-60.0, 61.0, 15.0), [phi], 5, "gaussian", 0.02, 9, axis_cls=mtr.AxisData, py=py)
    a = c.axes[0]
    x = a.x_coef.copy()
    if SLOPES[kind] is not None:
        x[3::4] = np.resize(SLOPES[kind], len(x) // 4)
    axes = [mtr.AxisData(x, a.y_coef, a.data)]
    got = ctx.reconstruct(axes, v, mtr.params(iter_times=1, sirt_inner=2, sirt_step=0.5, mace_step=0.7))
    assert rel_l2(got, oracle.reconstruct(oracle.FP64, axes, v, 1, 2, 0.5, 0.7)) < TOL
