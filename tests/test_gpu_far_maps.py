"""Maps that place the volume far off the detector.  Within +-1e9 px no tap falls
on it and nothing is reconstructed; beyond, the back-projection's windows cannot
hold the position and the launch is flagged.  Neither reads or writes outside
the windows, and the context works on."""
import numpy as np
import pytest

import cases
import mtr
import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu
P = dict(iter_times=1, sirt_inner=2, sirt_step=0.5, mace_step=0.7)


def _moved(c, which, offset):
    axes = []
    for a in c.axes:
        xc, yc = a.x_coef.copy(), a.y_coef.copy()
        (xc if which == "x" else yc)[0::4] += offset
        axes.append(mtr.AxisData(xc, yc, a.data))
    return axes


@pytest.mark.parametrize("case", ["mid", "mid_oblique"])
@pytest.mark.parametrize("which", ["x", "y"])
@pytest.mark.parametrize("offset", [1e8, -1e8])
def test_off_the_detector_gives_zeros(ctx, case, which, offset):
    c = cases.get(case)
    assert not ctx.reconstruct(_moved(c, which, offset), c.vol, mtr.params(**P)).any()


@pytest.mark.parametrize("case", ["mid_oblique", "leaning"])
@pytest.mark.parametrize("which", ["x", "y"])
@pytest.mark.parametrize("offset", [1.5e9, -5e9, 1e12, -1e300])
@pytest.mark.parametrize("prec", [mtr.PREC_FP32, mtr.PREC_MIXED_FP16])
def test_beyond_the_integers_is_refused_and_the_context_works_on(ctx, case, which, offset, prec):
    c = cases.tilt_axis_in_z(cases.get("mid_oblique")) if case == "leaning" else cases.get(case)
    with pytest.raises(mtr.MtrError):
        ctx.reconstruct(_moved(c, which, offset), c.vol, mtr.params(**P, precision=prec))
    want = oracle.reconstruct(oracle.REF_FAITHFUL, c.axes, c.vol, 1, 2, 0.5, 0.7)
    assert rel_l2(ctx.reconstruct(c.axes, c.vol, mtr.params(**P)), want) < 1e-4


def test_a_frame_far_along_x_keeps_the_windows(ctx):
    """The x offset itself is small; the volume's own coordinates carry it away."""
    c = cases.get("mid")
    v = mtr.VolumeSize.make(2_000_000_000, 2_000_000_064, 4, 52, 0, 20)
    r = mtr.Recon(ctx, c.axes[:1], v, mtr.params(**P))
    assert r.describe()[0]["back_projection"]["window_format"] != "line image"
    r.run()
    with pytest.raises(mtr.MtrError):
        r.download()
