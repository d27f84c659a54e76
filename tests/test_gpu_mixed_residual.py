"""The format of the residual in mixed precision follows from the axis and the
whole volume: not from tuning, the slab depth of a streamed run, or another axis
that rounds to the same key of the tuner's cache."""
import numpy as np
import pytest

import mtr
import phantom
from conftest import rel_l2, run_to_run_tol

pytestmark = pytest.mark.gpu

N = 13


def _run(ctx, vol, phi, data=None, **kw):
    xc, yc = phantom.axis_maps(256, 256, np.linspace(-60.0, 60.0, N), phi, vol)
    axis = mtr.AxisData(xc, yc, (N, 256, 256) if data is None else data)
    r = mtr.Recon(ctx, [axis], vol, mtr.params(iter_times=1, sirt_inner=3, sirt_step=0.5, mace_step=0.7,
                                               precision=mtr.PREC_MIXED_FP16, **kw))
    try:
        form = r.describe()[0]["back_projection"]["window_format"]
        r.run()
        return form, r.download()
    finally:
        r.close()


def test_tuned_untuned_and_streamed_runs_share_the_format(ctx, monkeypatch):
    vol = mtr.VolumeSize.make(0, 256, 0, 256, 0, 64)
    data = np.random.default_rng(3).random((N, 256, 256), dtype=np.float32)
    monkeypatch.setenv("MTR_AUTOTUNE", "0")  # (first: a tuned choice would be taken from the process' cache)
    untuned, want = _run(ctx, vol, 60.0, data)
    monkeypatch.delenv("MTR_AUTOTUNE")
    tuned, got = _run(ctx, vol, 60.0, data)
    streamed, got_streamed = _run(ctx, vol, 60.0, data, flags=mtr.FLAG_STREAM_SLABS, slab_depth=32)
    assert untuned == tuned == streamed == "fp16 pairs"
    tol = run_to_run_tol(mtr.PREC_MIXED_FP16)
    assert rel_l2(got, want) < tol
    assert rel_l2(got_streamed, want) < tol


@pytest.mark.parametrize("first", [5.738, 5.75])
def test_format_does_not_hang_on_the_order_of_calls(ctx, first):
    # sin 5.738 and sin 5.75 degrees lie on the two sides of 0.1 and round to one key
    vol = mtr.VolumeSize.make(0, 256, 0, 256, 0, 64 if first == 5.738 else 65)  # a geometry new to the process
    forms = {phi: _run(ctx, vol, phi)[0] for phi in sorted((5.738, 5.75), key=lambda p: p != first)}
    assert forms[5.75] == "fp16 pairs" and forms[5.738] != "fp16 pairs"
