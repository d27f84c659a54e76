"""Line back-projection whose pipeline waits give up at once (as the windowed
kernels' in test_gpu_failure.py): the launch flags itself, its producer drains
its own copies with the full bound before the epilogue reuses their memory, the
host reads MTR_ERR_TIMEOUT, and the same context then reconstructs correctly."""
import pytest

import cases
import mtr
import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def test_line_kernel_waits_that_give_up_report_timeout(ctx):
    c = cases.get("mid")  # 0 and 90 degrees: lines along Y and X
    p = mtr.params(iter_times=1, sirt_inner=2, sirt_step=0.5, mace_step=0.7)
    r = mtr.Recon(ctx, c.axes, c.vol, p)
    lib = ctx.lib
    try:
        assert all(d["back_projection"]["window_format"] == "line image" for d in r.describe())
        assert lib.mtr_set_wait_limit(0) == mtr.OK
        try:
            r.run()
            st = lib.mtr_recon_check(r.h)
        finally:
            lib.mtr_set_wait_limit(-1)
        assert st == mtr.ERR_TIMEOUT
    finally:
        r.close()
    got = ctx.reconstruct(c.axes, c.vol, p)
    want = oracle.reconstruct(oracle.REF_FAITHFUL, c.axes, c.vol, 1, 2, 0.5, 0.7)
    assert rel_l2(got, want) < 1e-4
