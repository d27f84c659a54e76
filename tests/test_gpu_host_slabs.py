"""Host buffers: slab entries into fresh, written, odd-addressed and pinned ones
give the same values and change nothing beside them; uploads from the host
equal uploads from the device."""
import ctypes as C

import numpy as np
import pytest
import torch

import cases
import mtr
import phantom

pytestmark = pytest.mark.gpu

# The same kernels on the same inputs; float atomics add in an unspecified order.
TOL = 1e-5


def _buffer(kind, n):
    """n floats with a guard of 64 on each side, and the whole array."""
    if kind == "fresh":
        whole = np.empty(n + 128, np.float32)
    elif kind == "pinned":
        whole = torch.full((n + 128,), 7.0).pin_memory().numpy()
    elif kind == "odd":  # 4-byte aligned only
        whole = np.full(n + 129, 7.0, np.float32)[1:]
    else:
        whole = np.full(n + 128, 7.0, np.float32)
    whole[:64] = whole[64 + n:] = 5.0
    return whole[64:64 + n], whole


@pytest.mark.parametrize("kind", ["fresh", "written", "odd", "pinned"])
@pytest.mark.parametrize("z", [(0, 1), None])
def test_slab_entries_into_any_host_buffer(ctx, kind, z):
    c = cases.get("mid")
    a, v = c.axes[0], c.vol
    z0, z1 = (v.Zstart, v.Zstart + 1) if z else (v.Zstart, v.Zend)
    n = (z1 - z0) * v.Y * v.X
    want = ctx.wbp(a, v, z0, z1).ravel()
    out, whole = _buffer(kind, n)
    s = a.c_struct()
    ctx.check(ctx.lib.mtr_wbp(ctx.h, C.byref(s), v, z0, z1, out.ctypes.data), "mtr_wbp")
    assert np.linalg.norm(out - want) <= TOL * np.linalg.norm(want)
    start = np.random.default_rng(3).random(n, dtype=np.float32)
    kept = start.copy()
    moved = ctx.sirt(a, v, start, 3, 0.5, z0, z1)
    assert np.array_equal(start, kept)
    out[:] = start
    ctx.check(ctx.lib.mtr_sirt(ctx.h, C.byref(s), v, z0, z1, 3, 0.5, out.ctypes.data), "mtr_sirt")
    assert np.linalg.norm(out - moved) <= TOL * np.linalg.norm(moved)
    assert (whole[:64] == 5.0).all() and (whole[64 + n:] == 5.0).all()


@pytest.mark.parametrize("prec", [mtr.PREC_FP32, mtr.PREC_MIXED_FP16])
@pytest.mark.parametrize("half", [False, True])
@pytest.mark.parametrize("px", [41, 47, 48])
@pytest.mark.parametrize("phi", [0.0, 30.0])
def test_host_uploads_equal_device_uploads(ctx, prec, half, px, phi):
    """Rows with and without padding, uploaded after a run on other values."""
    vol = mtr.VolumeSize.make(0, 36, 0, 30, 0, 9)
    c = phantom.make_case(vol, px, np.arange(-60.0, 61.0, 20.0), [phi], 3, "gaussian", 0.02, 4, axis_cls=mtr.AxisData,
                          py=44)
    a = c.axes[0]
    data = np.ascontiguousarray(a.data.astype(np.float16) if half else a.data)
    p = mtr.params(1, 2, 0.5, 0.7, prec)
    got = []
    for kind in (mtr.MEM_HOST, mtr.MEM_DEVICE):
        r = mtr.Recon(ctx, [mtr.AxisData(a.x_coef, a.y_coef, np.ones_like(a.data))], vol, p)
        r.run()
        d = data if kind == mtr.MEM_HOST else torch.from_numpy(data).cuda()
        torch.cuda.synchronize()
        (r.upload_half if half else r.upload)(0, d, kind)
        ctx.synchronize()
        r.run()
        got.append(r.download())
    assert np.linalg.norm(got[0] - got[1]) <= TOL * np.linalg.norm(got[1])
