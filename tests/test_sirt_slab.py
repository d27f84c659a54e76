"""Context.sirt's slab: planes [z0, z1) come from the library, what follows them
in the caller's array is returned as it was, and a slab too short for the planes
is refused before the library reads past its end."""
import ctypes as C

import numpy as np
import pytest

import cases
import mtr
from conftest import rel_l2

PLANE = 20 * 24


class _Library:
    """Stand-in for libmtr: adds one to the planes it is asked for."""

    def mtr_sirt_from(self, h, axis, vol, z0, z1, n_inner, step, src, dst):
        n = (z1 - z0) * vol.X * vol.Y
        a = np.ctypeslib.as_array(C.cast(src, C.POINTER(C.c_float)), (n,))
        np.ctypeslib.as_array(C.cast(dst, C.POINTER(C.c_float)), (n,))[:] = a + 1.0
        return mtr.OK


def _context():
    c = mtr.Context.__new__(mtr.Context)
    c.lib, c.h = _Library(), None
    c.check = lambda st, what: None
    return c


@pytest.mark.parametrize("z1", [1, 3, 8])
def test_planes_outside_the_range_keep_the_callers_values(z1):
    c = cases.get("single")
    whole = np.random.default_rng(1).random(c.vol.shape, dtype=np.float32)
    for _ in range(4):  # (memory that the heap hands out again)
        junk = np.full(c.vol.shape, -999.0, np.float32)
        del junk
        got = _context().sirt(c.axes[0], c.vol, whole, 1, 0.5, 0, z1)
        assert got.shape == whole.shape
        assert np.array_equal(got[:z1], whole[:z1] + 1.0) and np.array_equal(got[z1:], whole[z1:])


@pytest.mark.parametrize("n", [0, PLANE - 1])
def test_a_short_slab_is_refused(n):
    c = cases.get("single")
    with pytest.raises(ValueError):
        _context().sirt(c.axes[0], c.vol, np.zeros(n, np.float32), 1, 0.5, 0, 1)


@pytest.mark.gpu
def test_whole_volume_with_a_range(ctx):
    c = cases.get("single")
    whole = np.random.default_rng(2).random(c.vol.shape, dtype=np.float32)
    got = ctx.sirt(c.axes[0], c.vol, whole, 2, 0.5, 0, 3)
    assert np.array_equal(got[3:], whole[3:])
    assert rel_l2(got[:3], ctx.sirt(c.axes[0], c.vol, whole[:3], 2, 0.5, 0, 3)) < 1e-5
