"""The MACE step's consensus mean against FP64, over the axis counts with their
own kernel, the general one, sizes with a remainder, and states at the ends of
the FP32 range."""
import struct

import numpy as np
import pytest

import mtr

pytestmark = pytest.mark.gpu


def _states(rng, K, shape, kind):
    w = rng.standard_normal((K,) + shape).astype(np.float32)
    if kind == "wide":  # magnitudes over 30 decades, cancelling pairs
        w *= 10.0 ** rng.uniform(-15, 15, w.shape).astype(np.float32)
        w[-1] = -w[0] * np.float32(1.0000001)
    elif kind == "ends":
        pick = np.array([0.0, 1e-45, -3e-39, 1e-30, 2e-28, 1e36, -3e37, 1.7e38, np.inf, np.nan], np.float32)
        w = rng.choice(pick, w.shape).astype(np.float32)
    return w


@pytest.mark.parametrize("kind", ["plain", "wide", "ends"])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 5])
def test_consensus_mean(ctx, tmp_path, K, kind):
    rng = np.random.default_rng(K * 7 + len(kind))
    vol = mtr.VolumeSize.make(0, 37, 0, 11, 0, 5)  # 2035 voxels: a remainder after the 4-voxel steps
    xs, ys = mtr.geometry_from_tilts(np.array([-20.0, 0.0, 20.0]), 0.0, 40, 16, vol)
    axes = [mtr.AxisData(xs, ys, np.zeros((3, 16, 40), np.float32)) for _ in range(K)]
    w = _states(rng, K, vol.shape, kind)
    path = tmp_path / "state.ckpt"
    with open(path, "wb") as f:
        f.write(struct.pack("<8s7i4xq", b"MTRCKPT1", 1, K, vol.X, vol.Y, vol.Z, 0, 0, 0))
        np.zeros(vol.shape, np.float32).tofile(f)
        w.tofile(f)
    # no SIRT iteration: v = z = 2 * 0 - w, so the new states are rho * z + (1 - rho) * w in FP32
    rho = np.float32(0.25)
    r = mtr.Recon(ctx, axes, vol, mtr.params(1, 0, 0.5, float(rho)))
    r.load(path)
    r.run_outer(0, 1)
    got = r.download()
    with np.errstate(all="ignore"):
        z = -w
        new = rho * (np.float32(2) * z - z) + (np.float32(1) - rho) * w
        want = (new.astype(np.float64).sum(0) * (1.0 / K)).astype(np.float32)
    # both round an (almost) exact mean once: equal up to a rounding tie
    same = (got == want) | (np.isnan(got) & np.isnan(want))
    fine = np.isfinite(want) & ~same
    gap = np.abs(got[fine].astype(np.float64) - want[fine])
    assert (np.isfinite(want) | same).all()
    assert (gap <= np.spacing(np.abs(want[fine])).astype(np.float64)).all() and fine.sum() <= 2
