"""The footprint a server admits against is what a reconstruction allocates:
the row tables of a line axis (one per view where every view has its own y-map)
take no memory beside the arrays that are counted."""
import numpy as np
import pytest
import torch

import mtr

pytestmark = pytest.mark.gpu


def test_row_tables_take_no_memory_of_their_own():
    n, px, py, w = 1000, 16, 2048, 2000  # two axes: 81 MB of tables where each view has its own
    vol = mtr.VolumeSize.make(0, 8, 0, w, 0, 8)
    xc = np.tile([5.0, 1.0, 0.0, 0.0], n)
    used = {}
    for shared in (True, False):
        yc = np.tile([20.0, 0.0, 1.0, 0.0], n)
        if not shared:
            yc[0::4] += 1e-4 * np.arange(n)
        with mtr.Context(0) as ctx:
            before = torch.cuda.mem_get_info()[0]
            r = mtr.Recon(ctx, [mtr.AxisData(xc, yc, (n, py, px))] * 2, vol, mtr.params(iter_times=1, sirt_inner=1))
            assert all(d["back_projection"]["window_format"] == "line image" for d in r.describe())
            used[shared] = before - torch.cuda.mem_get_info()[0], r.footprint()
            r.close()
    assert used[True][1] == used[False][1]
    assert abs(used[True][0] - used[False][0]) < 40e6  # (the pool grows in steps of 32 MB at most)
