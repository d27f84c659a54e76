"""Two host threads, each with a context of its own, whose reconstructions launch
the same kernels with different amounts of shared memory (few and many views):
neither may lower the kernel's limit between the other's request and its launch."""
import threading

import numpy as np
import pytest

import mtr
import phantom
from conftest import rel_l2, run_to_run_tol

pytestmark = pytest.mark.gpu


def test_contexts_of_two_threads_share_kernels():
    vol = mtr.VolumeSize.make(0, 64, 0, 64, 0, 16)
    p = mtr.params(iter_times=1, sirt_inner=10, sirt_step=0.5, mace_step=0.7)
    rng = np.random.default_rng(4)
    jobs, want, errors = [], [], []
    for n in (9, 301):
        axes = []
        for phi in (0.0, 30.0):
            xc, yc = phantom.axis_maps(80, 80, np.linspace(-60.0, 60.0, n), phi, vol)
            axes.append(mtr.AxisData(xc, yc, rng.random((n, 80, 80), dtype=np.float32)))
        jobs.append(axes)
        with mtr.Context(0) as ctx:
            want.append(ctx.reconstruct(axes, vol, p))

    def work(i):
        try:
            with mtr.Context(0) as ctx:
                r = mtr.Recon(ctx, jobs[i], vol, p)
                for _ in range(200):
                    r.run()
                got = r.download()
                r.close()
            assert rel_l2(got, want[i]) < run_to_run_tol(mtr.PREC_FP32)
        except Exception as e:  # (to the test's own thread)
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
