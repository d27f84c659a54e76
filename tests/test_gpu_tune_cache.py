"""The tuner's cache file: an oblique axis, which is really tuned, is written
under its geometry's key and a second process takes its choice from the file;
a line axis is listed with the depths its kernels run at."""
import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import mtr
import phantom

pytestmark = pytest.mark.gpu

DESCRIBE = """
import json, sys
import numpy as np
sys.path[:0] = sys.argv[1:2]
import mtr, phantom
vol = mtr.VolumeSize.make(0, 45, 0, 37, 0, 23)
xc, yc = phantom.axis_maps(68, 68, np.linspace(-60.0, 60.0, 9), 50.0, vol)
with mtr.Context(0) as ctx:
    r = mtr.Recon(ctx, [mtr.AxisData(xc, yc, (9, 68, 68))], vol, mtr.params(iter_times=1, sirt_inner=1))
    print(json.dumps(r.describe()[0]))
    r.close()
"""


def _describe(cache):
    env = {k: v for k, v in os.environ.items() if not k.startswith("MTR_")} | {"MTR_AUTOTUNE_CACHE": str(cache)}
    out = subprocess.run([sys.executable, "-c", DESCRIBE, str(Path(mtr.__file__).parent)], env=env, check=True,
                         capture_output=True, text=True, timeout=300)
    return json.loads(out.stdout.strip().splitlines()[-1])


def test_a_second_process_takes_the_choice_from_the_file(tmp_path):
    cache = tmp_path / "tune.json"
    first = _describe(cache)
    d = json.loads(cache.read_text())
    (key, choice), = d.items()
    assert key.startswith("p68x68x9_v45x37x23")
    assert first["back_projection"]["depth"] == choice[0] and first["forward"]["depth"] == choice[1]
    # another valid choice than the one timed
    planted = [4 if choice[0] != 4 else 8, 8 if choice[1] != 8 else 16, 0, 1, 1]
    cache.write_text(json.dumps({key: planted}))
    second = _describe(cache)
    assert second["back_projection"]["depth"] == planted[0] and second["forward"]["depth"] == planted[1]
    assert second["back_projection"]["window_format"] == "pairs"


def test_line_axes_are_listed_with_their_own_depths(ctx, tmp_path, monkeypatch):
    cache = tmp_path / "tune.json"
    monkeypatch.setenv("MTR_AUTOTUNE_CACHE", str(cache))
    vol = mtr.VolumeSize.make(0, 60, 0, 52, 0, 11)
    xc, yc = phantom.axis_maps(76, 76, np.linspace(-60.0, 60.0, 9), 0.0, vol)
    r = mtr.Recon(ctx, [mtr.AxisData(xc, yc, (9, 76, 76))], vol, mtr.params(iter_times=1, sirt_inner=1))
    try:
        d = r.describe()[0]
        assert d["back_projection"]["window_format"] == "line image"
        entries = [v for k, v in json.loads(cache.read_text()).items()
                   if k.startswith("p76x76x9_v60x52x11") and k.endswith("_lines")]
        assert entries == [[d["back_projection"]["depth"], d["forward"]["depth"], 1, 1, 0]]
    finally:
        r.close()
