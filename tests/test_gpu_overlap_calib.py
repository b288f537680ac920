"""A calibration's bounces, whose closest hits are launched over the light samples before them, against launches that each end
before the next (CUDA_LAUNCH_BLOCKING, in a process of its own): the same images bit for bit, the same gradients."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = r'''
import sys
import numpy as np
from vtwin import dome
from vtwin.renderer import TwinRenderer

w, h, spp, depth, lights, replay = (int(a) for a in sys.argv[2:])
sc = dome.make_dome_scene(seed=3, width=w, height=h, level=4, with_instruments=3, tool_radius=0.03)
r = TwinRenderer.create(sc, nodes=False)
r.set_pose_array(dome.batch_pose_array(dome.instrument_poses(n_poses=1, n_tools=3, seed=5))[0])
info = r.calib_setup(n_nodes=130, lamp_samples=4)
albedo = np.clip(np.array([m["rho"] for m in sc["materials"]], np.float64), 0.05, 1.0)
lamp = np.full(info["n_lamps"], 50.0)
kw = dict(spp=spp, max_depth=depth, lightSamples=lights)
_, targets = r.calib_forward([0], albedo, lamp, **kw)
loss, images = r.calib_forward([0], 0.9 * albedo, 1.1 * lamp, targets=targets, replay=bool(replay), **kw)
ga, gl = r.calib_backward()
np.savez(sys.argv[1], loss=loss, image=np.array(images[0]), ga=ga, gl=gl)
'''


@pytest.mark.parametrize("args", [(9, 5, 2, 2, 1, 0), (161, 97, 3, 4, 2, 0), (161, 97, 3, 3, 4, 1)])
def test_overlapped_bounces_equal_separate_launches(tmp_path, args):
    runs = []
    for blocking in ("0", "1"):
        out = tmp_path / f"{blocking}.npz"
        env = dict(os.environ, CUDA_LAUNCH_BLOCKING=blocking, PYTHONPATH=os.path.join(ROOT, "veridien-twin_gb300"))
        subprocess.run([sys.executable, "-c", PROGRAM, str(out), *map(str, args)], check=True, env=env, timeout=300)
        runs.append(np.load(out))
    a, b = runs
    assert a["image"][..., :3].max() > 0 and np.array_equal(a["image"], b["image"])
    assert a["loss"] == b["loss"]
    for k in ("ga", "gl"):   # the same FP32 terms, summed in FP64 in another order
        assert np.abs(a[k] - b[k]).max() <= 1e-10 * np.abs(b[k]).max()
