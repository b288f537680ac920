"""The twin's frames with their caches, and a pose batch, whose kernels are launched over one another's tails, against kernels
launched each after the one before (the kernel profile): the same images, bit for bit."""
import numpy as np
import pytest

from vtwin import _abi as A
from vtwin import dome
from vtwin.renderer import TwinRenderer

pytestmark = pytest.mark.gpu


def _poses(n, tools, seed):
    return dome.batch_pose_array(dome.instrument_poses(n_poses=n, n_tools=tools, seed=seed))


@pytest.mark.parametrize("size", [(9, 5), (61, 37), (320, 200)])
@pytest.mark.parametrize("lights,refine", [(1, 0), (4, 6), (3, 1)])
def test_twin_frames(size, lights, refine):
    sc = dome.make_dome_scene(seed=2, width=size[0], height=size[1], level=4, with_instruments=3, tool_radius=0.03)
    P = _poses(3, 3, 5)
    frames = []
    for apart in (False, True):
        r = TwinRenderer.create(sc)
        r.kernel_profile(apart)
        mine = []
        # the second frame of a pose reads the caches that the first one filled
        for k in (0, 0, 1, 2, 2):
            r.set_pose_array(P[k])
            out = np.zeros((size[1], size[0], 4), np.float32)
            r.renderCamera(0, out=out, seed=4, spp=1, lightSamples=lights, refine=refine, refineLightSamples=1, refineShadows=True)
            mine.append(out)
        r.destroy()
        frames.append(mine)
    assert all(np.isfinite(f).all() for f in frames[0]) and frames[0][0][..., :3].max() > 0
    for a, b in zip(*frames):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("depth,poses", [(1, 2), (5, 4)])
def test_pose_batch(depth, poses):
    size = (61, 37)
    sc = dome.make_dome_scene(seed=1, width=size[0], height=size[1], level=3, with_instruments=4, tool_radius=0.04)
    sc["cameras"] = dome.batched_cameras(seed=3, n=2, width=size[0], height=size[1])
    r = TwinRenderer.create(sc, nodes=False)
    P = _poses(poses, 4, 11)
    got = r.render_batch([0, 1], P, spp=3, max_depth=depth, seed=7, radiance=True, use_graph=False)["radiance"]
    r.kernel_profile(True)
    for c in range(2):
        for q in range(poses):
            r.set_pose_array(P[q])
            r.renderCamera(c, spp=3, lightSamples=1, seed=7, mode=A.VT_SHADE_PATH, max_depth=depth)
            assert np.array_equal(got[c][q].reshape(size[1], size[0], 4), r.readback(c, "linear").reshape(size[1], size[0], 4))
    r.destroy()
