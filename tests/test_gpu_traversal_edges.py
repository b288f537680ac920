"""The traversal lanes at the edges of their ranges (one triangle a leaf to a leaf of the whole mesh, queues of less than a ray
a lane) and the bounces' overlapped launches against launches kept apart."""
import numpy as np
import pytest

from vtwin import _abi as A
from vtwin import dome
from vtwin.renderer import TwinRenderer

pytestmark = pytest.mark.gpu


def _scene(width, height, tools):
    return dome.make_dome_scene(seed=2, width=width, height=height, level=3, with_instruments=tools)


def _poses(tools):
    return np.concatenate([A.identity_poses(1), dome.instrument_poses(n_poses=1, n_tools=tools, seed=5)[0]]) if tools else A.identity_poses(1)


def _image(r, size, **o):
    out = np.zeros((size[1], size[0], 4), np.float32)
    r.renderCamera(0, out=out, seed=4, **o)
    return out


@pytest.mark.parametrize("size,tools", [((1, 1), 0), ((61, 37), 3), ((160, 120), 3)])
def test_leaf_sizes_give_one_image(size, tools):
    """Only the order of two triangles at one distance (a shared edge) may depend on the tree."""
    images = []
    for leaf in (1, 4, 64, 300):
        r = TwinRenderer.create(_scene(*size, tools), leafSize=leaf, nodes=False)
        r.set_pose_array(_poses(tools))
        images.append(_image(r, size, spp=2, lightSamples=2, mode=A.VT_SHADE_PATH, max_depth=4))
        r.destroy()
    assert np.isfinite(images[0]).all() and images[0][..., :3].max() > 0
    for im in images[1:]:
        assert np.mean((im != images[0]).any(-1)) <= 5e-3


@pytest.mark.parametrize("size", [(1, 1), (33, 17), (320, 200)])
@pytest.mark.parametrize("depth,lights", [(1, 1), (2, 3), (6, 1)])
def test_overlapped_bounces_equal_separate_launches(size, depth, lights):
    """The kernel profile launches every kernel after the one before: same image, bit for bit."""
    r = TwinRenderer.create(_scene(*size, 3), nodes=False)
    r.set_pose_array(_poses(3))
    o = dict(spp=3, lightSamples=lights, mode=A.VT_SHADE_PATH, max_depth=depth)
    want = _image(r, size, **o)
    r.kernel_profile(True)
    apart = _image(r, size, **o)
    r.kernel_profile(False)
    again = _image(r, size, **o)
    r.destroy()
    assert np.array_equal(want, apart) and np.array_equal(want, again)
