"""The packed 8-bit readback of a sensor image against its RGBA form, at pixel counts with every remainder of the packing's
four pixels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(16, 9), (15, 7), (19, 2), (9, 3)])
def test_rgb8_is_rgba8_without_alpha(width, height):
    from vtwin import _abi as A
    from vtwin import dome
    from vtwin.renderer import TwinRenderer

    r = TwinRenderer.create(dome.make_dome_scene(seed=1, width=width, height=height, level=2), nodes=False)
    r.set_pose_array(A.identity_poses(1))
    r.renderCamera(0, spp=1, lightSamples=1, mode=A.VT_SHADE_PATH, max_depth=2)
    r.sensor(0, exposure_s=2e-3, gain=1.0)
    rgba = r.readback(0, "rgba8")
    assert rgba[..., :3].std() > 0
    assert np.array_equal(r.readback(0, "rgb8"), rgba[..., :3])
    r.destroy()
