"""Renders and calibrations on one context when the memory for the refinement's wave is refused (on the host, vt_refuse): the
refinement in several waves gives the image of one wave, and a replayed calibration's backward still finds the state it needs."""
import numpy as np
import pytest

from vtwin import _abi as A
from vtwin import dome
from vtwin.renderer import TwinRenderer

pytestmark = pytest.mark.gpu

NONE = 2 ** 64 - 1


def _wave_bytes(paths, lights, n_pix):
    return paths * (128 + 48 * lights) + 36 * n_pix + 18 * 256


def _frame(r, size, **o):
    out = np.zeros((size[1], size[0], 4), np.float32)
    r.renderCamera(0, out=out, seed=4, **o)
    return out


# pass 1 and the refinement with more light samples than the other; an odd image; what pass 1 needs holds three of the seven
# sub-samples, or one
@pytest.mark.parametrize("mode", [A.VT_SHADE_TWIN, A.VT_SHADE_PATH])
@pytest.mark.parametrize("lights,refine_lights", [(4, 1), (1, 3)])
def test_refinement_in_several_waves(mode, lights, refine_lights):
    size = (61, 37)
    n_pix = 64 * 40   # in tiles of 8 x 4
    sc = dome.make_dome_scene(seed=2, width=size[0], height=size[1], level=4, with_instruments=3)
    o = dict(spp=2, lightSamples=lights, refine=7, refineLightSamples=refine_lights, refineShadows=True, mode=mode, max_depth=3)
    poses = dome.batch_pose_array(dome.instrument_poses(n_poses=1, n_tools=3, seed=5))[0]
    images = []
    least = max(_wave_bytes(2 * n_pix, lights, n_pix), _wave_bytes(n_pix, refine_lights, n_pix))
    assert least < _wave_bytes(4 * n_pix, refine_lights, n_pix)
    for limit in (NONE, least):
        r = TwinRenderer.create(sc)
        r.set_pose_array(poses)
        assert r.lib.vt_refuse(r._ctx, 0, limit) == A.VT_OK
        images.append([_frame(r, size, **o) for _ in range(2)])
        r.debugFlags(reset=True)
        _frame(r, size, **o)
        assert r.debugFlags()["refined"] > 100
        # the memory is there after all: one wave
        assert r.lib.vt_refuse(r._ctx, 0, NONE) == A.VT_OK
        images[-1].append(_frame(r, size, **o))
        # less than pass 1 needs, on a context that has the state already: no refusal to notice
        assert r.lib.vt_refuse(r._ctx, 0, 0) == A.VT_OK
        images[-1].append(_frame(r, size, **o))
        r.destroy()
    assert np.isfinite(images[0][0]).all() and images[0][0][..., :3].max() > 0
    for group in images:
        for im in group:
            assert np.array_equal(im, images[0][0])


def test_no_memory_at_all_is_an_error_and_the_context_lives():
    sc = dome.make_dome_scene(seed=2, width=48, height=32, level=3)
    r = TwinRenderer.create(sc, nodes=False)
    r.set_pose_array(A.identity_poses(1))
    o = dict(spp=1, mode=A.VT_SHADE_PATH, max_depth=2)
    assert r.lib.vt_refuse(r._ctx, 0, 1000) == A.VT_OK
    with pytest.raises(Exception, match="wavefront state"):
        _frame(r, (48, 32), **o)
    assert r.lib.vt_refuse(r._ctx, 7, 0) == A.VT_ERR_ARG
    assert r.lib.vt_refuse(r._ctx, 0, NONE) == A.VT_OK
    assert _frame(r, (48, 32), **o)[..., :3].max() > 0
    r.destroy()


@pytest.mark.parametrize("take_all", [False, True])
def test_replayed_backward_after_a_frame_that_was_refused_memory(take_all):
    """A replayed forward's wave state, then a refined frame that wants more and is refused, then the backward."""
    size = (64, 48)
    n_pix = size[0] * size[1]
    sc = dome.make_dome_scene(seed=3, width=size[0], height=size[1], level=3)
    r = TwinRenderer.create(sc, nodes=False)
    r.set_pose_array(A.identity_poses(1))
    info = r.calib_setup(n_nodes=130, lamp_samples=4)
    albedo = np.clip(np.array([m["rho"] for m in sc["materials"]], np.float64), 0.05, 1.0)
    lamp = np.full(info["n_lamps"], 50.0)
    kw = dict(spp=8, max_depth=3, lightSamples=1)
    _, targets = r.calib_forward([0], albedo, lamp, **kw)
    grads = []
    for frame in (False, True):
        r.calib_forward([0], 0.9 * albedo, 1.1 * lamp, targets=targets, replay=True, **kw)
        if frame:
            have = _wave_bytes(8 * n_pix, 1, 0)
            # wanted: 16 sub-samples of refinement with 4 light samples
            assert _wave_bytes(16 * n_pix, 4, n_pix) > have > _wave_bytes(2 * n_pix, 4, n_pix)
            r.lib.vt_refuse(r._ctx, 0, have)
            o = dict(spp=1, lightSamples=4, refine=16, refineLightSamples=4, mode=A.VT_SHADE_PATH, max_depth=2)
            first = _frame(r, size, **o)
            if take_all:   # a frame that cannot be had at all gives the state away
                with pytest.raises(Exception, match="wavefront state"):
                    _frame(r, size, spp=16, lightSamples=16, mode=A.VT_SHADE_PATH, max_depth=2)
            else:
                assert np.array_equal(first, _frame(r, size, **o))
        grads.append(r.calib_backward())
    if take_all:   # and without even the replay's own, an error
        r.calib_forward([0], 0.9 * albedo, 1.1 * lamp, targets=targets, replay=True, **kw)
        with pytest.raises(Exception, match="wavefront state"):
            _frame(r, size, spp=16, lightSamples=16, mode=A.VT_SHADE_PATH, max_depth=2)
        r.lib.vt_refuse(r._ctx, 0, 1000)
        with pytest.raises(Exception, match="wave state"):
            r.calib_backward()
    r.destroy()
    for a, b in zip(*grads):
        # the same FP32 terms, summed in FP64 in another order
        assert np.abs(a - b).max() <= 1e-10 * np.abs(b).max()
