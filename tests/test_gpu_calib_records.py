"""The path records of a calibration step at odd numbers of paths and nodes: kept, and traced again in chunks of sub-samples
that begin inside a group of 32 records."""
import numpy as np
import pytest

from vtwin import dome
from vtwin.renderer import TwinRenderer

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size,spp,depth,lights,nodes", [((17, 13), 5, 4, 4, 131), ((33, 7), 3, 1, 1, 130), ((61, 37), 7, 3, 2, 1001)])
def test_stored_and_replayed_records_agree(size, spp, depth, lights, nodes):
    sc = dome.make_dome_scene(seed=3, width=size[0], height=size[1], level=3)
    sc["cameras"] = dome.batched_cameras(seed=3, n=2, width=size[0], height=size[1])
    for cam in sc["cameras"]:
        cam["fx"] = cam["fy"] = 300.0 * cam["size"][0] / 640.0
    r = TwinRenderer.create(sc, nodes=False)
    info = r.calib_setup(n_nodes=nodes, lamp_samples=4)
    albedo = np.clip(np.array([m["rho"] for m in sc["materials"]], np.float64), 0.05, 1.0)
    lamp = np.full(info["n_lamps"], 50.0)
    kw = dict(spp=spp, max_depth=depth, lightSamples=lights)
    _, targets = r.calib_forward([0, 1], albedo, lamp, **kw)
    runs = []
    for replay in (False, 1, 2):
        loss, images = r.calib_forward([0, 1], 0.9 * albedo, 1.1 * lamp, targets=targets, replay=replay, **kw)
        runs.append((loss, [np.array(i) for i in images], r.calib_backward()))
    r.destroy()
    loss, images, grads = runs[0]
    assert loss > 0 and all(np.isfinite(g).all() for g in grads)
    for l, im, gr in runs[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(im, images))
        # the same FP32 terms, summed in FP64 in another order
        assert abs(l - loss) <= 1e-12 * loss
        for a, b in zip(gr, grads):
            assert np.abs(a - b).max() <= 1e-10 * max(np.abs(b).max(), 1e-300)
