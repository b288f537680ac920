"""The grid barrier of the FP32 solve's cooperative launch: blocks meet also where the count of arrivals passes 2^32, and a block that
never arrives ends the wait with an error that the context outlives."""
import time

import numpy as np
import pytest

from vtwin import _abi as A
from vtwin import dome
from vtwin.renderer import TwinRenderer

pytestmark = pytest.mark.gpu

BLOCKS, MEETINGS = 24, 6
LIMIT = 200_000_000   # 0.1 s of SM clocks


@pytest.fixture(scope="module")
def renderer():
    r = TwinRenderer.create(dome.make_dome_scene(seed=1, width=48, height=32, level=2), nodes=False)
    yield r
    r.destroy()


# from nothing, from the middle, and so that each of the meetings is the one that passes 2^32 or ends on it
@pytest.mark.parametrize("start", [0, 2 ** 31 - 30] + [2 ** 32 - BLOCKS * m - k for m in range(MEETINGS) for k in (0, 1, BLOCKS - 1) if m or k])
def test_blocks_meet(renderer, start):
    for _ in range(20):
        assert renderer.lib.vt_barrier_check(renderer._ctx, LIMIT, start, 0) == A.VT_OK


@pytest.mark.parametrize("start", [0, 2 ** 32 - 5])
@pytest.mark.parametrize("missing", [1, BLOCKS - 1])
def test_missing_block_times_out(renderer, start, missing):
    r = renderer
    t0 = time.perf_counter()
    assert r.lib.vt_barrier_check(r._ctx, 2_000_000, start, missing) == A.VT_ERR_TIMEOUT   # ~1 ms of waiting
    assert time.perf_counter() - t0 < 2.0
    assert b"did not arrive" in r.lib.vt_last_error(r._ctx)
    # the context is still usable
    assert r.lib.vt_barrier_check(r._ctx, LIMIT, start, 0) == A.VT_OK
    out = np.zeros((32, 48, 4), np.float32)
    r.renderCamera(0, out=out, spp=1, lightSamples=1, seed=0, mode=A.VT_SHADE_PATH, max_depth=2)
    assert np.all(np.isfinite(out)) and out[..., :3].max() > 0


def test_arguments(renderer):
    r = renderer
    assert r.lib.vt_barrier_check(r._ctx, 0, 0, 0) == A.VT_ERR_ARG
    assert r.lib.vt_barrier_check(r._ctx, LIMIT, 0, BLOCKS + 1) == A.VT_ERR_ARG
    assert r.lib.vt_barrier_check(r._ctx, LIMIT, 0, BLOCKS) == A.VT_OK   # nobody waits
