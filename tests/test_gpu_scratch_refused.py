"""Calls whose scratch is refused on the host (vt_refuse) and that have another way: the same answer, and no error left behind."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from vtwin import _abi as A  # noqa: E402
from vtwin import dome  # noqa: E402
from vtwin._lib import VtError  # noqa: E402
from vtwin.renderer import TwinRenderer  # noqa: E402

pytestmark = pytest.mark.gpu

NONE = 2 ** 64 - 1
SCRATCH = 2


def _renderer(width=16, height=16, **kw):
    return TwinRenderer.create(dome.make_dome_scene(seed=1, width=width, height=height, level=2), nodes=False, **kw)


# F's copy in aligned rows and the parts, or the parts alone: what the CUDA cores need is less
@pytest.mark.parametrize("n", [1541, 1540])
@pytest.mark.parametrize("host_f", [False, True])
def test_fp32_solve_of_several_columns(n, host_f):
    R = 4
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    F = torch.rand((n, n), device="cuda", generator=g) * (2.0 / n)
    if host_f:
        F = F.cpu().numpy()
    rho, E = (torch.rand(n, device="cuda", generator=g) * 0.8).cpu().numpy(), torch.rand((n, R), device="cuda", generator=g).cpu().numpy()

    def solve(limit):
        """(B, what is left as the context's last error) of a new context with at most that much scratch."""
        r = _renderer()
        r.lib.vt_refuse(r._ctx, SCRATCH, limit)
        try:
            B, info = r.solve_radiosity(F, rho, E, tol=1e-6, max_iters=60)
            assert info["status"] == A.VT_OK
        except VtError as e:
            assert "scratch" in str(e)
            B = None
        left = r.lib.vt_last_error(r._ctx)
        r.destroy()
        return B, left

    want, left = solve(NONE)
    assert left == b""
    refused, enough = 1000, 1 << 30   # for the tensor cores
    while enough - refused > 1:
        limit = (refused + enough) // 2
        B = solve(limit)[0]
        refused, enough = (refused, limit) if B is not None and np.array_equal(B, want) else (limit, enough)
    got, left = solve(refused)
    assert got is not None and left == b""
    # each is within its own residual of the solution: |B - B*| <= tol / (1 - 0.8) of |B|
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


def test_no_scratch_at_all_is_an_error():
    r = _renderer()
    r.lib.vt_refuse(r._ctx, SCRATCH, 1000)
    with pytest.raises(Exception, match="scratch"):
        r.solve_radiosity(np.zeros((64, 64), np.float32), np.zeros(64, np.float32), np.ones((64, 1), np.float32))
    r.lib.vt_refuse(r._ctx, SCRATCH, NONE)
    B, info = r.solve_radiosity(np.zeros((64, 64), np.float32), np.zeros(64, np.float32), np.ones((64, 1), np.float32))
    assert info["status"] == A.VT_OK and np.array_equal(B, np.ones((64, 1), np.float32))
    r.destroy()


@pytest.mark.parametrize("size", [(16, 9), (19, 2), (640, 480)])
def test_8_bit_readbacks(size):
    r = _renderer(*size)
    r.set_pose_array(A.identity_poses(1))
    r.renderCamera(0, spp=1, lightSamples=1, mode=A.VT_SHADE_PATH, max_depth=2)
    r.sensor(0, exposure_s=2e-3, gain=1.0)
    assert r.lib.vt_refuse(r._ctx, SCRATCH, 0) == A.VT_OK
    got, left = r.readback(0, "rgb8"), r.lib.vt_last_error(r._ctx)
    r.lib.vt_refuse(r._ctx, SCRATCH, NONE)
    rgba = r.readback(0, "rgba8")
    assert rgba[..., :3].std() > 0 and left == b""
    assert np.array_equal(got, rgba[..., :3]) and np.array_equal(r.readback(0, "rgb8"), got)
    r.destroy()
