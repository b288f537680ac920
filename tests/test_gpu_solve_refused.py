"""Dense solves when the host is refused what they would rather have (vt_refuse): the same answer the other way."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from vtwin import _abi as A  # noqa: E402
from vtwin import dome  # noqa: E402
from vtwin.renderer import TwinRenderer  # noqa: E402

pytestmark = pytest.mark.gpu

NONE = 2 ** 64 - 1
COOPERATIVE = 1


@pytest.fixture(scope="module")
def renderer():
    r = TwinRenderer.create(dome.make_dome_scene(seed=1, width=16, height=16, level=2), nodes=False)
    yield r
    r.destroy()


def _system(n, R):
    g = torch.Generator(device="cuda")
    g.manual_seed(n + R)
    F = torch.rand((n, n), device="cuda", generator=g) * (2.0 / n)
    return F, (torch.rand(n, device="cuda", generator=g) * 0.8).cpu().numpy(), torch.rand((n, R), device="cuda", generator=g).cpu().numpy()


@pytest.mark.parametrize("n", [1, 153, 1001, 4096])
@pytest.mark.parametrize("warm", [False, True])
def test_cooperative_launch(renderer, n, warm):
    """A launch per sweep sums every row in the same order: the same iterates bit for bit."""
    r = renderer
    F, rho, E = _system(n, 1)
    kw = dict(tol=1e-6, max_iters=50, check_every=3, B0=E * 0.5 if warm else None)
    want, a = r.solve_radiosity(F, rho, E, **kw)
    assert r.lib.vt_refuse(r._ctx, COOPERATIVE, 0) == A.VT_OK
    got, b = r.solve_radiosity(F, rho, E, **kw)
    assert r.lib.vt_refuse(r._ctx, COOPERATIVE, NONE) == A.VT_OK
    again, c = r.solve_radiosity(F, rho, E, **kw)
    assert a["status"] == A.VT_OK and a["iters"] > 1
    assert np.array_equal(want, got) and np.array_equal(want, again)
    assert (a["iters"], a["status"]) == (b["iters"], b["status"]) == (c["iters"], c["status"])
    assert abs(a["residual"] - b["residual"]) <= 1e-12 * a["residual"]
