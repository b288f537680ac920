"""Mixed-precision solves (BF16 / FP8 sweeps under an accurate residual): the iterate's own residual in FP64, at the edges of
the 128-row tiles, of a stage's 64 or 128 of K and of the runs that the CTAs take."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


# one stage in all; a ragged row tile and stage; more tiles than a stage's K; fewer and more stages than SMs; runs that cross
# tiles, with and without a remainder
@pytest.mark.parametrize("n", [16, 112, 128, 144, 1040, 2064, 4096, 6160])
@pytest.mark.parametrize("R", [1, 4, 64])
@pytest.mark.parametrize("precision", ["VT_PREC_BF16", "VT_PREC_FP8"])
def test_residual_against_fp64(n, R, precision):
    from vtwin import _abi as A
    from vtwin.renderer import solve_radiosity

    g = torch.Generator(device="cuda")
    g.manual_seed(n + R)
    F = torch.rand((n, n), device="cuda", generator=g) * (2.0 / n)   # row sums near 1
    rho = torch.rand(n, device="cuda", generator=g) * 0.8
    E = torch.rand((n, R), device="cuda", generator=g)
    tol = 1e-5
    B, info = solve_radiosity(F, rho.cpu().numpy(), E.cpu().numpy(), precision=getattr(A, precision), tol=tol)
    assert info["status"] == 0 and info["residual"] <= tol
    X = torch.from_numpy(B).cuda().double().reshape(n, R)
    r = E.double() + rho.double()[:, None] * (F.double() @ X) - X
    # the solver's residual takes F and X as two bf16 numbers each, without the product of the low parts: each product to
    # 3 x 2^-18, so rho F X (at most X in size) to 1.2e-5 of X
    assert float(r.norm() / X.norm()) <= tol + 1.2e-5
