"""Mixed-precision solves about the size and the number of columns where the combining kernels' blocks change their rows: the iterate's
own residual in FP64."""
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R", [(16, 20), (144, 60), (1040, 32), (4848, 16), (4848, 20), (4848, 64), (4864, 20)])
@pytest.mark.parametrize("precision", ["VT_PREC_BF16", "VT_PREC_FP8"])
def test_residual_against_fp64(n, R, precision):
    from vtwin import _abi as A
    from vtwin.renderer import solve_radiosity

    g = torch.Generator(device="cuda")
    g.manual_seed(n + R)
    F = torch.rand((n, n), device="cuda", generator=g) * (2.0 / n)
    rho = torch.rand(n, device="cuda", generator=g) * 0.8
    E = torch.rand((n, R), device="cuda", generator=g)
    tol = 1e-5
    B, info = solve_radiosity(F, rho.cpu().numpy(), E.cpu().numpy(), precision=getattr(A, precision), tol=tol)
    assert info["status"] == 0 and info["residual"] <= tol
    X = torch.from_numpy(B).cuda().double().reshape(n, R)
    r = E.double() + rho.double()[:, None] * (F.double() @ X) - X
    res = float(r.norm() / X.norm())
    # the solver's residual takes F and X as two bf16 numbers each, without the product of the low parts: 1.2e-5 of X
    assert res <= tol + 1.2e-5 and abs(res - info["residual"]) <= 1.2e-5
