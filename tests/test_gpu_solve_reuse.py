"""Mixed-precision solves that reuse one F's converted copies (reuse_f) in every order of the precisions, and with more columns than
the solve that made them: each call's iterate against its own residual in FP64."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [144, 1040])
@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("order", [["FP8", "BF16", "FP8"], ["BF16", "FP8", "BF16", "FP8"], ["FP8", "BF16", "BF16", "FP8", "FP8"]])
def test_precisions_in_turn(n, host, order):
    from vtwin import _abi as A
    from vtwin import dome
    from vtwin.renderer import TwinRenderer

    r = TwinRenderer.create(dome.make_dome_scene(seed=1, width=16, height=16, level=2), nodes=False)
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    F = torch.rand((n, n), device="cuda", generator=g) * (2.0 / n)
    rho = torch.rand(n, device="cuda", generator=g) * 0.8
    arg = F.cpu().numpy() if host else F
    tol = 1e-5
    for k, p in enumerate(order):
        R = (64, 4, 8, 1, 32)[k]   # the block of the first holds all
        E = torch.rand((n, R), device="cuda", generator=g)
        B, info = r.solve_radiosity(arg, rho.cpu().numpy(), E.cpu().numpy(), precision=getattr(A, "VT_PREC_" + p), tol=tol, max_iters=400,
                                    reuse_f=k > 0)
        assert info["status"] == 0 and info["residual"] <= tol, (k, p, info)
        X = torch.from_numpy(B).cuda().double().reshape(n, R)
        res = E.double() + rho.double()[:, None] * (F.double() @ X) - X
        # the solver's residual takes F and X as two bf16 numbers each, without the product of the low parts (1.2e-5 of X)
        assert float(res.norm() / X.norm()) <= tol + 1.2e-5
    r.destroy()
