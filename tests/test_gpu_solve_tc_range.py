"""FP32 sweeps with several right-hand sides over the range of the format: F and B near its smallest normal numbers and below them,
and so large that the tensor cores' sums overflow while float32 holds them."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _sweep(F, B0, rho, E):
    from vtwin.renderer import solve_radiosity

    B, info = solve_radiosity(F, rho, E, max_iters=1, tol=1e-30, B0=B0.cpu().numpy())
    assert info["iters"] == 1
    return torch.from_numpy(B).cuda().double()


# F of 2^-f, B of 2^-b: sums of n / 4 2^-(f + b)
@pytest.mark.parametrize("n,R", [(1537, 8), (2048, 64)])
@pytest.mark.parametrize("f,b", [(0, 0), (0, 110), (0, 118), (0, 130), (100, 0), (118, 0), (130, 0), (60, 58), (20, 98), (-40, -40), (-60, 100)])
def test_sweep_over_the_range(n, R, f, b):
    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    F = torch.rand((n, n), device="cuda", generator=g) * 2.0 ** -f
    B0 = torch.rand((n, R), device="cuda", generator=g) * 2.0 ** -b
    got = _sweep(F, B0, np.ones(n, np.float32), np.zeros((n, R), np.float32))
    want = F.double() @ B0.double()
    err = (got - want).abs() / want
    # the products to 2^-25, the sums over 32 of K to 2^-23, n / 64 additions of 2^-24 and the epilogue's; each of the sums is a
    # normal number
    assert float(want.min()) >= 2.0 ** -125
    assert float(err.max()) <= (n / 64 + 8) * 2.0 ** -24
    assert float(err.square().mean().sqrt()) <= 2.0 ** -22


@pytest.mark.parametrize("f,b", [(-60, -40), (-30, -75), (0, -113), (-113, 20)])
def test_large_values_take_the_cuda_core_sweep(f, b):
    """Past 2^96 a sum, or 2^112 a value: what the CUDA cores give, bit for bit (a copy of F one float off its alignment takes them)."""
    n, R = 1536, 4
    g = torch.Generator(device="cuda")
    g.manual_seed(5)
    other = torch.rand(n * n + 1, device="cuda", generator=g) * 2.0 ** -f
    F = other[1:].clone().view(n, n)
    B0 = torch.rand((n, R), device="cuda", generator=g) * 2.0 ** -b
    rho, E = np.ones(n, np.float32), np.ones((n, R), np.float32)
    got, want = _sweep(F, B0, rho, E), _sweep(other[1:].view(n, n), B0, rho, E)
    assert torch.isfinite(want).all() and torch.equal(got, want)
