"""FP32 sweeps with several right-hand sides on the tensor cores: against FP64, at the edges of the 128-row tiles, the
64-wide K stages and the kernel's smallest size, and where an infinity sends the solve to the CUDA-core sweeps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _inputs(n, R, signed, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    draw = torch.randn if signed else torch.rand
    F = draw((n, n), device="cuda", generator=g) / n
    B0 = draw((n, R), device="cuda", generator=g)
    rho = torch.rand(n, device="cuda", generator=g)
    E = torch.rand((n, R), device="cuda", generator=g)
    return F, rho.cpu().numpy(), E.cpu().numpy(), B0.cpu().numpy()


# the smallest size that takes the kernel, remainders of the tile, of the stage and of a row's 16 bytes, several tiles per
# block (6148)
@pytest.mark.parametrize("n,R", [(1536, 4), (1537, 8), (1540, 64), (1603, 20), (1666, 8), (2048, 60), (6148, 64)])
@pytest.mark.parametrize("signed", [False, True])
def test_one_sweep_against_fp64(n, R, signed):
    from vtwin.renderer import solve_radiosity

    F, rho, E, B0 = _inputs(n, R, signed, n + R)
    B, info = solve_radiosity(F, rho, E, max_iters=1, tol=1e-30, B0=B0)
    assert info["iters"] == 1
    F64, X = F.double(), torch.from_numpy(B0).cuda().double()
    r = torch.from_numpy(rho).cuda().double()[:, None]
    want = torch.from_numpy(E).cuda().double() + r * (F64 @ X)
    size = torch.from_numpy(E).cuda().double() + r * (F64.abs() @ X.abs())
    err = (torch.from_numpy(B).cuda().double() - want).abs() / size
    # the products to 2^-25, the tensor cores' sums over 32 of K and their drift to 2^-23, then n / 64 additions of 2^-24 of
    # the running sum each, the partials' and the epilogue's: a bound of (n / 64 + 8) 2^-24 on every element
    assert float(err.max()) <= (n / 64 + 8) * 2.0 ** -24
    # and on average well below it
    assert float(err.square().mean().sqrt()) <= 2.0 ** -22


@pytest.mark.parametrize("warm", [False, True])
def test_overflow_takes_the_cuda_core_sweeps(warm):
    """A system that diverges past float32's range gives what the CUDA-core sweeps give (an F one float off its alignment
    takes them from the start)."""
    from vtwin.renderer import solve_radiosity

    n, R = 1536, 8
    F, rho, E, B0 = _inputs(n, R, False, 3)
    F *= 3e30
    other = torch.empty(n * n + 1, device="cuda")
    other[1:] = F.reshape(-1)
    kw = dict(max_iters=4, check_every=2, tol=1e-6, B0=B0 if warm else None)
    got, a = solve_radiosity(F, rho, E, **kw)
    want, b = solve_radiosity(other[1:].view(n, n), rho, E, **kw)
    assert not np.isfinite(want).all()
    assert np.array_equal(got, want, equal_nan=True) and a["iters"] == b["iters"] and a["status"] == b["status"]
