"""One right-hand side, the sweeps between two checks in one launch: the iterate of k sweeps against k FP64 sweeps, at sizes
about the number of blocks, a row's remainders and the largest iterate that the launch holds, and checks that split the sweeps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 31, 152, 153, 500, 1001, 4096, 16384, 16385])
@pytest.mark.parametrize("check_every,sweeps", [(1, 3), (3, 7), (8, 8)])
def test_sweeps_against_fp64(n, check_every, sweeps):
    from vtwin.renderer import solve_radiosity

    g = torch.Generator(device="cuda")
    g.manual_seed(n)
    F = torch.rand((n, n), device="cuda", generator=g) / n
    rho = torch.rand(n, device="cuda", generator=g)
    E = torch.rand((n, 1), device="cuda", generator=g)
    B, info = solve_radiosity(F, rho.cpu().numpy(), E.cpu().numpy(), max_iters=sweeps, tol=1e-30, check_every=check_every)
    X, k = E.double(), info["iters"]
    assert 1 <= k < sweeps + check_every   # a single node may stand still before
    for _ in range(k):
        X = E.double() + rho.double()[:, None] * (F.double() @ X)
    # all terms positive: each sweep's sum is off by at most 2^-24 of itself for each of its additions in a row (n / 32 of a
    # lane and the lanes' tree) and adds the last sweep's error, which rho F (at most 1/2 in row sum, about) shrinks
    err = (torch.from_numpy(B).cuda().double().reshape(n, 1) - X).abs() / X
    assert float(err.max()) <= 2 * (n / 32 + 16) * 2.0 ** -24
