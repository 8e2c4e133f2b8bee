"""The residual of several right-hand sides: edges of the 256-row tile pairs, column groups, hard points.

Oracle: the dense FP64 matrix times x.  A sum of n products errs by at most n u sum_j |a_ij x_j|, with
u = 2^-53.  An entry itself is good to 8 u where it is a reciprocal (distance 3 u, the division's
argument 2 u, the division 2 u); an exponential takes its argument's error, 6 u, times that argument,
which is at most 16 in the unit cube: 8 u + 96 u.  The oracle errs by as much again.
"""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def run(pp, ctx, kernel, p0, pts, nrhs, update):
    n, dim = pts.shape
    rng = np.random.default_rng(n + nrhs)
    kid = pp.KERNELS[kernel]
    A = pp.KernelProblem(n, dim, kid, p0, 3.0, pts).dense()
    x, dx, b = (rng.standard_normal((n, nrhs)) for _ in range(3))
    xd, bd, r = torch.from_numpy(x).cuda(), torch.from_numpy(b).cuda(), torch.empty(n, nrhs, dtype=torch.float64).cuda()
    dxd = torch.from_numpy(dx).cuda() if update else None
    ctx.kernel_residual_batch([(kid, p0, 3.0, torch.from_numpy(pts).cuda(), xd, dxd, bd, r)])
    torch.cuda.synchronize()
    now = x + dx if update else x
    assert np.array_equal(xd.cpu().numpy(), now)
    entry = 8 if kernel in ("inv", "laplace") else 104
    bound = 2 * (n + entry) * 2.0**-53 * (np.abs(A) @ np.abs(now) + np.abs(b))
    assert (np.abs(r.cpu().numpy() - (b - A @ now)) <= bound).all()


@pytest.mark.parametrize("n", [1, 31, 255, 256, 257, 513, 800])
@pytest.mark.parametrize("nrhs,kernel,p0,dim", [(2, "inv", 1e-3, 2), (3, "exp", 0.1, 1), (8, "laplace", 1e-3, 3),
                                                (9, "matern32", 0.2, 3), (16, "inv", 1e-3, 1)])
def test_tile_edges(pp, gctx, n, nrhs, kernel, p0, dim):
    run(pp, gctx, kernel, p0, np.random.default_rng(n).uniform(0, 1, (n, dim)), nrhs, n % 2 == 1)


@pytest.mark.parametrize("kernel,p0", [("inv", 1e-3), ("laplace", 1e-3), ("exp", 0.1), ("matern32", 0.2)])
@pytest.mark.parametrize("nrhs", [2, 8])
def test_coincident_and_distant_points(pp, gctx, kernel, p0, nrhs):
    pts = np.random.default_rng(8).uniform(0, 1, (300, 3))
    pts[7], pts[9] = pts[270], pts[10]  # in different tiles, and side by side
    pts[20] = pts[21] = 0.0
    pts[21, 0] = 1e-20  # squared distance 1e-40, below the range of single precision
    pts[30] = 1e19      # squared distances near 1e38
    pts[40] = 1e150 if kernel == "matern32" else 1e160  # near 1e300; overflowing: entries are 0
    run(pp, gctx, kernel, p0, pts, nrhs, False)
