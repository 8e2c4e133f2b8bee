"""Entries of the residual at the ends of the distances' range: one answer whatever the number of
right-hand sides.  Oracle and bounds as in test_gpu_residual_wide."""
import numpy as np
import pytest
import torch

from test_gpu_residual_wide import run

pytestmark = pytest.mark.gpu

NRHS = [1, 2, 8, 16]


def residual(pp, ctx, kernel, p0, pts, x, b):
    r = torch.empty_like(torch.from_numpy(b)).cuda()
    ctx.kernel_residual_batch([(pp.KERNELS[kernel], p0, 0.5, torch.from_numpy(pts).cuda(), torch.from_numpy(x).cuda(), None,
                                torch.from_numpy(b).cuda(), r)])
    torch.cuda.synchronize()
    return r.cpu().numpy()


@pytest.mark.parametrize("nrhs", NRHS)
@pytest.mark.parametrize("kernel", ["inv", "laplace", "exp", "matern32"])
def test_zero_distance_below_a_tiny_parameter(pp, gctx, kernel, nrhs):
    """p0 = 1e-200: an entry at distance zero is K(0), 1e200 or 1 here, not that at a smallest distance."""
    pts = np.random.default_rng(3).uniform(0, 1, (300, 3))
    pts[5] = pts[290]
    run(pp, gctx, kernel, 1e-200, pts, nrhs, False)


@pytest.mark.parametrize("nrhs", NRHS)
@pytest.mark.parametrize("kernel,p0", [("inv", 1e-3), ("laplace", 1e-3), ("exp", 0.1), ("matern32", 0.2)])
def test_overflowing_distances(pp, gctx, kernel, p0, nrhs):
    """A squared distance past the largest double counts as 2^1023: entries of at most 1e-153."""
    rng = np.random.default_rng(4)
    pts, far = rng.uniform(0, 1, (300, 3)), [40, 281]
    near = np.delete(np.arange(300), far)
    x, b = rng.standard_normal((300, nrhs)), rng.standard_normal((300, nrhs))
    A = np.zeros((300, 300))
    A[np.ix_(near, near)] = pp.KernelProblem(298, 3, pp.KERNELS[kernel], p0, 0.5, pts[near]).dense()
    for i, at in zip(far, (1e160, -1e300)):
        pts[i] = at
        A[i, i] = pp.kernel_eval(pp.KERNELS[kernel], 0.0, p0) + 0.5
    r = residual(pp, gctx, kernel, p0, pts, x, b)
    assert (np.abs(r - (b - A @ x)) <= 2 * (300 + 104) * 2.0**-53 * (np.abs(A) @ np.abs(x) + np.abs(b))).all()


@pytest.mark.parametrize("kernel", ["inv", "laplace"])
def test_no_parameter_is_no_number_on_the_diagonal(pp, gctx, kernel):
    """p0 = 0 is accepted; K(0) is not finite then, nor is any row's residual, with one column or more."""
    rng = np.random.default_rng(5)
    pts, x, b = rng.uniform(0, 1, (300, 2)), rng.standard_normal((300, 8)), rng.standard_normal((300, 8))
    for q in (1, 2, 8):
        assert not np.isfinite(residual(pp, gctx, kernel, 0.0, pts, x[:, :q].copy(), b[:, :q].copy())).any()


@pytest.mark.parametrize("n", [5, 257, 300])
@pytest.mark.parametrize("nrhs", NRHS)
def test_places_past_the_last_point_are_of_no_account(pp, gctx, n, nrhs):
    """Points far from the origin and a kernel that grows with the distance (a negative length is accepted):
    an entry between a point and the origin would overflow, and nothing of it may reach a sum."""
    rng = np.random.default_rng(n)
    pts = 1000.0 + 0.01 * rng.uniform(0, 1, (n, 3))
    x, b = rng.standard_normal((n, nrhs)), rng.standard_normal((n, nrhs))
    d = np.sqrt(((pts[:, None, :] - pts[None, :, :]) ** 2).sum(-1))
    A = np.exp(d / 0.05) + 0.5 * np.eye(n)
    r = residual(pp, gctx, "exp", -0.05, pts, x, b)
    # entries to 8 u and their argument's 6 u; the coordinates' differences are exact
    assert (np.abs(r - (b - A @ x)) <= 2 * (n + 16) * 2.0 ** -53 * (np.abs(A) @ np.abs(x) + np.abs(b))).all()
