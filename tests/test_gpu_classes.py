"""Programs whose ready tasks are queued by priority class (work of at least 0.3 of what the CTAs could
do in the longest path's time): many small instances in one launch give the bits that each gives alone,
where its few tasks go through the one queue, run after run; and a matrix of 40 x 40 blocks, whose
instructions have more successors than a warp has lanes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_many_instances_equal_single_ones(pp, gctx):
    sizes = [256, 200, 320, 64] * 16
    alone, hs = [], []
    for i, n in enumerate(sizes):
        h, _ = pp.make_dense_problem(gctx, n=n, leaf=64, seed=i)
        h.upload()
        h.factor()
        h.sync()
        h.download()
        alone.append(h.host_arena().copy())
        h2, _ = pp.make_dense_problem(gctx, n=n, leaf=64, seed=i)
        h2.upload()
        h2.keep_original()
        hs.append(h2)
    batch = pp.Batch(gctx, hs)
    for _ in range(3):
        batch.restore()
        batch.factor()
        batch.sync()
        for h, want in zip(hs, alone):
            h.download()
            assert np.array_equal(h.host_arena(), want)


def test_many_successors(pp, gctx):
    n = 2560
    h, A = pp.make_dense_problem(gctx, n=n, leaf=64, seed=9)
    h.upload()
    h.factor()
    b = pp.rhs(n, 1)
    x = torch.empty((n, 1), dtype=torch.float64, device="cuda")
    h.solve(torch.from_numpy(b).cuda(), x)
    h.sync()
    r = b - A @ x.cpu().numpy()
    # a normwise backward error of a diagonally dominant elimination: a few n u
    assert np.abs(r).max() <= 8 * n * 2.0**-53 * (np.abs(A).sum(1).max() * np.abs(x.cpu().numpy()).max() + np.abs(b).max())
