"""LRTRUNC without a tolerance: the rank is the number of singular values above zero (at most the limit),
as it is with one, and the columns beyond it are zero."""
import numpy as np
import pytest

from test_gpu_lowrank import TOL, execute
from test_gpu_vm import dev, rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("k,r", [(8, 0), (8, 3), (17, 16), (32, 5), (1, 0)])
def test_no_tolerance_drops_what_is_zero(pp, gctx, k, r):
    """The columns beyond r are exactly zero, so is the rest of the Gram matrix: nothing is rounded."""
    rng = np.random.default_rng(k + r)
    U, V = np.linalg.qr(rng.standard_normal((64, k)))[0], rng.standard_normal((50, k))
    V[:, rng.permutation(k)[r:]] = 0.0
    dU, dV, dr = dev(U), dev(V), dev(np.full((1, 1), -1.0))
    execute(pp, gctx, dict(op=17, m=64, n=50, k=k, o=k, beta=0.0), {0: dU, 1: dV, 5: dr})
    assert dr.item() == r
    assert torch.count_nonzero(dU[:, r:]).item() == 0 and torch.count_nonzero(dV[:, r:]).item() == 0
    if r:
        assert rel(dU.cpu().numpy() @ dV.cpu().numpy().T, U @ V.T) < TOL


@pytest.mark.parametrize("k", [4, 17, 32])
def test_directions_are_orthonormal_to_rounding(pp, gctx, k):
    """The directions come from Jacobi rotations of a pair of rows until their cosine is below a few u.
    A rotation errs by at most 3 u in a row; a row takes part in k - 1 of them a sweep, and in the last two
    sweeps nothing corrects them any more: 6 k u, and the product with U as much as k u."""
    rng = np.random.default_rng(k)
    for grade in (0.0, 2.0, 6.0):
        U = np.linalg.qr(rng.standard_normal((90, k)))[0]
        s = 10.0 ** (-grade * np.arange(k) / k)
        V = (np.linalg.qr(rng.standard_normal((80, k)))[0] * s) @ np.linalg.qr(rng.standard_normal((k, k)))[0]
        dU, dV, dr = dev(U), dev(V), dev(np.full((1, 1), -1.0))
        execute(pp, gctx, dict(op=17, m=90, n=80, k=k, o=k, beta=1e-7), {0: dU, 1: dV, 5: dr})
        assert dr.item() == k
        Un, Vn = dU.cpu().numpy(), dV.cpu().numpy()
        assert np.abs(Un.T @ Un - np.eye(k)).max() <= 8 * k * 2.0 ** -53
        assert np.linalg.norm(Un @ Vn.T - U @ V.T, 2) <= 8 * k * 2.0 ** -53
