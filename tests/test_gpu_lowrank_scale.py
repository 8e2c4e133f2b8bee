"""The low-rank instructions on factors of very small and very large norm: they see a factor through its
Gram matrix, whose entries are squares, down to subnormal numbers (multiples of 2^-1074)."""
import numpy as np
import pytest

from test_gpu_lowrank import TOL, execute
from test_gpu_vm import dev, rel

pytestmark = pytest.mark.gpu
U53 = 2.0 ** -53


@pytest.mark.parametrize("e", [-400, -260, 260, 400])
@pytest.mark.parametrize("k", [2, 17, 32])
def test_truncation_does_not_depend_on_the_scale(pp, gctx, k, e):
    """Singular values 4^-i on random bases times 2^e: rank and error as they are for e = 0 (the bound of
    the unscaled case), in LRTRUNC and in the accumulation's adaptive form."""
    rng = np.random.default_rng(k)
    m, n, tol = 150, 120, 3e-5
    s = 4.0 ** -np.arange(k)
    r = int(np.count_nonzero(s > tol))
    U = np.linalg.qr(rng.standard_normal((m, k)))[0]
    V = (np.linalg.qr(rng.standard_normal((n, k)))[0] * s) @ np.linalg.qr(rng.standard_normal((k, k)))[0]
    bound = (np.sqrt(k) * tol if r < k else 0.0) + np.sqrt(k * U53)
    dU, dV, dr = dev(U), dev(V * 2.0 ** e), dev(np.full((1, 1), -1.0))
    execute(pp, gctx, dict(op=17, m=m, n=n, k=k, o=k, beta=tol), {0: dU, 1: dV, 5: dr})
    assert dr.item() == r
    Un, Vn = dU.cpu().numpy(), dV.cpu().numpy() * 2.0 ** -e
    assert np.linalg.norm(Un @ Vn.T - U @ V.T, 2) <= bound
    assert np.abs(Un[:, :r].T @ Un[:, :r] - np.eye(r)).max() < TOL
    # the same matrix as a sum of two: the sketch spans its column space
    c = rng.uniform(0.2, 0.8, k)
    d = [dev(a) for a in (U, V * c * 2.0 ** e, U, V * (1 - c) * 2.0 ** e, rng.uniform(-1, 1, (n, k)))]
    dr = dev(np.full((1, 1), -1.0))
    execute(pp, gctx, dict(op=9, m=m, n=n, k=k, l=k, alpha=1.0, beta=tol, flags=2), {**dict(enumerate(d)), 5: dr}, tmp=m * k)
    assert dr.item() == r
    Un, Vn = d[0].cpu().numpy(), d[1].cpu().numpy() * 2.0 ** -e
    assert np.linalg.norm(Un @ Vn.T - U @ V.T, 2) <= bound
    assert np.abs(Un[:, :r].T @ Un[:, :r] - np.eye(r)).max() < TOL
