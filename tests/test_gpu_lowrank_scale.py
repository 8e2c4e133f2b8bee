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


@pytest.mark.parametrize("e", [-505, -512, -520, -530])
@pytest.mark.parametrize("k", [2, 17, 32])
def test_accum_of_a_subnormal_sketch(pp, gctx, k, e):
    """The sketch scales with the right factors; three passes make its basis orthonormal whatever the
    first Gram matrix has lost, as long as it has digits left (here 2^-20 and less is lost)."""
    rng = np.random.default_rng(k)
    ny, nx = 90, 70
    U1, V1, U2, V2 = (rng.standard_normal(s) for s in ((ny, k), (nx, k), (ny, k), (nx, k)))
    R = rng.uniform(-1, 1, (nx, k))
    d = [dev(a) for a in (U1, V1 * 2.0 ** e, U2, V2 * 2.0 ** e, R)]
    execute(pp, gctx, dict(op=9, m=ny, n=nx, k=k, l=k, alpha=-1.0), dict(enumerate(d)), tmp=ny * k)
    M = U1 @ V1.T - U2 @ V2.T
    Q = np.linalg.qr(M @ R)[0]
    U, V = d[0].cpu().numpy(), d[1].cpu().numpy() * 2.0 ** -e
    assert np.isfinite(U).all() and np.isfinite(V).all()
    assert rel(U @ V.T, Q @ (Q.T @ M)) < TOL
    assert np.abs(U.T @ U - np.eye(k)).max() < TOL


@pytest.mark.parametrize("e", [-505, -512, -520, -530])
@pytest.mark.parametrize("m,k", [(40, 2), (600, 17), (1301, 32)])
def test_orth_of_a_subnormal_gram_matrix(pp, gctx, m, k, e):
    Y = np.random.default_rng(m).standard_normal((m, k))
    d = dev(Y * 2.0 ** e)
    execute(pp, gctx, dict(op=13, m=m, n=k, k=k), {0: d})
    Q = d.cpu().numpy()
    assert np.isfinite(Q).all()
    assert np.abs(Q.T @ Q - np.eye(k)).max() < TOL
    assert rel(Q @ (Q.T @ Y), Y) < TOL


@pytest.mark.parametrize("e", [-505, -512, -520, -525])
@pytest.mark.parametrize("k", [2, 17, 32])
def test_lrtrunc_of_a_subnormal_gram_matrix(pp, gctx, k, e):
    """Half of the singular values in [1/2, 1], the others zero, tolerance 1e-2: the rank is certain.  The
    Gram matrix errs by 2^-1075 at most per product, n products an entry, beside its rounding; what is
    dropped or turned with it has at most the root of k times that."""
    rng = np.random.default_rng(k)
    m, n, tol, r = 80, 60, 1e-2, k // 2
    s = np.r_[np.linspace(1.0, 0.5, r), np.zeros(k - r)]
    U = np.linalg.qr(rng.standard_normal((m, k)))[0]
    V = (np.linalg.qr(rng.standard_normal((n, k)))[0] * s) @ np.linalg.qr(rng.standard_normal((k, k)))[0]
    dU, dV, dr = dev(U), dev(V * 2.0 ** e), dev(np.full((1, 1), -1.0))
    execute(pp, gctx, dict(op=17, m=m, n=n, k=k, o=k, beta=tol), {0: dU, 1: dV, 5: dr})
    Un, Vn = dU.cpu().numpy(), dV.cpu().numpy() * 2.0 ** -e
    assert np.isfinite(Un).all() and np.isfinite(Vn).all()
    assert dr.item() == r
    assert np.linalg.norm(Un @ Vn.T - U @ V.T, 2) <= np.sqrt(k * (U53 + n * 2.0 ** (-1075 - 2 * e)))
    assert np.abs(Un[:, :r].T @ Un[:, :r] - np.eye(r)).max() < TOL
