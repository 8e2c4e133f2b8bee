"""The low-rank instructions at the edges of their rank blocks (16, 32), odd ranks, ragged and tall
row counts, transposed added terms, sketches in shared memory and in scratch."""
import numpy as np
import pytest

from test_gpu_vm import TaskBench, dev, rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

TOL = 1e-12  # relative Frobenius: the tolerance of the accumulation tests


def bench(pp, arrays, seed=0):
    tb = TaskBench(pp, seed=seed)
    for a in arrays:
        tb.host.append(np.ascontiguousarray(a))
        tb.devs.append(dev(tb.host[-1]))
    return tb


def execute(pp, gctx, fields, operands, tmp=0):
    t = np.zeros(1, dtype=pp.TASK_DTYPE)
    for k, v in fields.items():
        t[0][k] = v
    for s, a in operands.items():
        t[0]["p"][s], t[0]["ld"][s] = a.data_ptr(), a.shape[1]
    scratch = torch.zeros(max(tmp, 1), dtype=torch.float64, device="cuda")
    t[0]["tmp"] = scratch.data_ptr()
    gctx.vm_execute(t, np.zeros(0, np.int32), np.zeros(1, np.int32))


@pytest.mark.parametrize("trans", [0, 1])
@pytest.mark.parametrize("ny,nx,k1,k2", [(5, 7, 1, 1), (33, 40, 7, 16), (94, 93, 16, 15), (100, 64, 17, 8), (129, 130, 31, 32),
                                         (520, 300, 32, 32), (700, 90, 32, 5), (1300, 257, 16, 16)])
def test_accum_projects_onto_its_sketch(pp, gctx, ny, nx, k1, k2, trans):
    rng = np.random.default_rng(ny + k1)
    U1, V1, U2, V2 = (rng.standard_normal(s) for s in ((ny, k1), (nx, k1), (ny, k2), (nx, k2)))
    R = rng.uniform(-1, 1, (nx, k1))
    d = [dev(a) for a in (U1, V1, U2.T if trans else U2, V2.T if trans else V2, R)]
    execute(pp, gctx, dict(op=9, m=ny, n=nx, k=k1, l=k2, alpha=-1.0, flags=(0xC0 if trans else 0)), dict(enumerate(d)),
            tmp=ny * k1)
    M = U1 @ V1.T - U2 @ V2.T
    Q = np.linalg.qr(M @ R)[0]
    U, V = d[0].cpu().numpy(), d[1].cpu().numpy()
    assert rel(U @ V.T, Q @ (Q.T @ M)) < TOL
    assert np.abs(U.T @ U - np.eye(k1)).max() < TOL


@pytest.mark.parametrize("k", [1, 2, 15, 16, 17, 31, 32])
def test_lrtrunc_rank_and_error(pp, gctx, k):
    """Singular values 4^-i on random bases: the rank is the count above the tolerance, the error at
    most the dropped part (sqrt(k) times the first dropped value) plus the Gram matrix's rounding
    (sqrt(k u) of the largest)."""
    rng = np.random.default_rng(k)
    m, n, tol = 150, 203, 3e-5
    s = 4.0 ** -np.arange(k)
    U = np.linalg.qr(rng.standard_normal((m, k)))[0]
    V = (np.linalg.qr(rng.standard_normal((n, k)))[0] * s) @ np.linalg.qr(rng.standard_normal((k, k)))[0]
    dU, dV, dr = dev(U), dev(V), dev(np.full((1, 1), -1.0))
    execute(pp, gctx, dict(op=17, m=m, n=n, k=k, o=k, beta=tol), {0: dU, 1: dV, 5: dr})
    r = int(np.count_nonzero(s > tol))
    assert dr.item() == r
    Un, Vn = dU.cpu().numpy(), dV.cpu().numpy()
    assert np.all(Un[:, r:] == 0) and np.all(Vn[:, r:] == 0)
    assert np.linalg.norm(Un @ Vn.T - U @ V.T, 2) <= (np.sqrt(k) * tol if r < k else 0.0) + np.sqrt(k * 2.0 ** -53)
    assert np.abs(Un[:, :r].T @ Un[:, :r] - np.eye(r)).max() < TOL


def test_lrtrunc_limit_zero_matrix_and_nothing_to_do(pp, gctx):
    rng = np.random.default_rng(0)
    U, V = np.linalg.qr(rng.standard_normal((64, 8)))[0], rng.standard_normal((50, 8))
    dU, dV, dr = dev(U), dev(V), dev(np.full((1, 1), -1.0))
    execute(pp, gctx, dict(op=17, m=64, n=50, k=8, o=3, beta=0.0), {0: dU, 1: dV, 5: dr})
    assert dr.item() == 3
    w, sv, z = np.linalg.svd(U @ V.T)
    assert rel(dU.cpu().numpy() @ dV.cpu().numpy().T, (w[:, :3] * sv[:3]) @ z[:3]) < 1e-7  # sqrt of the Gram matrix's rounding
    dV.zero_()
    execute(pp, gctx, dict(op=17, m=64, n=50, k=8, o=8, beta=1e-7), {0: dU, 1: dV, 5: dr})
    assert dr.item() == 0 and torch.count_nonzero(dU).item() == 0
    dU, dV = dev(U), dev(V)
    execute(pp, gctx, dict(op=17, m=64, n=50, k=8, o=8, beta=0.0), {0: dU, 1: dV, 5: dr})
    assert dr.item() == 8
    assert rel(dU.cpu().numpy() @ dV.cpu().numpy().T, U @ V.T) < TOL


@pytest.mark.parametrize("m,k", [(1, 1), (40, 17), (600, 32), (1301, 16), (2000, 31)])
def test_orth_spans_its_columns(pp, gctx, m, k):
    rng = np.random.default_rng(m)
    Y = rng.standard_normal((m, k)) * 10.0 ** -(4.0 * np.arange(k) / k)
    d = dev(Y)
    execute(pp, gctx, dict(op=13, m=m, n=k, k=k), {0: d})
    Q = d.cpu().numpy()
    assert np.abs(Q.T @ Q - np.eye(k)).max() < TOL
    assert rel(Q @ (Q.T @ Y), Y) < TOL
