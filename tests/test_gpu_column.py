"""Products with one right-hand side (a matrix, a leaf's inverse triangle, whole or in part, in place or
not, the column stored as a column or as a row): every width of the lanes' split and its edges, aligned
pairs and odd strides.  Tolerance: two sums of k products differ by at most 2 k u sum_j |m_ij s_j|."""
import numpy as np
import pytest
import torch

from test_gpu_vm import dev

pytestmark = pytest.mark.gpu
TRMV, GEMM = 12, 6


def launch(pp, ctx, **f):
    t = np.zeros(1, dtype=pp.TASK_DTYPE)
    for k, v in f.items():
        if k in ("p", "ld"):
            for i, x in enumerate(v):
                t[0][k][i] = x.data_ptr() if k == "p" else x
        else:
            t[0][k] = v
    ctx.vm_execute(t, np.zeros(0, np.int32), np.zeros(1, np.int32))


@pytest.mark.parametrize("m", [1, 3, 4, 15, 16, 17, 32, 33, 64, 65, 94, 111, 128, 129, 256, 300, 1000])
@pytest.mark.parametrize("rows", [1, 8, 63, 257])
@pytest.mark.parametrize("pad,tB,alpha,beta", [(0, 0, -1.0, 1.0), (1, 1, 1.0, 0.0), (2, 1, -1.0, 1.0)])
def test_product(pp, gctx, m, rows, pad, tB, alpha, beta):
    rng = np.random.default_rng(m + rows)
    A, x, y = rng.standard_normal((rows, m + pad)), rng.standard_normal((m, 3)), rng.standard_normal((rows, 2))
    s = np.ascontiguousarray(x[:, :1].T) if tB else x
    out = dev(y)
    launch(pp, gctx, op=GEMM, flags=1 | (tB << 6), m=rows, n=1, k=m, alpha=alpha, beta=beta, p=[out, dev(A), dev(s)],
           ld=[2, m + pad, s.shape[1]])
    want = beta * y[:, 0] + alpha * (A[:, :m] @ x[:, 0])
    bound = 2 * (m + 2) * 2.0**-53 * (np.abs(A[:, :m]) @ np.abs(x[:, 0]) + np.abs(y[:, 0]))
    got = out.cpu().numpy()
    assert (np.abs(got[:, 0] - want) <= bound).all() and np.array_equal(got[:, 1], y[:, 1])


@pytest.mark.parametrize("m", [1, 8, 16, 31, 64, 94, 111, 128, 129, 200, 256])
@pytest.mark.parametrize("upper", [0, 1])
@pytest.mark.parametrize("part", [None, (0, 5), (3, 64), (-7, 7)])
def test_triangle(pp, gctx, m, upper, part):
    rng = np.random.default_rng(m)
    pad = m % 3
    A, x = rng.standard_normal((m, m + pad)), rng.standard_normal((m, 1))
    T = np.triu(A[:, :m]) if upper else np.tril(A[:, :m])
    A[:, :m][(np.tril(np.ones((m, m)), -1) if upper else np.triu(np.ones((m, m)), 1)) > 0] = np.nan  # not to be read as a value
    want, bound = T @ x[:, 0], 2 * (m + 2) * 2.0**-53 * (np.abs(T) @ np.abs(x[:, 0]))
    if part is None:
        out = dev(x)
        launch(pp, gctx, op=TRMV, m=m, n=1, ctrl=upper, p=[out, dev(A)], ld=[1, m + pad])
        assert (np.abs(out.cpu().numpy()[:, 0] - want) <= bound).all()
        return
    o = part[0] % m
    n = min(part[1], m - o)
    out = dev(np.full((n, 1), 7.0))
    launch(pp, gctx, op=TRMV, m=m, n=1, o=o, l=n, ctrl=upper, p=[out, dev(A), dev(x)], ld=[1, m + pad, 1])
    assert (np.abs(out.cpu().numpy()[:, 0] - want[o : o + n]) <= bound[o : o + n]).all()


@pytest.mark.parametrize("n", [1, 2, 9])
@pytest.mark.parametrize("tri", [0, 1, 2])
@pytest.mark.parametrize("m", [5, 30, 94, 200])
def test_infinite_entry_stays_in_its_rows(pp, gctx, m, n, tri):
    """An infinity in the right-hand side reaches the rows whose coefficients meet it, and no other."""
    rng = np.random.default_rng(m)
    A, x = rng.uniform(1, 2, (m, m)), rng.uniform(1, 2, (m, n))
    T = [np.tril, np.triu, np.array][tri](A)
    x[m // 2, 0] = np.inf
    out = dev(np.zeros((m, n)))
    if tri == 2:
        launch(pp, gctx, op=GEMM, flags=1, m=m, n=n, k=m, alpha=1.0, beta=0.0, p=[out, dev(A), dev(x)], ld=[n, m, n])
    else:
        launch(pp, gctx, op=TRMV, m=m, n=n, o=0, l=m, ctrl=tri, p=[out, dev(A), dev(x)], ld=[n, m, n])
    got, meets = out.cpu().numpy(), T[:, m // 2] != 0
    assert np.isposinf(got[meets, 0]).all() and np.isfinite(got[~meets, 0]).all() and np.isfinite(got[:, 1:]).all()
