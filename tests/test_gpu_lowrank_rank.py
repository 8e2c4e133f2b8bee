"""The truncation's rank decision and accuracy where the factor is rank deficient or graded in a basis
that does not show it.  Reference: the factor's singular values in 64 bits."""
import numpy as np
import pytest

from test_gpu_lowrank import execute
from test_gpu_vm import dev

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
U53 = 2.0 ** -53


def spectrum(kind, k):
    h = max(1, k // 4)
    if kind == "deficient":
        return np.r_[np.ones(h), np.zeros(k - h)]
    g = max(1, k // 2)  # decades down to 1e-5, then zeros
    return np.r_[10.0 ** -(5.0 * np.arange(g) / max(1, g - 1)), np.zeros(k - g)]


def problems(kind, k, count, m=72, n=64):
    s = spectrum(kind, k)
    for seed in range(count):
        rng = np.random.default_rng(seed)
        U = np.linalg.qr(rng.standard_normal((m, k)))[0]
        V = (np.linalg.qr(rng.standard_normal((n, k)))[0] * s) @ np.linalg.qr(rng.standard_normal((k, k)))[0]
        yield rng, U, V


def run_all(pp, gctx, tasks):
    gctx.vm_execute(tasks, np.zeros(0, np.int32), np.zeros(len(tasks), np.int32))


def check(kind, k, tol, items):
    """Rank: the singular values are 1e-5 and more, or zero; a computed zero is at most the root of the
    Gram matrix's error, n u of it at most and a few u in earnest, so 1e-6 and 3e-7 lie between.  Error:
    V S^T S differs from V by what the dropped directions hold of V.  The Gram matrix and its factor err by
    (n + k) u, which turns a kept direction of size s by as much / s^2, s s_dropped of which is zero, so
    the error is at most that angle times the s it belongs to: (n + k) u / 1e-5, plus the products' rounding."""
    s = spectrum(kind, k)
    r, n = int(np.count_nonzero(s)), items[0][3].shape[0]
    bound = (n + k) * U53 * (1.0 / s[r - 1] + np.sqrt(k))
    ranks = [int(dr.item()) for dr, *_ in items]
    assert ranks == [r] * len(items), f"{sum(q != r for q in ranks)} of {len(items)} ranks are not {r}"
    for dr, dU, U, V, dV in items:
        err = np.linalg.norm(dU.cpu().numpy() @ dV.cpu().numpy().T - U @ V.T, 2)
        assert err <= bound


@pytest.mark.parametrize("tol", [1e-6, 3e-7])
@pytest.mark.parametrize("kind,k", [("deficient", 32), ("deficient", 17), ("graded", 32), ("graded", 16), ("deficient", 5)])
def test_lrtrunc(pp, gctx, kind, k, tol):
    items = []
    for _, U, V in problems(kind, k, 200):
        items.append((dev(np.full((1, 1), -1.0)), dev(U), U, V, dev(V)))
    t = np.zeros(len(items), dtype=pp.TASK_DTYPE)
    for i, (dr, dU, U, V, dV) in enumerate(items):
        t[i]["op"], t[i]["m"], t[i]["n"], t[i]["k"], t[i]["o"], t[i]["beta"] = 17, U.shape[0], V.shape[0], k, k, tol
        for slot, a in ((0, dU), (1, dV), (5, dr)):
            t[i]["p"][slot], t[i]["ld"][slot] = a.data_ptr(), a.shape[1]
    run_all(pp, gctx, t)
    check(kind, k, tol, items)


@pytest.mark.parametrize("tol", [1e-6, 3e-7])
@pytest.mark.parametrize("kind,k", [("deficient", 32), ("graded", 32), ("graded", 16)])
def test_adaptive_accum(pp, gctx, kind, k, tol):
    """The same matrix as the sum of two halves, from its sketch."""
    items, keep = [], []
    probs = list(problems(kind, k, 100))
    t = np.zeros(len(probs), dtype=pp.TASK_DTYPE)
    for i, (rng, U, V) in enumerate(probs):
        d = [dev(a) for a in (U, 0.5 * V, U, 0.5 * V, rng.uniform(-1, 1, V.shape))]
        dr, scratch = dev(np.full((1, 1), -1.0)), torch.zeros(U.size, dtype=torch.float64, device="cuda")
        t[i]["op"], t[i]["m"], t[i]["n"], t[i]["k"], t[i]["l"] = 9, U.shape[0], V.shape[0], k, k
        t[i]["alpha"], t[i]["beta"], t[i]["flags"], t[i]["tmp"] = 1.0, tol, 2, scratch.data_ptr()
        for slot, a in list(enumerate(d)) + [(5, dr)]:
            t[i]["p"][slot], t[i]["ld"][slot] = a.data_ptr(), a.shape[1]
        items.append((dr, d[0], U, V, d[1]))
        keep.append((d, scratch))
    run_all(pp, gctx, t)
    check(kind, k, tol, items)
