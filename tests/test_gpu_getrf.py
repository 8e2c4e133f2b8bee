"""The unpivoted block factorization at the edges of its eight-column panels, and with values that leave
the range of its quotients (zero and tiny pivots, infinities, subnormals): the oracle's bits."""
import numpy as np
import pytest

from test_gpu_vm import TaskBench

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


@pytest.mark.parametrize("m,n", [(1, 1), (1, 64), (64, 1), (7, 7), (8, 8), (9, 9), (8, 17), (17, 8), (31, 33), (33, 31),
                                 (40, 64), (64, 40), (57, 63), (64, 64)])
@pytest.mark.parametrize("pad", [0, 3])
def test_panel_edges(pp, oracle, gctx, m, n, pad):
    tb = TaskBench(pp, seed=64 * m + n)
    a = tb.operand(m, n, kind="diag", ld_pad=pad)
    d, h = tb.run(gctx, oracle, dict(op=1, m=m, n=n), {0: a})[a[0]]
    assert np.array_equal(d, h)


@pytest.mark.parametrize("kind", ["zero pivot", "tiny", "huge", "infinite", "zero column"])
@pytest.mark.parametrize("n", [5, 30, 64])
def test_out_of_range(pp, oracle, gctx, kind, n):
    tb = TaskBench(pp, seed=n)
    a = tb.operand(n, n, kind="diag", ld_pad=1)
    x, at = tb.host[a[0]], n // 2
    if kind == "zero pivot":
        x[at, : at + 1] = 0.0
    elif kind == "tiny":
        x[at, : n] *= 1e-300
        x[at + 1 :, at] *= 1e-310
    elif kind == "huge":
        x[:, at] *= 1e290
        x[0, :n] *= 1e-290
    elif kind == "infinite":
        x[n - 1, at] = np.inf
    else:
        x[at:, at] = 0.0
        x[:at, at] = 0.0
    tb.devs[a[0]].copy_(__import__("torch").from_numpy(x))
    d, h = tb.run(gctx, oracle, dict(op=1, m=n, n=n), {0: a})[a[0]]
    assert np.array_equal(d, h, equal_nan=True)
