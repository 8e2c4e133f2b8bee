"""Triangular solves and pivoted GETRF at the edges of their blocks (8 positions, 8 lines per warp,
64 lines per pass), bitwise equal to the oracle's divisions — also where the quotients' exponents
leave the range of the multiplicative form and the routines divide instead."""
import numpy as np
import pytest

from test_gpu_vm import TaskBench, dev

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")

SCALES = {"plain": (1.0, 1.0), "tiny rows": (2.0 ** -700, 1.0), "huge triangle": (1.0, 2.0 ** 500),
          "tiny triangle": (2.0 ** -300, 2.0 ** -500), "zeros": (0.0, 1.0)}


def scaled(tb, idx, factor):
    tb.host[idx] *= factor
    tb.devs[idx] = dev(tb.host[idx])


@pytest.mark.parametrize("scale", sorted(SCALES))
@pytest.mark.parametrize("op", [2, 3, 4, 5])
@pytest.mark.parametrize("size,lines", [(1, 1), (7, 9), (8, 8), (9, 64), (63, 65), (64, 130)])
def test_triangular_bitwise(pp, oracle, gctx, op, size, lines, scale):
    fb, ft = SCALES[scale]
    tb = TaskBench(pp, seed=100 * op + size)
    m, n = (lines, size) if op == 3 else (size, lines)
    b, t = tb.operand(m, n), tb.operand(size, size, kind="diag")
    scaled(tb, b[0], fb)
    scaled(tb, t[0], ft)
    d, h = tb.run(gctx, oracle, dict(op=op, m=m, n=n), {0: b, 1: t})[b[0]]
    assert np.array_equal(d, h, equal_nan=True)


@pytest.mark.parametrize("scale", ["plain", "tiny rows", "zeros"])
@pytest.mark.parametrize("m,n", [(1, 1), (8, 8), (9, 9), (33, 33), (64, 64), (40, 64), (64, 24)])
def test_pivoted_getrf_bitwise(pp, oracle, gctx, m, n, scale):
    tb = TaskBench(pp, seed=m + 3 * n)
    a, p = tb.operand(m, n), tb.operand(m, 1, ld_pad=0)
    if scale == "tiny rows":  # quotients of every magnitude below 1
        tb.host[a[0]] *= 2.0 ** -(20.0 * np.arange(m))[:, None]
    elif scale == "zeros" and m > 2:  # an exactly zero column below an exactly zero pivot candidate
        tb.host[a[0]][1:, 0] = 0.0
    tb.devs[a[0]] = dev(tb.host[a[0]])
    out = tb.run(gctx, oracle, dict(op=1, flags=4, m=m, n=n), {0: a, 1: p})
    for d, h in (out[a[0]], out[p[0]]):
        assert np.array_equal(d, h, equal_nan=True)
