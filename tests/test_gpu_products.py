"""The VM's product routine at the edges of its tile shapes (128 x 16, 64 x 32, 128 x 32, 16 x 128,
64 x 64), of its k chunks (64) and passes (8), aligned and odd strides: bitwise equal to the oracle's
ascending chain; free-order products of small outputs (k split over 2, 4 or 8 warps) within the
rounding of two summation orders."""
import numpy as np
import pytest

from test_gpu_vm import TaskBench

pytestmark = pytest.mark.gpu
pytest.importorskip("torch")


def product(pp, oracle, gctx, m, n, k, tA, tB, flags, alpha, beta, pad):
    tb = TaskBench(pp, seed=m * 1000 + n * 10 + k)
    c = tb.operand(m, n, ld_pad=pad)
    a = tb.operand(k, m, ld_pad=pad) if tA else tb.operand(m, k, ld_pad=pad)
    b = tb.operand(n, k, ld_pad=pad) if tB else tb.operand(k, n, ld_pad=pad)
    flags |= (tA << 5) | (tB << 6)
    d, h = tb.run(gctx, oracle, dict(op=6, flags=flags, m=m, n=n, k=k, alpha=alpha, beta=beta), {0: c, 1: a, 2: b})[c[0]]
    size = np.abs(tb.host[a[0]]).max() * np.abs(tb.host[b[0]]).max() * k + np.abs(h).max()
    return d, h, size


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("tA,tB", [(0, 0), (1, 0), (0, 1), (1, 1)])
@pytest.mark.parametrize("m,n,k", [(128, 16, 64), (129, 15, 65), (64, 32, 63), (65, 17, 72), (16, 65, 8), (16, 64, 129),
                                   (64, 64, 7), (65, 65, 64), (17, 33, 1), (260, 1, 200)])
def test_product_bitwise(pp, oracle, gctx, m, n, k, tA, tB, pad):
    d, h, _ = product(pp, oracle, gctx, m, n, k, tA, tB, 0, -1.0, 1.0, pad)
    assert np.array_equal(d, h)


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("tA,tB", [(0, 0), (1, 0), (0, 1)])
@pytest.mark.parametrize("k", [63, 64, 65, 512, 1000])
@pytest.mark.parametrize("m,n", [(16, 16), (17, 16), (16, 17), (32, 32), (1, 24), (33, 8)])
def test_product_free_order(pp, oracle, gctx, m, n, k, tA, tB, pad):
    """Two sums of the same k products differ by at most 2 k u times the sum of their magnitudes."""
    d, h, size = product(pp, oracle, gctx, m, n, k, tA, tB, 1, 1.0, 1.0, pad)
    assert np.abs(d - h).max() <= 2 * k * 2.0 ** -53 * size


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (7, 8, 9), (8, 1, 64), (65, 9, 65), (200, 16, 130), (256, 4, 32), (64, 8, 512),
                                   (40, 3, 1024), (40, 3, 1025)])
def test_rows_times_few_columns(pp, oracle, gctx, m, n, k, pad):
    """Free-order products with at most 16 columns (rows straight from global memory, the columns staged;
    above k = 1024 the general product): within the rounding of two summation orders."""
    for alpha, beta in ((-1.0, 1.0), (1.0, 0.0)):
        d, h, size = product(pp, oracle, gctx, m, n, k, 0, 0, 1, alpha, beta, pad)
        assert np.abs(d - h).max() <= 2 * k * 2.0 ** -53 * size


@pytest.mark.parametrize("pad", [0, 1])
@pytest.mark.parametrize("tA,tB", [(0, 0), (0, 1)])
@pytest.mark.parametrize("m,n,k", [(16, 128, 64), (16, 129, 64), (9, 300, 72), (1, 1000, 200)])
def test_flat_product_bitwise(pp, oracle, gctx, m, n, k, tA, tB, pad):
    """Outputs of at most 16 rows over several tiles: every warp stays inside its own tile."""
    d, h, _ = product(pp, oracle, gctx, m, n, k, tA, tB, 0, 1.0, 1.0, pad)
    assert np.array_equal(d, h)
