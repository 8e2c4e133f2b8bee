"""The quotients of the triangular instructions against the processor's division, bit for bit: TRSMR with a
diagonal matrix divides every column by its own number (the updates between columns subtract zeros), GETRF
of one column divides it by its first entry.  Exponents on both sides of the range in which the
instructions use their own quotients (biased 600 to 1445), special mantissas, signed zeros, subnormals."""
import numpy as np
import pytest

from test_gpu_vm import dev

pytestmark = pytest.mark.gpu

ONES = (1 << 52) - 1
IN, OUT = [600, 601, 1022, 1023, 1024, 1444, 1445], [0, 1, 599, 1446, 1447, 2046]


def doubles(rng, shape, exponents, mantissas=None):
    e = rng.choice(exponents, shape).astype(np.uint64) if exponents is not None else rng.integers(600, 1446, shape).astype(np.uint64)
    m = rng.integers(0, 1 << 52, shape).astype(np.uint64)
    if mantissas is not None:
        pick = rng.integers(0, len(mantissas) + 1, shape)
        for i, v in enumerate(mantissas):
            m[pick == i] = v
    s = rng.integers(0, 2, shape).astype(np.uint64)
    return ((s << np.uint64(63)) | (e << np.uint64(52)) | m).view(np.float64)


def trsmr(pp, gctx, sets):
    """sets: (B, t): B[:, j] / t[j] for every j, all of them in one launch."""
    t = np.zeros(len(sets), dtype=pp.TASK_DTYPE)
    keep = []
    for i, (B, d) in enumerate(sets):
        keep.append((dev(B), dev(np.diag(d))))
        t[i]["op"], t[i]["m"], t[i]["n"] = pp.OP_NAMES.index("trsmr"), B.shape[0], B.shape[1]
        for slot, a in enumerate(keep[-1]):
            t[i]["p"][slot], t[i]["ld"][slot] = a.data_ptr(), a.shape[1]
    gctx.vm_execute(t, np.zeros(0, np.int32), np.zeros(len(sets), np.int32))
    return [a.cpu().numpy() for a, _ in keep]


def same(got, B, d):
    with np.errstate(all="ignore"):
        want = B / d
    bad = np.argwhere(got.view(np.uint64) != want.view(np.uint64))
    assert bad.size == 0, f"{len(bad)} quotients differ, first {B[tuple(bad[0])]!r} / {d[bad[0][1]]!r}"


def test_millions_of_pairs(pp, gctx):
    rng = np.random.default_rng(1)
    sets = [(doubles(rng, (4096, 64), None), doubles(rng, 64, None, [0, 1, 2, ONES - 1])) for _ in range(24)]
    for (B, d), got in zip(sets, trsmr(pp, gctx, sets)):
        same(got, B, d)


def test_special_mantissas_and_limits(pp, gctx):
    rng = np.random.default_rng(2)
    m = [0, 1, 2, ONES - 2, ONES - 1, ONES, 1 << 51, (1 << 51) - 1]
    sets = [(doubles(rng, (1024, 64), IN, m), doubles(rng, 64, IN, [v for v in m if v != ONES])) for _ in range(24)]
    sets += [(doubles(rng, (64, 64), IN, m), doubles(rng, 64, IN, m)) for _ in range(24)]  # the divisor of all ones too
    for (B, d), got in zip(sets, trsmr(pp, gctx, sets)):
        same(got, B, d)


@pytest.mark.parametrize("xe,te", [(OUT, IN), (IN, OUT), (IN + OUT, IN + OUT)])
def test_beyond_the_limits(pp, gctx, xe, te):
    """One column per instruction: a quotient that overflows would meet the zeros beside it."""
    rng = np.random.default_rng(3)
    m = [0, 1, ONES - 1, ONES]
    sets = [(doubles(rng, (40, 1), xe, m), doubles(rng, 1, te, m)) for _ in range(500)]
    sets = [(B, d) for B, d in sets if d[0] != 0.0]
    for i, (B, _) in enumerate(sets):
        B[i % 40], B[(i + 7) % 40] = 0.0, -0.0
    for (B, d), got in zip(sets, trsmr(pp, gctx, sets)):
        same(got, B, d)


@pytest.mark.parametrize("exponents", [None, IN, OUT])
def test_getrf_column(pp, gctx, exponents):
    rng = np.random.default_rng(4)
    cols = [doubles(rng, (64, 1), exponents, [0, 1, ONES - 1, ONES]) for _ in range(2000)]
    for i, c in enumerate(cols):
        c[1 + i % 63] = 0.0 if i % 2 else -0.0
        if c[0] == 0.0:
            c[0] = 1.5
    t = np.zeros(len(cols), dtype=pp.TASK_DTYPE)
    ds = [dev(c) for c in cols]
    for i, a in enumerate(ds):
        t[i]["op"], t[i]["m"], t[i]["n"] = pp.OP_NAMES.index("getrf"), 64, 1
        t[i]["p"][0], t[i]["ld"][0] = a.data_ptr(), 1
    gctx.vm_execute(t, np.zeros(0, np.int32), np.zeros(len(cols), np.int32))
    for c, a in zip(cols, ds):
        got = a.cpu().numpy()
        assert got[0] == c[0]
        same(got[1:], c[1:], c[0])
