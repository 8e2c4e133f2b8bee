"""The work that programs built on this engine have it do, as cases that can be timed and compared.

Every case goes through the public Python entry points (the C ABI behind them):

  dense    an all-dense block tree: restore, factor, one direct solve
  pivot    the same with partial pivoting inside the GETRF blocks, refined against the dense matrix
  kernel   one kernel-matrix job: restore, factor, FP64 refinement to 1e-10 (weak or standard
           admissibility, FP64 or the mixed BF16 form)
  rebuild  the same, with the matrix built on the device from its points first (a program that
           changes the points or the kernel between solves)
  resolve  further right-hand sides against factors that are already on the device
  batch    many jobs of one shape in merged launches, a fixed number of refinement solves
  gmres    an uneven batch whose factors are too coarse for refinement: GMRES cycles around the
           merged solve
  product  the matrix-free residual r = b - A x alone (FP64)
  serve    requests through the server: H-matrices built, factored and solved at admission

Matrices are seeded: points U[0,1]^dim in Morton order, right-hand sides U[-1,1], the diagonal
shift twice the largest off-diagonal row sum unless a case gives one.
"""
import importlib
import math

import numpy as np
import torch

pp = importlib.import_module("pastel-palettes_b200")

_kept = {}


def _ctx():
    """One device context per process, as a program keeps it."""
    if "ctx" not in _kept:
        torch.cuda.init()
        _kept["ctx"] = pp.Context(device=0)
        _kept["ctx"].set_device_dag(True)
    return _kept["ctx"]


def _server():
    """One server per process (four slots), on a context of its own."""
    if "server" not in _kept:
        torch.cuda.init()
        _kept["server_ctx"] = pp.Context(device=0)
        _kept["server"] = pp.Server(_kept["server_ctx"], hbm_budget_bytes=16 << 30, max_inflight=4)
    return _kept["server_ctx"], _kept["server"]


def listed():
    return [
        # the smallest job a caller has: latency of one factor and one solve launch
        dict(name="dense_256", family="dense", n=256, leaf=64, nrhs=1),
        # the plain FP64 block LU configuration
        dict(name="dense_1024", family="dense", n=1024, leaf=256, nrhs=1),
        # a matrix that is not diagonally dominant, ragged leaves
        dict(name="pivot_1000", family="pivot", n=1000, leaf=128, nrhs=4),
        # one mid-sized weakly admissible job, ragged size, one right-hand side
        dict(name="hodlr_3001", family="kernel", n=3001, dim=2, kernel="laplace", p0=1e-3, leaf=128, rank=16,
             admissibility=0, rank_tol=0.0, nrhs=1, precision="fp64"),
        # the HODLR configuration as a batch of jobs in merged launches
        dict(name="batch_32x8192", family="batch", count=32, n=8192, dim=2, kernel="inv", p0=1e-3, leaf=256, rank=16,
             nrhs=1, solves=4),
        # an uneven batch with coarse factors: the exponential kernel with a small shift
        dict(name="gmres_16", family="gmres", count=16, nmin=1024, nmax=4096, sizes=5, p0=0.1, shift=1e-2, leaf=128,
             rank=24, rank_tol=1e-7, restart=32, cycles=3),
        # standard admissibility in 3-D with 512 leaves: the plain FP64 form
        dict(name="standard_fp64_8192", family="kernel", n=8192, dim=3, kernel="laplace", p0=1e-3, leaf=512, rank=32,
             admissibility=1, rank_tol=1e-8, nrhs=8, precision="fp64"),
        # the same in the mixed BF16 form, the largest job of the list
        dict(name="standard_bf16_32768", family="kernel", n=32768, dim=3, kernel="laplace", p0=1e-3, leaf=512, rank=32,
             admissibility=1, rank_tol=1e-8, nrhs=8, precision="bf16"),
        # a served job's follow-up right-hand sides
        dict(name="resolve_16384", family="resolve", n=16384, dim=3, kernel="exp", p0=0.1, leaf=128, rank=32,
             admissibility=0, rank_tol=1e-7, nrhs=4, precision="fp64"),
        # points or kernel changed: build, factor, solve
        dict(name="rebuild_5000", family="rebuild", n=5000, dim=3, kernel="matern32", p0=0.2, leaf=128, rank=32,
             admissibility=0, rank_tol=1e-7, nrhs=2, precision="fp64"),
        # the refinement's matrix-free product at the size of the largest configuration
        dict(name="product_65536", family="product", n=65536, dim=3, kernel="laplace", p0=1e-3, nrhs=8),
        # six requests of uneven size arriving together
        dict(name="serve_6", family="serve", count=6, nmin=2048, nmax=6144, sizes=3, leaf=128, rank=32, rank_tol=1e-7),
    ]


KERNELS = [("laplace", 1e-3), ("exp", 0.1), ("matern32", 0.2)]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["dense", "pivot", "kernel", "kernel", "mixed", "rebuild", "resolve", "batch", "gmres", "product",
                         "serve"])
    if family == "dense":
        return dict(family="dense", n=_log_int(rng, 200, 2048), leaf=rng.choice([64, 128, 256]),
                    nrhs=rng.choice([1, 2, 5, 8]))
    if family == "pivot":
        return dict(family="pivot", n=_log_int(rng, 200, 1600), leaf=rng.choice([64, 128, 256]),
                    nrhs=rng.choice([1, 3, 4, 8]))
    if family == "kernel":
        if rng.random() < 0.5:  # weak admissibility, any size
            return dict(family="kernel", n=_log_int(rng, 1024, 12000), dim=2, kernel=rng.choice(["inv", "laplace"]),
                        p0=1e-3, leaf=rng.choice([128, 256]), rank=16, admissibility=0, rank_tol=0.0,
                        nrhs=rng.choice([1, 2, 4]), precision="fp64")
        return dict(family="kernel", n=_log_int(rng, 3000, 9000), dim=3, kernel="laplace", p0=1e-3,
                    leaf=rng.choice([256, 512]), rank=32, admissibility=1, rank_tol=1e-8, nrhs=rng.choice([1, 4, 8, 11]),
                    precision="fp64")
    if family == "mixed":  # the sizes whose leaves have exactly 512 rows
        return dict(family="kernel", n=rng.choice([4096, 8192, 16384]), dim=3, kernel=rng.choice(["laplace", "inv"]),
                    p0=1e-3, leaf=512, rank=32, admissibility=1, rank_tol=1e-8, nrhs=rng.randint(1, 8), precision="bf16")
    if family in ("rebuild", "resolve"):
        kernel, p0 = rng.choice(KERNELS)
        hi = 8000 if family == "rebuild" else 16384
        return dict(family=family, n=_log_int(rng, 2048, hi), dim=3, kernel=kernel, p0=p0, leaf=128, rank=32,
                    admissibility=0, rank_tol=1e-7, nrhs=rng.randint(1, 16), precision="fp64")
    if family == "batch":
        return dict(family="batch", count=rng.randint(4, 32), n=_log_int(rng, 1024, 8192), dim=2, kernel="inv", p0=1e-3,
                    leaf=rng.choice([128, 256]), rank=rng.choice([8, 16]), nrhs=rng.choice([1, 1, 2]), solves=4)
    if family == "gmres":
        return dict(family="gmres", count=rng.randint(4, 16), nmin=1024, nmax=_log_int(rng, 2000, 4096),
                    sizes=rng.randint(0, 999), p0=0.1, shift=1e-2, leaf=128, rank=24, rank_tol=1e-7, restart=32, cycles=3)
    if family == "product":
        kernel, p0 = rng.choice(KERNELS)
        return dict(family="product", n=_log_int(rng, 4096, 65536), dim=rng.choice([2, 3]), kernel=kernel, p0=p0,
                    nrhs=rng.choice([1, 3, 4, 8]))
    return dict(family="serve", count=rng.randint(2, 6), nmin=2048, nmax=6144, sizes=rng.randint(0, 999), leaf=128,
                rank=32, rank_tol=1e-7)


# ----------------------------------------------------------------------------- inputs
def _device_rhs(n, nrhs, seed):
    return torch.from_numpy(pp.rhs(n, nrhs, seed=seed)).cuda()


def _kernel_problem(ctx, c, seed, construct):
    return pp.make_kernel_problem(ctx, c["n"], c["dim"], c["kernel"], c["p0"], c["leaf"], c["rank"],
                                  c.get("admissibility", 0), 1.0, shift=c.get("shift"), seed=seed,
                                  rank_tol=c.get("rank_tol") or None, construct=construct)


def _uneven(c):
    """The sizes of an uneven batch: log-uniform, any integer."""
    r = np.random.default_rng(c["sizes"])
    return [int(round(math.exp(r.uniform(math.log(c["nmin"]), math.log(c["nmax"]))))) for _ in range(c["count"])]


def _requests(c, seed):
    """Per request of a serving case: (n, kernel, p0, right-hand-side sets)."""
    r = np.random.default_rng(c["sizes"] + 1)
    for i, n in enumerate(_uneven(c)):
        kernel, p0 = KERNELS[int(r.integers(0, 3))]
        nrhs, sets = int(r.integers(1, 17)), 1 + int(r.integers(0, 3))
        yield n, kernel, p0, np.random.default_rng(seed + 977 * i).uniform(-1.0, 1.0, (sets, n, nrhs))


class _DeviceBlocks:
    """The blocks of an H-matrix on the device as an array-interface object; holds the matrix, which
    owns the memory, for as long as a tensor made from it lives."""

    def __init__(self, h):
        self.h = h
        self.__cuda_array_interface__ = {"shape": (h.arena_bytes() // 8,), "typestr": "<f8", "version": 3,
                                         "data": (int(h.device_arena_ptr()), False)}


def prepare(case, seed):
    c, family = case, case["family"]
    if family == "serve":
        ctx, server = _server()
        jobs = []
        for i, (n, kernel, p0, rhs) in enumerate(_requests(c, seed)):
            _, prob = pp.make_kernel_problem(ctx, n, 3, kernel, p0, c["leaf"], c["rank"], seed=seed + 31 * i,
                                             construct="none")
            prob.points_dev = None
            jobs.append((prob, rhs))
        return dict(case=c, ctx=ctx, server=server, jobs=jobs)
    ctx = _ctx()
    if family in ("dense", "pivot"):
        h, a = pp.make_dense_problem(ctx, c["n"], c["leaf"], seed=seed, shift=0.0 if family == "pivot" else None)
        if family == "pivot":
            h.set_pivoting()
        h.upload()
        h.keep_original()
        b = _device_rhs(c["n"], c["nrhs"], seed + 1)
        state = dict(case=c, h=h, b=b)
        if family == "pivot":
            state["refiner"] = pp.Refiner(h, ctx, dense=a)
        else:
            state["x"] = torch.empty_like(b)
            state["lu"] = torch.as_tensor(_DeviceBlocks(h), device="cuda")
        return state
    if family == "product":
        rng = np.random.default_rng(seed)
        pts = torch.from_numpy(rng.uniform(0.0, 1.0, (c["n"], c["dim"]))).cuda()
        x, b = _device_rhs(c["n"], c["nrhs"], seed + 1), _device_rhs(c["n"], c["nrhs"], seed + 2)
        return dict(case=c, ctx=ctx, pts=pts, x=x, b=b, r=torch.empty_like(b), kernel=pp.KERNELS[c["kernel"]])
    if family in ("batch", "gmres"):
        hs, probs, bs = [], [], []
        for i, n in enumerate(_uneven(c) if family == "gmres" else [c["n"]] * c["count"]):
            d = dict(c, n=n, dim=2, kernel="exp") if family == "gmres" else c
            h, prob = _kernel_problem(ctx, d, seed + 31 * i, "device")
            if family == "batch":
                h.set_gemm_tile(128)
            h.keep_original()
            hs.append(h)
            probs.append(prob)
            bs.append(_device_rhs(n, c.get("nrhs", 1), seed + 7 * i + 1))
        batch = pp.Batch(ctx, hs)
        if family == "batch":
            return dict(case=c, batch=batch, bs=bs, refiner=pp.BatchRefiner(batch, probs))
        return dict(case=c, batch=batch, bs=bs, gmres=pp.BatchGMRES(batch, probs, m=c["restart"]))
    # kernel / rebuild / resolve
    h, prob = _kernel_problem(ctx, c, seed, "device")
    if c["precision"] == "bf16":
        h.set_precision(pp.BF16)
    h.set_gemm_tile(128)
    b = _device_rhs(c["n"], c["nrhs"], seed + 1)
    state = dict(case=c, h=h, prob=prob, b=b, refiner=pp.Refiner(h, ctx, prob))
    if family == "kernel":
        h.keep_original()
    elif family == "resolve":
        h.factor()
    return state


# ----------------------------------------------------------------------------- one pass
def run(state):
    c, family = state["case"], state["case"]["family"]
    if family == "dense":
        h = state["h"]
        h.restore()
        h.factor()
        h.solve(state["b"], state["x"])
        return {"lu": state["lu"], "x": state["x"]}
    if family == "product":
        state["ctx"].kernel_residual_batch([(state["kernel"], c["p0"], 1.0, state["pts"], state["x"], None, state["b"],
                                             state["r"])])
        return {"r": state["r"]}
    if family == "batch":
        state["batch"].restore()
        state["batch"].factor()
        xs, _ = state["refiner"].run(state["bs"], c["solves"])
        return {"x": xs}
    if family == "gmres":
        state["batch"].restore()
        state["batch"].factor()
        xs, _ = state["gmres"].run(state["bs"], c["cycles"])
        return {"x": xs}
    if family == "serve":
        server, ids = state["server"], []
        for prob, rhs in state["jobs"]:
            h = pp.Hierarchical.geometric(state["ctx"], prob.points, c["leaf"], kmax=c["rank"])
            h.set_rank_tolerance(c["rank_tol"])
            ids.append(server.submit(h, prob, rhs, tol=1e-10))
        server.wait_all()
        return {"x": [server.result(i) for i in ids]}
    h = state["h"]
    if family == "rebuild":
        h.construct(state["prob"], state["prob"].points_dev)
    elif family != "resolve":
        h.restore()
    if family != "resolve":
        h.factor()
    x, _ = state["refiner"].solve(state["b"], tol=1e-10)
    return {"x": x}


# ----------------------------------------------------------------------------- what a pass cannot do without
def _hodlr_work(n, leaf, rank, nrhs, factor=True, solves=1):
    """Bytes and FP64 operations of a weakly admissible job: leaves and factors read and written
    once by the factorization and read once by each solve; every residual evaluates half the
    matrix (about 20 operations an entry and 4 for each right-hand side)."""
    levels = max(1, math.ceil(math.log2(n / leaf)))
    m = n / 2 ** levels
    entries = n * m + 2.0 * n * rank * levels
    flops = solves * (4.0 * entries * nrhs + 0.5 * n * n * (20 + 4 * nrhs))
    if factor:
        flops += 2 / 3 * n * m * m + n * levels * (2 * m * rank + levels * 4 * rank * rank + 20 * rank * rank)
    return 8.0 * entries * ((2 if factor else 0) + solves) + 8.0 * n * (3 * nrhs + 3) * solves, flops


def work(case):
    c, family = case, case["family"]
    n, nrhs = c.get("n", 0), c.get("nrhs", 1)
    if family in ("dense", "pivot"):
        return {"bytes": 8.0 * (2.0 * n * n + 2.0 * n * nrhs), "flops": 2 / 3 * n ** 3 + 2.0 * n * n * nrhs}
    if family == "product":
        return {"bytes": 8.0 * n * (c["dim"] + 3 * nrhs), "flops": 0.5 * n * n * (20 + 4 * nrhs)}
    if family in ("batch", "gmres", "serve"):
        sizes = [n] * c["count"] if family == "batch" else _uneven(c)
        solves = c["solves"] if family == "batch" else c["cycles"] * c["restart"] if family == "gmres" else 2
        parts = [_hodlr_work(k, c["leaf"], c["rank"], nrhs if family != "serve" else 8, True, solves) for k in sizes]
        return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}
    if c["admissibility"] == 1:  # mostly dense at these sizes
        return {"bytes": 8.0 * n * n * 3, "flops": 2 / 3 * n ** 3 + 0.5 * n * n * (20 + 4 * nrhs) + 2.0 * n * n * nrhs}
    b, f = _hodlr_work(n, c["leaf"], c["rank"], nrhs, family != "resolve", 2)
    return {"bytes": b, "flops": f + (8.0 * n * n * c["rank"] if family == "rebuild" else 0.0)}


# ----------------------------------------------------------------------------- 64-bit answers
def _entry(kind, d, p0):
    if kind == "inv":
        return 1.0 / (d + p0)
    if kind == "laplace":
        return 1.0 / (4.0 * math.pi * (d + p0))
    if kind == "exp":
        return torch.exp(-d / p0)
    s = math.sqrt(3.0) * d / p0
    return (1.0 + s) * torch.exp(-s)


def _slab(kind, p0, x, y):
    d2 = torch.zeros(x.shape[0], y.shape[0], dtype=torch.float64, device=x.device)
    for k in range(x.shape[1]):
        d2 += (x[:, k, None] - y[None, :, k]) ** 2
    return _entry(kind, d2.sqrt_(), p0)


def _morton(pts):
    n, dim = pts.shape
    q = np.clip((pts * (1 << 21)).astype(np.uint64), 0, (1 << 21) - 1)
    key = np.zeros(n, dtype=np.uint64)
    for b in range(21):
        for d in range(dim):
            key |= ((q[:, d] >> np.uint64(b)) & np.uint64(1)) << np.uint64(b * dim + d)
    return pts[np.argsort(key, kind="stable")]


def _kernel_solution(n, dim, kernel, p0, shift, seed, b):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    pts = torch.from_numpy(_morton(np.random.default_rng(seed).uniform(0.0, 1.0, (n, dim)))).to(dev)
    a = torch.empty(n, n, dtype=torch.float64, device=dev)
    for r in range(0, n, 4096):
        a[r:r + 4096] = _slab(kernel, p0, pts[r:r + 4096], pts)
    if shift is None:
        shift = 2.0 * float((a.sum(1) - a.diagonal()).max())
    a.diagonal().add_(shift)
    # symmetric positive definite after the shift
    return torch.cholesky_solve(torch.from_numpy(b).to(dev), torch.linalg.cholesky(a)).cpu().numpy()


def _dense_layout(lu, leaf):
    """The factored matrix in the storage order of the all-dense tree: quadrants in row-major order
    down to the leaf, each block row-major from a multiple of four elements."""
    parts, at = [], 0

    def emit(r, m, col, k):
        nonlocal at
        if m <= leaf and k <= leaf:
            pad = -at % 4
            parts.append(np.zeros(pad))
            parts.append(lu[r:r + m, col:col + k].reshape(-1))
            at += pad + m * k
            return
        for i, mi in ((0, m // 2), (m // 2, m - m // 2)):
            for j, kj in ((0, k // 2), (k // 2, k - k // 2)):
                emit(r + i, mi, col + j, kj)

    emit(0, lu.shape[0], 0, lu.shape[1])
    return np.concatenate(parts)


def exact(case, seed):
    c, family = case, case["family"]
    n = c.get("n", 0)
    if family in ("dense", "pivot"):
        a = np.random.default_rng(seed).uniform(-1.0, 1.0, (n, n)) + (0.0 if family == "pivot" else n) * np.eye(n)
        x = np.linalg.solve(a, np.random.default_rng(seed + 1).uniform(-1.0, 1.0, (n, c["nrhs"])))
        if family == "pivot":
            return {"x": x}
        lu = a.copy()
        for i in range(n - 1):
            lu[i + 1:, i] /= lu[i, i]
            lu[i + 1:, i + 1:] -= np.outer(lu[i + 1:, i], lu[i, i + 1:])
        return {"lu": _dense_layout(lu, c["leaf"]), "x": x}
    if family == "product":
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        pts = torch.from_numpy(np.random.default_rng(seed).uniform(0.0, 1.0, (n, c["dim"]))).to(dev)
        x, b = (torch.from_numpy(np.random.default_rng(seed + k).uniform(-1.0, 1.0, (n, c["nrhs"]))).to(dev) for k in (1, 2))
        r = b - x  # the shift of 1
        for i in range(0, n, 4096):
            r[i:i + 4096] -= _slab(c["kernel"], c["p0"], pts[i:i + 4096], pts) @ x
        return {"r": r}
    if family == "serve":
        return {"x": [np.stack([_kernel_solution(k, 3, kernel, p0, None, seed + 31 * i, b) for b in rhs])
                      for i, (k, kernel, p0, rhs) in enumerate(_requests(c, seed))]}
    if family in ("batch", "gmres"):
        sizes = _uneven(c) if family == "gmres" else [n] * c["count"]
        dim, kernel = (2, "exp") if family == "gmres" else (c["dim"], c["kernel"])
        return {"x": [_kernel_solution(k, dim, kernel, c["p0"], c.get("shift"), seed + 31 * i,
                                       np.random.default_rng(seed + 7 * i + 1).uniform(-1.0, 1.0, (k, c.get("nrhs", 1))))
                      for i, k in enumerate(sizes)]}
    b = np.random.default_rng(seed + 1).uniform(-1.0, 1.0, (n, c["nrhs"]))
    return {"x": _kernel_solution(n, c["dim"], c["kernel"], c["p0"], None, seed, b)}
