"""Performance cases of the KKT solve path, through the public Python API.

Six kinds of work, each a thing that an interior-point program does with this
library; K = [[H + delta I, A'], [A, -gamma I]] throughout, from the seeded
generator (A: `per_col` N(0,1) entries per column, half of them in a band of
half-width `band` when it is positive; H log-uniform in [hmin, hmax]):

  spmv     y = K x                                        CsrOperator.spmv
  dual     r = c - A' y (the dual residual)               CsrOperator.spmv, transposed
  factor   K from (A, x, s), its factor, one M^-1 b       KktAssembly, Factor
  apply    the three preconditioner stages one by one     Factor.apply
  solve    SQMR with 1 or several right-hand sides        sqmr_solve, sqmr_solve_multi
  batch    many uneven systems, factored and solved       batch_factor_solve_graph

The SQMR cases run a fixed number of iterations (an inexact inner solve: the
tolerance is never met within them), few enough that the iterates do not yet
depend on the order of the sums.
"""
import math

import numpy as np
import torch

import culip_b200 as cb

LISTED = [
    # the smallest product: the benchmark's small system, where a call's latency is all there is
    dict(name="spmv small f64", kind="spmv", n=2000, m=1000, per_col=4, band=0, precision="f64", sell=False),
    # the product of the mixed-precision workload's matrix on the SELL copy, as the benchmark's spmv line: bandwidth
    dict(name="spmv mixed f64 sell", kind="spmv", n=1000000, m=500000, per_col=6, band=32, precision="f64", sell=True),
    # the dual residual at the size of the scale workload, odd sizes, single precision, alpha and beta in use
    dict(name="dual residual f32", kind="dual", n=200003, m=99991, per_col=6, band=32, precision="f32"),
    # one interior-point iteration's matrix work on a small system: launches and gaps between them
    dict(name="factor small f64", kind="factor", n=2000, m=1000, per_col=4, band=0, hmin=1e-2, hmax=1e2, block=4,
         reg=1e-8, precision="f64", pivot="bk", graph=False),
    # the same at the size of the scale workload, replayed from the factor's graph
    dict(name="factor scale f64", kind="factor", n=200000, m=100000, per_col=6, band=32, hmin=1e-6, hmax=1e6,
         block=32, reg=1e-8, precision="f64", pivot="bk", graph=True),
    # a ragged system of medium size in single precision, blocks that divide neither part, rook pivots
    dict(name="factor ragged f32", kind="factor", n=77777, m=38889, per_col=5, band=32, hmin=1e-2, hmax=1e2,
         block=23, precision="f32", pivot="rook", graph=True),
    # the preconditioner alone, for a caller with an iteration of its own: the scale workload's factor
    dict(name="apply scale f64", kind="apply", n=200000, m=100000, per_col=6, band=32, hmin=1e-6, hmax=1e6, block=32,
         reg=1e-8, precision="f64"),
    # the largest factor, in single precision: the mixed-precision workload's
    dict(name="apply mixed f32", kind="apply", n=1000000, m=500000, per_col=6, band=32, hmin=1e-2, hmax=1e2, block=32,
         precision="f32"),
    # the smallest solve: the time of an iteration is its chain of dependent steps
    dict(name="solve small f64", kind="solve", n=2000, m=1000, per_col=4, band=0, hmin=1e-2, hmax=1e2, block=4,
         reg=1e-8, precision="f64", nrhs=1, its=24),
    # the headline solve
    dict(name="solve scale f64", kind="solve", n=200000, m=100000, per_col=6, band=32, hmin=1e-6, hmax=1e6, block=32,
         reg=1e-8, precision="f64", nrhs=1, its=32),
    # predictor, corrector and two centrality corrections of one iteration: four right-hand sides, mixed precision
    dict(name="solve 4 rhs f32", kind="solve", n=123457, m=61729, per_col=6, band=32, hmin=1e-4, hmax=1e4, block=32,
         precision="f32", nrhs=4, its=24),
    # many uneven systems at once: sizes log-uniform as in the served trace, up to the batched workload's largest
    dict(name="batch 256 f32", kind="batch", count=256, nmin=500, nmax=20000, band=32, hmin=1e-4, hmax=1e4, block=32,
         precision="f32", its=12),
]


def listed():
    return [dict(c) for c in LISTED]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds, its sizes log-uniform over their whole range."""
    kind = rng.choice(["spmv", "dual", "factor", "apply", "solve", "batch"])
    precision = rng.choice(["f64", "f32"])
    if kind == "batch":
        lo = _log_int(rng, 200, 2000)
        return dict(kind=kind, count=_log_int(rng, 8, 192), nmin=lo, nmax=lo * rng.randint(2, 10), band=32,
                    hmin=1e-4, hmax=1e4, block=rng.choice([8, 16, 24, 32]), precision=precision,
                    its=rng.randint(6, 12))
    top = {"spmv": 900000, "dual": 400000, "factor": 180000, "apply": 500000, "solve": 150000}[kind]
    n = _log_int(rng, 500, top)
    case = dict(kind=kind, n=n, m=max(100, int(n * rng.uniform(0.3, 0.7))), per_col=rng.randint(4, 8),
                band=rng.choice([0, 32]), precision=precision)
    if kind == "spmv":
        case["sell"] = rng.random() < 0.5
    if kind in ("factor", "apply", "solve"):
        h = rng.choice([1e1, 1e2, 1e4])
        case.update(hmin=1 / h, hmax=h, block=rng.choice([4, 8, 16, 24, 32, rng.randint(4, 32)]))
    if kind == "factor":
        case.update(pivot=rng.choice(["bk", "rook"]), graph=rng.random() < 0.5)
    if kind == "solve":
        case.update(nrhs=rng.choice([1, 1, 2, 3, 4]), its=rng.randint(8, 24))
    return case


# ---------------------------------------------------------------------------
# inputs


def _system(case, seed):
    """K (host CSR) with H from the case's range where it has one."""
    reg = _regularisation(case)
    return cb.kkt_generate(case["n"], case["m"], case["per_col"], case["band"], case.get("hmin", 1e-2),
                           case.get("hmax", 1e2), delta=reg, gamma=reg, seed=seed)


def _constraints(case, seed):
    """The m x n constraint matrix A as host CSR: K's rows n.. without their diagonal entry, the last of each row."""
    rowptr, colidx, val = _system(case, seed)
    n, m = case["n"], case["m"]
    first = int(rowptr[n])
    keep = np.ones(len(colidx) - first, bool)
    keep[rowptr[n + 1:] - 1 - first] = False
    rp = (rowptr[n:] - first - np.arange(m + 1)).astype(np.int32)
    return rp, np.ascontiguousarray(colidx[first:][keep]), np.ascontiguousarray(val[first:][keep])


def _dtype(case):
    return torch.float64 if case["precision"] == "f64" else torch.float32


def _precision(case):
    return cb.F64 if case["precision"] == "f64" else cb.F32


def _regularisation(case):
    # delta = gamma: the benchmark systems' 1e-8 where a case says so.  The factor replaces pivots below 1e-8, which
    # 1e-8 is in single precision, so the others keep above it
    return case.get("reg", 1e-6)


def _randn(seed, *shape):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)


def _uniform(seed, *shape):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    return torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _log_uniform(seed, size, lo, hi):
    return torch.exp(math.log(lo) + _uniform(seed, size) * (math.log(hi) - math.log(lo)))


def _cuda(*arrays):
    return [torch.from_numpy(a).cuda() for a in arrays]


def _iterate(case, seed):
    """A strictly positive iterate (x, s) with s / x log-uniform in the case's range."""
    x = _log_uniform(seed + 1, case["n"], 1e-1, 1e1)
    return x, x * _log_uniform(seed + 2, case["n"], case["hmin"], case["hmax"])


def _batch_systems(case, seed):
    sizes = np.random.default_rng(case["count"])  # the sizes belong to the case, the entries to the seed
    reg, systems = _regularisation(case), []
    for i in range(case["count"]):
        n = int(round(math.exp(sizes.uniform(math.log(case["nmin"]), math.log(case["nmax"])))))
        rp, ci, v = cb.kkt_generate(n, n // 2, int(sizes.integers(4, 9)), case["band"], case["hmin"], case["hmax"],
                                    delta=reg, gamma=reg, seed=seed + 1 + i)
        systems.append((rp, ci, v, cb.kkt_blocking(n, n // 2, case["block"])))
    return systems


def prepare(case, seed):
    handle = cb.Handle(0)
    kind, dtype = case["kind"], _dtype(case)
    s = dict(case=case, kind=kind, handle=handle)
    if kind == "spmv":
        rp, ci, v = _cuda(*_system(case, seed))
        s["A"] = cb.CsrOperator(handle, rp, ci, v.to(dtype))
        if case["sell"]:
            s["A"].set_format(cb.FMT_SELL)
        s["x"] = _randn(seed + 3, case["n"] + case["m"]).to(dtype)
        s["y"] = torch.empty_like(s["x"])
    elif kind == "dual":
        rp, ci, v = _cuda(*_constraints(case, seed))
        s["A"] = cb.CsrOperator(handle, rp, ci, v.to(dtype), ncols=case["n"], explicit_transpose=True)
        s["y"] = _randn(seed + 3, case["m"]).to(dtype)
        s["c"] = _randn(seed + 4, case["n"]).to(dtype)
        s["r"] = torch.empty_like(s["c"])
    elif kind == "factor":
        rp, ci, v = _cuda(*_constraints(case, seed))
        s["aval"] = v
        s["x"], s["s"] = _iterate(case, seed)
        s["asm"] = cb.KktAssembly(handle, case["m"], case["n"], rp, ci)
        s["kval"] = torch.empty(s["asm"].nnz, dtype=dtype, device="cuda")
        s["F"] = cb.Factor(cb.Pattern(handle, *s["asm"].structure(), cb.kkt_blocking(case["n"], case["m"],
                                                                                     case["block"]),
                                      0, 1.0, _precision(case)))
        s["pivot"] = {"bk": cb.PIV_BK, "rook": cb.PIV_ROOK}[case["pivot"]]
        s["b"] = _randn(seed + 3, case["n"] + case["m"]).to(dtype)
        s["t"] = [torch.empty_like(s["b"]) for _ in range(3)]
    elif kind in ("apply", "solve"):
        rp, ci, v = _system(case, seed)
        N = case["n"] + case["m"]
        s["F"] = cb.Factor(cb.Pattern(handle, rp, ci, cb.kkt_blocking(case["n"], case["m"], case["block"]), 0, 1.0,
                                      _precision(case)))
        d_rp, d_ci, d_v = _cuda(rp, ci, v)
        s["F"].compute(d_v.to(dtype))
        if kind == "apply":
            s["b"] = _randn(seed + 3, N).to(dtype)
            s["t"] = [torch.empty_like(s["b"]) for _ in range(3)]
        else:
            s["A"] = cb.CsrOperator(handle, d_rp, d_ci, d_v)
            s["b"] = _randn(seed + 3, case["nrhs"], N)
            s["x"] = torch.empty_like(s["b"])
    elif kind == "batch":
        rp, ci, v, starts, offsets = cb.union_systems(_batch_systems(case, seed))
        pattern = cb.Pattern(handle, rp, ci, starts, 0, 1.0, _precision(case), system_row_offsets=offsets)
        s["F"] = cb.Factor(pattern)
        s["B"] = cb.Batch(pattern, offsets)
        d_rp, d_ci, d_v = _cuda(rp, ci, v)
        s["vals"] = d_v.to(dtype)
        s["A"] = cb.CsrOperator(handle, d_rp, d_ci, d_v)
        s["b"] = _randn(seed + 3, len(rp) - 1)
        s["x"] = torch.empty_like(s["b"])
    return s


def run(s):
    case, kind = s["case"], s["kind"]
    if kind == "spmv":
        return s["A"].spmv(s["x"], s["y"])
    if kind == "dual":
        s["r"].copy_(s["c"])
        return s["A"].spmv(s["y"], s["r"], alpha=-1.0, beta=1.0, transpose=True)
    if kind == "factor":
        reg = _regularisation(case)
        s["asm"].assemble(s["aval"], s["kval"], x=s["x"], s=s["s"], delta=reg, gamma=reg)
        if case["graph"]:
            s["F"].compute_graph(s["kval"], s["pivot"])
        else:
            s["F"].compute(s["kval"], pivot=s["pivot"])
        left, middle, right = s["t"]
        s["F"].apply(cb.LEFT, s["b"], left)
        s["F"].apply(cb.MIDDLE, left, middle)
        s["F"].apply(cb.RIGHT, middle, right)
        return {"kval": s["kval"], "x": right}
    if kind == "apply":
        left, middle, right = s["t"]
        s["F"].apply(cb.LEFT, s["b"], left)
        s["F"].apply(cb.MIDDLE, left, middle)
        s["F"].apply(cb.RIGHT, middle, right)
        return {"left": left, "middle": middle, "right": right}
    if kind == "solve":
        if case["nrhs"] == 1:
            res, its, status = cb.sqmr_solve(s["handle"], s["A"], s["F"], s["b"][0], s["x"][0], 1e-14, case["its"])
        else:
            res, its, status = cb.sqmr_solve_multi(s["handle"], s["A"], s["F"], s["b"], s["x"], 1e-14, case["its"])
        return {"x": s["x"], "residual": res, "iterations": its, "status": status}
    res, its, status = cb.batch_factor_solve_graph(s["B"], s["A"], s["F"], s["vals"], s["b"], s["x"], 1e-14,
                                                   case["its"])
    return {"x": s["x"], "residual": res, "iterations": its, "status": status}


# ---------------------------------------------------------------------------
# what a pass cannot do without


def _apply_bytes(N, nnz_u, m, block, v):
    """The three stages: U and U' once each with their row offsets, the pivot tiles' triangles twice, D, and every
    stage's input and output vector."""
    return 2 * (nnz_u * (v + 4) + 4 * N) + 2 * v * m * (block + 1) // 2 + 3 * v * N + 6 * v * N


def _iteration(N, nnz_k, nnz_u, m, block, v, nrhs):
    """One SQMR iteration: K, U, U', the tiles and D once, eleven passes over vectors for each right-hand side."""
    b = nnz_k * 12 + 4 * N + 2 * (nnz_u * (v + 4) + 4 * N) + v * m * (block + 1) + 3 * v * N + 88 * N * nrhs
    return b, nrhs * (2 * nnz_k + 4 * nnz_u + 2 * m * (block + 1) + 30 * N)


def work(case):
    kind, v = case["kind"], 8 if case["precision"] == "f64" else 4
    if kind == "batch":
        N = nnz_k = nnz_u = m = 0
        for i in range(case["count"]):  # the distribution's quantiles; 6 entries per column on average
            n = case["nmin"] * (case["nmax"] / case["nmin"]) ** ((i + 0.5) / case["count"])
            N, m, nnz_u = N + 1.5 * n, m + n / 2, nnz_u + 6 * n
        nnz_k = 2 * nnz_u + N
        b, f = _iteration(N, nnz_k, nnz_u, m, case["block"], v, 1)
        fb = nnz_k * (v + 4) + nnz_u * (v + 4) + v * m * (case["block"] + 1) / 2 + 3 * v * N
        return {"bytes": fb + case["its"] * b, "flops": 2 * 6 * nnz_u + case["its"] * f}
    n, m, k = case["n"], case["m"], case["per_col"]
    N, nnz_a = n + m, n * k
    nnz_k = 2 * nnz_a + N
    if kind == "spmv":
        return {"bytes": nnz_k * (v + 4) + 4 * (N + 1) + 2 * v * N, "flops": 2 * nnz_k}
    if kind == "dual":
        return {"bytes": nnz_a * (v + 4) + 4 * (n + 1) + v * (m + 2 * n), "flops": 2 * nnz_a + n}
    block = min(case["block"], m)
    if kind == "apply":
        return {"bytes": _apply_bytes(N, nnz_a, m, block, v), "flops": 4 * nnz_a + 2 * m * (block + 1) + 4 * N}
    if kind == "factor":
        # A's values and the iterate in, K's values out and read back with their columns, U, the tiles and D out
        b = nnz_a * 8 + 16 * n + 2 * nnz_k * v + nnz_k * 4
        b += nnz_a * (v + 4) + 4 * N + v * m * (block + 1) // 2 + 3 * v * N
        return {"bytes": b + _apply_bytes(N, nnz_a, m, block, v),
                "flops": 2 * k * nnz_a + m * block * block // 3 + 4 * nnz_a + 2 * m * (block + 1)}
    b, f = _iteration(N, nnz_k, nnz_a, m, block, v, case["nrhs"])
    return {"bytes": case["its"] * b, "flops": case["its"] * f}


# ---------------------------------------------------------------------------
# the same in plain 64-bit torch


def _rows_of(rowptr):
    counts = torch.from_numpy(np.diff(rowptr).astype(np.int64)).cuda()
    return torch.repeat_interleave(torch.arange(len(rowptr) - 1, device="cuda"), counts)


def _preconditioner_solve(rp, ci, aval, d, gamma, block, b):
    """M^-1 b for M = [[D, A'], [A, A D^-1 A' + S]], S the diagonal blocks of -gamma I - A D^-1 A': what the block
    factor of fill level 0 is in exact arithmetic for K in its natural order."""
    m, n = len(rp) - 1, len(d)
    rows, cols = _rows_of(rp), torch.from_numpy(ci.astype(np.int64)).cuda()
    starts = cb.kkt_blocking(n, m, block).astype(np.int64)
    starts = torch.from_numpy(starts[np.searchsorted(starts, n):] - n).cuda()
    nb = len(starts) - 1
    of_row = torch.bucketize(torch.arange(m, device="cuda"), starts, right=True) - 1
    width = int((starts[1:] - starts[:-1]).max())
    # A as one dense strip per block over the columns that its rows touch
    key, column = torch.unique(of_row[rows] * n + cols, return_inverse=True)
    strip = key // n
    first = torch.searchsorted(strip, torch.arange(nb, device="cuda"))
    wide = int(torch.bincount(strip, minlength=nb).max())
    S = torch.eye(width, device="cuda", dtype=torch.float64).repeat(nb, 1, 1) * -1.0
    local = torch.arange(m, device="cuda") - starts[of_row]
    S[of_row, local, local] = -gamma
    step = max(1, (1 << 27) // (width * wide))
    for k0 in range(0, nb, step):
        k1 = min(nb, k0 + step)
        here = (of_row[rows] >= k0) & (of_row[rows] < k1)
        W = torch.zeros(k1 - k0, width, wide, device="cuda", dtype=torch.float64)
        blk = of_row[rows[here]]
        W[blk - k0, local[rows[here]], column[here] - first[blk]] = aval[here] / torch.sqrt(d[cols[here]])
        S[k0:k1] -= W @ W.transpose(1, 2)
    top = b[:n] / d
    rhs = b[n:].clone()
    rhs.index_add_(0, rows, -aval * top[cols])
    padded = torch.zeros(nb, width, 1, device="cuda", dtype=torch.float64)
    padded[of_row, local, 0] = rhs
    low = torch.linalg.solve(S, padded)[of_row, local, 0]
    out = torch.cat([b[:n], low])
    out[:n].index_add_(0, cols, -aval * low[rows])
    out[:n] /= d
    return out


def exact(case, seed):
    kind, dtype = case["kind"], _dtype(case)

    def held(t):  # as the program holds it
        return t.to(dtype).double()

    if kind == "spmv":
        rp, ci, v = _system(case, seed)
        x = held(_randn(seed + 3, case["n"] + case["m"]))
        y = torch.zeros_like(x)
        return y.index_add_(0, _rows_of(rp), held(torch.from_numpy(v).cuda()) * x[torch.from_numpy(ci).cuda().long()])
    if kind == "dual":
        rp, ci, v = _constraints(case, seed)
        y, r = held(_randn(seed + 3, case["m"])), held(_randn(seed + 4, case["n"]))
        return r.index_add_(0, torch.from_numpy(ci).cuda().long(), -held(torch.from_numpy(v).cuda()) * y[_rows_of(rp)])
    if kind == "factor":
        n, m, reg = case["n"], case["m"], _regularisation(case)
        rp, ci, v = _constraints(case, seed)
        x, s = _iterate(case, seed)
        d, aval = s / x + reg, torch.from_numpy(v).cuda()
        rows, cols = _rows_of(rp), torch.from_numpy(ci.astype(np.int64)).cuda()
        every = torch.arange(n + m, device="cuda")
        key = torch.cat([every * (n + m) + every, (n + rows) * (n + m) + cols, cols * (n + m) + n + rows])
        values = torch.cat([d, torch.full((m,), -reg, device="cuda", dtype=torch.float64), aval, aval])
        b = held(_randn(seed + 3, n + m))
        return {"kval": values[torch.argsort(key)],
                "x": _preconditioner_solve(rp, ci, held(aval), held(d), reg, case["block"], b)}
    if kind == "apply":
        n, m = case["n"], case["m"]
        rowptr, _, val = _system(case, seed)
        rp, ci, v = _constraints(case, seed)
        d = held(torch.from_numpy(val[rowptr[:n]]).cuda())  # the diagonal leads each of the first n rows
        b = held(_randn(seed + 3, n + m))
        gamma = float(held(torch.tensor(-val[-1])))
        # the split of M between the stages depends on the pivots: only their product is defined
        return {"left": None, "middle": None,
                "right": _preconditioner_solve(rp, ci, held(torch.from_numpy(v).cuda()), d, gamma, case["block"], b)}
    return None  # SQMR's iterates before convergence are no function of the system alone
