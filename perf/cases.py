"""The work a user of this framework has it do, as cases that can be timed and checked.

A case names one public call (`op`) on one kind of matrix:

  op       mv        y = A x on device vectors, FP64, merge-path CRS
           mv_f32    the same with FP32 values and vectors
           mv_host   y = A x on the caller's (pageable) host arrays
           power     `it` power iterations on device vectors
           solve     power solve to a residual, mixed precision, host start vector
           csb, coh  y = A x on device vectors in the CSB / CO-H formats
           load      triplets in any order, on the device -> CRS and its plan, then one y = A x
           service   a batch of power solves of many small matrices through the serving loop
  matrix   poisson   the 5-point Poisson matrix of an m x n grid (generatePoissonMatrix)
           stencil   a 5- or 9-point stencil with a coefficient of its own for every entry
           irregular lognormal row lengths, part of the columns in a band, the rest anywhere
           mixed     (service) Poisson grids and random matrices side by side

Matrices, vectors and coefficients come from the seed alone.
"""
import math

import numpy as np
import torch

from thesis_spmv_gb300.matrix import PREC_MIXED, COHCuda, CRSCuda, CSBCuda
from thesis_spmv_gb300.service import Service

DEV = "cuda"
TOL = 1e-10
SERVICE_ROUND = 8


def listed():
    return [
        # the reference's unit tests and first steps of a user: a few thousand rows, where one call is launches and latency
        {"name": "mv_poisson_64x48", "op": "mv", "matrix": "poisson", "m": 64, "n": 48},
        # the headline SpMV: 84 M nonzeros, streamed from HBM
        {"name": "mv_poisson_4096", "op": "mv", "matrix": "poisson", "m": 4096, "n": 4096},
        # the irregular headline: 67 M nonzeros, most of whose gathers go anywhere in a 32 MB x
        {"name": "mv_irregular_4m", "op": "mv", "matrix": "irregular", "rows": 4194304, "mean": 16.0, "band": 0.3},
        # single-precision product of a discretised operator with varying coefficients on an odd grid
        {"name": "mv_f32_stencil9_1999x1501", "op": "mv_f32", "matrix": "stencil", "m": 1999, "n": 1501, "points": 9},
        # the reference's distributed and OpenMP drivers: a power method on a matrix that fits the L2
        {"name": "power_poisson_512", "op": "power", "matrix": "poisson", "m": 512, "n": 512, "it": 100},
        # the same on a large ragged grid with varying coefficients, an odd number of iterations
        {"name": "power_stencil5_3001x2777", "op": "power", "matrix": "stencil", "m": 3001, "n": 2777, "points": 5,
         "it": 25},
        # dominant eigenpair of an irregular matrix to 1e-10, low-precision iterations first
        {"name": "solve_irregular_1m", "op": "solve", "matrix": "irregular", "rows": 1048576, "mean": 16.0, "band": 0.3},
        # the reference's blocked formats on the two kinds of matrix
        {"name": "csb_poisson_4096", "op": "csb", "matrix": "poisson", "m": 4096, "n": 4096},
        {"name": "coh_irregular_1m", "op": "coh", "matrix": "irregular", "rows": 1000003, "mean": 16.0, "band": 0.3},
        # the reference's drivers hold x and y in host memory (new[]): both cross the host link on every call
        {"name": "mv_host_poisson_4096", "op": "mv_host", "matrix": "poisson", "m": 4096, "n": 4096},
        # a matrix assembled on the device in no particular order, made ready and used once
        {"name": "load_poisson_2048", "op": "load", "matrix": "poisson", "m": 2048, "n": 2048},
        # the serving loop: grids that run to their iteration limit beside random matrices that converge quickly
        {"name": "service_32_solves", "op": "service", "matrix": "mixed", "grids": 16, "side": 512, "randoms": 16,
         "rows": 32768, "it": 1000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["mv", "mv", "mv", "mv_f32", "power", "power", "solve", "csb", "coh", "mv_host", "load", "service"])
    if op == "service":
        return {"op": op, "matrix": "mixed", "grids": rng.randint(1, 16), "side": rng.randint(48, 512),
                "randoms": rng.randint(0, 16), "rows": _log(rng, 1024, 32768), "it": 8 * rng.randint(16, 125)}
    kind = "irregular" if op == "solve" else rng.choice(["poisson", "stencil", "irregular"])
    big = {"csb": 4.0e6, "coh": 4.0e6, "solve": 1.5e6, "load": 4.0e6}.get(op, 1.6e7)
    case = {"op": op, "matrix": kind}
    if kind == "irregular":
        case["rows"] = _log(rng, 1024, min(big, 4.1e6))
        case["mean"] = float(rng.choice([4.0, 8.0, 16.0]))
        case["band"] = float(rng.choice([0.0, 0.3, 0.9]))
    else:
        rows = math.exp(rng.uniform(math.log(1024), math.log(big)))
        m = int(round(math.sqrt(rows) * math.exp(rng.uniform(-0.7, 0.7))))
        case["m"] = max(4, m)
        case["n"] = max(4, int(rows / case["m"]))
        if kind == "stencil":
            case["points"] = rng.choice([5, 9]) if rows < 8.0e6 else 5
    if op == "power":
        case["it"] = rng.randint(2, 40)
    return case


# ---- matrices, in torch alone ------------------------------------------------

def _generator(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _grid_triplets(m, n, points, g):
    """Entries of a 5- or 9-point stencil in CRS order; g: one coefficient per entry from it (None: 4 and -1)."""
    size = m * n
    row = torch.arange(size, device=DEV, dtype=torch.int32)
    i, j = row % m, row // m
    offs = [(dj, di) for dj in (-1, 0, 1) for di in (-1, 0, 1) if points == 9 or di == 0 or dj == 0]
    mask = torch.empty((size, len(offs)), device=DEV, dtype=torch.bool)
    cols = torch.empty((size, len(offs)), device=DEV, dtype=torch.int32)
    for k, (dj, di) in enumerate(offs):
        mask[:, k] = (i + di >= 0) & (i + di < m) & (j + dj >= 0) & (j + dj < n)
        cols[:, k] = row + (dj * m + di)
    counts = mask.sum(1)
    rows = torch.repeat_interleave(row, counts)
    cols = cols[mask]
    diag = cols == rows
    if g is None:
        vals = torch.where(diag, 4.0, -1.0).to(torch.float64)
    else:
        u = torch.rand(rows.numel(), device=DEV, dtype=torch.float64, generator=g)
        vals = torch.where(diag, (points - 1) + u, -0.5 - u)
    return size, rows, cols, vals


def _random_triplets(n, lengths, band, g):
    """Entries in CRS order, no coordinate twice: `band` of the columns within 4096 of the diagonal, the rest anywhere."""
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), lengths)
    k = rows.numel()
    near = torch.rand(k, device=DEV, generator=g) < band
    cols = torch.where(near, rows + torch.randint(-4096, 4097, (k,), device=DEV, generator=g),
                       torch.randint(0, n, (k,), device=DEV, generator=g)) % n
    key = torch.sort(rows * n + cols).values
    keep = torch.ones(k, dtype=torch.bool, device=DEV)
    keep[1:] = key[1:] != key[:-1]
    key = key[keep]
    vals = 1.0 - torch.rand(key.numel(), device=DEV, dtype=torch.float64, generator=g)
    return n, (key // n).to(torch.int32), (key % n).to(torch.int32), vals


def _triplets(case, g):
    """(order, rows, cols, vals) of the case's matrix, in CRS order."""
    if case["matrix"] == "poisson":
        return _grid_triplets(case["m"], case["n"], 5, None)
    if case["matrix"] == "stencil":
        return _grid_triplets(case["m"], case["n"], case["points"], g)
    n, mean, sigma = case["rows"], case["mean"], 1.2
    z = torch.randn(n, device=DEV, generator=g)
    lengths = torch.exp(math.log(mean) - 0.5 * sigma * sigma + sigma * z).round().clamp(1, min(20000, n)).long()
    return _random_triplets(n, lengths, case["band"], g)


def _counts(case):
    """(rows, entries) of the case's matrix, the expected ones where it is random."""
    if case["matrix"] == "irregular":
        return case["rows"], case["rows"] * case["mean"]
    m, n = case["m"], case["n"]
    entries = m * n + 2 * (m - 1) * n + 2 * m * (n - 1)
    if case.get("points") == 9:
        entries += 4 * (m - 1) * (n - 1)
    return m * n, entries


def _load(handle, case, g):
    """The matrix into the handle, as a program that has it on the device does; the handle works on torch's stream."""
    if case["matrix"] == "poisson":
        handle.generatePoissonMatrix(case["m"], case["n"])
        n = case["m"] * case["n"]
    else:
        n, rows, cols, vals = _triplets(case, g)
        torch.cuda.synchronize()
        handle.loadFromDeviceTriplets(n, n, rows.numel(), rows.data_ptr(), cols.data_ptr(), vals.data_ptr())
    handle.set_stream(torch.cuda.current_stream().cuda_stream)
    return n


def _vector(n, seed):
    """Seeded start vector, uniform in [0, 1)."""
    return torch.rand(n, device=DEV, dtype=torch.float64, generator=_generator(2 * int(seed) + 1))


# ---- the serving batch ---------------------------------------------------------

class _Csr:
    def __init__(self, nor, row_start, col_ind, data):
        self.nor, self.row_start, self.col_ind, self.data = nor, row_start, col_ind, data


def _grid_sides(case):
    lo, hi, k = 32, case["side"], case["grids"]
    return [int(round(lo * (hi / lo) ** ((i + 1) / k))) for i in range(k)]


def _random_orders(case):
    lo, hi, k = 512, case["rows"], case["randoms"]
    return [int(round(lo * (hi / lo) ** ((i + 1) / k))) for i in range(k)]


def _service_random(n, g):
    lengths = torch.poisson(torch.full((n,), 8.0, device=DEV), generator=g).clamp(1, n).long()
    return _random_triplets(n, lengths, 0.0, g)


def _service_start(n, seed, k):
    return np.random.default_rng([int(seed), 7, k]).random(n)


# ---- prepare / run -----------------------------------------------------------

def prepare(case, seed):
    op, g = case["op"], _generator(2 * int(seed))
    state = {"op": op}
    if op == "service":
        state["service"] = Service(hbm_budget_bytes=32 << 30, round_iterations=SERVICE_ROUND)
        state["it"] = case["it"]
        state["grids"] = [(s, _service_start(s * s, seed, k)) for k, s in enumerate(_grid_sides(case))]
        state["randoms"] = []
        for k, n in enumerate(_random_orders(case)):
            _, rows, cols, vals = _service_random(n, g)
            start = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
            start[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
            a = _Csr(n, start.to(torch.int32).cpu().numpy(), cols.cpu().numpy(), vals.cpu().numpy())
            state["randoms"].append((a, _service_start(n, seed, 1000 + k)))
        return state
    if op == "load":
        n, rows, cols, vals = _triplets(case, g)
        p = torch.randperm(rows.numel(), device=DEV, generator=g)
        state["triplets"] = (n, rows[p], cols[p], vals[p])
        state["handle"] = CRSCuda()
        state["handle"].set_stream(torch.cuda.current_stream().cuda_stream)
    else:
        state["handle"] = {"csb": CSBCuda, "coh": COHCuda}.get(op, CRSCuda)()
        n = _load(state["handle"], case, g)
    x = _vector(n, seed)
    if op in ("mv_host", "solve"):
        state["x"] = x.cpu().numpy()
        state["y"] = np.zeros(n)
        return state
    dtype = torch.float32 if op == "mv_f32" else torch.float64
    state["x"] = x.to(dtype)
    state["y"] = torch.empty(n, device=DEV, dtype=dtype)
    if op == "power":
        state["it"] = case["it"]
        state["v"] = torch.empty(n, device=DEV, dtype=dtype)
    return state


def run(state):
    op = state["op"]
    if op == "service":
        svc = state["service"]
        ids = [svc.submit_poisson(s, s, max_it=state["it"], tol=TOL, precision=PREC_MIXED, x0=x0, keep_vector=True)
               for s, x0 in state["grids"]]
        ids += [svc.submit_csr(a, max_it=state["it"], tol=TOL, precision=PREC_MIXED, x0=x0, keep_vector=True)
                for a, x0 in state["randoms"]]
        svc.run_until_idle()
        got = [svc.result(i, want_vector=True) for i in ids]
        for i in ids:
            svc.release(i)
        return {"lambda": np.array([r.lambda_ for r, _ in got]), "vectors": np.concatenate([u for _, u in got]),
                "iterations": np.array([r.iterations for r, _ in got]),
                "converged": np.array([r.converged for r, _ in got])}
    h, x, y = state["handle"], state["x"], state["y"]
    if op == "mv_host":
        h.mv(x, y)
        return y
    if op == "solve":
        u = x.copy()
        info = h.solve(u, 500, TOL, PREC_MIXED)
        return {"vector": u, "lambda": np.array([info.lambda_]), "iterations": info.iterations,
                "converged": info.converged}
    if op == "power":
        v = state["v"]
        v.copy_(x)
        h.power_device(v.data_ptr(), y.data_ptr(), state["it"])
        return [v, y]
    if op == "load":
        n, rows, cols, vals = state["triplets"]
        h.loadFromDeviceTriplets(n, n, rows.numel(), rows.data_ptr(), cols.data_ptr(), vals.data_ptr())
    if op == "mv_f32":
        h.mv_device_f32(x.data_ptr(), y.data_ptr())
    else:
        h.mv_device(x.data_ptr(), y.data_ptr())
    return y


# ---- work --------------------------------------------------------------------

def work(case):
    if case["op"] == "service":
        byts = flops = 0.0
        for s in _grid_sides(case):
            # a grid's power steps run to the limit
            byts += case["it"] * (12.0 * 5 * s * s + 20.0 * s * s)
            flops += case["it"] * 10.0 * s * s
        for n in _random_orders(case):
            byts += 24 * (12.0 * 8 * n + 20.0 * n)
            flops += 24 * 16.0 * n
        return {"bytes": byts, "flops": flops}
    n, nnz = _counts(case)
    entry = 4.0 + (4.0 if case["op"] == "mv_f32" else 8.0)
    vec = 4.0 if case["op"] == "mv_f32" else 8.0
    one = entry * nnz + 4.0 * (n + 1) + 2 * vec * n
    steps = {"power": case.get("it", 1), "solve": 24}.get(case["op"], 1)
    byts, flops = steps * one, steps * 2.0 * nnz
    if case["op"] == "load":
        byts += 16.0 * nnz + 12.0 * nnz + 4.0 * n  # the triplets read, the CRS arrays written
    return {"bytes": byts, "flops": flops}


# ---- the same in plain torch, 64 bits -------------------------------------------

def _product(rows, cols, vals, n):
    rows, cols = rows.long(), cols.long()

    def mv(x):
        return torch.zeros(n, device=DEV, dtype=torch.float64).index_add_(0, rows, vals * x[cols])
    return mv


def _iterate(mv, x, steps):
    """The last two of `steps` power iterates, normalised: (newest, the one before)."""
    prev = x
    for _ in range(steps):
        y = mv(x)
        prev, x = x, y / torch.linalg.vector_norm(y)
    return x, prev


def exact(case, seed):
    op, g = case["op"], _generator(2 * int(seed))
    if op == "service":
        lams, vecs = [], []
        grids = [(s, k, None) for k, s in enumerate(_grid_sides(case))]
        randoms = [(n, 1000 + k, _service_random(n, g)) for k, n in enumerate(_random_orders(case))]
        for size, k, t in grids + randoms:
            n = size * size if t is None else size
            x = torch.from_numpy(_service_start(n, seed, k)).to(DEV)
            if t is None:
                # 5-point Laplacian by slices; the grid stops at its limit, rounded up to whole rounds
                pad = torch.zeros((size + 2, size + 2), device=DEV, dtype=torch.float64)

                def mv(v, pad=pad, size=size):
                    pad[1:-1, 1:-1] = v.view(size, size)
                    c = pad[1:-1, 1:-1]
                    return (4 * c - pad[:-2, 1:-1] - pad[2:, 1:-1] - pad[1:-1, :-2] - pad[1:-1, 2:]).reshape(-1)
                steps = -(-case["it"] // SERVICE_ROUND) * SERVICE_ROUND - 1
            else:
                mv = _product(t[1], t[2], t[3], n)
                steps = 80  # to the converged eigenvector
            u = _iterate(mv, x, steps)[0]
            lams.append(torch.dot(u, mv(u)))
            vecs.append(u)
        return {"lambda": torch.stack(lams), "vectors": torch.cat(vecs), "iterations": None, "converged": None}
    n, rows, cols, vals = _triplets(case, g)
    mv = _product(rows, cols, vals, n)
    x = _vector(n, seed)
    if op == "power":
        last, prev = _iterate(mv, x, case["it"])
        return [prev, last] if case["it"] % 2 else [last, prev]
    if op == "solve":
        u = _iterate(mv, x, 80)[0]
        return {"vector": u, "lambda": torch.dot(u, mv(u)).reshape(1), "iterations": None, "converged": None}
    return mv(x)
