"""Performance cases of the solver path: what is timed and how its results are checked.

Every case is one call a user's program makes through the package's public
entry points on the GPU: a sparse matrix-vector product, a residual, one
application of a preconditioner, a matrix taken into a solver, a whole solve,
or a batch of solves. Sizes follow the benchmark's configurations (32^3 with
64 tiles, 128^3 with 1024, 192^3 with 2368, the 100^3 LDU mesh) and generic
grids with three different, also odd, edges; ``draw`` spreads over the same
ranges. ``exact`` restates each case in 64 bits with torch alone, taking from
the package only the inputs (the generated coefficients and the tile map).

A case's keys:

* ``op``: ``spmv`` | ``residual`` | ``ilu`` | ``gs`` | ``factor`` |
  ``pbicgstab`` | ``mpir`` | ``batch``
* ``kind``: ``poisson`` | ``var`` (cell coefficients log-normal, sigma 1.5) |
  ``convdiff`` (velocity 0.5, 0.25, 0.125) | ``ldu`` (permuted hexahedral mesh)
* ``nx, ny, nz, tiles``: the grid and the number of tiles
* ``dtype``: ``float32`` | ``float64``, of the coefficients and the vectors
* ``matrix_seed``: the matrix is this one and only the vectors follow the
  run's seed (large grids, whose host-side generation would dominate);
  without it the matrix follows the run's seed too
* ``pre``: the preconditioner of a ``pbicgstab`` solve
* ``systems, edge_lo, edge_hi, edge_seed``: the batch's systems and their
  grid edges; the coefficients follow the run's seed
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import graphene_b200 as gb

_GEN = {"poisson": (gb.GEN_POISSON, ()), "var": (gb.GEN_VAR_POISSON, (1.5,)),
        "convdiff": (gb.GEN_CONVDIFF, (0.5, 0.25, 0.125))}
_SWEEPS = 2  # Gauss-Seidel sweeps of a preconditioner application


def listed():
    return [
        # The smallest call: one product on a 32^3 grid, where the launch and
        # the return to the host are what a user waits for.
        {"name": "spmv_32", "op": "spmv", "kind": "poisson", "nx": 32, "ny": 32, "nz": 32, "tiles": 64,
         "dtype": "float32"},
        # The unstructured mesh in LDU form: face ordering, scattered columns.
        {"name": "spmv_mesh_100", "op": "spmv", "kind": "ldu", "nx": 100, "ny": 100, "nz": 100, "tiles": 1024,
         "dtype": "float32", "matrix_seed": 4},
        # A plain float64 product with three odd edges and ragged tiles.
        {"name": "spmv_odd_f64", "op": "spmv", "kind": "convdiff", "nx": 141, "ny": 97, "nz": 123, "tiles": 827,
         "dtype": "float64", "matrix_seed": 1},
        # The outer residual of mixed-precision refinement: x in float64,
        # coefficients, b and r in float32, computed in float64.
        {"name": "residual_192", "op": "residual", "kind": "var", "nx": 192, "ny": 192, "nz": 192, "tiles": 2368,
         "dtype": "float32", "matrix_seed": 2},
        # One block-ILU(0) application, the largest part of every Krylov
        # iteration, at the largest configuration.
        {"name": "ilu_192", "op": "ilu", "kind": "var", "nx": 192, "ny": 192, "nz": 192, "tiles": 2368,
         "dtype": "float32", "matrix_seed": 2},
        # The same in float64 (the plain FP64 solver), nonsymmetric.
        {"name": "ilu_128_f64", "op": "ilu", "kind": "convdiff", "nx": 128, "ny": 128, "nz": 128, "tiles": 1024,
         "dtype": "float64", "matrix_seed": 1},
        # Two Gauss-Seidel sweeps from a given x, as smoother and
        # preconditioner of the convection-diffusion configuration.
        {"name": "gs_128", "op": "gs", "kind": "convdiff", "nx": 128, "ny": 128, "nz": 128, "tiles": 1024,
         "dtype": "float32", "matrix_seed": 1},
        # Gauss-Seidel on the unstructured mesh in float64: rows of uneven
        # length, levels without a stencil's regularity.
        {"name": "gs_mesh_100_f64", "op": "gs", "kind": "ldu", "nx": 100, "ny": 100, "nz": 100, "tiles": 1024,
         "dtype": "float64", "matrix_seed": 4},
        # A solver taken on a resident matrix and applied once: what a time
        # step with new coefficients pays before its first iteration.
        {"name": "factor_97", "op": "factor", "kind": "var", "nx": 97, "ny": 96, "nz": 95, "tiles": 432,
         "dtype": "float32", "matrix_seed": 2},
        # A small whole solve, bound by the latency of its many short kernels.
        {"name": "pbicgstab_32", "op": "pbicgstab", "kind": "poisson", "nx": 32, "ny": 32, "nz": 32, "tiles": 64,
         "dtype": "float32", "pre": "ILU"},
        # Many small uneven systems from host memory in one batch.
        {"name": "batch_24", "op": "batch", "kind": "var", "systems": 24, "edge_lo": 16, "edge_hi": 48,
         "dtype": "float32", "edge_seed": 7},
        # The headline: matrix resident, solver created, refined to 1e-10.
        {"name": "mpir_192", "op": "mpir", "kind": "var", "nx": 192, "ny": 192, "nz": 192, "tiles": 2368,
         "dtype": "float32", "matrix_seed": 2},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: an op at a grid of three drawn edges, 400 to 3400 rows a
    tile, either type where the op has both."""
    op = rng.choice(["spmv", "residual", "ilu", "gs", "factor", "pbicgstab", "mpir", "batch", "ilu", "gs"])
    if op == "batch":
        lo = rng.randint(12, 24)
        return {"op": op, "kind": rng.choice(["var", "poisson"]), "systems": rng.randint(3, 32), "edge_lo": lo,
                "edge_hi": lo + rng.randint(4, 32), "dtype": rng.choice(["float32", "float64"]),
                "edge_seed": rng.randint(1, 99)}
    hi = {"pbicgstab": 96, "mpir": 112}.get(op, 176)
    edge = _log_int(rng, 14, hi)
    dims = [max(8, min(hi, int(edge * rng.uniform(0.8, 1.25)))) for _ in range(3)]
    rows = dims[0] * dims[1] * dims[2]
    kinds = {"residual": ["var"], "mpir": ["var", "poisson"], "factor": ["var", "convdiff"],
             "pbicgstab": ["poisson", "var", "convdiff"]}.get(op, ["var", "convdiff", "ldu"])
    kind = rng.choice(kinds)
    if kind == "ldu" and rows > 1_000_000:
        kind = "convdiff"
    case = {"op": op, "kind": kind, "nx": dims[0], "ny": dims[1], "nz": dims[2],
            "tiles": max(1, rows // _log_int(rng, 400, 3400)),
            "dtype": "float32" if op in ("residual", "mpir") else rng.choice(["float32", "float64"]),
            "matrix_seed": rng.randint(1, 9)}
    if op == "pbicgstab":
        case["pre"] = rng.choice(["ILU", "ILU", "GS"])
    return case


# -- inputs ------------------------------------------------------------------

@functools.lru_cache(maxsize=6)
def _fixed_host(kind, nx, ny, nz, tiles, dtype, seed):
    return _new_host(kind, nx, ny, nz, tiles, dtype, seed)


def _new_host(kind, nx, ny, nz, tiles, dtype, seed):
    t = gb.parseType(dtype)
    if kind == "ldu":
        return gb.generateLduMesh(nx, ny, nz, seed, seed + 1, seed + 2, numTiles=tiles, valueType=t)
    gen, params = _GEN[kind]
    h = gb.generateMatrix(gen, nx, ny, nz, params, seed, tiles)
    return h if t == gb.FLOAT32 else h.astype(t)


def _host(case, seed):
    at = (case["kind"], case["nx"], case["ny"], case["nz"], case["tiles"], case["dtype"])
    return _fixed_host(*at, case["matrix_seed"]) if "matrix_seed" in case else _new_host(*at, seed)


def _uniform(n, seed, dtype):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.rand(n, generator=g, device="cuda", dtype=torch.float64).mul_(2.0).sub_(1.0).to(dtype)


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.float64


def _pre(name):
    return {"type": "ILU"} if name == "ILU" else {"type": "GaussSeidel", "numFixedIterations": _SWEEPS}


def _config(case):
    op = case["op"]
    if op in ("ilu", "factor"):
        return {"type": "ILU"}
    if op == "gs":
        return _pre("GS")
    if op == "mpir":
        return {"type": "IterativeRefinement", "relResidual": 1e-10, "maxIterations": 50,
                "extendedPrecisionType": "float64",
                "innerSolver": {"type": "PBiCGStab", "maxIterations": 500, "relResidual": 1e-4,
                                "preconditioner": _pre("ILU")}}
    return {"type": "PBiCGStab", "maxIterations": 1000, "relResidual": 1e-6,
            "preconditioner": _pre(case.get("pre", "ILU"))}


def _batch_hosts(case, seed):
    t = gb.parseType(case["dtype"])
    edges = np.random.default_rng(case["edge_seed"]).integers(case["edge_lo"], case["edge_hi"] + 1, case["systems"])
    gen, params = _GEN[case["kind"]]
    hosts = []
    for i, e in enumerate(int(v) for v in edges):
        h = gb.generateMatrix(gen, e, e, e, params, seed + i, max(1, e ** 3 // 512))
        hosts.append(h if t == gb.FLOAT32 else h.astype(t))
    return hosts


def _batch_rhs(case, hosts, seed):
    """b = A x for a seeded x, on the host: a batch takes host vectors."""
    out = []
    for i, h in enumerate(hosts):
        rp, col, off, dg = h.globalCrs()
        x = np.random.default_rng([seed, i]).uniform(-1.0, 1.0, h.numRows)
        b = dg * x + np.add.reduceat(np.append(off * x[col], 0.0), rp[:-1])
        out.append(b.astype(np.float32 if case["dtype"] == "float32" else np.float64))
    return out


def prepare(case, seed):
    op, dtype = case["op"], _dtype(case)
    if op == "batch":
        hosts = _batch_hosts(case, seed)
        return {"op": op, "batch": gb.Batch(hosts, _config(case)), "b": _batch_rhs(case, hosts, seed)}
    h = _host(case, seed)
    A = h.copyToTile()
    n = h.numRows
    state = {"op": op, "A": A}
    if op == "spmv":
        state["x"] = _uniform(n, seed, dtype)
        state["y"] = torch.empty_like(state["x"])
    elif op == "residual":
        state["x"] = _uniform(n, seed, torch.float64)
        state["b"] = _uniform(n, seed + 1, torch.float32)
    elif op in ("ilu", "factor"):
        state["b"] = _uniform(n, seed, dtype)
    elif op == "gs":
        state["x0"] = _uniform(n, seed, dtype)
        state["b"] = _uniform(n, seed + 1, dtype)
    else:  # a solve: b = A x of a seeded x
        state["b"] = A * _uniform(n, seed, dtype)
    if op in ("ilu", "gs", "pbicgstab"):
        state["solver"] = gb.Solver(A, _config(case))
    else:
        state["config"] = _config(case)
    return state


def run(state):
    op = state["op"]
    if op == "batch":
        return state["batch"].solveHost(state["b"])[0]
    A = state["A"]
    if op == "spmv":
        A.spmv(state["x"], state["y"])
        return state["y"]
    if op == "residual":
        return A.residual(state["x"], state["b"], destType=gb.FLOAT32, intermediateType=gb.FLOAT64)
    if op == "gs":
        x = state["x0"].clone()
    elif op == "ilu":
        x = torch.empty_like(state["b"])
    else:
        x = torch.zeros_like(state["b"])
    if "solver" in state:
        state["solver"].solve(x, state["b"])
    else:
        A.solve(x, state["b"], state["config"])
    return x


# -- bytes and operations ----------------------------------------------------

def work(case):
    """Bytes and operations of one pass, every operand once: coefficients with
    a 32-bit column each, and the vectors. Whole solves count the iterations
    that their tolerances take on these systems, about 0.72 (PBiCGStab to
    1e-6) and 1.42 (refinement to 1e-10) an edge."""
    if case["op"] == "batch":
        total = {"bytes": 0.0, "flops": 0.0}
        edge = 0.5 * (case["edge_lo"] + case["edge_hi"])
        one = work({"op": "pbicgstab", "kind": case["kind"], "nx": edge, "ny": edge, "nz": edge,
                    "tiles": max(1.0, edge ** 3 / 512), "dtype": case["dtype"]})
        for k in total:
            total[k] = one[k] * case["systems"]
        return total
    a, b, c, P = case["nx"], case["ny"], case["nz"], case["tiles"]
    n = a * b * c
    m = 2 * (3 * n - a * b - b * c - c * a)
    inner = max(0.0, 6.0 * (n - P * (n / P) ** (2.0 / 3.0)))  # couplings inside cubic tiles
    v = 4 if case["dtype"] == "float32" else 8
    e = v + 4
    op = case["op"]
    spmv = {"bytes": e * m + 3 * v * n, "flops": 2 * m + n}
    ilu = {"bytes": e * inner + 3 * v * n, "flops": 2 * inner + 2 * n}
    gs = {"bytes": e * m + 4 * v * n, "flops": 2 * m + 2 * n}
    if op == "spmv":
        return spmv
    if op == "residual":
        return {"bytes": e * m + (4 + 8 + 4 + 4) * n, "flops": 2 * m + 2 * n}
    if op == "ilu":
        return ilu
    if op == "gs":
        return {k: _SWEEPS * gs[k] for k in gs}
    factor = {"bytes": 2 * e * inner + 3 * v * n, "flops": 4 * inner}
    if op == "factor":
        return {k: factor[k] + ilu[k] for k in ilu}
    pre = ilu if case.get("pre", "ILU") == "ILU" else {k: _SWEEPS * gs[k] for k in gs}
    its = max(1.0, (1.42 if op == "mpir" else 0.72) * n ** (1.0 / 3.0))
    # Two preconditioner applications and products, and the vector updates.
    return {"bytes": its * (2 * pre["bytes"] + 2 * spmv["bytes"] + 16 * v * n),
            "flops": its * (2 * pre["flops"] + 2 * spmv["flops"] + 20 * n)}


# -- the same in 64 bits -----------------------------------------------------

class _System:
    """The matrix in tile order as padded rows of (column, value) on the GPU,
    float64: cols and vals [n, K] sorted by column (n: padding), diag [n],
    tile [n]."""

    def __init__(self, h, dtype):
        dev = "cuda"
        n = h.numRows
        rp, col, off, dg = (torch.from_numpy(v).to(dev) for v in h.globalCrs())
        if dtype == "float32":
            off, dg = off.float().double(), dg.float().double()
        ids = torch.from_numpy(h.decomposeVector(np.arange(n, dtype=np.float64), gb.FLOAT64)).to(dev).long()
        pos = torch.empty_like(ids)
        pos[ids] = torch.arange(n, device=dev)
        self.n, self.ids = n, ids
        self.tile = torch.from_numpy(h.rowToTile()).to(dev).long()[ids]
        self.diag = dg[ids]
        length = (rp[1:] - rp[:-1])
        K = max(1, int(length.max()))
        at = torch.arange(K, device=dev)
        src = rp[:-1][ids][:, None] + at[None, :]
        real = at[None, :] < length[ids][:, None]
        src = torch.where(real, src, torch.zeros_like(src)).clamp_(max=max(0, col.numel() - 1))
        self.cols = torch.where(real, pos[col[src]], torch.full_like(src, n))
        self.vals = torch.where(real, off[src], torch.zeros((), dtype=torch.float64, device=dev))
        self.cols, order = self.cols.sort(dim=1)
        self.vals = torch.gather(self.vals, 1, order)
        rows = torch.arange(n, device=dev)[:, None]
        tile = torch.cat([self.tile, self.tile.new_full((1,), -1)])
        own = tile[self.cols] == self.tile[:, None]
        self.lower, self.upper = own & (self.cols < rows), own & (self.cols > rows)

    def gather(self, x):
        return torch.cat([x, x.new_zeros(1)])[self.cols]

    def product(self, x):
        return self.diag * x + (self.vals * self.gather(x)).sum(1)

    def levels(self, mask):
        """Rows in an order of rounds in which each row's masked columns come
        in earlier rounds."""
        lev = torch.zeros(self.n, dtype=torch.long, device=self.cols.device)
        while True:
            new = torch.where(mask, torch.cat([lev, lev.new_zeros(1)])[self.cols] + 1, 0).amax(1)
            if torch.equal(new, lev):
                break
            lev = new
        order = lev.argsort(stable=True)
        return torch.split(order, torch.bincount(lev).tolist())


def _ilu(S, b):
    n, K = S.n, S.cols.shape[1]
    F = torch.where(S.lower | S.upper, S.vals, 0.0)
    F = torch.cat([F, F.new_zeros(1, K)])
    cols = torch.cat([S.cols, S.cols.new_full((1, K), n)])
    D = torch.cat([S.diag, S.diag.new_ones(1)])
    down = S.levels(S.lower)
    for rows in down:
        for s in range(K):
            on = S.lower[rows, s]
            r = rows[on]
            if not len(r):
                continue
            k = cols[r, s]
            a = F[r, s] / D[k]
            F[r, s] = a
            # a[k, j] for every later column j of the row, and for j = row
            for t in range(s + 1, K):
                j = torch.where(S.lower[r, t] | S.upper[r, t], cols[r, t], -1)
                F[r, t] -= a * (F[k] * (cols[k] == j[:, None])).sum(1)
            D[r] -= a * (F[k] * (cols[k] == r[:, None])).sum(1)
    y = torch.cat([b, b.new_zeros(1)])
    L, U = torch.where(S.lower, F[:n], 0.0), torch.where(S.upper, F[:n], 0.0)
    for rows in down:
        y[rows] -= (L[rows] * y[cols[rows]]).sum(1)
    for rows in S.levels(S.upper):
        y[rows] = (y[rows] - (U[rows] * y[cols[rows]]).sum(1)) / D[rows]
    return y[:n]


def _gauss_seidel(S, x, b):
    down = S.levels(S.lower)
    for _ in range(_SWEEPS):
        old = b - torch.where(S.lower, 0.0, S.vals * S.gather(x)).sum(1)
        y = torch.cat([x, x.new_zeros(1)])
        for rows in down:
            L = torch.where(S.lower[rows], S.vals[rows] * y[S.cols[rows]], 0.0).sum(1)
            y[rows] = (old[rows] - L) / S.diag[rows]
        x = y[:-1]
    return x


def _solution(S, b, symmetric, rounds=12000):
    """A x = b with Jacobi-preconditioned conjugate gradients, or BiCGStab
    for a nonsymmetric A, to a relative residual of 1e-14; None when that is
    not reached."""
    x, r = torch.zeros_like(b), b.clone()
    goal = 1e-14 * torch.linalg.vector_norm(b)
    if symmetric:
        z = r / S.diag
        p, rz = z.clone(), torch.dot(r, z)
        for i in range(rounds):
            q = S.product(p)
            a = rz / torch.dot(p, q)
            x += a * p
            r -= a * q
            if i % 25 == 24 and torch.linalg.vector_norm(r) < goal:
                return x
            z = r / S.diag
            rz, was = torch.dot(r, z), rz
            p = z + (rz / was) * p
        return None
    r0, p, rho = r.clone(), r.clone(), torch.dot(r, r)
    for i in range(rounds):
        y = p / S.diag
        v = S.product(y)
        a = rho / torch.dot(r0, v)
        s = r - a * v
        z = s / S.diag
        t = S.product(z)
        w = torch.dot(t, s) / torch.dot(t, t)
        x += a * y + w * z
        r = s - w * t
        if torch.linalg.vector_norm(r) < goal:
            return x
        rho, was = torch.dot(r0, r), rho
        p = r + (rho / was) * (a / w) * (p - w * v)
    return None


def exact(case, seed):
    op, kind = case["op"], case["kind"]
    if op == "batch":
        hosts = _batch_hosts(case, seed)
        out = []
        for h, b in zip(hosts, _batch_rhs(case, hosts, seed)):
            S = _System(h, case["dtype"])
            x = _solution(S, torch.from_numpy(b).cuda().double()[S.ids], True)
            if x is None:
                out.append(None)
                continue
            natural = torch.empty_like(x)
            natural[S.ids] = x
            out.append(natural.cpu().numpy())
        return out
    state = prepare(case, seed)
    S = _System(_host(case, seed), case["dtype"])
    if op == "spmv":
        return S.product(state["x"].double())
    if op == "residual":
        return state["b"].double() - S.product(state["x"])
    b = state["b"].double()
    if op in ("ilu", "factor"):
        return _ilu(S, b)
    if op == "gs":
        return _gauss_seidel(S, state["x0"].double(), b)
    return _solution(S, b, kind != "convdiff")
