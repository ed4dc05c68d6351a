"""The direct sweeps (kernels_direct.cu): their row records and step tables,
replayed on the host over the matrices they accept."""
import ctypes as C

import numpy as np
import pytest

import graphene_b200 as gb

ILU, GS, GS_ZERO = 0, 1, 2


def check_direct(h, sweep, dilu=False, warps=2):
    st, sec, ip = C.c_int32(), C.c_int32(), C.c_int32()
    gb._lib.check(gb._lib.lib().gr_host_matrix_check_direct(h._h, sweep, int(dilu), warps, C.byref(st), C.byref(sec),
                                                            C.byref(ip)))
    return st.value, bool(sec.value), bool(ip.value)


def sparse_coo(n, per_row, seed, symmetric):
    """A random pattern of at most six off-diagonals a row."""
    rng = np.random.default_rng(seed)
    count = np.zeros(n, int)
    pairs = set()
    for i in range(n):
        for j in rng.integers(max(0, i - 60), min(n, i + 60), per_row):
            new = [(i, j), (j, i)] if symmetric else [(i, j)]
            if i == j or any(q in pairs or count[q[0]] >= 6 for q in new):
                continue
            pairs.update(new)
            for a, _ in new:
                count[a] += 1
    r, c = np.array(sorted(pairs)).T
    rows = np.concatenate([r, np.arange(n)])
    return n, rows, np.concatenate([c, np.arange(n)]), np.concatenate([rng.uniform(-1, 1, len(r)),
                                                                        rng.uniform(8, 16, n)])


@pytest.mark.parametrize("dims,tiles,part", [
    ((16, 16, 16), 8, gb.PART_RCB),
    ((13, 11, 7), 6, gb.PART_BFS),
    ((12, 10, 8), 1, gb.PART_AUTO),
    ((20, 20, 20), 200, gb.PART_RCB),
    ((5, 4, 3), 60, gb.PART_RCB),
    ((33, 17, 9), 5, gb.PART_CONTIGUOUS),
    ((1, 1, 1), 1, gb.PART_AUTO),
])
@pytest.mark.parametrize("warps", [1, 2, 4])
def test_replay_grids(dims, tiles, part, warps):
    h = gb.generate3DPoissonMatrix(gb.FLOAT32, *dims, tiles, part)
    for sweep in (ILU, GS, GS_ZERO):
        for dilu in (False, True):
            steps, _, in_place = check_direct(h, sweep, dilu, warps)
            assert steps >= 1
            assert in_place == (sweep != ILU)


@pytest.mark.parametrize("seed", [0, 1, 2])
@pytest.mark.parametrize("symmetric,tiles", [(True, 7), (True, 1), (False, 1)])
def test_replay_unstructured(seed, symmetric, tiles):
    coo = sparse_coo(500, 2 if symmetric else 5, seed, symmetric)
    h = gb.HostMatrix.from_coo(*coo, tiles, partitioner=gb.PART_BFS if tiles > 1 else gb.PART_AUTO)
    assert check_direct(h, ILU)[1]
    check_direct(h, ILU, True, 1)
    check_direct(h, GS_ZERO, False, 4)
    mesh = gb.generateLduMesh(9, 8, 7, numTiles=5, partitioner=gb.PART_RCB)
    for sweep in (ILU, GS, GS_ZERO):
        assert check_direct(mesh, sweep, False, 1 + seed % 2)[1]


def test_long_rows_and_warps_are_refused():
    n, per = 64, 20
    rows = np.repeat(np.arange(n), per)
    cols = (rows + 1 + np.tile(np.arange(per), n)) % n
    keep = np.concatenate([rows, cols, np.arange(n)]), np.concatenate([cols, rows, np.arange(n)])
    uniq = np.unique(np.stack(keep), axis=1)
    h = gb.HostMatrix.from_coo(n, uniq[0], uniq[1], np.ones(uniq.shape[1]), 1)
    for sweep in (ILU, GS, GS_ZERO):
        with pytest.raises(gb.GrapheneError):
            check_direct(h, sweep)
    p = gb.generate3DPoissonMatrix(gb.FLOAT32, 4, 4, 4, 1)
    for warps in (0, 3, 5):
        with pytest.raises(gb.GrapheneError):
            check_direct(p, ILU, False, warps)


# ---- on the GPU: the automatic kernel against the level schedules ----------------------

def _systems():
    """Sizes on each side of the shapes directShape picks from: tiles an SM
    (below 1, 2, 4, above), rows a level, tiles of a single row, rows of one
    to six entries, one tile, ragged last tiles."""
    mesh = gb.generateLduMesh
    pois = gb.generate3DPoissonMatrix
    yield "one_row_tiles", lambda: pois(gb.FLOAT32, 5, 4, 3, 60, gb.PART_RCB)
    yield "one_tile", lambda: pois(gb.FLOAT32, 13, 12, 11, 1)
    yield "two_warps", lambda: pois(gb.FLOAT32, 24, 23, 22, 40)
    yield "four_warps", lambda: pois(gb.FLOAT32, 40, 41, 42, 18, gb.PART_RCB)
    yield "some_tiles_an_sm", lambda: pois(gb.FLOAT32, 37, 36, 35, 200, gb.PART_RCB)
    yield "many_tiles_an_sm", lambda: pois(gb.FLOAT32, 33, 32, 31, 700, gb.PART_RCB)
    yield "mesh", lambda: mesh(21, 20, 19, numTiles=23, partitioner=gb.PART_RCB)
    yield "mesh_many", lambda: mesh(29, 28, 27, numTiles=650, partitioner=gb.PART_RCB)
    yield "unstructured", lambda: gb.HostMatrix.from_coo(*sparse_coo(700, 2, 5, True), 9, partitioner=gb.PART_BFS)
    yield "nonsymmetric", lambda: gb.HostMatrix.from_coo(*sparse_coo(600, 5, 6, False), 1)


SYSTEMS = dict(_systems())


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SYSTEMS))
@pytest.mark.parametrize("types", ["f32", "f64", "f32_vec64"])
def test_direct_sweeps_equal_level_schedules(name, types):
    """Same operations in the same order: bit for bit, for vectors aligned to
    16 bytes and not."""
    import torch
    h = SYSTEMS[name]()
    if types == "f64":
        h = h.astype(gb.FLOAT64)
    A = h.copyToTile()
    dt = torch.float32 if types == "f32" else torch.float64
    n = h.numRows
    g = torch.Generator().manual_seed(3)
    b, x0 = (torch.rand(n + 4, generator=g, dtype=torch.float64).mul(2).sub(1).to(dt).cuda() for _ in range(2))
    configs = [{"type": "ILU"}, {"type": "ILU", "diagonalBased": True},
               {"type": "GaussSeidel", "numFixedIterations": 2},
               {"type": "GaussSeidel", "numFixedIterations": 1, "seed": "diag"},
               {"type": "GaussSeidel", "numFixedIterations": 2, "halo": "drop"}]
    for cfg in configs:
        direct, levels = gb.Solver(A, cfg), gb.Solver(A, {**cfg, "kernel": "levels"})
        for off in (0, 1):  # the second: not 16-byte aligned
            got, want = x0.clone()[off:off + n], x0.clone()[off:off + n]
            direct.solve(got, b[off:off + n])
            levels.solve(want, b[off:off + n])
            assert torch.equal(got, want), (cfg, off)
    for pre in ({"type": "ILU"}, {"type": "GaussSeidel", "numFixedIterations": 2}):
        # The fused p / s updates, and sweeps from x = 0.
        xs = []
        for kernel in ({}, {"kernel": "levels"}):
            x = torch.zeros(n, dtype=dt, device="cuda")
            gb.Solver(A, {"type": "PBiCGStab", "maxIterations": 4, "preconditioner": {**pre, **kernel}}).solve(x, b[:n])
            xs.append(x)
        assert torch.equal(*xs), pre


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("dilu", [False, True])
@pytest.mark.parametrize("first_rows", [False, True])
def test_factorisation_of_zeros_and_infinities(dtype, dilu, first_rows):
    """A zero diagonal, signed zeros and overflowing quotients go through the
    factorisation as through the level-scheduled one: the same bits, NaN where
    it has NaN."""
    import torch
    h = gb.generate3DPoissonMatrix(gb.parseType(dtype), 9, 8, 7, 6, gb.PART_RCB)
    rp, col, off, dg = h.globalCrs()
    rng = np.random.default_rng(5)
    off = off * rng.uniform(0.5, 2.0, len(off))
    off[rng.integers(0, len(off), 40)] = -0.0
    off[rng.integers(0, len(off), 10)] = 1e38 if dtype == "float32" else 1e308
    dg = dg.copy()
    dg[rng.integers(0, len(dg), 4)] = 0.0
    dg[rng.integers(0, len(dg), 4)] = 1e-38 if dtype == "float32" else 1e-308
    if first_rows:  # rows that others divide by before anything is subtracted from them
        lower = h.levels()[0]
        natural = h.decomposeVector(np.arange(h.numRows, dtype=np.float64), gb.FLOAT64).astype(int)
        dg[natural[lower == 0][:3]] = 0.0
    A = h.copyToTile()
    A.updateGlobalValues(off, dg)
    b = torch.from_numpy(rng.uniform(-1, 1, h.numRows)).to(getattr(torch, dtype)).cuda()
    got, want = torch.empty_like(b), torch.empty_like(b)
    cfg = {"type": "ILU", "diagonalBased": dilu}
    gb.Solver(A, cfg).solve(got, b)
    gb.Solver(A, {**cfg, "kernel": "levels"}).solve(want, b)
    assert not first_rows or not torch.isfinite(want).all()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got.nan_to_num(1.5), want.nan_to_num(1.5))
