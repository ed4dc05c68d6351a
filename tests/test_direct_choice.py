"""The automatic choice between the direct sweeps and the other kernels
(directShape, direct.cpp): the shape it gives for matrices on each side of its
lines, and what solvers then run."""
import ctypes as C
import subprocess
import sys

import pytest

import graphene_b200 as gb

ILU, GS = 0, 1
F32, F64 = gb.FLOAT32, gb.FLOAT64
B200 = (148, 233472)


def shape(h, sweep, coef, vec, sms=B200[0]):
    w, d = C.c_int32(), C.c_int32()
    gb._lib.check(gb._lib.lib().gr_host_matrix_direct_shape(h._h, sweep, coef, vec, sms, B200[1], C.byref(w),
                                                            C.byref(d)))
    return w.value, d.value


def grid(n, tiles):
    return gb.generate3DPoissonMatrix(F32, n, n, n, tiles, gb.PART_RCB)


def mesh(n, tiles):
    return gb.generateLduMesh(n, n, n, numTiles=tiles, partitioner=gb.PART_RCB)


# Where the level rings measured faster (figures at directShape) they are
# taken: (matrix, sweep, coefficients, vectors).
@pytest.mark.parametrize("make,sweep,coef,vec", [
    (lambda: grid(96, 432), GS, F64, F64),
    (lambda: grid(80, 400), GS, F64, F64),
    (lambda: grid(80, 256), GS, F64, F64),
    (lambda: mesh(80, 400), GS, F64, F64),
    (lambda: mesh(40, 64), GS, F64, F64),
    (lambda: gb.generate3DPoissonMatrix(F32, 109, 80, 107, 931, gb.PART_RCB), GS, F64, F64),
    (lambda: grid(96, 560), ILU, F64, F64),
    (lambda: grid(112, 300), ILU, F64, F64),
    (lambda: gb.generate3DPoissonMatrix(F32, 101, 122, 116, 599, gb.PART_RCB), ILU, F64, F64),
    (lambda: grid(112, 300), ILU, F32, F64),
    (lambda: grid(128, 700), ILU, F32, F32),
])
def test_ring_where_it_is_faster(make, sweep, coef, vec):
    assert shape(make(), sweep, coef, vec) == (0, 0)


@pytest.mark.parametrize("make,sweep,coef,vec,want", [
    (lambda: grid(32, 64), ILU, F32, F32, (2, 8)),
    (lambda: grid(64, 64), ILU, F32, F32, (4, 8)),
    (lambda: grid(64, 64), ILU, F32, F64, (4, 8)),
    (lambda: grid(64, 512), ILU, F32, F32, (1, 8)),
    (lambda: grid(112, 300), ILU, F32, F32, (2, 8)),
    (lambda: mesh(80, 256), ILU, F64, F64, (4, 8)),
    (lambda: grid(96, 148), ILU, F64, F64, (4, 8)),
    (lambda: grid(96, 1200), ILU, F64, F64, (1, 4)),
    (lambda: gb.generate3DPoissonMatrix(F32, 130, 107, 112, 609, gb.PART_RCB), ILU, F64, F64, (1, 8)),
    (lambda: grid(64, 64), GS, F32, F32, (4, 4)),
    (lambda: grid(96, 432), GS, F32, F64, (2, 4)),
    (lambda: grid(64, 512), GS, F32, F32, (1, 4)),
    (lambda: grid(64, 1000), GS, F64, F64, (1, 4)),
    (lambda: mesh(60, 64), GS, F64, F64, (4, 4)),
    (lambda: mesh(100, 1024), GS, F64, F64, (1, 4)),
])
def test_direct_where_it_is_faster(make, sweep, coef, vec, want):
    assert shape(make(), sweep, coef, vec) == want


def test_depth_by_waves():
    """Four steps ahead where the tiles then need a wave less."""
    h = grid(96, 592)  # 11 tiles an SM with 8 steps ahead, 15 with 4
    got = {sms: shape(h, ILU, F32, F32, sms) for sms in (54, 45, 36, 27, 20)}
    assert got == {54: (1, 8), 45: (1, 4), 36: (1, 8), 27: (1, 8), 20: (1, 4)}


@pytest.mark.gpu
def test_double_vectors_over_float_coefficients():
    """One solver, float vectors through the direct kernel and double ones
    through the ring: both as the level schedules, also after new values and
    within PBiCGStab's captured iterations."""
    import torch
    h = grid(112, 300)
    A = h.copyToTile()
    s, p = gb.Solver(A, {"type": "ILU"}), gb.Solver(A, {"type": "PBiCGStab", "maxIterations": 4,
                                                      "preconditioner": {"type": "ILU"}})
    assert s.sweepKernel(F32) == "direct 2x8 factor" and s.sweepKernel(F64) == "ring"
    assert p.sweepKernel(F64) == "ring"
    g = torch.Generator().manual_seed(7)
    b = torch.rand(h.numRows, generator=g, dtype=torch.float64).mul(2).sub(1).cuda()
    rp, col, off, dg = h.globalCrs()
    for scale in (1.0, 1.25):
        A.updateGlobalValues(off * scale, dg)
        s.refresh()
        p.refresh()
        for dt in (torch.float64, torch.float32, torch.float64):
            want, got = (torch.zeros(h.numRows, dtype=dt, device="cuda") for _ in range(2))
            gb.Solver(A, {"type": "ILU", "kernel": "levels"}).solve(want, b.to(dt))
            s.solve(got, b.to(dt))
            assert torch.equal(got, want)
            want.zero_()
            got.zero_()
            gb.Solver(A, {"type": "PBiCGStab", "maxIterations": 4,
                          "preconditioner": {"type": "ILU", "kernel": "levels"}}).solve(want, b.to(dt))
            p.solve(got, b.to(dt))
            assert torch.equal(got, want)
    assert s.sweepKernel(F64) == "ring"


@pytest.mark.gpu
def test_no_tables_for_a_sweep_that_does_not_fit():
    """Tiles whose step tables outgrow shared memory: the matrix keeps no
    direct tables (about 125 MB here) beside what the automatic choice makes
    when an option of the ring kernel rules them out."""
    import torch
    from cuda.bindings import runtime
    torch.cuda.init()
    pool = runtime.cudaDeviceGetDefaultMemPool(0)[1]
    h = gb.generate3DPoissonMatrix(F32, 256000, 1, 1, 16, gb.PART_CONTIGUOUS)

    def held(cfg):
        A = h.copyToTile()
        before = int(runtime.cudaMemPoolGetAttribute(pool, runtime.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)[1])
        s = gb.Solver(A, cfg)
        after = int(runtime.cudaMemPoolGetAttribute(pool, runtime.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)[1])
        return after - before, s.sweepKernel(F32), A, s

    auto = held({"type": "ILU"})
    assert not auto[1].startswith("direct")
    same = held({"type": "ILU", "tilesPerBlock": 1})
    assert same[1] == auto[1]
    assert auto[0] - same[0] < 8 << 20


FOOTPRINT = """
import sys
import numpy as np
import torch
from cuda.bindings import runtime
import graphene_b200 as gb
torch.cuda.init()
pool = runtime.cudaDeviceGetDefaultMemPool(0)[1]
def held():
    return int(runtime.cudaMemPoolGetAttribute(pool, runtime.cudaMemPoolAttr.cudaMemPoolAttrUsedMemCurrent)[1])
nx, ny, tiles, t = map(int, sys.argv[1:5])
h = gb.generate3DPoissonMatrix(t, nx, ny, 1, tiles, gb.PART_CONTIGUOUS)
cfg = {"type": "PBiCGStab", "maxIterations": 2, "preconditioner": {"type": "ILU"}}
dt = np.float64 if t or len(sys.argv) > 5 else np.float32
before = held()
A = h.copyToTile()
s = gb.Solver(A, cfg)
s.solveHost(np.zeros(h.numRows, dt), np.ones(h.numRows, dt))
used = held() - before
assert s.sweepKernel(t).startswith("direct")
srv = gb.Server(slots=1)
print(used, srv.wait(srv.submit(h, cfg, np.ones(h.numRows, dt)))[2]["footprint_bytes"])
srv.close()
"""


@pytest.mark.gpu
@pytest.mark.parametrize("args", [("65536", "1", "64", "0"), ("65536", "1", "64", "1"), ("20000", "3", "100", "0"),
                                  ("20000", "3", "100", "0", "double"), ("300", "300", "60", "1")])
def test_server_admits_by_no_less_than_a_pair_holds(args):
    """Narrow levels, each padded to eight records: what the matrix and its
    solver hold (in a process of its own, with no blocks kept from before)
    stays within the estimate that the server admits by."""
    out = subprocess.run([sys.executable, "-c", FOOTPRINT, *args], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    used, estimate = map(int, out.stdout.split())
    assert 0 < used <= estimate


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [F32, F64])
@pytest.mark.parametrize("dims,tiles,factor", [((3000, 1, 1), 2, True), ((6000, 1, 1), 300, False),
                                               ((16, 16, 16), 1, True), ((40, 38, 3), 7, True)])
def test_packing_of_narrow_and_wide_steps(dims, tiles, factor, dtype):
    """Several blocks a tile, eight lanes or a warp a step, chains with and
    without the fused factorisation: as the level schedules, bit for bit, also
    after new values."""
    import torch
    h = gb.generate3DPoissonMatrix(dtype, *dims, tiles, gb.PART_CONTIGUOUS)
    A = h.copyToTile()
    dt = torch.float64 if dtype == F64 else torch.float32
    b = torch.linspace(-1, 1, h.numRows, dtype=dt, device="cuda")
    rp, col, off, dg = h.globalCrs()
    ilu, gs = {"type": "ILU"}, {"type": "GaussSeidel", "numFixedIterations": 2}
    solvers = [gb.Solver(A, c) for c in (ilu, gs)]
    assert solvers[0].sweepKernel(dtype).endswith("factor") == factor
    for scale in (1.0, 1.5):
        A.updateGlobalValues(off * scale, dg * 2)
        for c, s in zip((ilu, gs), solvers):
            s.refresh()
            got, want = torch.ones_like(b), torch.ones_like(b)
            s.solve(got, b)
            gb.Solver(A, {**c, "kernel": "levels"}).solve(want, b)
            assert torch.equal(got, want)


@pytest.mark.gpu
def test_refresh_of_long_chains():
    """New values in a Gauss-Seidel solver of few tiles and many narrow levels
    take tens of microseconds (a block a tile took a millisecond)."""
    import time
    h = gb.generate3DPoissonMatrix(F32, 65536, 1, 1, 16, gb.PART_CONTIGUOUS)
    s = gb.Solver(h.copyToTile(), {"type": "GaussSeidel", "numFixedIterations": 1})
    assert s.sweepKernel() == "direct 4x4"
    best = 1.0
    for _ in range(10):
        t0 = time.perf_counter()
        s.refresh()
        best = min(best, time.perf_counter() - t0)
    assert best < 3e-4


# Every shape the ILU rule can give, each at its smallest matrix or nearly so.
SHAPES = {
    "direct 2x8": (lambda: grid(24, 27), F32),
    "direct 4x8": (lambda: grid(32, 8), F32),
    "direct 1x8": (lambda: gb.generate3DPoissonMatrix(F32, 29, 28, 27, 330, gb.PART_RCB), F32),
    "direct 1x4": (lambda: gb.generate3DPoissonMatrix(F32, 36, 35, 34, 2900, gb.PART_RCB), F32),
    "direct 2x4": (lambda: mesh(100, 800), F64),
    "direct 4x4": (lambda: grid(96, 160), F64),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(SHAPES))
def test_every_ilu_shape(name):
    """Taken, and as the level schedules, in either type of vectors."""
    import torch
    make, coef = SHAPES[name]
    h = make() if coef == F32 else make().astype(coef)
    A = h.copyToTile()
    n = h.numRows
    g = torch.Generator().manual_seed(9)
    b64 = torch.rand(n + 1, generator=g, dtype=torch.float64).mul(2).sub(1).cuda()
    for cfg in ({"type": "ILU"}, {"type": "ILU", "diagonalBased": True}):
        s, want = gb.Solver(A, cfg), gb.Solver(A, {**cfg, "kernel": "levels"})
        assert s.sweepKernel(coef) == name + " factor"
        for dt in (torch.float32, torch.float64)[0 if coef == F32 else 1:]:
            for off in (0, 1):  # the second: not 16-byte aligned
                b = b64.to(dt)[off:off + n]
                x, y = (torch.zeros(n + 1, dtype=dt, device="cuda")[off:off + n] for _ in range(2))
                s.solve(x, b)
                want.solve(y, b)
                assert torch.equal(x, y)
