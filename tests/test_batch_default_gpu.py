"""Batches on the automatically chosen preconditioner kernels: the direct
sweeps, whose blocks look up their tile's system and return once it is done.
Every system as alone, and as with the ring kernel, bit for bit."""
import numpy as np
import pytest

import graphene_b200 as gb

pytestmark = pytest.mark.gpu

PRE = {"ILU": {"type": "ILU"}, "DILU": {"type": "ILU", "diagonalBased": True},
       "GS": {"type": "GaussSeidel", "numFixedIterations": 2}}
# Uneven sizes, none a whole number of 32-row chunks but the fifth (the others
# get a tile of padding rows), one that is done early.
SPEC = [(12, 11, 9, 4, 1), (20, 21, 20, 16, 2), (5, 4, 3, 1, 3), (17, 13, 10, 8, 4), (32, 32, 8, 24, 5), (7, 9, 11, 3, 6)]
# Many small systems: more than four tiles an SM, where double Gauss-Seidel
# runs direct too.
MANY = [(9 + k % 5, 8 + k % 7, 10 + k % 3, 12 + k % 4, 50 + k) for k in range(56)]


def hosts(vt, spec):
    return [gb.generateMatrix(gb.GEN_VAR_POISSON, nx, ny, nz, (1.0,), seed, tiles, gb.PART_AUTO, vt)
            for nx, ny, nz, tiles, seed in spec]


def check(hs, cfg, ring, dt, direct, seed):
    bs = [gb.randomVector(seed + k, h.numRows).astype(dt) for k, h in enumerate(hs)]
    t = gb.FLOAT32 if dt == np.float32 else gb.FLOAT64
    B, R = gb.Batch(hs, cfg), gb.Batch(hs, ring)
    assert B.sweepKernel(t).startswith("direct") == direct
    assert R.sweepKernel(t) == "ring"
    (xs, sts), (xr, sr) = B.solveHost(bs), R.solveHost(bs)
    (again, _) = B.solveHost(bs)
    counts = set()
    for h, b, x, y, z, st, rt in zip(hs, bs, xs, xr, again, sts, sr):
        alone = np.zeros(h.numRows, dt)
        sa = gb.Solver(h.copyToTile(), cfg).solveHost(alone, b)
        np.testing.assert_array_equal(x, alone)
        np.testing.assert_array_equal(x, y)
        np.testing.assert_array_equal(x, z)
        assert st.iterations == sa.iterations == rt.iterations
        assert st.innerIterations == sa.innerIterations == rt.innerIterations
        assert st.finalResidual == sa.finalResidual == rt.finalResidual
        assert st.converged and sa.converged
        counts.add((st.iterations, st.innerIterations))
    assert len(counts) > 1  # some systems are done while others run on


def pbicgstab(pre, dt):
    return {"type": "PBiCGStab", "maxIterations": 300, "relTolerance": 1e-5 if dt == np.float32 else 1e-9, "norm": "L2",
            "preconditioner": pre}


@pytest.mark.parametrize("pre", sorted(PRE))
@pytest.mark.parametrize("vt,dt", [(gb.FLOAT32, np.float32), (gb.FLOAT64, np.float64), (gb.FLOAT32, np.float64)])
def test_pbicgstab(pre, vt, dt):
    p = PRE[pre]
    direct = not (pre == "GS" and vt == gb.FLOAT64)
    check(hosts(vt, SPEC), pbicgstab(p, dt), pbicgstab({**p, "kernel": "ring"}, dt), dt, direct, 11)


@pytest.mark.parametrize("pre", ["ILU", "GS"])
@pytest.mark.parametrize("vt,dt", [(gb.FLOAT32, np.float32), (gb.FLOAT64, np.float64)])
def test_many_small_systems(pre, vt, dt):
    p = PRE[pre]
    check(hosts(vt, MANY), pbicgstab(p, dt), pbicgstab({**p, "kernel": "ring"}, dt), dt, True, 300)


@pytest.mark.parametrize("pre", sorted(PRE))
def test_refinement(pre):
    def cfg(p):
        return {"type": "IterativeRefinement", "relResidual": 1e-10, "maxIterations": 30,
                "extendedPrecisionType": "float64",
                "innerSolver": {"type": "PBiCGStab", "maxIterations": 300, "relResidual": 1e-4, "preconditioner": p}}
    p = PRE[pre]
    check(hosts(gb.FLOAT32, SPEC), cfg(p), cfg({**p, "kernel": "ring"}), np.float32, True, 31)


def test_refusal_names_what_a_batch_takes():
    with pytest.raises(gb.GrapheneError, match="automatic or ring kernel"):
        gb.Batch(hosts(gb.FLOAT32, SPEC[:2]), pbicgstab({"type": "ILU", "kernel": "levels"}, np.float32))
