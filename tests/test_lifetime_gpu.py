"""A solver keeps its device matrix alive: the handles may go in either order,
as when Python's collector finalises a cycle that holds both."""
import gc

import pytest

import graphene_b200 as gb

pytestmark = pytest.mark.gpu

CONFIGS = [{"type": "ILU"}, {"type": "GaussSeidel", "numFixedIterations": 2},
           {"type": "PBiCGStab", "maxIterations": 20, "preconditioner": {"type": "ILU"}}]


@pytest.mark.parametrize("cfg", CONFIGS, ids=[c["type"] for c in CONFIGS])
def test_solver_outlives_its_matrix_handle(cfg):
    import torch
    h = gb.generate3DPoissonMatrix(gb.FLOAT32, 12, 11, 10, 8)
    b = torch.linspace(-1, 1, h.numRows, device="cuda")
    A = h.copyToTile()
    s = gb.Solver(A, cfg)
    want, got = torch.zeros_like(b), torch.zeros_like(b)
    s.solve(want, b)
    A.__del__()
    s.solve(got, b)
    assert torch.equal(got, want)
    s.__del__()
    torch.cuda.synchronize()


def test_collected_in_a_cycle():
    import torch
    for _ in range(4):
        h = gb.generate3DPoissonMatrix(gb.FLOAT32, 9, 8, 7, 4)
        cycle = {"matrix": h.copyToTile()}
        cycle["solver"] = gb.Solver(cycle["matrix"], CONFIGS[2])
        cycle["self"] = cycle
        del cycle, h
        gc.collect()
    x = torch.zeros(504, device="cuda")
    h = gb.generate3DPoissonMatrix(gb.FLOAT32, 9, 8, 7, 4)
    gb.Solver(h.copyToTile(), CONFIGS[0]).solve(x, torch.ones_like(x))
    torch.cuda.synchronize()
