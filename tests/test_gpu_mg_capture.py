"""The dense matrices of small multigrid levels under stream capture: a captured
V-cycle combines them when its graph runs, so neither recording one nor
replaying one of another stage may leave matrices that a later call takes for
the current stage's."""
import numpy as np
import pytest


def _solver(op):
    from tdsez_gb300.propagator import Solver
    # a degree-2 coarsest polynomial: its error depends on the stage's matrices.
    # One batch is trained, only to open coarse_gain()
    s = Solver(op, pc="mg", precision="fp32", rtol=1e-10, mg_coarse_its=2, mg_learned=True)
    s.train_coarse(pairs=8, epochs=1, lr=1e-3, seed=3)
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["record", "replay"])
def test_captured_vcycle_leaves_no_matrices(cuda, order):
    import torch
    from tdsez_gb300.operators import Operator
    from tdsez_gb300.space import Space
    from tdsez_gb300.workloads import heterostructure
    w = heterostructure(nel=(16, 16, 32))
    S = Space(w.knots, w.p, w.nq)
    op = Operator(S, w.phys)
    # the field's weight in the matrices differs (0.15 Ha at the ends of the box)
    a, b = (1.0, 0.25j, [0.0]), (1.0, 0.25j, [0.0005])
    op.set_stage(*a)
    s0, s = _solver(op), _solver(op)
    op.set_stage(*b)
    want = s0.coarse_gain(trials=4, seed=9)[0]
    op.set_stage(*a)
    rng = np.random.default_rng(4)
    r = torch.tensor(rng.standard_normal(S.ndof) + 1j * rng.standard_normal(S.ndof), device=cuda)
    z, zc = torch.empty_like(r), torch.empty_like(r)
    s.precondition(r, z)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    if order == "record":      # stage a applied, stage b recorded but not run
        op.set_stage(*b)
        with torch.cuda.graph(graph):
            s.precondition(r, zc)
    else:                      # stage a recorded, b applied, a replayed
        with torch.cuda.graph(graph):
            s.precondition(r, zc)
        op.set_stage(*b)
        s.precondition(r, torch.empty_like(r))
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.linalg.norm(zc - z) <= 1e-5 * torch.linalg.norm(z)   # FP32 products, the same launches
    # the same Chebyshev steps on the same right-hand sides: equal but for the
    # FP32 rounding of another run, far below the effect of the stage
    assert abs(s.coarse_gain(trials=4, seed=9)[0] - want) <= 1e-4 * want
