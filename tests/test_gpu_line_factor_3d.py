"""The stored line factor on row-planar buffers (3D, tensor-core transforms):
substitution (the plain call) against the elimination inside the application (a
captured call), for line counts off the CTAs' 32 lines, row pitches with padding
and lines from a few rows up."""
import numpy as np
import pytest

from tests.cases import product_of
from tests.test_gpu_mg_dense import _case


@pytest.mark.gpu
@pytest.mark.parametrize("p,nel", [(2, (1, 1, 6)), (2, (9, 14, 33)), (3, (5, 6, 8)), (3, (30, 13, 17)), (3, (17, 29, 60)),
                                   (4, (2, 9, 7)), (4, (21, 12, 41)), (5, (3, 4, 9)), (5, (12, 19, 30))])
def test_stored_factor_planar(cuda, p, nel):
    import torch
    from tdsez_gb300.propagator import Solver
    S, op = product_of(_case("layered", p, nel))
    rng = np.random.default_rng(p + nel[2])
    b = torch.tensor(rng.standard_normal(S.ndof) + 1j * rng.standard_normal(S.ndof), device=cuda)
    op.set_stage(1.0, 0.05j, [0.03])
    s = Solver(op, pc="fdm", precision="fp32", rtol=1e-12, maxit=30)
    for g in (0.05j, 0.02j):
        op.set_stage(1.0, g, [0.03])
        plain, captured = torch.empty_like(b), torch.empty_like(b)
        s.precondition(b, plain)
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            s.precondition(b, captured)
        graph.replay()
        torch.cuda.synchronize()
        # two FP32 eliminations of systems of condition below 1e3: the bar of the 2D test
        assert torch.linalg.norm(plain - captured) < 1e-4 * torch.linalg.norm(captured)
