"""The two FDM line-solve kernels against each other: the substitution with the
stored factor (the plain call) and the elimination inside the application (a
captured call, which must not depend on the stored factor), and the stored
factor after a change of the stage coefficients."""
import numpy as np
import pytest

from oracle import bspline as ob
from tests.cases import product_of


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [False, True])
@pytest.mark.parametrize("p,nel_y", [(2, 1), (2, 17), (3, 2), (3, 16), (3, 45), (4, 1), (4, 13), (4, 30), (5, 16), (5, 31)])
def test_stored_factor_and_elimination(cuda, p, nel_y, cap):
    import torch
    from tdsez_gb300.propagator import Solver
    nel_x, Lx, Ly = 37 + p, 20.0, 0.5 * nel_y + 8.0
    c = dict(knots=[ob.uniform_knots(nel_x, -Lx, Lx, p), ob.uniform_knots(nel_y, -Ly, Ly, p)], p=p, nq=p + 1,
             charge=-1.0, mass=1.0, V=[lambda x: 0.05 * x, lambda y: 0.02 * y * y], coupled=(1,))
    if cap:
        c.update(cap_kmin=1.0, bounds=[(-Lx, Lx), (-Ly, Ly)])
    S, op = product_of(c)
    rng = np.random.default_rng(10 * p + nel_y)
    b = torch.tensor(rng.standard_normal(S.ndof) + 1j * rng.standard_normal(S.ndof), device=cuda)
    op.set_stage(1.0, 0.05j, [0.03])
    s = Solver(op, pc="fdm", precision="fp32", rtol=1e-12, maxit=30)
    z = {}
    for g in (0.05j, 0.02j, 0.05j):   # the factor of one stage must not serve another
        op.set_stage(1.0, g, [0.03])
        plain, captured = torch.empty_like(b), torch.empty_like(b)
        s.precondition(b, plain)
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):
            s.precondition(b, captured)
        graph.replay()
        torch.cuda.synchronize()
        # Two FP32 eliminations of systems of condition below 1e3 (1e4 with the
        # eigenvectors of complex pencils), 60 roundings per row: the bar of
        # the comparison with the FP64 solve, and ten times that
        tol = 1e-3 if cap else 1e-4
        assert torch.linalg.norm(plain - captured) < tol * torch.linalg.norm(captured)
        if g in z:
            assert torch.equal(plain, z[g])
        z[g] = plain
    assert torch.linalg.norm(z[0.02j] - z[0.05j]) > 1e-2 * torch.linalg.norm(z[0.05j])
