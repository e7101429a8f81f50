"""The FDM line solves at their edges: lines from the shortest axis (one
element) through both sides of a block boundary of the two halves, line
counts off the 64-line blocks, real and complex axis pencils."""
import numpy as np
import pytest
import scipy.sparse.linalg as sla

from oracle import bspline as ob
from tests.cases import oracle_of, product_of


@pytest.mark.gpu
@pytest.mark.parametrize("cap", [False, True])
@pytest.mark.parametrize("p,nel_y", [(2, 1), (2, 14), (2, 15), (3, 1), (3, 3), (3, 15), (3, 16), (3, 33), (4, 1),
                                     (4, 12), (4, 13), (4, 29), (5, 1), (5, 15), (5, 16), (5, 35)])
def test_line_solve_edges(cuda, p, nel_y, cap):
    import torch
    from tdsez_gb300.propagator import Solver
    nel_x, Lx, Ly = 61 + p, 30.0, 0.5 * nel_y + 8.0
    c = dict(knots=[ob.uniform_knots(nel_x, -Lx, Lx, p), ob.uniform_knots(nel_y, -Ly, Ly, p)], p=p, nq=p + 1,
             charge=-1.0, mass=1.0, V=[lambda x: 0.05 * x, lambda y: 0.02 * y * y], coupled=(1,))
    if cap:
        c.update(cap_kmin=1.0, bounds=[(-Lx, Lx), (-Ly, Ly)])
    S, ph, A = oracle_of(c)
    PS, op = product_of(c)
    g = 0.05j
    op.set_stage(1.0, g, [0.03])
    Am = (A.M + g * (A.H_total() + 0.03 * A.terms()[0])).tocsc()
    rng = np.random.default_rng(100 * p + nel_y)
    b = rng.standard_normal(S.ndof) + 1j * rng.standard_normal(S.ndof)
    xref = sla.spsolve(Am, b)
    s = Solver(op, pc="fdm", precision="fp32", rtol=1e-12, maxit=30)
    bd = torch.tensor(b, device=cuda)
    zd = torch.empty_like(bd)
    s.precondition(bd, zd)
    # FP32 arithmetic on systems of condition below 1e3 (the bar of the longer lines' test);
    # complex pencils add the condition of their eigenvectors, so there FGMRES decides
    if not cap:
        assert np.linalg.norm(zd.cpu().numpy() - xref) < 1e-4 * np.linalg.norm(xref)
    xd = torch.zeros_like(bd)
    its, reason, rn = s.solve(bd, xd)
    assert reason > 0 and its <= 4, (its, reason, rn)
    assert np.linalg.norm(xd.cpu().numpy() - xref) < 1e-9 * np.linalg.norm(xref)
