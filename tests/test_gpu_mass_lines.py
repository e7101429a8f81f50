"""The Kronecker inverse of the overlap at the edges of its line tiles: line
counts around the 16-line tiles, the shortest axes, every degree, and axes too
long for a tile in shared memory, against dense FP64 solves."""
import numpy as np
import pytest

from oracle import bspline as ob


@pytest.mark.gpu
@pytest.mark.parametrize("p,nel", [(2, (1, 1, 1)), (3, (13, 14, 15)), (3, (12, 1, 40)), (5, (11, 28, 2)), (4, (40, 3, 9)),
                                   (2, (31, 45)), (5, (1, 27)), (2, (3, 1400)), (7, (100,)), (1, (30,)), (2, (1800,))])
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_mass_solve_edges(cuda, p, nel, prec):
    import torch
    from tdsez_gb300.operators import Operator, Physics
    from tdsez_gb300.space import Space
    kn = [ob.uniform_knots(n, -3.0, 5.0, p) for n in nel]
    op = Operator(Space(kn, p, p + 1), Physics(charge=-1.0, coupled=()))
    shape = [len(k) - p - 1 for k in reversed(kn)]
    rng = np.random.default_rng(sum(nel) + p)
    b = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    want, cond = b, 1.0
    for d, k in enumerate(kn):
        ax = ob.Axis(k, p, p + 1)
        N = np.asarray(ax.basis_matrix().todense())
        M = N.T @ (ax.wq.reshape(-1, 1) * N)
        cond *= np.linalg.cond(M)
        axis = len(nel) - 1 - d
        want = np.moveaxis(np.tensordot(np.linalg.inv(M), want, axes=(1, axis)), 0, axis)
    dt = torch.complex64 if prec == "fp32" else torch.complex128
    x = torch.tensor(b.reshape(-1), dtype=dt, device=cuda)
    op.mass_solve(x)
    err = np.linalg.norm(x.cpu().numpy() - want.reshape(-1)) / np.linalg.norm(want)
    # Cholesky solves of condition kappa per axis: a few eps kappa each
    assert err < 4 * (2.0 ** -24 if prec == "fp32" else 2.0 ** -53) * cond, (err, cond)
