"""The soft-core term's kernels at their edges: the 2D stencil on grids around
its 32 x 8 tiles, with interface knots, other Gauss rules and two centres; the
3D column kernel on tiles of one to nine elements and several z chunks. The
library's H with and without the centres differ by the term, which the test
forms by dense quadrature."""
import numpy as np
import pytest

from oracle import bspline as ob

CENTRES = [(1.0, 0.3, -0.4, 0.2, 0.7), (0.5, -2.0, 1.0, -1.0, 1.5)]


def _term(knots, p, nq, centres, x):
    """V_q x by interpolation to every Gauss point and back (FP64)."""
    ax = [ob.Axis(k, p, nq) for k in knots]
    N = [np.asarray(a.basis_matrix().todense()) for a in ax]
    f = x.reshape([a.n for a in reversed(ax)])
    dim = len(ax)
    for d in range(dim):
        f = np.moveaxis(np.tensordot(N[d], f, axes=(1, dim - 1 - d)), 0, dim - 1 - d)
    pts = np.meshgrid(*[a.xq.ravel() for a in reversed(ax)], indexing="ij")[::-1]
    w = 1.0
    for m in np.meshgrid(*[a.wq.ravel() for a in reversed(ax)], indexing="ij"):
        w = w * m
    v = sum(-c[0] / np.sqrt(sum((pts[d] - c[1 + d]) ** 2 for d in range(dim)) + c[4]) for c in centres)
    f = f * w * v
    for d in range(dim):
        f = np.moveaxis(np.tensordot(N[d].T, f, axes=(1, dim - 1 - d)), 0, dim - 1 - d)
    return f.reshape(-1)


def _check(knots, p, nq, dtype, tol, cuda):
    import torch
    from tdsez_gb300 import _lib
    from tdsez_gb300.operators import Operator, Physics
    from tdsez_gb300.space import Space
    cs = CENTRES if len(knots) == 3 else [(z, a, b, 0.0, s) for z, a, b, _, s in CENTRES]
    out = []
    for soft in ((), cs):
        S = Space(knots, p, nq)
        op = Operator(S, Physics(charge=-1.0, coupled=(), softcore=soft))
        rng = np.random.default_rng(S.ndof)
        x = rng.standard_normal(S.ndof) + 1j * rng.standard_normal(S.ndof)
        op.set_stage(0.0, 0.3 + 0.7j, [])
        xd = torch.tensor(x, dtype=dtype, device=cuda)
        yd = torch.empty_like(xd)
        op.apply(_lib.TDZ_STAGE, xd, yd)
        out.append(yd.cpu().numpy())
    want = (0.3 + 0.7j) * _term(knots, p, nq, cs, x)
    # the bars of the apply parity tests, on the scale of the whole operator
    assert np.abs(out[1] - out[0] - want).max() < 2 * tol * max(np.abs(out[1]).max(), np.abs(want).max())


@pytest.mark.gpu
@pytest.mark.parametrize("p,nel,nq", [(2, (1, 1), 3), (2, (30, 6), 3), (3, (29, 13), 4), (3, (30, 14), 6),
                                      (4, (28, 5), 5), (5, (27, 3), 2), (5, (60, 12), 6)])
@pytest.mark.parametrize("interface", [False, True])
def test_stencil_2d_edges(cuda, p, nel, nq, interface):
    import torch
    if interface and min(nel) > 2:
        kn = [ob.interface_knots(-8.0, 8.0, n, p, [0.5, 3.0]) for n in nel]
    else:
        kn = [ob.uniform_knots(n, -8.0, 8.0, p) for n in nel]
    _check(kn, p, nq, torch.complex128, 1e-12, cuda)
    _check(kn, p, nq, torch.complex64, 1e-6, cuda)


@pytest.mark.gpu
@pytest.mark.parametrize("p,nel", [(2, (1, 8, 3)), (2, (9, 7, 40)), (3, (8, 9, 1)), (3, (7, 1, 33)), (4, (8, 8, 9)),
                                   (4, (9, 2, 30)), (5, (8, 3, 9)), (5, (1, 9, 8))])
def test_columns_3d_edges(cuda, p, nel):
    import torch
    kn = [ob.uniform_knots(n, -6.0, 6.0, p) for n in nel]
    _check(kn, p, p + 1, torch.complex64, 1e-6, cuda)
