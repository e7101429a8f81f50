"""The native FP64 3D apply with inner-axis terms on both sides of the rule that
skips tile rows past the grid: grids of a few rows, tiles two fifths empty and a
little less, full ones, against products of sparse 1D matrices in FP64."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import bspline as ob
from tests.cases import product_of

V = [lambda x: 0.05 * x * x, lambda y: 0.1 * y, lambda z: 0.02 * z]


def _apply(axes, mats, x):
    """The product of one 1D matrix per axis (x, y, z) and the vector, x fastest."""
    u = x.reshape([a["M"].shape[0] for a in reversed(axes)])
    for k, m in enumerate(mats):
        u = np.moveaxis(u, 2 - k, 0)
        u = np.moveaxis((m @ u.reshape(u.shape[0], -1)).reshape(u.shape), 0, 2 - k)
    return u.reshape(-1)


def stage(knots, p, mass, alpha, g, fields, x):
    axes = []
    for kn, v in zip(knots, V):
        a = ob.Axis(kn, p, p + 1)
        N, D, w, q = a.basis_matrix(0), a.basis_matrix(1), a.wq.reshape(-1), a.xq.reshape(-1)
        form = lambda B, f: sp.csr_matrix(B.T @ sp.diags(w * f) @ B)   # noqa: E731
        axes.append({"M": form(N, 1.0 + 0 * q), "H": form(D, 0.5 / mass + 0 * q) + form(N, v(q)), "X": form(N, q)})
    y = alpha * _apply(axes, [a["M"] for a in axes], x)
    for k in range(3):   # charge -1: + field times position
        m = [a["M"] for a in axes]
        m[k] = axes[k]["H"] + fields[k] * axes[k]["X"]
        y = y + g * _apply(axes, m, x)
    return y


@pytest.mark.gpu
@pytest.mark.parametrize("p,ny", [(2, 1), (2, 14), (2, 15), (3, 1), (3, 6), (3, 7), (3, 13), (3, 16), (3, 17), (4, 5),
                                  (4, 6), (4, 15), (4, 28), (5, 4), (5, 5), (5, 14), (5, 15)])
def test_rows_past_the_grid(cuda, p, ny):
    import torch
    from tdsez_gb300 import _lib
    kn = [ob.uniform_knots(n, -8.0 - d, 8.0 + d, p) for d, n in enumerate((9, ny, 11))]
    c = dict(knots=kn, p=p, nq=p + 1, charge=-1.0, mass=0.5, coupled=(0, 1, 2), V=V)
    PS, op = product_of(c)
    rng = np.random.default_rng(10 * p + ny)
    x = rng.standard_normal(PS.ndof) + 1j * rng.standard_normal(PS.ndof)
    alpha, g, cc = 1.0 + 0.1j, 0.02 + 0.3j, [0.03, -0.02, 0.01]
    op.set_stage(alpha, g, cc)
    want = stage(kn, p, 0.5, alpha, g, cc, x)
    xd = torch.tensor(x, device=cuda)
    yd = torch.full_like(xd, float("nan"))
    op.apply(_lib.TDZ_STAGE, xd, yd)
    assert np.abs(yd.cpu().numpy() - want).max() < 1e-12 * np.abs(want).max()   # the bar of the apply parity tests
