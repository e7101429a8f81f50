"""The native FP64 3D apply with inner-axis terms on both sides of the rule that
skips tile rows past the grid: grids of a few rows, tiles two fifths empty and a
little less, full ones, against the oracle."""
import numpy as np
import pytest

from oracle import bspline as ob
from tests.cases import oracle_of, product_of


@pytest.mark.gpu
@pytest.mark.parametrize("p,ny", [(2, 1), (2, 14), (2, 15), (3, 1), (3, 6), (3, 7), (3, 13), (3, 16), (3, 17), (4, 5),
                                  (4, 6), (4, 15), (4, 28), (5, 4), (5, 5), (5, 14), (5, 15)])
def test_rows_past_the_grid(cuda, p, ny):
    import torch
    from tdsez_gb300 import _lib
    kn = [ob.uniform_knots(n, -8.0 - d, 8.0 + d, p) for d, n in enumerate((9, ny, 11))]
    c = dict(knots=kn, p=p, nq=p + 1, charge=-1.0, mass=0.5, coupled=(0, 1, 2),
             V=[lambda x: 0.05 * x * x, lambda y: 0.1 * y, lambda z: 0.02 * z])
    S, ph, A = oracle_of(c)
    PS, op = product_of(c)
    rng = np.random.default_rng(10 * p + ny)
    x = rng.standard_normal(S.ndof) + 1j * rng.standard_normal(S.ndof)
    alpha, g, cc = 1.0 + 0.1j, 0.02 + 0.3j, [0.03, -0.02, 0.01]
    op.set_stage(alpha, g, cc)
    want = alpha * (A.M @ x) + g * (A.H_total() @ x + sum(ck * (T @ x) for ck, T in zip(cc, A.terms())))
    xd = torch.tensor(x, device=cuda)
    yd = torch.full_like(xd, float("nan"))
    op.apply(_lib.TDZ_STAGE, xd, yd)
    assert np.abs(yd.cpu().numpy() - want).max() < 1e-12 * np.abs(want).max()   # the bar of the apply parity tests
