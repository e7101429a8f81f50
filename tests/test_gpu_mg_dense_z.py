"""The z kernel of the dense-axis Chebyshev steps on both sides of its rule: many
columns (16 per CTA, matrices in stages), few columns (8 per CTA, matrices
whole), few columns with an axis too long to hold them whole; last stages and
row groups with remainders."""
import numpy as np
import pytest

from tests.cases import product_of
from tests.test_gpu_mg_dense import _case


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["layered", "const"])
@pytest.mark.parametrize("p,nel", [(2, (36, 34, 21)), (2, (36, 34, 31)), (3, (9, 12, 13)), (2, (10, 9, 140)), (2, (9, 9, 105))])
def test_vcycle_fp32_equals_fp64(cuda, kind, p, nel):
    import torch
    from tdsez_gb300.propagator import Solver
    z = []
    for prec in ("fp32", "fp64"):
        PS, op = product_of(_case(kind, p, nel))
        op.set_stage(1.0, 0.2j, [0.03] * len(op.coupled))
        s = Solver(op, pc="mg", precision=prec, mg_levels=2)
        rng = np.random.default_rng(6)
        r = torch.tensor(rng.standard_normal(PS.ndof) + 1j * rng.standard_normal(PS.ndof), device=cuda)
        out = torch.empty_like(r)
        s.precondition(r, out)
        z.append(out.cpu().numpy())
    # the bound of the other sizes: Chebyshev steps of FP32 products and mass
    # solves (condition up to 1e3 per level)
    assert np.linalg.norm(z[0] - z[1]) < 2e-3 * np.linalg.norm(z[1]), np.linalg.norm(z[0] - z[1]) / np.linalg.norm(z[1])
