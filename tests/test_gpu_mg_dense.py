"""The dense-axis Chebyshev steps of small multigrid levels: one V-cycle with
FP32 levels (which take them) equals the V-cycle with FP64 levels (which never
do) to FP32 rounding, for a mass layered along z and for a constant mass with
inner-axis potentials and fields, on axis lengths off the kernels' groups of 2,
8, 16 and 32, with real and complex stages; and with an absorbing layer or a
soft-core centre, where the general step runs."""
import numpy as np
import pytest

from oracle import bspline as ob
from tests.cases import product_of


def _case(kind, p, nel):
    kn = [ob.uniform_knots(n, -8.0 - d, 8.0 + d, p) for d, n in enumerate(nel)]
    c = dict(knots=kn, p=p, nq=p + 1, charge=-1.0, coupled=(0, 2))
    if kind == "layered":
        c.update(knots=kn[:2] + [ob.interface_knots(-10.0, 10.0, nel[2], p, [-2.0, 3.0])], mass_axis=2, coupled=(2,),
                 inv_mass=lambda z: 11.0 if -2.0 < z < 3.0 else 14.0,
                 V=[None, None, lambda z: -0.2 if -2.0 < z < 3.0 else 0.1])
    else:
        c.update(mass=0.5, V=[lambda x: 0.05 * x * x, None, lambda z: 0.02 * z])
        if kind == "cap":
            c.update(cap_kmin=1.0, bounds=[(k[0], k[-1]) for k in kn])
        if kind == "soft":
            c.update(soft=[(1.0, 0.3, 0.2, -0.1, 0.8)])
    return c


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["layered", "const", "cap", "soft"])
@pytest.mark.parametrize("p,nel", [(2, (12, 13, 30)), (3, (30, 14, 40)), (3, (17, 33, 21)), (4, (9, 21, 28))])
@pytest.mark.parametrize("g", [0.2j, 0.1 + 0.2j])
def test_vcycle_fp32_equals_fp64(cuda, kind, p, nel, g):
    import torch
    from tdsez_gb300.propagator import Solver
    z = []
    for prec in ("fp32", "fp64"):
        PS, op = product_of(_case(kind, p, nel))
        op.set_stage(1.0, g, [0.03] * len(op.coupled))
        s = Solver(op, pc="mg", precision=prec, mg_levels=3)
        rng = np.random.default_rng(5)
        r = torch.tensor(rng.standard_normal(PS.ndof) + 1j * rng.standard_normal(PS.ndof), device=cuda)
        out = torch.empty_like(r)
        s.precondition(r, out)
        z.append(out.cpu().numpy())
    # 28 Chebyshev steps of FP32 products and mass solves (condition up to 1e3 per level)
    assert np.linalg.norm(z[0] - z[1]) < 2e-3 * np.linalg.norm(z[1]), np.linalg.norm(z[0] - z[1]) / np.linalg.norm(z[1])
