"""The dense-axis Chebyshev steps of small multigrid levels do run where they are
meant to: two launches a step instead of four, so a V-cycle with them takes fewer
launches than the V-cycle of the same grid with an absorbing layer, which never
takes them."""
import numpy as np
import pytest

from tests.cases import product_of
from tests.test_gpu_mg_dense import _case


@pytest.mark.gpu
@pytest.mark.parametrize("p,nel,levels", [(2, (12, 13, 30), 3), (3, (30, 14, 40), 3), (3, (17, 33, 21), 3),
                                          (4, (9, 21, 28), 3), (2, (36, 34, 31), 2), (2, (10, 9, 140), 2)])
def test_dense_steps_run(cuda, p, nel, levels):
    import torch
    from tdsez_gb300 import _lib
    from tdsez_gb300.propagator import Solver
    lib = _lib.load()
    n = {}
    for kind in ("layered", "const", "cap"):
        S, op = product_of(_case(kind, p, nel))
        op.set_stage(1.0, 0.2j, [0.03] * len(op.coupled))
        s = Solver(op, pc="mg", precision="fp32", mg_levels=levels, mg_smooth=4, mg_coarse_its=8)
        r = torch.tensor(np.random.default_rng(5).standard_normal(S.ndof) + 0j, device=cuda)
        z = torch.empty_like(r)
        s.precondition(r, z)
        before = lib.tdz_launch_count()
        s.precondition(r, z)
        n[kind] = lib.tdz_launch_count() - before
    # at least the coarsest level (7 steps) and another one (6) take them, two
    # launches less each, for one launch per level that combines the matrices
    for kind in ("layered", "const"):
        assert n[kind] <= n["cap"] - 2 * (7 + 6) + levels, n


@pytest.mark.gpu
@pytest.mark.parametrize("p,nel", [(2, (90, 88, 30)), (3, (85, 85, 100))])
def test_general_steps_run(cuda, p, nel):
    """Past the line the general step is the shorter one: as many launches as with
    an absorbing layer."""
    import torch
    from tdsez_gb300 import _lib
    from tdsez_gb300.propagator import Solver
    lib = _lib.load()
    n = []
    for kind in ("layered", "cap"):
        S, op = product_of(_case(kind, p, nel))
        op.set_stage(1.0, 0.2j, [0.03] * len(op.coupled))
        s = Solver(op, pc="mg", precision="fp32", mg_levels=1, mg_coarse_its=8)
        r = torch.tensor(np.random.default_rng(5).standard_normal(S.ndof) + 0j, device=cuda)
        z = torch.empty_like(r)
        s.precondition(r, z)
        before = lib.tdz_launch_count()
        s.precondition(r, z)
        n.append(lib.tdz_launch_count() - before)
    assert n[0] == n[1], n
