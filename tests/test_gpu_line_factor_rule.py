"""Which kernels the FDM line solves take, by launches: with a stored factor an
application at the stage of the last one takes one line-solve launch and one at
a new stage three, an elimination two at either; on both sides of the rule's
line in the number of lines (32 per SM, 64 at degree 5)."""
import numpy as np
import pytest

from tests.cases import product_of
from tests.test_gpu_mg_dense import _case


@pytest.mark.gpu
@pytest.mark.parametrize("p", [2, 3, 4, 5])
@pytest.mark.parametrize("over", [False, True])
def test_line_count_rule(cuda, p, over):
    import torch
    from tdsez_gb300 import _lib
    from tdsez_gb300.propagator import Solver
    lib = _lib.load()
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    most = (64 if p == 5 else 32) * sms
    nx = 64
    ny = most // nx + (1 if over else 0)          # axis lengths nx, ny
    S, op = product_of(_case("layered", p, (nx - p, ny - p, 9)))
    op.set_stage(1.0, 0.05j, [0.03])
    s = Solver(op, pc="fdm", precision="fp32")
    r = torch.tensor(np.random.default_rng(p).standard_normal(S.ndof) + 0j, device=cuda)
    z = torch.empty_like(r)

    def launches():
        before = lib.tdz_launch_count()
        s.precondition(r, z)
        return lib.tdz_launch_count() - before
    s.precondition(r, z)
    again = launches()
    op.set_stage(1.0, 0.04j, [0.03])
    new = launches()
    assert new - again == (0 if over else 2), (again, new)
