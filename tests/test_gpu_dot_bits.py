"""The FP64 dots keep FP64 partial sums over threads: vectors whose products and
sums are whole multiples of one power of two, within FP64's 53 bits and beyond
the 48 or so of a double-float, have exact dots."""
import ctypes as C

import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("k", [1, 2, 3, 5, 8, 13, 16])
@pytest.mark.parametrize("n", [1, 31, 200, 256])
def test_dots_exact(cuda, n, k):
    import torch
    from tdsez_gb300 import _lib
    lib = _lib.load()
    rng = np.random.default_rng(1000 * n + k)
    # 46-bit integers: one element per thread, whose split into two FP32 numbers is
    # exact; sums of at most 256 below 2^53 in magnitude for random signs
    w = rng.integers(-2 ** 46, 2 ** 46, (2, n))
    unit = rng.choice([1, 1j, -1, -1j], (k, n))
    wr, wi = w[0].astype(object), w[1].astype(object)
    want = []
    for i in range(k):
        a, b = unit[i].real.astype(int).astype(object), unit[i].imag.astype(int).astype(object)
        re, im = int(np.sum(a * wr + b * wi)), int(np.sum(a * wi - b * wr))
        assert max(abs(re), abs(im)) < 2 ** 53
        want.append(complex(re, im) * 2.0 ** -40)
    V = [torch.tensor(u, device=cuda) for u in unit]
    wd = torch.tensor((w[0] + 1j * w[1]) * 2.0 ** -40, device=cuda)
    out = torch.zeros(k, dtype=torch.complex128, device=cuda)
    ptrs = (C.c_void_p * k)(*[v.data_ptr() for v in V])
    _lib.check(lib.tdz_vec_mdot(ptrs, k, C.c_void_p(wd.data_ptr()), n, _lib.TDZ_FP64, C.c_void_p(out.data_ptr()),
                                C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert out.cpu().numpy().tolist() == want


@pytest.mark.gpu
@pytest.mark.parametrize("outer", ["fp64", "df"])
def test_gram_schmidt_widths(cuda, outer):
    """A solve through every width of the fused Gram-Schmidt pass (16 vectors with
    the norm are 34 sums, more than a warp has lanes) and the separate passes
    beyond: the solution's residual is the one reported."""
    import torch
    from oracle import bspline as ob
    from tdsez_gb300 import _lib
    from tdsez_gb300.operators import Operator, Physics
    from tdsez_gb300.propagator import Solver
    from tdsez_gb300.space import Space
    p = 3
    kn = [ob.uniform_knots(n, -10.0, 10.0, p) for n in (40, 30, 20)]
    S = Space(kn, p, p + 1)
    op = Operator(S, Physics(charge=-1.0, coupled=(2,), potential=[lambda x: 0.1 * x * x, None, None]))
    op.set_stage(1.0, 0.08j, [0.05])
    rng = np.random.default_rng(1)
    b = torch.tensor(rng.standard_normal(S.ndof) + 1j * rng.standard_normal(S.ndof), device=cuda)
    x, r = torch.zeros_like(b), torch.empty_like(b)
    its, reason, rn = Solver(op, pc="mass", rtol=1e-8, restart=60, maxit=60, outer=outer).solve(b, x)
    assert reason > 0 and 18 <= its < 60, (its, reason)
    op.apply(_lib.TDZ_STAGE, x, r)
    true = torch.linalg.norm(b - r).item()
    # FP64 solution, FP32 preconditioner: the recurrence's residual and the true one
    # differ by some 1e-14 |A||x|, far below 1e-8 |b|
    assert true <= 1.01 * 1e-8 * torch.linalg.norm(b).item(), (true, rn)
