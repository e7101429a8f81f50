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
