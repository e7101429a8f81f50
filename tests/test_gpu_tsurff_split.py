"""The face contractions of the GPU t-SURFF sampler where their thread groups
have ragged ends: node counts off the 32-lane groups, momenta off the groups
of four, faces large enough for the four-momenta variant, one momentum."""
import math

import numpy as np
import pytest

from oracle import bspline as ob
from oracle import tsurff as ots


def _field(t):
    return [0.05 * math.sin(0.3 * t), 0.02 * math.cos(0.2 * t), -0.03 * math.sin(0.1 * t + 1.0)]


@pytest.mark.gpu
@pytest.mark.parametrize("p,nel,nk", [(2, (5,), (1,)), (7, (40,), (65,)), (3, (30, 7), (33, 1)), (5, (6, 45), (3, 70)),
                                      (2, (12, 14, 11), (5, 1, 2)), (3, (16, 15, 17), (9, 10, 11))])
def test_tsurff_ragged_groups(cuda, p, nel, nk):
    import torch
    from tdsez_gb300.space import Space
    from tdsez_gb300.tsurff import TSurff
    dim = len(nel)
    kn = [ob.uniform_knots(n, -20.0 - d, 20.0 + d, p) for d, n in enumerate(nel)]
    S = ob.Space([ob.Axis(k, p, p + 1) for k in kn])
    kg = [(-1.5, 1.2 + 0.1 * d, n) for d, n in enumerate(nk)]
    ks = [np.linspace(lo, hi, n) if n > 1 else np.array([lo]) for lo, hi, n in kg]
    ora = ots.OracleTSurff(S, 13.0, ks, 0.8, 0.05, 1.0, _field, 0.1)
    gpu = TSurff(Space(kn, p, p + 1), 13.0, kg, _field, 0.1, mass=0.8, v0=0.05, charge=-1.0)
    rng = np.random.default_rng(9)
    amp = np.zeros(int(np.prod(nk)), dtype=complex)
    for t in (0.0, 0.3, 0.4):
        psi = rng.standard_normal(S.ndof) + 1j * rng.standard_normal(S.ndof)
        amp = ora.add_flux(t, psi, ks, amp)
        gpu.sample(t, torch.tensor(psi, device=cuda))
    a = gpu.amplitudes()
    # sums of at most 1e4 FP64 products per face, the existing parity bar
    assert np.abs(a - amp).max() <= 1e-11 * np.abs(amp).max()
