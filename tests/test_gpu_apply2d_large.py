"""2D applies on both sides of the line between the tile kernel and the
row-streaming one: few rows past the line, ragged last tiles and row chunks,
grids too narrow for the streaming kernel, and each combination of streams and
coefficient kinds, against products of sparse 1D matrices in FP64."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import bspline as ob

G, FIELD = 0.1 + 0.3j, 0.02


def _axis(knots, p):
    a = ob.Axis(knots, p, p + 1)
    N, D, w, x = a.basis_matrix(0), a.basis_matrix(1), a.wq.reshape(-1), a.xq.reshape(-1)
    form = lambda B, f: sp.csr_matrix(B.T @ sp.diags(w * f) @ B)   # noqa: E731
    return {"M": form(N, 1.0 + 0 * x), "S": form(D, 1.0 + 0 * x), "x": x, "form": lambda f: form(N, f),
            "dform": lambda f: form(D, f), "X": form(N, x)}


def _case(kind, p, nx, ny):
    from tdsez_gb300.operators import Physics, cap_profile
    kn = [ob.uniform_knots(nx, -30.0, 30.0, p), ob.uniform_knots(ny, -40.0, 40.0, p)]
    A, B = _axis(kn[0], p), _axis(kn[1], p)
    vx, vy = (lambda x: 0.01 * x * x), (lambda y: 0.02 * y)
    terms = []   # (coefficient, y matrix, x matrix) of H + c D
    if kind in ("layered", "both"):
        inv = lambda y: np.where(y < 0.0, 2.0, 3.0)   # noqa: E731
        terms += [(0.5, B["form"](inv(B["x"])), A["S"]), (0.5, B["dform"](inv(B["x"])), A["M"])]
        ph = dict(mass_axis=1, inv_mass_fn=lambda y: float(inv(np.array(y))))
    else:
        terms += [(0.5 / 0.8, B["M"], A["S"]), (0.5 / 0.8, B["S"], A["M"])]
        ph = dict(mass=0.8)
    axis = 1 if kind == "layered" else 0
    ph.update(coupled=(axis,), potential=[None if kind == "layered" else vx, vy], charge=-1.0)
    terms.append((1.0, B["form"](vy(B["x"])), A["M"]))
    terms.append((FIELD, B["X"], A["M"]) if axis else (FIELD, B["M"], A["X"]))
    if kind != "layered":
        terms.append((1.0, B["M"], A["form"](vx(A["x"]))))
    if kind == "cap":
        bounds = [(-30.0, 30.0), (-40.0, 40.0)]
        ph.update(cap_kmin=1.0, bounds=bounds)
        W = [np.array([cap_profile(v, lo, hi, 1.0) for v in ax["x"]]) for ax, (lo, hi) in zip((A, B), bounds)]
        terms += [(-1j / 0.8, B["M"], A["form"](W[0])), (-1j / 0.8, B["form"](W[1]), A["M"])]
    return kn, Physics(**ph), terms, A, B


@pytest.mark.gpu
@pytest.mark.parametrize("kind,p,nx,ny,prec", [
    ("const", 2, 1005, 1300, "fp32"),     # past the line, ragged tiles
    ("const", 3, 1021, 1150, "fp32"),     # just below it
    ("const", 5, 1149, 1300, "fp32"),
    ("const", 3, 130, 11000, "fp32"),     # past it, too narrow
    ("const", 4, 20000, 64, "fp32"),      # few rows: one chunk a tile
    ("layered", 4, 1532, 2000, "fp32"),
    ("mass", 3, 1700, 1801, "fp32"),
    ("cap", 4, 765, 690, "fp64"),
    ("cap", 2, 900, 1250, "fp64"),
    ("const", 5, 1020, 850, "fp64"),
    ("layered", 4, 2300, 2451, "fp64"),
    ("mass", 5, 1340, 1400, "fp64"),
    ("both", 3, 1530, 1601, "fp64"),
    ("both", 2, 1280, 1101, "fp32"),
])
def test_large_2d_apply(cuda, kind, p, nx, ny, prec):
    import torch
    from tdsez_gb300 import _lib
    from tdsez_gb300.operators import Operator
    from tdsez_gb300.space import Space
    kn, ph, terms, A, B = _case("const" if kind == "mass" else kind, p, nx, ny)
    op = Operator(Space(kn, p, p + 1), ph)
    op.set_stage(1.0, G, [FIELD])
    rng = np.random.default_rng(nx + p)
    x = rng.standard_normal((B["M"].shape[0], A["M"].shape[0])) + 1j * rng.standard_normal((B["M"].shape[0], A["M"].shape[0]))
    if prec == "fp32":
        x = x.astype(np.complex64).astype(complex)
    both = lambda my, mx: (mx @ (my @ x).T).T   # noqa: E731
    want = both(B["M"], A["M"])
    if kind != "mass":
        want = want + G * sum(c * both(my, mx) for c, my, mx in terms)
    xd = torch.tensor(x.reshape(-1), dtype=torch.complex64 if prec == "fp32" else torch.complex128, device=cuda)
    yd = torch.full_like(xd, complex(float("nan"), 0.0))
    op.apply(_lib.TDZ_MASS if kind == "mass" else _lib.TDZ_STAGE, xd, yd)
    err = np.abs(yd.cpu().numpy() - want.reshape(-1)).max() / np.abs(want).max()
    assert err < (1e-6 if prec == "fp32" else 1e-12), err   # the bars of the apply parity tests
