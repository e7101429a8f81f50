"""Performance cases of the propagation library: what a propagation run asks of it.

Each case is a dict of plain values. ``listed()`` gives the fixed ones,
``draw(rng)`` another of the same ranges, ``prepare(case, seed)`` what a
program holds before the call (operator, solver or sampler handles, inputs
from the seed), ``run(state)`` one pass through the public entry points,
``work(case)`` the bytes and operations that pass cannot do without and
``exact(case, seed)`` its result from dense 64-bit linear algebra that shares
no code with the library.

Families:

  apply   y = A x of the stage operator: the matrix product inside every
          Krylov iteration (FP32 vectors: smoothers and residuals of the
          mixed-precision multigrid; "df": FGMRES residuals and right-hand
          sides in double-float; "fp64": the library's default outer
          arithmetic), on the z-layered heterostructure and on the 3D
          soft-core atom
  mass    x = M^-1 b, FP32 (every smoother step of the multigrid) or FP64
          (projection of initial states)
  cn      one Crank-Nicolson step of the heterostructure, with the
          fast-diagonalisation inverse as the benchmark runs it, or with the
          library's default multigrid
  pade    one Pade(2,2) step of the 2D soft-core atom with absorbing layers
  batch   one step of an intensity scan: independent 2D runs stepped together
  tsurff  photoelectron spectra: flux samples through the surface and the
          amplitudes
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tdsez_gb300 import _lib
from tdsez_gb300.operators import MA_C, Operator, Physics
from tdsez_gb300.propagator import BatchPropagator, Propagator
from tdsez_gb300.space import Space, symexp_knots, uniform_knots
from tdsez_gb300.tsurff import TSurff
from tdsez_gb300.workloads import heterostructure

DEV = "cuda"
FIELD = 0.02          # field strength of the applies' stage (a.u.)
G_APPLY = 0.025j      # g of the applies' stage: i dt / 2 at dt = 0.05


def listed():
    return [
        # one smoother application on a coarse multigrid level: launch latency
        {"name": "apply_fp32_small", "family": "apply", "op": "layered", "nx": 16, "ny": 20, "nz": 40, "p": 3,
         "precision": "fp32"},
        # the same on the finest level of the benchmark heterostructure
        {"name": "apply_fp32_large", "family": "apply", "op": "layered", "nx": 160, "ny": 160, "nz": 320, "p": 3,
         "precision": "fp32"},
        # FGMRES residual of a degree-4 run on a ragged grid
        {"name": "apply_df_ragged", "family": "apply", "op": "layered", "nx": 97, "ny": 83, "nz": 171, "p": 4,
         "precision": "df"},
        # the default outer arithmetic on a middle-sized grid
        {"name": "apply_fp64_mid", "family": "apply", "op": "layered", "nx": 64, "ny": 64, "nz": 128, "p": 2,
         "precision": "fp64"},
        # stage of the 3D soft-core atom: separable part and quadrature term
        {"name": "apply_softcore3d", "family": "apply", "op": "softcore", "nx": 96, "ny": 96, "nz": 96, "p": 4,
         "precision": "fp32"},
        # the Kronecker inverse of the overlap in a smoother step
        {"name": "mass_fp32", "family": "mass", "nx": 120, "ny": 120, "nz": 240, "p": 3, "precision": "fp32"},
        # a small run's step: host and launch latency
        {"name": "cn_fdm_small", "family": "cn", "nx": 24, "ny": 24, "nz": 48, "p": 3, "pc": "fdm"},
        # the benchmark step
        {"name": "cn_fdm_large", "family": "cn", "nx": 160, "ny": 160, "nz": 320, "p": 3, "pc": "fdm"},
        # the default solver (multigrid) on a middle-sized grid
        {"name": "cn_mg_mid", "family": "cn", "nx": 48, "ny": 48, "nz": 96, "p": 3, "pc": "mg"},
        # 2D soft-core atom with absorbing layers, half the size of the strong-field configuration
        {"name": "pade_2d", "family": "pade", "nel": 256, "p": 4},
        # a small intensity scan
        {"name": "batch_scan", "family": "batch", "runs": 6, "nel_min": 48, "nel_max": 128},
        # spectra of the strong-field configuration
        {"name": "tsurff_2d", "family": "tsurff", "dim": 2, "nel": 256, "p": 4, "nk": 128},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    fam = rng.choice(["apply", "apply", "apply", "apply", "mass", "cn", "cn", "pade", "batch", "tsurff"])
    if fam in ("apply", "mass", "cn"):
        hi = {"apply": 150, "mass": 120, "cn": 120}[fam]
        nx, ny = _log(rng, 14, hi), _log(rng, 14, hi)
        nz = _log(rng, 32, 2 * hi)
        p = rng.choice([2, 3, 3, 4, 5])
        if fam == "apply":
            prec = rng.choice(["fp32", "fp32", "df", "df", "fp64"])
            if rng.random() < 0.25:
                n = _log(rng, 16, 96)
                return {"family": fam, "op": "softcore", "nx": n, "ny": n, "nz": n, "p": p,
                        "precision": "df" if prec == "df" else "fp32"}
            return {"family": fam, "op": "layered", "nx": nx, "ny": ny, "nz": nz, "p": p, "precision": prec}
        if fam == "mass":
            return {"family": fam, "nx": nx, "ny": ny, "nz": nz, "p": p,
                    "precision": rng.choice(["fp32", "fp32", "fp64"])}
        if rng.random() < 0.25:
            return {"family": fam, "nx": _log(rng, 24, 48), "ny": _log(rng, 24, 48), "nz": _log(rng, 48, 96),
                    "p": rng.choice([2, 3]), "pc": "mg"}
        return {"family": fam, "nx": nx, "ny": ny, "nz": nz, "p": rng.choice([2, 3, 3, 4]), "pc": "fdm"}
    if fam == "pade":
        return {"family": fam, "nel": _log(rng, 64, 256), "p": rng.choice([3, 4, 5])}
    if fam == "batch":
        lo = _log(rng, 32, 64)
        return {"family": fam, "runs": rng.randint(3, 8), "nel_min": lo, "nel_max": _log(rng, lo + 8, 128)}
    if rng.random() < 0.3:
        return {"family": "tsurff", "dim": 3, "nel": _log(rng, 16, 40), "p": rng.choice([2, 3, 4]),
                "nk": _log(rng, 8, 24)}
    return {"family": "tsurff", "dim": 2, "nel": _log(rng, 64, 320), "p": rng.choice([3, 4, 5]),
            "nk": _log(rng, 24, 160)}


# ------------------------------------------------------------------ workloads
class Problem:
    """Knots, physics and time step of a case."""

    def __init__(self, knots, p, phys, dt, field, t0):
        self.knots, self.p, self.phys, self.dt, self.field, self.t0 = knots, p, phys, dt, field, t0
        self.shape = tuple(len(k) - p - 1 for k in reversed(knots))     # (z, y, x) or (y, x)

    @property
    def n(self):
        return int(np.prod(self.shape))


def _pulse(e0, phase=0.0):
    length = 4 * 2 * math.pi / 0.057

    def field(t):
        t = t % length
        return [e0 * math.sin(math.pi * t / length) ** 2 * math.cos(0.057 * t + phase)]
    return field, length


def layered(case):
    w = heterostructure((case["nx"], case["ny"], case["nz"]), case["p"])
    return Problem(w.knots, case["p"], w.phys, w.dt, _pulse(w.meta["E0"])[0], 100.0)


def softcore3d(case):
    L, p = 60.0, case["p"]
    knots = [symexp_knots(-L, L, case[a], 0.9, p) for a in ("nx", "ny", "nz")]
    phys = Physics(charge=-1.0, mass=1.0, coupled=(2,), softcore=[(1.0, 0.0, 0.0, 0.0, 0.5)])
    return Problem(knots, p, phys, 0.02, _pulse(0.053)[0], 100.0)


def softcore2d(nel, p, dt, cap=False, e0=0.05, phase=0.0):
    L = 100.0
    knots = [uniform_knots(nel, -L, L, p)] * 2
    kmin = MA_C / (2.0 * 0.2 * 20.0)     # layers of 20 a.u.
    phys = Physics(charge=-1.0, mass=1.0, coupled=(0,), softcore=[(1.0, 0.0, 0.0, 0.0, 1.0)],
                   cap_kmin=kmin if cap else None, bounds=[(-L, L)] * 2 if cap else ())
    return Problem(knots, p, phys, dt, _pulse(e0, phase)[0], 100.0)


def problem(case):
    f = case["family"]
    if f == "apply" and case["op"] == "softcore":
        return softcore3d(case)
    if f in ("apply", "mass", "cn"):
        return layered(case)
    return softcore2d(case["nel"], case["p"], 0.02, cap=True)


def scan(case):
    """The runs of a scan: grids between the case's two sizes, degrees 3 to 5,
    field strengths and carrier phases spread over the run index."""
    out = []
    for r in range(case["runs"]):
        s = r / max(1, case["runs"] - 1)
        nel = int(round(case["nel_min"] + s * (case["nel_max"] - case["nel_min"])))
        out.append(softcore2d(nel, 3 + r % 3, 0.05, e0=10 ** (-2 + s), phase=2.4 * r))
    return out


def normal(shape, seed, dtype):
    """Complex normal coefficients: a residual or Krylov vector."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = torch.randn(tuple(shape) + (2,), generator=g, device=DEV, dtype=torch.float64)
    return torch.view_as_complex(r).to(dtype).reshape(-1).contiguous()


def packet(prob, seed):
    """A moving Gaussian packet: its values at the Greville abscissae as
    coefficients, of unit 2-norm."""
    rng = np.random.default_rng(seed)
    psi = None
    for U in reversed(prob.knots):
        x = np.array([U[i + 1:i + prob.p + 1].mean() for i in range(len(U) - prob.p - 1)])
        half = 0.5 * (U[-1] - U[0])
        c, w, k = half * rng.uniform(-0.2, 0.2), half * rng.uniform(0.08, 0.2), rng.uniform(-0.3, 0.3)
        v = torch.tensor(np.exp(-((x - c) / w) ** 2 / 2 + 1j * k * x), device=DEV)
        psi = v if psi is None else torch.outer(psi, v).reshape(-1)
    return (psi / torch.linalg.vector_norm(psi)).contiguous()


def operator(prob):
    return Operator(Space(prob.knots, prob.p, prob.p + 1), prob.phys)


def surface(case):
    """Sampler settings: radius, momentum axis and time step (half the box of
    the 3D cases, the strong-field configuration's square in 2D)."""
    return (80.0 if case["dim"] == 2 else 20.0), (-1.5, 1.5, case["nk"]), 0.5


def surface_space(case):
    L = 100.0 if case["dim"] == 2 else 40.0
    return [uniform_knots(case["nel"], -L, L, case["p"])] * case["dim"]


def surface_field(dim):
    f = _pulse(0.05)[0]
    return lambda t: f(t) + [0.0] * (dim - 1)


SAMPLES = 4


# -------------------------------------------------------------------- passes
def prepare(case, seed):
    fam = case["family"]
    if fam == "batch":
        probs = scan(case)
        props = [Propagator(operator(q), "cn", field=q.field, pc="fdm", precision="fp32", outer="df",
                            guess_order=-1) for q in probs]
        psis = [packet(q, seed + 1000 * i) for i, q in enumerate(probs)]
        return {"family": fam, "batch": BatchPropagator(props, threads=8), "psis": psis, "t": probs[0].t0,
                "dt": probs[0].dt}
    if fam == "tsurff":
        R, grid, dt = surface(case)
        knots = surface_space(case)
        prob = Problem(knots, case["p"], None, dt, None, 0.0)
        ts = TSurff(Space(knots, case["p"], case["p"] + 1), R, [grid] * case["dim"], surface_field(case["dim"]), dt)
        return {"family": fam, "ts": ts, "dt": dt, "t": 100.0,
                "psis": [packet(prob, seed + 1000 * i) for i in range(SAMPLES)]}
    prob = problem(case)
    op = operator(prob)
    if fam == "apply":
        op.set_stage(1.0, G_APPLY, [FIELD])
        x = normal(prob.shape, seed, torch.complex64 if case["precision"] == "fp32" else torch.complex128)
        return {"family": fam, "op": op, "x": x, "y": torch.empty_like(x), "df": case["precision"] == "df"}
    if fam == "mass":
        b = normal(prob.shape, seed, torch.complex64 if case["precision"] == "fp32" else torch.complex128)
        return {"family": fam, "op": op, "b": b, "x": torch.empty_like(b)}
    if fam == "pade":
        prop = Propagator(op, "pade22", field=prob.field, pc="fdm", precision="fp32", outer="df", guess_order=-1)
    elif case["pc"] == "fdm":
        prop = Propagator(op, "cn", field=prob.field, pc="fdm", precision="fp32", rtol=1e-10, outer="df",
                          relaxed=True, guess_order=-1)
    else:
        prop = Propagator(op, "cn", field=prob.field, pc=case["pc"])
    return {"family": fam, "prop": prop, "psi": packet(prob, seed), "t": prob.t0, "dt": prob.dt}


def run(state):
    fam = state["family"]
    if fam == "apply":
        return state["op"].apply(_lib.TDZ_STAGE, state["x"], state["y"], df=state["df"])
    if fam == "mass":
        return state["op"].mass_solve(state["x"].copy_(state["b"]))
    if fam == "tsurff":
        for psi in state["psis"]:
            state["ts"].sample(state["t"], psi)
            state["t"] += state["dt"]
        return state["ts"].amplitudes()
    t, state["t"] = state["t"], state["t"] + state["dt"]
    if fam == "batch":
        return state["batch"].step(state["psis"], t, state["dt"])
    return state["prop"].step(state["psi"], t, state["dt"])


def work(case):
    """Bytes: inputs read and outputs written once. Operations: the band
    contractions of the sum-factorised operators, the dense transforms and
    line solves of the inverses, the surface and momentum contractions."""
    fam = case["family"]
    if fam == "tsurff":
        d, q, nk = case["dim"], case["nel"] * (case["p"] + 1) * (0.8 if case["dim"] == 2 else 0.5), case["nk"]
        face = 8.0 * q * nk if d == 2 else 8.0 * q * nk * (q + nk)
        n = (case["nel"] + case["p"]) ** (d - 1) * (case["p"] + 1)
        return {"bytes": SAMPLES * 2 * d * 16.0 * n + 16.0 * nk ** d,
                "flops": SAMPLES * (2 * d * (2 * face + 10.0 * nk ** d) + 14.0 * nk ** d)}
    probs = scan(case) if fam == "batch" else [problem(case)]
    b = f = 0.0
    for prob in probs:
        bw, n, dim = 2 * prob.p + 1, prob.n, len(prob.shape)
        apply_f = 4.0 * bw * (8 if dim == 3 else 5) * n
        if prob.phys.softcore:
            apply_f += 4.0 * (prob.p + 1) * 2 * dim * n
        if fam == "apply":
            b += (16.0 if case["precision"] == "fp32" else 32.0) * n
            f += apply_f
        elif fam == "mass":
            b += (16.0 if case["precision"] == "fp32" else 32.0) * n
            f += 3 * 4.0 * bw * n
        else:
            solves = 2 if fam == "pade" else 1
            inverse = 4.0 * 2 * sum(prob.shape[1:]) * n + 8.0 * 4 * prob.p * prob.p * n
            b += 32.0 * n
            f += solves * (2 * apply_f + inverse)
    return {"bytes": b, "flops": f}


# --------------------------------------------- the same results in 64 bits
def basis(U, p, x):
    """Values and first derivatives (len(x), n) of the B-splines on the knots
    U at points inside the knot range (Cox-de Boor recursion)."""
    U, x = np.asarray(U, dtype=np.float64), np.asarray(x, dtype=np.float64)
    n = len(U) - p - 1
    spans = np.clip(np.searchsorted(U, x, side="right") - 1, p, n - 1)
    B = np.zeros((len(x), len(U) - 1))
    B[np.arange(len(x)), spans] = 1.0
    low = None
    for q in range(1, p + 1):
        low = B
        m = len(U) - 1 - q
        d0, d1 = U[q:q + m] - U[:m], U[q + 1:q + 1 + m] - U[1:1 + m]
        a = np.where(d0 > 0, (x[:, None] - U[:m]) / np.where(d0 > 0, d0, 1), 0.0)
        b = np.where(d1 > 0, (U[q + 1:q + 1 + m] - x[:, None]) / np.where(d1 > 0, d1, 1), 0.0)
        B = a * low[:, :m] + b * low[:, 1:1 + m]
    d0, d1 = U[p:p + n] - U[:n], U[p + 1:p + 1 + n] - U[1:1 + n]
    D = p * (low[:, :n] * np.where(d0 > 0, 1 / np.where(d0 > 0, d0, 1), 0.0)
             - low[:, 1:1 + n] * np.where(d1 > 0, 1 / np.where(d1 > 0, d1, 1), 0.0))
    return B, D


def points(U, q, lo=-math.inf, hi=math.inf):
    """q Gauss points and weights of every non-empty span inside [lo, hi]."""
    gx, gw = np.polynomial.legendre.leggauss(q)
    x, w = [], []
    for a, b in zip(U[:-1], U[1:]):
        a, b = max(a, lo), min(b, hi)
        if b > a:
            x.append(0.5 * (a + b) + 0.5 * (b - a) * gx)
            w.append(0.5 * (b - a) * gw)
    return np.concatenate(x), np.concatenate(w)


def absorber(x, lo, hi, kmin):
    """Manolopoulos' transmission-free absorbing potential, layers of width
    c / (2 delta kmin), delta = 0.2, at both walls."""
    c = MA_C
    a, b = 1 - 16 / c ** 3, (1 - 17 / c ** 3) / c ** 2
    width = c / (2 * 0.2 * kmin)
    u = width - np.minimum(x - lo, hi - x)
    r = c * np.clip(u / width, 0.0, 1 - 1e-10)
    w = 0.5 * kmin ** 2 * (a * r - b * r ** 3 + 4 / (c - r) ** 2 - 4 / (c + r) ** 2)
    return np.where(u > 0, w, 0.0)


class Exact:
    """Dense 1D matrices of a problem and its operators in 64 bits."""

    def __init__(self, prob):
        self.prob, ph, p = prob, prob.phys, prob.p
        self.dim = len(prob.knots)
        self.M, self.H, self.X, self.N, self.xq, self.wq, self.S = [], [], [], [], [], [], []
        for d, U in enumerate(prob.knots):
            x, w = points(U, p + 1)
            N, D = basis(U, p, x)
            band = lambda B, f: B.T @ ((w * f)[:, None] * B)   # noqa: E731
            f = ph.potential[d] if d < len(ph.potential) else None
            v = ph.sign * np.array([f(t) for t in x]) if f else np.zeros_like(x)
            minv = np.array([ph.inv_mass_fn(t) for t in x]) if ph.mass_axis == d else np.full_like(x, 1.0 / ph.mass)
            H = 0.5 * band(D, minv) + band(N, v)
            if ph.cap_kmin is not None:
                H = H - 1j / ph.mass * band(N, absorber(x, *ph.bounds[d], ph.cap_kmin))
            self.M.append(band(N, np.ones_like(x)))
            self.S.append(band(D, np.ones_like(x)))
            self.X.append(band(N, x))
            self.H.append(H)
            if ph.mass_axis == d:
                self.Mm = band(N, minv)
            self.N.append(N)
            self.xq.append(x)
            self.wq.append(w)

    @staticmethod
    def dev(a):
        return torch.as_tensor(a, device=DEV).to(torch.complex128)

    def along(self, a, x, d):
        """Matrix a on axis d (0 = x, the last index of the array)."""
        k = self.dim - 1 - d
        y = torch.movedim(torch.tensordot(self.dev(a), x, dims=([1], [k])), 0, k)
        return y

    def kron(self, mats, x):
        for d, a in enumerate(mats):
            x = self.along(a, x, d)
        return x

    def mass(self, x):
        return self.kron(self.M, x)

    def separable(self, x, c, axis):
        """H x without the soft-core term, with the field c on one axis."""
        ph, out = self.prob.phys, 0
        H = [h + c * xx if d == axis else h for d, (h, xx) in enumerate(zip(self.H, self.X))]
        if ph.mass_axis is None:
            for d in range(self.dim):
                out = out + self.kron([H[e] if e == d else self.M[e] for e in range(self.dim)], x)
            return out
        # the mass layered along z: its weight on the kinetic terms of x and y
        out = self.kron([self.M[0], self.M[1], H[2]], x)
        out = out + self.kron([0.5 * self.S[0], self.M[1], self.Mm], x)
        return out + self.kron([self.M[0], 0.5 * self.S[1], self.Mm], x)

    def softcore(self, x):
        f = self.kron(self.N, x)
        v = 0
        for Z, cx, cy, cz, a in self.prob.phys.softcore:
            r2 = a
            for d, cc in zip(range(self.dim), (cx, cy, cz)):
                sh = [1] * self.dim
                sh[self.dim - 1 - d] = -1
                r2 = r2 + torch.as_tensor((self.xq[d] - cc) ** 2, device=DEV).reshape(sh)
            v = v - Z / torch.sqrt(r2)
        for d in range(self.dim):
            sh = [1] * self.dim
            sh[self.dim - 1 - d] = -1
            v = v * torch.as_tensor(self.wq[d], device=DEV).reshape(sh)
        return self.prob.phys.sign * self.kron([N.T for N in self.N], f * v)

    def stage(self, x, alpha, g, c, axis):
        y = self.separable(x, c, axis)
        if self.prob.phys.softcore:
            y = y + self.softcore(x)
        return alpha * self.mass(x) + g * y

    # -- solves of (M + g H_E) X = b
    def solver(self, g, c, axis):
        inverse = self.layered_inverse(g, c) if self.prob.phys.mass_axis is not None else self.pencil_inverse(g, c, axis)

        def solve(b):
            x = inverse(b)
            norm = torch.linalg.vector_norm(b)
            for _ in range(60):     # what the inverse leaves out: the soft-core term, rounding
                r = b - self.stage(x, 1.0, g, c, axis)
                x = x + inverse(r)
                if torch.linalg.vector_norm(r) < 1e-14 * norm:
                    break
            return x
        return solve

    def pencil_inverse(self, g, c, axis):
        """Eigenvectors of every axis pencil (H_d, M_d)."""
        V, lam = [], []
        for d in range(self.dim):
            H = self.H[d] + (c * self.X[d] if d == axis else 0)
            if np.iscomplexobj(H):
                l, v = np.linalg.eig(np.linalg.solve(self.M[d], H))
            else:
                C = np.linalg.inv(np.linalg.cholesky(self.M[d]))
                l, v = np.linalg.eigh(C @ H @ C.T)
                v = C.T @ v
            V.append(v)
            lam.append(l)
        left = [np.linalg.inv(self.M[d] @ V[d]) for d in range(self.dim)]
        den = 1.0
        for d in range(self.dim):
            sh = [1] * self.dim
            sh[self.dim - 1 - d] = -1
            den = den + g * self.dev(lam[d]).reshape(sh)
        return lambda b: self.kron(V, self.kron(left, b) / den)

    def layered_inverse(self, g, c):
        """Eigenvectors of (S, M) along x and y, banded elimination along z of
        M + g (H_z + c X) + g (lam_x + lam_y) / 2 Mm, all lines together."""
        V, lam = [], []
        for d in (0, 1):
            C = np.linalg.inv(np.linalg.cholesky(self.M[d]))
            l, v = np.linalg.eigh(C @ self.S[d] @ C.T)
            V.append(C.T @ v)
            lam.append(l)
        eye = np.eye(self.M[2].shape[0])
        B, Cz, p = self.M[2] + g * (self.H[2] + c * self.X[2]), g * 0.5 * self.Mm, self.prob.p
        s = torch.as_tensor(lam[1][:, None] + lam[0][None, :], device=DEV).to(torch.complex128)
        n = B.shape[0]
        U = []                       # rows of the unit upper factor and the reciprocal pivots
        for k in range(n):
            row = {j: B[k, j] + s * Cz[k, j] for j in range(max(0, k - p), min(n, k + p + 1))}
            low = {}
            for j in range(max(0, k - p), k):
                low[j] = f = row[j]
                for q, u in U[j][1].items():
                    row[q] = row[q] - f * u
            inv = 1.0 / row[k]
            U.append((inv, {j: row[j] * inv for j in row if j > k}, low))

        def inverse(b):
            y = self.kron([V[0].T, V[1].T, eye], b)
            for k in range(n):
                for j, f in U[k][2].items():
                    y[k] -= f * y[j]
                y[k] *= U[k][0]
            for k in range(n - 1, -1, -1):
                for j, u in U[k][1].items():
                    y[k] -= u * y[j]
            return self.kron([V[0], V[1], eye], y)
        return inverse

    def cn(self, psi, c, axis):
        X = self.solver(0.5j * self.prob.dt, c, axis)(self.mass(psi))
        return 2 * X - psi

    def pade(self, psi, c, axis):
        g = [self.prob.dt * complex(s * math.sqrt(3.0), 3.0) / 12.0 for s in (-1, 1)]
        for k in (0, 1):
            psi = self.solver(g[k], c, axis)(2 * self.mass(psi) - self.stage(psi, 1.0, g[1 - k], c, axis))
        return psi


def exact(case, seed):
    fam = case["family"]
    if fam == "tsurff":
        return exact_tsurff(case, seed)
    if fam == "batch":
        out = []
        for i, q in enumerate(scan(case)):
            c = q.phys.sign * q.field(q.t0 + 0.5 * q.dt)[0]
            out.append(Exact(q).cn(packet(q, seed + 1000 * i).reshape(q.shape), c, 0).reshape(-1))
        return out
    prob = problem(case)
    E = Exact(prob)
    axis = prob.phys.coupled[0]
    if fam in ("apply", "mass"):
        x = normal(prob.shape, seed, torch.complex64 if case["precision"] == "fp32" else torch.complex128)
        x = x.to(torch.complex128).reshape(prob.shape)
        if fam == "apply":
            return E.stage(x, 1.0, G_APPLY, FIELD, axis).reshape(-1)
        return E.kron([np.linalg.inv(m) for m in E.M], x).reshape(-1)
    psi = packet(prob, seed).reshape(prob.shape)
    c = prob.phys.sign * prob.field(prob.t0 + 0.5 * prob.dt)[0]
    return (E.pade if fam == "pade" else E.cn)(psi, c, axis).reshape(-1)


def exact_tsurff(case, seed):
    """Flux amplitudes through |x_d| = R: at every sample the surface integral
    against the Volkov states, then the trapezoid rule in time."""
    dim, p = case["dim"], case["p"]
    R, (k0, k1, nk), dt = surface(case)
    knots, field = surface_space(case), surface_field(dim)
    prob = Problem(knots, p, None, dt, None, 0.0)
    k = np.linspace(k0, k1, nk)
    xs, ws = points(knots[0], p + 1, -R, R)     # every axis has the same knots
    N = basis(knots[0], p, xs)[0]
    wall = [basis(knots[0], p, np.array([x])) for x in (-R, R)]
    wave = np.exp(-1j * np.outer(k, xs))
    K = np.meshgrid(*[k] * dim, indexing="ij")
    # A' = -E (charge -1), B' = A, C' = |A|^2 / 2 from rest at t = 0, by
    # Runge-Kutta steps of at most dt / 2

    def advance(y, t, t1):
        def rhs(t, y):
            A = y[:3]
            E = np.array(field(t) + [0.0] * (3 - dim))
            return np.concatenate([-E, A, [0.5 * A @ A]])
        m = max(1, math.ceil((t1 - t) / (0.5 * dt) - 1e-9))
        h = (t1 - t) / m
        for i in range(m):
            u = t + i * h
            a = rhs(u, y)
            b = rhs(u + h / 2, y + h / 2 * a)
            c = rhs(u + h / 2, y + h / 2 * b)
            d = rhs(u + h, y + h * c)
            y = y + h / 6 * (a + 2 * b + 2 * c + d)
        return y
    vol, tv, t, prev, amp = np.zeros(7), 0.0, 100.0, None, np.zeros([nk] * dim, dtype=complex)
    for i in range(SAMPLES):
        psi = packet(prob, seed + 1000 * i).cpu().numpy().reshape(prob.shape)
        psi = np.transpose(psi)                  # axes x, y, z
        vol, tv = advance(vol, tv, t), t
        A, B, C = vol[:3], vol[3:6], vol[6]
        cur = 0
        for a in range(dim):
            for side, sg in ((0, -1.0), (1, 1.0)):
                face = []
                for j in (0, 1):                 # value and normal derivative on the wall's nodes
                    f = np.tensordot(wall[side][j][0], psi, axes=(0, a))
                    for ax in range(dim - 1):
                        f = np.moveaxis(np.tensordot(N, f, axes=(1, ax)), 0, ax)
                    face.append(f)
                g = [-sg * face[1], -1j * sg * face[0]]
                rest = [d for d in range(dim) if d != a]
                for ax, d in enumerate(rest):
                    e = ws * np.exp(-1j * A[d] * xs)
                    g = [np.moveaxis(np.tensordot(wave * e, f, axes=(1, ax)), 0, ax) for f in g]
                g = [np.expand_dims(f, a) for f in g]
                ka = K[a] + A[a]
                cur = cur + np.exp(-1j * ka * sg * R) * (g[0] + ka * g[1])
        phase = C + sum(tv * K[d] ** 2 / 2 + K[d] * B[d] for d in range(dim))
        cur = 0.5j * (2 * math.pi) ** (-dim / 2) * np.exp(1j * phase) * cur
        if prev is not None:
            amp = amp + 0.5 * dt * (prev + cur)
        prev, t = cur, t + dt
    return amp.reshape(-1)
