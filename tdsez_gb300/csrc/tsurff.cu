// t-SURFF surface flux on the device (FP64): trace of psi and (1/m) d_n psi
// at the surface Gauss points, the factorised flux of FluxGrid
// (src/tsurff.cpp:478-534) as two small contractions per face, and the
// trapezoid accumulation of AddFlux (src/tsurff.cpp:439-469). The Volkov
// integrals (RK4, src/tsurff.cpp:395-428) are advanced on the host.
#include "tsurff.h"

#include <array>
#include <cmath>

#include "cplx.cuh"

namespace tdz {

namespace {

__device__ __forceinline__ double2 cexpi(double a) {
    double s, c;
    sincos(a, &s, &c);
    return make_double2(c, s);
}
__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

struct AxisView {
    int n, p, Q;
    const int *off;
    const double *val, *der;    // [Q][p+1]
};

struct FaceParams {
    AxisView b, c;
    int a, side;                 // normal axis, side (0: -R, 1: +R)
    int stride[3];               // coefficient strides per axis
    int wall_off;                // first basis index of the normal axis at the wall
    int pa;                      // degree of the normal axis
    const double *wval, *wder;   // p+1 values / derivatives at the wall
    const double *xb, *xc, *wb, *wc;   // node coordinates and weights
    double Ab, Ac;
    int nb, nc;                  // momenta along b and c
    const double2 *eb, *ec;      // exp(-i k x_q) along b and c: [nk][Q]
    size_t goff, hoff, toff;     // this face's place in g, H and T
};
struct Faces {
    FaceParams f[6];
    int nf;
    double inv_mass;
};

struct KGrid {
    int nk[3];
    const double *k[3];
};

// per-momentum phases of one sample, one axis after the other:
// wall[k] = exp(-i (k + A_d) R) and fin[k] = exp(i (t k^2 / 2m + k B_d / m)),
// so the kernels over the momentum grid multiply table entries instead of
// calling sincos 2 dim + 1 times per momentum
struct PhaseParams {
    KGrid kg;
    double A[3], B[3], R, t, inv2m, invm;
    double2 *wall, *fin;
};

// g[0] = -e (1/m) d_n psi, g[1] = -i sigma e psi / m with e = w exp(-i A_t.x_t)
// at every surface node of every face (blockIdx.y; the row past the last face
// fills the phase tables). `lanes` threads per node share its (p+1)^(dim-1)
// tangential products and reduce by shuffles: with a few thousand nodes the
// kernel is bound by the latency of the gathered loads, which one thread per
// node issued one after the other (22 us per face at 1024 nodes of degree 4;
// all four faces of that case take 12 us now).
__global__ void __launch_bounds__(256) k_trace(const Faces fs, const PhaseParams pp, int lanes,
                                               const double2 *__restrict__ psi, double2 *__restrict__ gall) {
    const int gid = blockIdx.x * blockDim.x + threadIdx.x;
    if ((int)blockIdx.y == fs.nf) {
        int i = gid;
        for (int d = 0; d < 3; ++d) {
            if (i >= 0 && i < pp.kg.nk[d]) {
                const double k = pp.kg.k[d][i];
                const int o = (d > 0 ? pp.kg.nk[0] : 0) + (d > 1 ? pp.kg.nk[1] : 0) + i;
                pp.wall[o] = cexpi(-(k + pp.A[d]) * pp.R);
                pp.fin[o] = cexpi(pp.t * k * k * pp.inv2m + k * pp.B[d] * pp.invm);
            }
            i -= pp.kg.nk[d];
        }
        return;
    }
    const FaceParams &f = fs.f[blockIdx.y];
    const int Qb = f.b.Q, Qc = f.c.Q;
    const int idx = gid / lanes, lane = gid % lanes;
    const bool valid = idx < Qb * Qc;
    const int ib = valid ? idx / Qc : 0, ic = valid ? idx % Qc : 0;
    const int ob = f.b.off[ib], oc = f.c.off[ic];
    const size_t sa = (size_t)f.stride[f.a], sb = (size_t)f.stride[f.a == 0 ? 1 : 0], sc = (size_t)f.stride[f.a == 2 ? 1 : 2];
    double2 v = make_double2(0, 0), dn = make_double2(0, 0);
    const int nbc = (f.b.p + 1) * (f.c.p + 1);
    for (int e = lane; valid && e < nbc; e += lanes) {
        const int jb = e / (f.c.p + 1), jc = e % (f.c.p + 1);
        const double vt = f.b.val[ib * (f.b.p + 1) + jb] * f.c.val[ic * (f.c.p + 1) + jc];
        const double2 *q = psi + (size_t)f.wall_off * sa + (size_t)(ob + jb) * sb + (size_t)(oc + jc) * sc;
        double2 sv = make_double2(0, 0), sd = make_double2(0, 0);
#pragma unroll 4
        for (int ja = 0; ja <= f.pa; ++ja) {
            const double2 ps = q[(size_t)ja * sa];
            const double va = f.wval[ja], da = f.wder[ja];
            sv.x += va * ps.x; sv.y += va * ps.y;
            sd.x += da * ps.x; sd.y += da * ps.y;
        }
        v.x += vt * sv.x; v.y += vt * sv.y;
        dn.x += vt * sd.x; dn.y += vt * sd.y;
    }
    for (int o = lanes / 2; o > 0; o >>= 1) {
        v.x += __shfl_down_sync(0xffffffffu, v.x, o);
        v.y += __shfl_down_sync(0xffffffffu, v.y, o);
        dn.x += __shfl_down_sync(0xffffffffu, dn.x, o);
        dn.y += __shfl_down_sync(0xffffffffu, dn.y, o);
    }
    if (!valid || lane != 0) return;
    const double sm = (f.side ? 1.0 : -1.0) * fs.inv_mass;
    dn.x *= sm;
    dn.y *= sm;
    const double xb = f.xb[ib], xc = f.xc[ic];
    double2 e = cexpi(-(f.Ab * xb + f.Ac * xc));
    const double w = f.wb[ib] * f.wc[ic];
    e.x *= w; e.y *= w;
    const double2 g1 = cmul(e, dn);
    // -i sigma e psi / m
    const double2 ev = cmul(e, v);
    double2 *g = gall + f.goff;
    g[idx] = make_double2(-g1.x, -g1.y);
    g[(size_t)Qb * Qc + idx] = make_double2(sm * ev.y, -sm * ev.x);
}

// The momentum contractions of every face (blockIdx.y), the same form twice:
//   STAGE 0: H[s][kc][ib] = sum_ic g[s][ib][ic] Ec[kc][ic]
//   STAGE 1: T[s][kb][kc] = sum_ib H[s][kc][ib] Eb[kb][ib]
// `lanes` threads split the contracted index (contiguous in both operands)
// and compute J momenta of one row; FP64 products, the partial sums reduced
// by shuffles. One thread per output with the whole sum left a 2D face 256
// serial chains of 1024 dependent FP64 products (515 us per face; 26 us for
// all four faces split this way). J = 4 reuses the row operand where the
// outputs fill the chip anyway, which halves the L2 reads of 3D faces.
template <int STAGE, int J>
__global__ void __launch_bounds__(256) k_face(const Faces fs, int lanes, const double2 *__restrict__ inall,
                                              double2 *__restrict__ outall) {
    const FaceParams &f = fs.f[blockIdx.y];
    const int Q = STAGE == 0 ? f.c.Q : f.b.Q;
    const int rows = STAGE == 0 ? f.b.Q : f.nc, nj = STAGE == 0 ? f.nc : f.nb;
    const double2 *E = STAGE == 0 ? f.ec : f.eb;
    const double2 *in = inall + (STAGE == 0 ? f.goff : f.hoff);
    double2 *out = outall + (STAGE == 0 ? f.hoff : f.toff);
    const int ng = (nj + J - 1) / J;
    const long long gid = (blockIdx.x * (long long)blockDim.x + threadIdx.x) / lanes;
    const int lane = threadIdx.x % lanes;
    const bool valid = gid < 2LL * ng * rows;
    const int r = (int)(gid % rows);
    const int j0 = (int)((gid / rows) % ng) * J, s = (int)(gid / ((long long)rows * ng));
    double2 acc[J];
#pragma unroll
    for (int j = 0; j < J; ++j) acc[j] = make_double2(0, 0);
    if (valid) {
        const double2 *ir = in + ((size_t)s * rows + r) * Q;
        for (int q = lane; q < Q; q += lanes) {
            const double2 a = ir[q];
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const double2 b = E[(size_t)min(j0 + j, nj - 1) * Q + q];
                acc[j].x += a.x * b.x - a.y * b.y;
                acc[j].y += a.x * b.y + a.y * b.x;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < J; ++j)
        for (int o = lanes / 2; o > 0; o >>= 1) {
            acc[j].x += __shfl_down_sync(0xffffffffu, acc[j].x, o);
            acc[j].y += __shfl_down_sync(0xffffffffu, acc[j].y, o);
        }
    if (!valid || lane != 0) return;
#pragma unroll
    for (int j = 0; j < J; ++j)
        if (j0 + j < nj) out[((size_t)s * nj + j0 + j) * rows + r] = acc[j];
}

struct Finish {
    double2 pre;       // the common factor
    double h;          // trapezoid weight
    int have_prev;
};

// flux(k) = sum over faces of exp(-i (k_a + A_a) sigma R) (T_1 + (k_a + A_a) T_2),
// faces 2 a and 2 a + 1 being the sides of axis a
__device__ __forceinline__ double2 flux_at(const Faces &fs, const PhaseParams &pp, const int *kk, const double2 *Tall) {
    double2 o = make_double2(0, 0);
    int woff = 0;
    for (int a = 0; 2 * a < fs.nf; ++a) {
        const double2 ph = pp.wall[woff + kk[a]];
        const double ka = pp.kg.k[a][kk[a]] + pp.A[a];
        woff += pp.kg.nk[a];
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            const FaceParams &f = fs.f[2 * a + side];
            const int b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
            const double2 *T = Tall + f.toff;
            const size_t e = (size_t)kk[b] * f.nc + kk[c];
            const double2 t1 = T[e], t2 = T[(size_t)f.nb * f.nc + e];
            const double2 v = cmul(make_double2(ph.x, side ? ph.y : -ph.y),
                                   make_double2(t1.x + ka * t2.x, t1.y + ka * t2.y));
            o.x += v.x;
            o.y += v.y;
        }
    }
    return o;
}
__device__ __forceinline__ void k_index(const KGrid &kg, size_t idx, int *kk) {
    kk[2] = (int)(idx % kg.nk[2]);
    kk[1] = (int)((idx / kg.nk[2]) % kg.nk[1]);
    kk[0] = (int)(idx / ((size_t)kg.nk[2] * kg.nk[1]));
}
// pre times the Volkov factor prod_d exp(i (t k_d^2 / 2m + k_d B_d / m))
__device__ __forceinline__ double2 volkov_at(const PhaseParams &pp, const int *kk, double2 pre) {
    const int *nk = pp.kg.nk;
    const double2 a = cmul(pre, pp.fin[kk[0]]);
    return cmul(cmul(a, pp.fin[nk[0] + kk[1]]), pp.fin[nk[0] + nk[1] + kk[2]]);
}

// one sample: c = pre Volkov(k) flux(k); amp += h (prev + c); prev = c
__global__ void k_accumulate(const Faces fs, const PhaseParams pp, const double2 *__restrict__ T, Finish fin,
                             double2 *prev, double2 *amp) {
    const size_t tot = (size_t)pp.kg.nk[0] * pp.kg.nk[1] * pp.kg.nk[2];
    const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (idx >= tot) return;
    int kk[3];
    k_index(pp.kg, idx, kk);
    const double2 c = cmul(volkov_at(pp, kk, fin.pre), flux_at(fs, pp, kk, T));
    if (fin.have_prev) {
        const double2 p = prev[idx];
        double2 a = amp[idx];
        a.x += fin.h * (p.x + c.x);
        a.y += fin.h * (p.y + c.y);
        amp[idx] = a;
    }
    prev[idx] = c;
}

// end term: amp[q_e] += w_e pre Volkov(k) flux(k); the entries of one node
// name distinct momenta
__global__ void k_end_acc(const Faces fs, const PhaseParams pp, const double2 *__restrict__ T, double2 pre,
                          const int *__restrict__ q, const double *__restrict__ w, int m, double2 *__restrict__ amp) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m) return;
    const size_t idx = (size_t)q[e];
    int kk[3];
    k_index(pp.kg, idx, kk);
    const double2 c = cmul(volkov_at(pp, kk, pre), flux_at(fs, pp, kk, T));
    double2 a = amp[idx];
    a.x += w[e] * c.x;
    a.y += w[e] * c.y;
    amp[idx] = a;
}

inline int blocks_for(size_t n, int t = 256) { return (int)((n + t - 1) / t); }

}  // namespace

void TSurff::setup(const Space &s, const tdz_tsurff_opts &o, tdz_field_fn f, void *ctx) {
    dim = s.dim;
    R = o.radius;
    mass = o.mass > 0 ? o.mass : 1.0;
    V0 = o.v0;
    sign = -o.charge;
    dt = o.dt;
    TDZ_CHECK(dt > 0, TDZ_ERR_ARG, "t-SURFF needs the time step");
    TDZ_CHECK(R > 0, TDZ_ERR_ARG, "t-SURFF radius must be positive");
    field = f;
    field_ctx = ctx;
    nq = o.nquad > 0 ? o.nquad : s.nquad;
    std::vector<double> gx, gw;
    gauss_legendre(nq, gx, gw);
    nktot = 1;
    for (int d = 0; d < 3; ++d) {
        AxisTables &T = ax[d];
        nodes[d].clear();
        weights[d].clear();
        k[d].clear();
        if (d >= dim) {
            nodes[d] = {0.0};
            weights[d] = {1.0};
            k[d] = {0.0};
            nk[d] = 1;
            T.n = 1; T.p = 0; T.Q = 1;
            upload(T.off, std::vector<int>{0});
            upload(T.val, std::vector<double>{1.0});
            upload(T.der, std::vector<double>{0.0});
            T.wall_off[0] = T.wall_off[1] = 0;
            T.wall_val[0] = T.wall_val[1] = {1.0};
            T.wall_der[0] = T.wall_der[1] = {0.0};
        } else {
            const Axis1D &A = s.ax[d];
            TDZ_CHECK(A.U.front() < -R && A.U.back() > R, TDZ_ERR_ARG, "t-SURFF surface is not inside the box");
            for (size_t j = 0; j + 1 < A.U.size(); ++j) {
                const double lo = std::max(A.U[j], -R), hi = std::min(A.U[j + 1], R);
                if (hi <= lo) continue;
                for (int q = 0; q < nq; ++q) {
                    nodes[d].push_back(0.5 * (lo + hi) + 0.5 * (hi - lo) * gx[q]);
                    weights[d].push_back(0.5 * (hi - lo) * gw[q]);
                }
            }
            T.n = A.n;
            T.p = A.p;
            T.Q = (int)nodes[d].size();
            std::vector<int> off(T.Q);
            std::vector<double> val((size_t)T.Q * (A.p + 1)), der((size_t)T.Q * (A.p + 1)), tmp(2 * (A.p + 1));
            for (int q = 0; q < T.Q; ++q) {
                const int sp = find_span(A.U, A.p, A.n, nodes[d][q]);
                ders_basis(A.U, A.p, sp, nodes[d][q], 1, tmp.data());
                off[q] = sp - A.p;
                for (int r = 0; r <= A.p; ++r) { val[(size_t)q * (A.p + 1) + r] = tmp[r]; der[(size_t)q * (A.p + 1) + r] = tmp[A.p + 1 + r]; }
            }
            upload(T.off, off);
            upload(T.val, val);
            upload(T.der, der);
            hoff[d] = off;
            hval[d].assign(val.begin(), val.end());
            for (int side = 0; side < 2; ++side) {
                const double x = side ? R : -R;
                const int sp = find_span(A.U, A.p, A.n, x);
                ders_basis(A.U, A.p, sp, x, 1, tmp.data());
                T.wall_off[side] = sp - A.p;
                T.wall_val[side].assign(tmp.begin(), tmp.begin() + A.p + 1);
                T.wall_der[side].assign(tmp.begin() + A.p + 1, tmp.begin() + 2 * (A.p + 1));
            }
            nk[d] = std::max(1, o.nk[d]);
            for (int i = 0; i < nk[d]; ++i)
                k[d].push_back(nk[d] == 1 ? o.kmin[d] : o.kmin[d] + i * (o.kmax[d] - o.kmin[d]) / (nk[d] - 1));
        }
        n[d] = T.n;
        // exp(-i k x_q) table
        std::vector<double2> ek((size_t)nk[d] * T.Q);
        for (int i = 0; i < nk[d]; ++i)
            for (int q = 0; q < T.Q; ++q) {
                const double a = -k[d][i] * nodes[d][q];
                ek[(size_t)i * T.Q + q] = make_double2(std::cos(a), std::sin(a));
            }
        upload(T.ek, ek);
        nktot *= nk[d];
    }
    size_t gtot = 0, htot = 0, ttot = 0;   // work arrays of all 2 dim faces
    for (int a = 0; a < dim; ++a) {
        const int b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
        gtot += (size_t)4 * ax[b].Q * ax[c].Q;
        htot += (size_t)4 * ax[b].Q * nk[c];
        ttot += (size_t)4 * nk[b] * nk[c];
    }
    g.alloc(gtot * sizeof(double2));
    H.alloc(htot * sizeof(double2));
    T.alloc(ttot * sizeof(double2));
    tab.alloc((size_t)2 * (nk[0] + nk[1] + nk[2]) * sizeof(double2));
    for (DevBuf *b : {&prev, &amp}) b->alloc(nktot * sizeof(double2));
    TDZ_CUDA(cudaMemset(amp.ptr, 0, nktot * sizeof(double2)));
    // wall values and node coordinates / weights per axis
    std::vector<double> wv, wd;
    for (int d = 0; d < 3; ++d)
        for (int side = 0; side < 2; ++side) {
            wv.insert(wv.end(), ax[d].wall_val[side].begin(), ax[d].wall_val[side].end());
            wd.insert(wd.end(), ax[d].wall_der[side].begin(), ax[d].wall_der[side].end());
            wv.resize(wv.size() + (16 - ax[d].wall_val[side].size()), 0.0);
            wd.resize(wd.size() + (16 - ax[d].wall_der[side].size()), 0.0);
        }
    upload(wallv, wv);
    upload(walld, wd);
    std::vector<double> xw;
    for (int d = 0; d < 3; ++d) xw.insert(xw.end(), nodes[d].begin(), nodes[d].end());
    for (int d = 0; d < 3; ++d) xw.insert(xw.end(), weights[d].begin(), weights[d].end());
    std::vector<double> kall;
    for (int d = 0; d < 3; ++d) kall.insert(kall.end(), k[d].begin(), k[d].end());
    upload(phase, xw);        // node coordinates then weights
    kdev_host = kall;
    upload(kdev, kall);
}

namespace {
using Volkov7 = std::array<double, 7>;   // A_x, A_y, A_z, B_x, B_y, B_z, C
// one classical fourth-order Runge-Kutta step (Kutta's tableau) of y' = f(t, y)
template <class F> Volkov7 rk4_step(const F &f, double t, const Volkov7 &y, double h) {
    auto along = [&](const Volkov7 &s, double c) {
        Volkov7 r;
        for (int i = 0; i < 7; ++i) r[i] = y[i] + c * s[i];
        return r;
    };
    const Volkov7 s1 = f(t, y);
    const Volkov7 s2 = f(t + 0.5 * h, along(s1, 0.5 * h));
    const Volkov7 s3 = f(t + 0.5 * h, along(s2, 0.5 * h));
    const Volkov7 s4 = f(t + h, along(s3, h));
    Volkov7 out;
    for (int i = 0; i < 7; ++i) out[i] = y[i] + h * (s1[i] + 2.0 * (s2[i] + s3[i]) + s4[i]) / 6.0;
    return out;
}
}  // namespace

// Volkov phases of the surface states from the last sample time to t:
// A' = -s E(t), B' = A, C' = |A|^2 / 2m + V0, by Runge-Kutta substeps of at
// most dt/2 (the substep rule of AdvanceVolkov, src/tsurff.cpp:395-428, which
// the flux's parity with the reference depends on)
void TSurff::advance_volkov(double t) {
    const double span = t - vt;
    if (span <= 0) return;
    const int substeps = std::max(1, (int)std::ceil(span / (0.5 * dt) - 1e-9));
    const double ds = span / substeps;
    auto deriv = [&](double tt, const Volkov7 &y) {
        Volkov7 d{};
        double a2 = 0.0;
        for (int a = 0; a < 3; ++a) {
            d[a] = (a < dim && field) ? -sign * field(a, tt, field_ctx) : 0.0;
            d[3 + a] = y[a];
            a2 += y[a] * y[a];
        }
        d[6] = a2 / (2.0 * mass) + V0;
        return d;
    };
    Volkov7 y{A[0], A[1], A[2], B[0], B[1], B[2], C};
    for (int k = 0; k < substeps; ++k) y = rk4_step(deriv, vt + k * ds, y, ds);
    for (int a = 0; a < 3; ++a) { A[a] = y[a]; B[a] = y[3 + a]; }
    C = y[6];
    vt = t;
}

KGridHost TSurff::kgrid() const {
    KGridHost kg;
    size_t ka = 0;
    for (int d = 0; d < 3; ++d) {
        kg.nk[d] = nk[d];
        kg.k[d] = kdev.as<double>() + ka;
        ka += k[d].size();
    }
    return kg;
}

namespace {
// smallest power of two >= v, at most 32: threads that share one sum of v terms
inline int lanes_for(int v) {
    int l = 1;
    while (l < v && l < 32) l *= 2;
    return l;
}

Faces make_faces(const TSurff &ts) {
    const double *xw = ts.phase.as<double>();
    size_t xoff[3], woff[3], acc = 0;
    for (int d = 0; d < 3; ++d) { xoff[d] = acc; acc += ts.nodes[d].size(); }
    for (int d = 0; d < 3; ++d) { woff[d] = acc; acc += ts.weights[d].size(); }
    Faces fs{};
    fs.nf = 2 * ts.dim;
    fs.inv_mass = 1.0 / ts.mass;
    size_t go = 0, ho = 0, to = 0;
    for (int a = 0; a < ts.dim; ++a)
        for (int side = 0; side < 2; ++side) {
            const int b = a == 0 ? 1 : 0, c = a == 2 ? 1 : 2;
            FaceParams &f = fs.f[2 * a + side];
            auto view = [&](int d) {
                const auto &t = ts.ax[d];
                return AxisView{t.n, t.p, t.Q, t.off.as<int>(), t.val.as<double>(), t.der.as<double>()};
            };
            f.b = view(b);
            f.c = view(c);
            f.a = a;
            f.side = side;
            f.stride[0] = 1;
            f.stride[1] = ts.n[0];
            f.stride[2] = ts.n[0] * ts.n[1];
            f.wall_off = ts.ax[a].wall_off[side];
            f.pa = ts.ax[a].p;
            f.wval = ts.wallv.as<double>() + (a * 2 + side) * 16;
            f.wder = ts.walld.as<double>() + (a * 2 + side) * 16;
            f.xb = xw + xoff[b];
            f.xc = xw + xoff[c];
            f.wb = xw + woff[b];
            f.wc = xw + woff[c];
            f.Ab = ts.A[b];
            f.Ac = ts.A[c];
            f.nb = ts.nk[b];
            f.nc = ts.nk[c];
            f.eb = ts.ax[b].ek.as<double2>();
            f.ec = ts.ax[c].ek.as<double2>();
            f.goff = go;
            f.hoff = ho;
            f.toff = to;
            go += (size_t)2 * f.b.Q * f.c.Q;
            ho += (size_t)2 * f.b.Q * f.nc;
            to += (size_t)2 * f.nb * f.nc;
        }
    return fs;
}

PhaseParams make_phases(const TSurff &ts) {
    PhaseParams pp{};
    const KGridHost kh = ts.kgrid();
    int tot = 0;
    for (int d = 0; d < 3; ++d) {
        pp.kg.nk[d] = kh.nk[d];
        pp.kg.k[d] = kh.k[d];
        pp.A[d] = ts.A[d];
        pp.B[d] = ts.B[d];
        tot += kh.nk[d];
    }
    pp.R = ts.R;
    pp.t = ts.vt;
    pp.inv2m = 0.5 / ts.mass;
    pp.invm = 1.0 / ts.mass;
    pp.wall = ts.tab.as<double2>();
    pp.fin = pp.wall + tot;
    return pp;
}

template <int STAGE> void contract_faces(const Faces &fs, const double2 *in, double2 *out, cudaStream_t st) {
    int qmax = 1;
    long long gmax1 = 0, gmax4 = 0;
    for (int i = 0; i < fs.nf; ++i) {
        const FaceParams &f = fs.f[i];
        const long long rows = STAGE == 0 ? f.b.Q : f.nc, nj = STAGE == 0 ? f.nc : f.nb;
        qmax = std::max(qmax, STAGE == 0 ? f.c.Q : f.b.Q);
        gmax1 = std::max(gmax1, 2 * rows * nj);
        gmax4 = std::max(gmax4, 2 * rows * ((nj + 3) / 4));
    }
    const int lanes = lanes_for(qmax);
    // four momenta per group once that still leaves 16 warps per SM
    const bool four = gmax4 * lanes * fs.nf >= (long long)16 * 32 * sm_count();
    const dim3 grid(blocks_for((size_t)(four ? gmax4 : gmax1) * lanes), fs.nf);
    if (four) k_face<STAGE, 4><<<grid, 256, 0, st>>>(fs, lanes, in, out);
    else k_face<STAGE, 1><<<grid, 256, 0, st>>>(fs, lanes, in, out);
    TDZ_CUDA(cudaGetLastError());
    count_launch();
}

// T = the face contractions of psi at the current Volkov time (FluxGrid), and
// the phase tables of the momentum grid
void face_contractions(const TSurff &ts, const Faces &fs, const PhaseParams &pp, const double2 *psi, cudaStream_t st) {
    int nodes = 1, nbc = 1;
    for (int i = 0; i < fs.nf; ++i) {
        nodes = std::max(nodes, fs.f[i].b.Q * fs.f[i].c.Q);
        nbc = std::max(nbc, (fs.f[i].b.p + 1) * (fs.f[i].c.p + 1));
    }
    const int lanes = lanes_for(nbc);
    const int kt = pp.kg.nk[0] + pp.kg.nk[1] + pp.kg.nk[2];
    double2 *g = ts.g.as<double2>(), *H = ts.H.as<double2>();
    k_trace<<<dim3(blocks_for(std::max((size_t)nodes * lanes, (size_t)kt)), fs.nf + 1), 256, 0, st>>>(fs, pp, lanes, psi, g);
    TDZ_CUDA(cudaGetLastError());
    count_launch();
    // below 3D axis c is a single node and momentum with factor one: H = g
    if (ts.dim == 3) contract_faces<0>(fs, g, H, st);
    contract_faces<1>(fs, ts.dim == 3 ? H : g, ts.T.as<double2>(), st);
}
}  // namespace

void TSurff::sample(double t, const double2 *psi, cudaStream_t st) {
    if (have_prev && t == prevT) return;
    TDZ_CHECK(!have_prev || t > prevT, TDZ_ERR_ARG, "t-SURFF sample times must increase");
    advance_volkov(t);
    const Faces fs = make_faces(*this);
    const PhaseParams pp = make_phases(*this);
    face_contractions(*this, fs, pp, psi, st);
    const double two_pi = 2.0 * std::acos(-1.0);
    const double pref = 0.5 * std::pow(two_pi, -0.5 * dim);
    // pre = (i/2) (2 pi)^{-d/2} exp(i C)
    const Finish fin{make_double2(-pref * std::sin(C), pref * std::cos(C)), 0.5 * (t - prevT), have_prev ? 1 : 0};
    k_accumulate<<<blocks_for(nktot), 256, 0, st>>>(fs, pp, T.as<double2>(), fin, prev.as<double2>(), amp.as<double2>());
    TDZ_CUDA(cudaGetLastError());
    count_launch();
    prevT = t;
    have_prev = true;
    ++samples;
}

void TSurff::add_weighted_flux(const double2 *phi, const int *q, const double *w, int m, cudaStream_t st) {
    if (m <= 0) return;
    const Faces fs = make_faces(*this);
    const PhaseParams pp = make_phases(*this);
    face_contractions(*this, fs, pp, phi, st);
    const double pref = 0.5 * std::pow(2.0 * std::acos(-1.0), -0.5 * dim);
    const double2 pre = make_double2(-pref * std::sin(C), pref * std::cos(C));
    k_end_acc<<<blocks_for((size_t)m), 256, 0, st>>>(fs, pp, T.as<double2>(), pre, q, w, m, amp_end.as<double2>());
    TDZ_CUDA(cudaGetLastError());
    count_launch();
}

namespace {
// out[a][k][b] = sum_i F[k][i] in[a][i][b] (complex, double-float arithmetic)
__global__ void k_axis_dense(const double2 *__restrict__ F, const double2 *__restrict__ in, double2 *__restrict__ out,
                             long long A, int nk, int ni, long long B) {
    const long long total = A * nk * B;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const long long b = t % B, r = t / B;
        const int k = (int)(r % nk);
        const long long a = r / nk;
        cdff acc = czero<cdff>();
        const double2 *fk = F + (size_t)k * ni;
        const double2 *ia = in + (size_t)a * ni * B + b;
        for (int i = 0; i < ni; ++i) {
            const cdff f = load_c<cdff, double2>(fk[i]);
            const cdff v = load_c<cdff, double2>(ia[(size_t)i * B]);
            cfma(acc, f, v);
        }
        out[t] = store_c<double2, cdff>(cnorm(acc));
    }
}
}  // namespace

void TSurff::interior(const double2 *psi, std::vector<cd> &out, cudaStream_t st) {
    // F_d[k][i] = sum_q w_q exp(-i (k + A_d) x_q) B_i(x_q) over the in-box nodes
    for (int d = 0; d < 3; ++d) {
        std::vector<double2> f((size_t)nk[d] * n[d], make_double2(0.0, 0.0));
        if (d >= dim) {
            f[0] = make_double2(1.0, 0.0);
        } else {
            const int pp = ax[d].p + 1;
            for (size_t q = 0; q < nodes[d].size(); ++q)
                for (int kk = 0; kk < nk[d]; ++kk) {
                    const double ph = -(k[d][kk] + A[d]) * nodes[d][q];
                    const cd e = weights[d][q] * cd(std::cos(ph), std::sin(ph));
                    for (int b = 0; b < pp; ++b) {
                        const int i = hoff[d][q] + b;
                        const cd v = e * hval[d][q * pp + b];
                        double2 &z = f[(size_t)kk * n[d] + i];
                        z.x += v.real();
                        z.y += v.imag();
                    }
                }
        }
        upload(F[d], f);
    }
    // contract x, then y, then z: [z][y][x] -> [z][y][kx] -> [z][ky][kx] -> [kz][ky][kx]
    const size_t w0 = (size_t)n[2] * n[1] * nk[0], w1 = (size_t)n[2] * nk[1] * nk[0];
    if (work[0].bytes < w0 * sizeof(double2)) work[0].alloc(w0 * sizeof(double2));
    if (work[1].bytes < std::max(w1, nktot) * sizeof(double2)) work[1].alloc(std::max(w1, nktot) * sizeof(double2));
    auto pass = [&](const double2 *src, double2 *dst, long long a, int d, long long b) {
        const long long total = a * nk[d] * b;
        const int blocks = (int)std::min<long long>((total + 255) / 256, 16LL * sm_count());
        k_axis_dense<<<blocks, 256, 0, st>>>(F[d].as<double2>(), src, dst, a, nk[d], n[d], b);
        TDZ_CUDA(cudaGetLastError());
        count_launch();
    };
    pass(psi, work[0].as<double2>(), (long long)n[2] * n[1], 0, 1);
    pass(work[0].as<double2>(), work[1].as<double2>(), n[2], 1, nk[0]);
    pass(work[1].as<double2>(), work[0].as<double2>(), 1, 2, (long long)nk[1] * nk[0]);
    std::vector<double2> h(nktot);
    TDZ_CUDA(cudaMemcpyAsync(h.data(), work[0].ptr, nktot * sizeof(double2), cudaMemcpyDeviceToHost, st));
    TDZ_CUDA(cudaStreamSynchronize(st));
    // times the Volkov phase (2 pi)^(-d/2) exp(i (C + T k^2 / 2m + k.B / m)), k_x slowest
    const double norm = std::pow(2.0 * M_PI, -0.5 * dim);
    out.assign(nktot, cd(0.0));
    for (int i = 0; i < nk[0]; ++i)
        for (int j = 0; j < nk[1]; ++j)
            for (int l = 0; l < nk[2]; ++l) {
                const double kv[3] = {k[0][i], k[1][j], k[2][l]};
                double ph = C;
                for (int d = 0; d < dim; ++d) ph += vt * kv[d] * kv[d] / (2.0 * mass) + kv[d] * B[d] / mass;
                const double2 g = h[((size_t)l * nk[1] + j) * nk[0] + i];
                out[((size_t)i * nk[1] + j) * nk[2] + l] = norm * cd(std::cos(ph), std::sin(ph)) * cd(g.x, g.y);
            }
}

}  // namespace tdz
