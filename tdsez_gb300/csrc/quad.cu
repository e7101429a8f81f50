// Non-separable soft-core potential term by per-element quadrature (quad.h).
// 3D: one CTA per element (k_quad): gather the (p+1)^3 coefficients,
// interpolate to the Q^3 Gauss points axis by axis (sum factorisation, shared
// memory ping-pong), multiply by w V with V from the closed form, project back
// axis by axis and add coef * result to y with atomics (neighbouring elements
// share coefficients); or, for ordinary knots, the streaming kernel below.
// 2D: the assembled stencil (k_stencil2), or for tables beyond kQuad2Table one
// CTA per element (k_quad2).
#include "quad.h"

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cplx.cuh"

namespace tdz {

namespace {

constexpr int kMaxQ = 10;      // Gauss points per element and axis
constexpr int kQThreads = 64;

template <class T> struct QuadParams {
    const void *x;
    void *y;
    int n[3], nel[3], nq;
    const int *off[3];
    const T *N[3], *w[3], *xq[3];
    int nsoft;
    T soft[kMaxSoft][5];
    T cre, cim;
    double cre_d, cim_d;
};

__device__ __forceinline__ void atomic_add_c(float2 *p, float2 v) {
    atomicAdd(&p->x, v.x);
    atomicAdd(&p->y, v.y);
}
__device__ __forceinline__ void atomic_add_c(double2 *p, double2 v) {
    atomicAdd(&p->x, v.x);
    atomicAdd(&p->y, v.y);
}

template <class T> __device__ __forceinline__ T rsqrt_t(T v);
template <> __device__ __forceinline__ float rsqrt_t<float>(float v) { return rsqrtf(v); }
template <> __device__ __forceinline__ double rsqrt_t<double>(double v) { return 1.0 / sqrt(v); }

template <class T, int P>
__global__ void __launch_bounds__(kQThreads) k_quad(const QuadParams<T> prm) {
    using C = typename CT<T>::type;
    constexpr int NP = P + 1;
    constexpr int M = NP > kMaxQ ? NP : kMaxQ;
    constexpr int CAP = M * M * M;
    __shared__ C bufA[CAP], bufB[CAP];
    __shared__ T sN[3][kMaxQ * NP], sW[3][kMaxQ], sX[3][kMaxQ];
    const int Q = prm.nq, tid = threadIdx.x;
    int e = blockIdx.x;
    int el[3] = {0, 0, 0};
    for (int d = 0; d < 3; ++d) { el[d] = e % prm.nel[d]; e /= prm.nel[d]; }
    int o[3] = {0, 0, 0};
    for (int d = 0; d < 3; ++d) o[d] = prm.off[d][el[d]];
    for (int d = 0; d < 3; ++d)
        for (int i = tid; i < Q * NP; i += kQThreads) sN[d][i] = prm.N[d][(size_t)el[d] * Q * NP + i];
    for (int d = 0; d < 3; ++d)
        for (int i = tid; i < Q; i += kQThreads) {
            sW[d][i] = prm.w[d][(size_t)el[d] * Q + i];
            sX[d][i] = prm.xq[d][(size_t)el[d] * Q + i];
        }
    const C *X = static_cast<const C *>(prm.x);
    C *Y = static_cast<C *>(prm.y);
    // extents of the local tensor [z][y][x] during the passes
    for (int i = tid; i < NP * NP * NP; i += kQThreads) {
        const int kx = i % NP, ky = (i / NP) % NP, kz = i / (NP * NP);
        bufA[i] = X[((size_t)(o[2] + kz) * prm.n[1] + (o[1] + ky)) * prm.n[0] + o[0] + kx];
    }
    __syncthreads();
    // x: A[kz][ky][kx] -> B[kz][ky][qx]
    for (int i = tid; i < NP * NP * Q; i += kQThreads) {
        const int qx = i % Q, r = i / Q;
        C acc = czero<C>();
        for (int k = 0; k < NP; ++k) rfma(acc, sN[0][qx * NP + k], bufA[r * NP + k]);
        bufB[i] = acc;
    }
    __syncthreads();
    // y: B[kz][ky][qx] -> A[kz][qy][qx]
    for (int i = tid; i < NP * Q * Q; i += kQThreads) {
        const int qx = i % Q, qy = (i / Q) % Q, kz = i / (Q * Q);
        C acc = czero<C>();
        for (int k = 0; k < NP; ++k) rfma(acc, sN[1][qy * NP + k], bufB[(kz * NP + k) * Q + qx]);
        bufA[i] = acc;
    }
    __syncthreads();
    // z: A[kz][qy][qx] -> B[qz][qy][qx], times w V
    for (int i = tid; i < Q * Q * Q; i += kQThreads) {
        const int qx = i % Q, qy = (i / Q) % Q, qz = i / (Q * Q);
        C acc = czero<C>();
        for (int k = 0; k < NP; ++k) rfma(acc, sN[2][qz * NP + k], bufA[(k * Q + qy) * Q + qx]);
        T v = T(0);
        for (int c = 0; c < prm.nsoft; ++c) {
            const T dx = sX[0][qx] - prm.soft[c][1], dy = sX[1][qy] - prm.soft[c][2], dz = sX[2][qz] - prm.soft[c][3];
            v -= prm.soft[c][0] * rsqrt_t<T>(dx * dx + dy * dy + dz * dz + prm.soft[c][4]);
        }
        const T f = sW[0][qx] * sW[1][qy] * sW[2][qz] * v;
        acc.x *= f;
        acc.y *= f;
        bufB[i] = acc;
    }
    __syncthreads();
    // back z: B[qz][qy][qx] -> A[kz][qy][qx]
    for (int i = tid; i < NP * Q * Q; i += kQThreads) {
        const int qx = i % Q, qy = (i / Q) % Q, kz = i / (Q * Q);
        C acc = czero<C>();
        for (int q = 0; q < Q; ++q) rfma(acc, sN[2][q * NP + kz], bufB[(q * Q + qy) * Q + qx]);
        bufA[i] = acc;
    }
    __syncthreads();
    // back y: A[kz][qy][qx] -> B[kz][ky][qx]
    for (int i = tid; i < NP * NP * Q; i += kQThreads) {
        const int qx = i % Q, ky = (i / Q) % NP, kz = i / (Q * NP);
        C acc = czero<C>();
        for (int q = 0; q < Q; ++q) rfma(acc, sN[1][q * NP + ky], bufA[(kz * Q + q) * Q + qx]);
        bufB[i] = acc;
    }
    __syncthreads();
    // back x and scatter: B[kz][ky][qx] -> y
    for (int i = tid; i < NP * NP * NP; i += kQThreads) {
        const int kx = i % NP, r = i / NP, ky = r % NP, kz = r / NP;
        C acc = czero<C>();
        for (int q = 0; q < Q; ++q) rfma(acc, sN[0][q * NP + kx], bufB[r * Q + q]);
        C out;
        out.x = prm.cre * acc.x - prm.cim * acc.y;
        out.y = prm.cre * acc.y + prm.cim * acc.x;
        atomic_add_c(&Y[((size_t)(o[2] + kz) * prm.n[1] + (o[1] + ky)) * prm.n[0] + o[0] + kx], out);
    }
}

// the same in 2D, for stencils that would take too much memory
template <class T, int P>
__global__ void __launch_bounds__(kQThreads) k_quad2(const QuadParams<T> prm) {
    using C = typename CT<T>::type;
    constexpr int NP = P + 1, M = NP > kMaxQ ? NP : kMaxQ;
    __shared__ C bufA[M * M], bufB[M * M];
    __shared__ T sN[2][kMaxQ * NP], sW[2][kMaxQ], sX[2][kMaxQ];
    const int Q = prm.nq, tid = threadIdx.x;
    const int el[2] = {(int)(blockIdx.x % prm.nel[0]), (int)(blockIdx.x / prm.nel[0])};
    const int ox = prm.off[0][el[0]], oy = prm.off[1][el[1]];
    for (int d = 0; d < 2; ++d) {
        for (int i = tid; i < Q * NP; i += kQThreads) sN[d][i] = prm.N[d][(size_t)el[d] * Q * NP + i];
        for (int i = tid; i < Q; i += kQThreads) {
            sW[d][i] = prm.w[d][(size_t)el[d] * Q + i];
            sX[d][i] = prm.xq[d][(size_t)el[d] * Q + i];
        }
    }
    const C *X = static_cast<const C *>(prm.x);
    C *Y = static_cast<C *>(prm.y);
    for (int i = tid; i < NP * NP; i += kQThreads) bufA[i] = X[(size_t)(oy + i / NP) * prm.n[0] + ox + i % NP];
    __syncthreads();
    // x: A[ky][kx] -> B[ky][qx]
    for (int i = tid; i < NP * Q; i += kQThreads) {
        const int qx = i % Q, ky = i / Q;
        C acc = czero<C>();
        for (int k = 0; k < NP; ++k) rfma(acc, sN[0][qx * NP + k], bufA[ky * NP + k]);
        bufB[i] = acc;
    }
    __syncthreads();
    // y: B[ky][qx] -> A[qy][qx], times w V
    for (int i = tid; i < Q * Q; i += kQThreads) {
        const int qx = i % Q, qy = i / Q;
        C acc = czero<C>();
        for (int k = 0; k < NP; ++k) rfma(acc, sN[1][qy * NP + k], bufB[k * Q + qx]);
        T v = T(0);
        for (int c = 0; c < prm.nsoft; ++c) {
            const T dx = sX[0][qx] - prm.soft[c][1], dy = sX[1][qy] - prm.soft[c][2];
            v -= prm.soft[c][0] * rsqrt_t<T>(dx * dx + dy * dy + prm.soft[c][4]);
        }
        const T f = sW[0][qx] * sW[1][qy] * v;
        acc.x *= f;
        acc.y *= f;
        bufA[i] = acc;
    }
    __syncthreads();
    // back y: A[qy][qx] -> B[ky][qx]
    for (int i = tid; i < NP * Q; i += kQThreads) {
        const int qx = i % Q, ky = i / Q;
        C acc = czero<C>();
        for (int q = 0; q < Q; ++q) rfma(acc, sN[1][q * NP + ky], bufA[q * Q + qx]);
        bufB[i] = acc;
    }
    __syncthreads();
    // back x and scatter
    for (int i = tid; i < NP * NP; i += kQThreads) {
        const int kx = i % NP, ky = i / NP;
        C acc = czero<C>();
        for (int q = 0; q < Q; ++q) rfma(acc, sN[0][q * NP + kx], bufB[ky * Q + q]);
        C out;
        out.x = prm.cre * acc.x - prm.cim * acc.y;
        out.y = prm.cre * acc.y + prm.cim * acc.x;
        atomic_add_c(&Y[(size_t)(oy + ky) * prm.n[0] + ox + kx], out);
    }
}

// ---------------------------------------------------------------- 2D stencil
// The term couples a coefficient to the (2p+1)^2 around it. Its entries are
// stored one triangle only, entry-major (entry e of every coefficient is
// contiguous): e = 0 the diagonal, then the offsets (dx, dy) with dy > 0 or
// dy = 0 and dx > 0; the mirrored ones are read at the partner coefficient.
//
// Bound by GB300's FP64 pipe (FP64 vectors): 2 (2p+1)^2 products per
// coefficient, against 2 (p+1)^2 (4 (p+1)) products and (p+1)^2 potential
// values (FP64 square root and division) per element when the quadrature is
// redone in every apply, which took 251 us on 256^2 elements of degree 4 with
// atomics; the stencil takes 26 us there, and is deterministic.
inline int quad2_entries(int p) { return ((2 * p + 1) * (2 * p + 1) + 1) / 2; }
// entry e >= 0 of the triangle <-> offset (dx, dy): e = dy (2p+1) + dx, dx in -p..p
// (dy = 0: dx >= 0), so that e runs over 0 .. quad2_entries - 1
__host__ __device__ constexpr int quad2_entry(int p, int dx, int dy) { return dy * (2 * p + 1) + dx; }

struct Asm2Params {
    int n0, n1, Q, p;
    const int *off[2], *elo[2], *ehi[2];   // element windows; elements of each coefficient's support
    const double *N[2], *w[2], *xq[2];
    int nel0, nel1, nsoft;
    double soft[kMaxSoft][5];
    double *wv;                            // w V at the Gauss points, [nel1 Q][nel0 Q]
    double *st64;                          // tables to fill (null: not held)
    float *st32;
};

__global__ void k_wv2(const Asm2Params prm) {
    const size_t n = (size_t)prm.nel0 * prm.Q * prm.nel1 * prm.Q;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < n; e += (size_t)gridDim.x * blockDim.x) {
        const int qx = (int)(e % ((size_t)prm.nel0 * prm.Q)), qy = (int)(e / ((size_t)prm.nel0 * prm.Q));
        double v = 0.0;
        for (int c = 0; c < prm.nsoft; ++c) {
            const double dx = prm.xq[0][qx] - prm.soft[c][1], dy = prm.xq[1][qy] - prm.soft[c][2];
            v -= prm.soft[c][0] / sqrt(dx * dx + dy * dy + prm.soft[c][4]);
        }
        prm.wv[e] = prm.w[0][qx] * prm.w[1][qy] * v;
    }
}

// one thread per coefficient and entry (blockIdx.y)
__global__ void __launch_bounds__(128) k_assemble2(const Asm2Params prm) {
    const size_t N = (size_t)prm.n0 * prm.n1;
    const size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (idx >= N) return;
    const int bw = 2 * prm.p + 1, np = prm.p + 1, Q = prm.Q;
    const int e = blockIdx.y;
    // dy (2p+1) + dx with dx in -p..p
    const int dy = (e + prm.p) / bw, dx = e - dy * bw;
    const int i = (int)(idx % prm.n0), j = (int)(idx / prm.n0);
    const int i2 = i + dx, j2 = j + dy;
    double sum = 0.0;
    if (i2 >= 0 && i2 < prm.n0 && j2 < prm.n1) {
        const int x0 = max(prm.elo[0][i], prm.elo[0][i2]), x1 = min(prm.ehi[0][i], prm.ehi[0][i2]);
        const int y0 = max(prm.elo[1][j], prm.elo[1][j2]), y1 = min(prm.ehi[1][j], prm.ehi[1][j2]);
        for (int ey = y0; ey <= y1; ++ey) {
            const double *Ny = prm.N[1] + (size_t)ey * Q * np - prm.off[1][ey];
            for (int qy = 0; qy < Q; ++qy) {
                const double fy = Ny[qy * np + j] * Ny[qy * np + j2];
                const double *wv = prm.wv + ((size_t)ey * Q + qy) * prm.nel0 * Q;
                double row = 0.0;
                for (int ex = x0; ex <= x1; ++ex) {
                    const double *Nx = prm.N[0] + (size_t)ex * Q * np - prm.off[0][ex];
                    for (int qx = 0; qx < Q; ++qx) row = fma(wv[ex * Q + qx], Nx[qx * np + i] * Nx[qx * np + i2], row);
                }
                sum = fma(fy, row, sum);
            }
        }
    }
    if (prm.st64) prm.st64[(size_t)e * N + idx] = sum;
    if (prm.st32) prm.st32[(size_t)e * N + idx] = (float)sum;
}

// y += coef * V_q x from the stencil; a 32 x 8 tile of coefficients per CTA
constexpr int kStX = 32, kStY = 8;
template <class T, int P>
__global__ void __launch_bounds__(kStX *kStY) k_stencil2(const T *__restrict__ st, int n0, int n1, T cre, T cim,
                                                         const typename CT<T>::type *__restrict__ x,
                                                         typename CT<T>::type *__restrict__ y) {
    using C = typename CT<T>::type;
    constexpr int RX = kStX + 2 * P, RY = kStY + 2 * P;
    __shared__ C sx[RY][RX];
    const int tilesX = (n0 + kStX - 1) / kStX;
    const int x0 = (blockIdx.x % tilesX) * kStX, y0 = (blockIdx.x / tilesX) * kStY;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int e = ty * kStX + tx; e < RY * RX; e += kStX * kStY) {
        const int gy = y0 - P + e / RX, gx = x0 - P + e % RX;
        sx[e / RX][e % RX] = gy >= 0 && gy < n1 && gx >= 0 && gx < n0 ? x[(size_t)gy * n0 + gx] : czero<C>();
    }
    __syncthreads();
    const int gx = x0 + tx, gy = y0 + ty;
    if (gx >= n0 || gy >= n1) return;
    const size_t N = (size_t)n0 * n1, idx = (size_t)gy * n0 + gx;
    C up = czero<C>(), lo = czero<C>();   // the triangle and its mirror
#pragma unroll
    for (int dy = 0; dy <= P; ++dy)
#pragma unroll
        for (int dx = -P; dx <= P; ++dx) {
            if (dy == 0 && dx < 0) continue;
            const T *row = st + (size_t)quad2_entry(P, dx, dy) * N;
            rfma(up, row[idx], sx[ty + P + dy][tx + P + dx]);
            if (dy == 0 && dx == 0) continue;
            // the partner (gx - dx, gy - dy); outside the grid x is zero there
            const bool in = gx - dx >= 0 && gx - dx < n0 && gy - dy >= 0;
            rfma(lo, in ? row[idx - (size_t)dy * n0 - dx] : T(0), sx[ty + P - dy][tx + P - dx]);
        }
    up.x += lo.x;
    up.y += lo.y;
    C o = y[idx];
    o.x += cre * up.x - cim * up.y;
    o.y += cre * up.y + cim * up.x;
    y[idx] = o;
}

template <class T, int P> void launch_stencil2(const QuadTerm &q, cd coef, const void *x, void *y, cudaStream_t st) {
    using C = typename CT<T>::type;
    const long long tiles = (long long)((q.n[0] + kStX - 1) / kStX) * ((q.n[1] + kStY - 1) / kStY);
    TDZ_CHECK(tiles < (1LL << 31), TDZ_ERR_UNSUPPORTED, "too many coefficients for the quadrature term");
    const T *tab = static_cast<const T *>((sizeof(T) == 8 ? q.st64 : q.st32).ptr);
    k_stencil2<T, P><<<(unsigned)tiles, dim3(kStX, kStY), 0, st>>>(tab, q.n[0], q.n[1], (T)coef.real(), (T)coef.imag(),
                                                                   static_cast<const C *>(x), static_cast<C *>(y));
}

// ---------------------------------------------------------------- streaming 3D kernel
// For axes whose elements own consecutive coefficient windows (no repeated
// knots) and Q = p + 1 Gauss points. A CTA owns TE x TE elements in (x, y)
// and streams a chunk of their z column. Interpolation of a coefficient plane
// to the tile's (TE Q)^2 quadrature points (x, then y) is done once per
// plane and kept in a ring of p + 1 planes; per z element every quadrature
// column is interpolated along z, multiplied by w V (V from the closed form)
// and projected back along z into a ring of p + 1 accumulator planes; a
// coefficient plane whose elements are all done is projected back along y
// and x and added to y with one atomic per coefficient and tile (the tiles
// overlap by p coefficients per axis, chunk ends by p planes). Versus one CTA
// per element: each interpolated plane serves p + 1 elements and the
// coefficients receive (1 + p/TE)^2 atomic adds instead of (p+1)^3.
// Double-float arithmetic on FP64 vectors (the FGMRES applies: 1/sqrt of the
// potential by rsqrtf and one Newton step in double-float, about 48 bits);
// FP32 vectors take the column kernel below.
template <class A> struct QArith;
template <> struct QArith<dff> {
    using C = cdff;
    using MC = double2;
    using TT = double;
    __device__ static dff from(TT v) { return dff_split(v); }
    __device__ static dff one() { return dff(1.f); }
    __device__ static dff mul(dff a, dff b) { return renorm(tfma(a, b, dff(0.f))); }
    __device__ static dff pot(const QuadParams<TT> &prm, dff x, dff y, dff z) {
        dff v(0.f);
        for (int k = 0; k < prm.nsoft; ++k) {
            const dff dx = renorm(tfma(dff(1.f), x, dff_split(-prm.soft[k][1])));
            const dff dy = renorm(tfma(dff(1.f), y, dff_split(-prm.soft[k][2])));
            const dff dz = renorm(tfma(dff(1.f), z, dff_split(-prm.soft[k][3])));
            const dff r2 = renorm(tfma(dx, dx, tfma(dy, dy, tfma(dz, dz, dff_split(prm.soft[k][4])))));
            // 1/sqrt(r2): rsqrtf, then one Newton step y1 = y0 - y0 (r2 y0^2 - 1) / 2 in double-float
            const float y0 = rsqrtf(r2.hi);
            const dff t = renorm(tfma(dff(y0), dff(y0), dff(0.f)));            // y0^2, exact
            const dff u = renorm(tfma(r2, t, dff(-1.f)));                       // r2 y0^2 - 1
            const dff yi = renorm(tfma(dff(-0.5f * y0), u, dff(y0)));
            v = renorm(tfma(dff_split(-prm.soft[k][0]), yi, v));
        }
        return v;
    }
    __device__ static void scale(cdff &f, dff w) {
        cdff r = czero<cdff>();
        rfma(r, w, f);
        f = cnorm(r);
    }
    __device__ static void atomic_out(double2 *dst, cdff a, double cre, double cim) {
        const double ax = dff_to_double(a.re()), ay = dff_to_double(a.im());
        atomicAdd(&dst->x, cre * ax - cim * ay);
        atomicAdd(&dst->y, cre * ay + cim * ax);
    }
};

template <class A, int P, int TE> struct QStream {
    using C = typename QArith<A>::C;
    static constexpr int NP = P + 1, Q = P + 1, TQ = TE * Q, TC = TE + P, PL = TQ * TQ;
    static constexpr size_t smem = sizeof(C) * ((size_t)2 * NP * PL + TC * TC + TC * TQ);
};
constexpr int kQsThreads = 512;
// tile side in elements: the two rings of (TE (p+1))^2 points fit the 227 KB of shared memory
template <class A, int P> constexpr int qs_te() {
    return P <= 3 ? 7 : (P == 4 ? 6 : 4);
}

template <class A, int P, int TE>
__global__ void __launch_bounds__(kQsThreads) k_quad3_stream(const QuadParams<typename QArith<A>::TT> prm,
                                                             int zchunk) {
    using Q3 = QArith<A>;
    using C = typename Q3::C;
    using MC = typename Q3::MC;
    using S = QStream<A, P, TE>;
    constexpr int NP = S::NP, Q = S::Q, TQ = S::TQ, TC = S::TC, PL = S::PL;
    extern __shared__ __align__(16) unsigned char qs_raw[];
    C *sV = reinterpret_cast<C *>(qs_raw);   // [NP][PL] x,y-interpolated coefficient planes (ring, row qy, column qx)
    C *sG = sV + NP * PL;                    // [NP][PL] z-projected accumulators (ring)
    C *sX = sG + NP * PL;                    // [TC][TC] staged coefficient plane
    C *sU = sX + TC * TC;                    // [TC][TQ] x-interpolated rows, then the back-y rows
    __shared__ A sNx[TE * Q * NP], sNy[TE * Q * NP], sNz[Q * NP];
    __shared__ A sWx[TQ], sWy[TQ], sXx[TQ], sXy[TQ], sWz[Q], sXz[Q];
    const int tid = threadIdx.x;
    const int nelx = prm.nel[0], nely = prm.nel[1], nelz = prm.nel[2];
    const int tilesX = (nelx + TE - 1) / TE;
    const int ex0 = (blockIdx.x % tilesX) * TE, ey0 = (blockIdx.x / tilesX) * TE;
    const int ez0 = blockIdx.y * zchunk, ez1 = min(nelz, ez0 + zchunk);
    if (ez0 >= ez1) return;
    const int n0 = prm.n[0], n1 = prm.n[1], n2 = prm.n[2];
    const int cx0 = prm.off[0][ex0], cy0 = prm.off[1][ey0];
    const A zero = A(0.f);
    // per-tile tables (elements past the grid: zero rows, no contribution)
    for (int i = tid; i < TE * Q * NP; i += kQsThreads) {
        const int e = i / (Q * NP), r = i % (Q * NP);
        sNx[i] = ex0 + e < nelx ? Q3::from(prm.N[0][(size_t)(ex0 + e) * Q * NP + r]) : zero;
        sNy[i] = ey0 + e < nely ? Q3::from(prm.N[1][(size_t)(ey0 + e) * Q * NP + r]) : zero;
    }
    for (int i = tid; i < TQ; i += kQsThreads) {
        const int e = i / Q;
        const bool inx = ex0 + e < nelx, iny = ey0 + e < nely;
        sWx[i] = inx ? Q3::from(prm.w[0][(size_t)ex0 * Q + i]) : zero;
        sXx[i] = inx ? Q3::from(prm.xq[0][(size_t)ex0 * Q + i]) : zero;
        sWy[i] = iny ? Q3::from(prm.w[1][(size_t)ey0 * Q + i]) : zero;
        sXy[i] = iny ? Q3::from(prm.xq[1][(size_t)ey0 * Q + i]) : zero;
    }
    for (int i = tid; i < NP * PL; i += kQsThreads) sG[i] = czero<C>();
    const MC *X = static_cast<const MC *>(prm.x);
    MC *Y = static_cast<MC *>(prm.y);
    __syncthreads();

    // coefficient plane kz -> sV[kz % NP]
    auto interpolate_plane = [&](int kz) {
        for (int i = tid; i < TC * TC; i += kQsThreads) {
            const int iy = i / TC, ix = i % TC, gy = cy0 + iy, gx = cx0 + ix;
            sX[i] = (gy < n1 && gx < n0 && kz < n2) ? load_c<C, MC>(X[((size_t)kz * n1 + gy) * n0 + gx]) : czero<C>();
        }
        __syncthreads();
        for (int i = tid; i < TC * TQ; i += kQsThreads) {   // x: sU[iy][qx]
            const int iy = i / TQ, qx = i % TQ, e = qx / Q;
            const A *nx = sNx + qx * NP;
            C a = czero<C>();
#pragma unroll
            for (int c = 0; c < NP; ++c) rfma(a, nx[c], sX[iy * TC + e + c]);
            sU[i] = cnorm(a);
        }
        __syncthreads();
        C *v = sV + (size_t)(kz % NP) * PL;
        for (int i = tid; i < PL; i += kQsThreads) {        // y: v[qy][qx]
            const int qy = i / TQ, qx = i % TQ, e = qy / Q;
            const A *ny = sNy + qy * NP;
            C a = czero<C>();
#pragma unroll
            for (int c = 0; c < NP; ++c) rfma(a, ny[c], sU[(e + c) * TQ + qx]);
            v[i] = cnorm(a);
        }
        __syncthreads();
    };
    // complete coefficient plane kz in sG[kz % NP]: back along y and x, add to y, clear
    auto flush_plane = [&](int kz) {
        C *g = sG + (size_t)(kz % NP) * PL;
        for (int i = tid; i < TC * TQ; i += kQsThreads) {   // back y: sU[iy][qx]
            const int iy = i / TQ, qx = i % TQ;
            C a = czero<C>();
#pragma unroll
            for (int c = 0; c < NP; ++c) {
                const int e = iy - c;
                if (e < 0 || e >= TE) continue;
#pragma unroll
                for (int q = 0; q < Q; ++q) rfma(a, sNy[(e * Q + q) * NP + c], g[(e * Q + q) * TQ + qx]);
            }
            sU[i] = cnorm(a);
        }
        __syncthreads();
        for (int i = tid; i < TC * TC; i += kQsThreads) {   // back x, add to y
            const int iy = i / TC, ix = i % TC, gy = cy0 + iy, gx = cx0 + ix;
            C a = czero<C>();
#pragma unroll
            for (int c = 0; c < NP; ++c) {
                const int e = ix - c;
                if (e < 0 || e >= TE) continue;
#pragma unroll
                for (int q = 0; q < Q; ++q) rfma(a, sNx[(e * Q + q) * NP + c], sU[iy * TQ + e * Q + q]);
            }
            if (gy < n1 && gx < n0 && kz < n2)
                Q3::atomic_out(&Y[((size_t)kz * n1 + gy) * n0 + gx], cnorm(a), prm.cre_d, prm.cim_d);
        }
        for (int i = tid; i < PL; i += kQsThreads) g[i] = czero<C>();
        __syncthreads();
    };

    const int cz0 = prm.off[2][ez0];
    for (int c = 0; c < P; ++c) interpolate_plane(cz0 + c);
    for (int ez = ez0; ez < ez1; ++ez) {
        const int cz = prm.off[2][ez];
        interpolate_plane(cz + P);
        for (int i = tid; i < Q * NP; i += kQsThreads) sNz[i] = Q3::from(prm.N[2][(size_t)ez * Q * NP + i]);
        for (int i = tid; i < Q; i += kQsThreads) {
            sWz[i] = Q3::from(prm.w[2][(size_t)ez * Q + i]);
            sXz[i] = Q3::from(prm.xq[2][(size_t)ez * Q + i]);
        }
        __syncthreads();
        // z: interpolate, times w V, project back, per quadrature column
        for (int i = tid; i < PL; i += kQsThreads) {
            const int qy = i / TQ, qx = i % TQ;
            C v[NP], g[NP];
#pragma unroll
            for (int c = 0; c < NP; ++c) {
                v[c] = sV[(size_t)((cz + c) % NP) * PL + i];
                g[c] = czero<C>();
            }
            const A wxy = Q3::mul(sWx[qx], sWy[qy]);
#pragma unroll
            for (int qz = 0; qz < Q; ++qz) {
                C f = czero<C>();
#pragma unroll
                for (int c = 0; c < NP; ++c) rfma(f, sNz[qz * NP + c], v[c]);
                f = cnorm(f);
                const A wv = Q3::mul(Q3::mul(wxy, sWz[qz]), Q3::pot(prm, sXx[qx], sXy[qy], sXz[qz]));
                Q3::scale(f, wv);
#pragma unroll
                for (int c = 0; c < NP; ++c) rfma(g[c], sNz[qz * NP + c], f);
            }
#pragma unroll
            for (int c = 0; c < NP; ++c) {
                C &d = sG[(size_t)((cz + c) % NP) * PL + i];
                rfma(d, Q3::one(), cnorm(g[c]));
                d = cnorm(d);
            }
        }
        __syncthreads();
        flush_plane(cz);   // no later element of the chunk touches plane cz
    }
    // planes with contributions from the chunk's last elements
    const int czl = prm.off[2][ez1 - 1];
    for (int c = 1; c <= P; ++c) flush_plane(czl + c);
}

// ---------------------------------------------------------------- column 3D kernel
// The FP32 form of the streaming kernel, with the rings in registers. A CTA owns
// 8 x 8 elements in (x, y) and streams a chunk of their z column; thread (ex,
// qy) owns the Q quadrature columns of element ex at quadrature row qy, so a
// column's interpolated planes (v, the last p + 1) and its z-projected
// accumulators (g, the next p + 1) stay in its registers (degrees 2 and 3; 24
// bytes of a thread are spilled at degree 4, 424 at degree 5), and the
// contractions along x at either end are register loops too. Per coefficient
// plane: y interpolation through shared memory (sX -> sY), then per thread the
// x interpolation, the z element (interpolate, times w V from the closed form,
// project back), the x projection, and a rotation over the 8 lanes of a row
// that adds up the coefficients shared by neighbouring elements; the finished
// row sums (sS) are projected along y and added to y with one atomic per
// coefficient and tile. Two barriers per plane: the y projection of the last
// plane runs beside the y interpolation of the next. Complex products are
// packed FP32 (one issue slot for both components).
//
// Bound by issue slots (about 760 instructions per thread and plane at p = 4,
// 10 warps per SM). The kernel above, with both rings in shared memory and
// five barriers per plane, took 657 us for 96^3 elements of degree 4; this one
// 305 us. Double-float keeps the rings in shared memory: they would need 200
// registers.
template <int P> struct QCols {
    static constexpr int NP = P + 1, Q = P + 1, TE = 8, TQ = TE * Q, TC = TE + P, NT = TE * TQ;
    static constexpr int PY = 24;            // row pitch of sY: two rows of 8 lanes hit different banks
    static constexpr int NZ = Q * NP + 2 * Q;   // z tables of one element: N, w, x
};
__device__ __forceinline__ float2 pfma(float a, float2 v, float2 acc) { return __ffma2_rn(make_float2(a, a), v, acc); }

template <int P>
__global__ void __launch_bounds__(QCols<P>::NT, P <= 3 ? 2 : 1) k_quad3_cols(const QuadParams<float> prm, int zchunk) {
    using S = QCols<P>;
    constexpr int NP = S::NP, Q = S::Q, TE = S::TE, TQ = S::TQ, TC = S::TC, NT = S::NT, PY = S::PY, NZ = S::NZ;
    __shared__ float2 sX[TC * TC], sY[TQ * PY], sS[TQ * TC];
    __shared__ float sNy[TQ * NP], sZ[NZ];
    constexpr bool kNxReg = P <= 4;          // x tables in registers, or (degree 5) in shared memory
    __shared__ float sNx[kNxReg ? 1 : Q * NP * TE];
    const int tid = threadIdx.x, ex = tid & 7, qy = tid >> 3;
    const int nelx = prm.nel[0], nely = prm.nel[1], nelz = prm.nel[2];
    const int tilesX = (nelx + TE - 1) / TE;
    const int ex0 = (blockIdx.x % tilesX) * TE, ey0 = (blockIdx.x / tilesX) * TE;
    const int ez0 = blockIdx.y * zchunk, nelc = min(nelz, ez0 + zchunk) - ez0;
    if (nelc <= 0) return;
    const int n0 = prm.n[0], n1 = prm.n[1], n2 = prm.n[2];
    const int cx0 = prm.off[0][ex0], cy0 = prm.off[1][ey0], cz0 = prm.off[2][ez0];
    const float2 *__restrict__ X = static_cast<const float2 *>(prm.x);
    float2 *__restrict__ Y = static_cast<float2 *>(prm.y);
    // this thread's element and row (elements past the grid: zero tables, no contribution)
    const bool inx = ex0 + ex < nelx, iny = ey0 + qy / Q < nely;
    float nxr[kNxReg ? Q * NP : 1], wxy[Q], xx[Q];
    if constexpr (kNxReg) {
#pragma unroll
        for (int i = 0; i < Q * NP; ++i) nxr[i] = inx ? prm.N[0][(size_t)(ex0 + ex) * Q * NP + i] : 0.f;
    } else {
        for (int i = tid; i < Q * NP * TE; i += NT)
            sNx[i] = ex0 + i % TE < nelx ? prm.N[0][(size_t)(ex0 + i % TE) * Q * NP + i / TE] : 0.f;
    }
    auto nx = [&](int q, int c) {
        if constexpr (kNxReg) return nxr[q * NP + c];
        else return sNx[(q * NP + c) * TE + ex];
    };
    const float wy = iny ? prm.w[1][(size_t)ey0 * Q + qy] : 0.f, yy = iny ? prm.xq[1][(size_t)ey0 * Q + qy] : 0.f;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        wxy[q] = inx ? prm.w[0][(size_t)(ex0 + ex) * Q + q] * wy : 0.f;
        xx[q] = inx ? prm.xq[0][(size_t)(ex0 + ex) * Q + q] : 0.f;
    }
    for (int i = tid; i < TQ * NP; i += NT)
        sNy[i] = ey0 + i / (Q * NP) < nely ? prm.N[1][(size_t)ey0 * Q * NP + i] : 0.f;
    // coefficient plane k of the chunk: one element per thread, a plane ahead
    const int lx = cx0 + tid % TC, ly = cy0 + tid / TC;
    const bool ldr = tid < TC * TC && lx < n0 && ly < n1;
    const int nplanes = nelc + P;
    auto load_x = [&](int k) {
        return ldr && k < nplanes && cz0 + k < n2 ? X[((size_t)(cz0 + k) * n1 + ly) * n0 + lx] : make_float2(0.f, 0.f);
    };
    auto load_z = [&](int e) {   // z tables of element ez0 + e
        if (tid >= NZ || e < 0 || e >= nelc) return 0.f;
        const size_t el = ez0 + e;
        return tid < Q * NP ? prm.N[2][el * Q * NP + tid]
                            : tid < Q * NP + Q ? prm.w[2][el * Q + tid - Q * NP] : prm.xq[2][el * Q + tid - Q * NP - Q];
    };
    if (tid < TC * TC) sX[tid] = load_x(0);
    float2 px = load_x(1);
    float pz = load_z(-P);
    __syncthreads();

    float2 v[Q][NP], g[Q][NP];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int c = 0; c < NP; ++c) v[q][c] = g[q][c] = make_float2(0.f, 0.f);

    // step k: plane k enters the rings, element k - P is integrated, plane
    // k - P leaves (the last P steps only drain)
#pragma unroll 1
    for (int k = 0; k < nelc + 2 * P + 1; ++k) {
        // y interpolation of plane k; y projection of the plane that left in the last step
        if (k < nplanes)
            for (int i = tid; i < TQ * TC; i += NT) {
                const int r = i / TC, ix = i % TC, e = r / Q;
                float2 a = make_float2(0.f, 0.f);
#pragma unroll
                for (int c = 0; c < NP; ++c) a = pfma(sNy[r * NP + c], sX[(e + c) * TC + ix], a);
                sY[r * PY + ix] = a;
            }
        if (tid < NZ) sZ[tid] = pz;
        const int i = NT - 1 - tid, kz = cz0 + k - 1 - P;
        if (k > P && i < TC * TC) {
            const int iy = i / TC, ix = i % TC, gy = cy0 + iy, gx = cx0 + ix;
            float2 a = make_float2(0.f, 0.f);
#pragma unroll
            for (int c = 0; c < NP; ++c) {
                const int e = iy - c;
                if (e < 0 || e >= TE) continue;
#pragma unroll
                for (int q = 0; q < Q; ++q) a = pfma(sNy[(e * Q + q) * NP + c], sS[(e * Q + q) * TC + ix], a);
            }
            if (gy < n1 && gx < n0 && kz < n2)
                atomicAdd(&Y[((size_t)kz * n1 + gy) * n0 + gx],
                          make_float2(prm.cre * a.x - prm.cim * a.y, prm.cre * a.y + prm.cim * a.x));
        }
        __syncthreads();
        if (k == nelc + 2 * P) break;
        // the next plane and the next element's z tables
        if (tid < TC * TC) sX[tid] = px;
        px = load_x(k + 2);
        pz = load_z(k + 1 - P);
        // x interpolation of this thread's element
#pragma unroll
        for (int q = 0; q < Q; ++q) {
#pragma unroll
            for (int c = 0; c < P; ++c) v[q][c] = v[q][c + 1];
            v[q][P] = make_float2(0.f, 0.f);
        }
        if (k < nplanes) {
#pragma unroll
            for (int c = 0; c < NP; ++c) {
                const float2 u = sY[qy * PY + ex + c];
#pragma unroll
                for (int q = 0; q < Q; ++q) v[q][P] = pfma(nx(q, c), u, v[q][P]);
            }
        }
        if (k < P) {
            __syncthreads();
            continue;
        }
        if (k < nplanes) {
#pragma unroll
            for (int qz = 0; qz < Q; ++qz) {
                const float wz = sZ[Q * NP + qz], zz = sZ[Q * NP + Q + qz];
                float pot[Q];
#pragma unroll
                for (int q = 0; q < Q; ++q) pot[q] = 0.f;
                for (int m = 0; m < prm.nsoft; ++m) {
                    const float dy = yy - prm.soft[m][2], dz = zz - prm.soft[m][3];
                    const float r = fmaf(dz, dz, fmaf(dy, dy, prm.soft[m][4]));
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        const float dx = xx[q] - prm.soft[m][1];
                        pot[q] = fmaf(-prm.soft[m][0], rsqrtf(fmaf(dx, dx, r)), pot[q]);
                    }
                }
                float nz[NP];
#pragma unroll
                for (int c = 0; c < NP; ++c) nz[c] = sZ[qz * NP + c];
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    float2 f = make_float2(0.f, 0.f);
#pragma unroll
                    for (int c = 0; c < NP; ++c) f = pfma(nz[c], v[q][c], f);
                    const float wv = wxy[q] * wz * pot[q];
                    f = __fmul2_rn(f, make_float2(wv, wv));
#pragma unroll
                    for (int c = 0; c < NP; ++c) g[q][c] = pfma(nz[c], f, g[q][c]);
                }
            }
        }
        // plane k - P is complete: project along x. part(c) belongs to
        // coefficient ex + c; rotated by c lanes it lands on lane (ex + c) & 7,
        // as coefficient ex + c (main) or, past the eighth, 8 + lane (over)
        float2 main = make_float2(0.f, 0.f), over = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < NP; ++c) {
            float2 part = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < Q; ++q) part = pfma(nx(q, c), g[q][0], part);
            float2 r;
            r.x = __shfl_sync(0xffffffffu, part.x, (ex - c) & 7, 8);
            r.y = __shfl_sync(0xffffffffu, part.y, (ex - c) & 7, 8);
            if (ex >= c) main = __fadd2_rn(main, r);
            else over = __fadd2_rn(over, r);
        }
        sS[qy * TC + ex] = main;
        if (ex < P) sS[qy * TC + TE + ex] = over;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
#pragma unroll
            for (int c = 0; c < P; ++c) g[q][c] = g[q][c + 1];
            g[q][P] = make_float2(0.f, 0.f);
        }
        __syncthreads();
    }
}

// the streaming kernel applies: 3D, Q = p + 1, consecutive element offsets on every axis
bool stream_ok(const QuadTerm &q) { return q.dim == 3 && q.nq == q.p + 1 && q.consecutive; }

template <int P> void launch_q3c(const QuadTerm &q, const QuadParams<float> &prm, cudaStream_t st) {
    using S = QCols<P>;
    const int tiles = ((q.nel[0] + S::TE - 1) / S::TE) * ((q.nel[1] + S::TE - 1) / S::TE);
    // z chunks: the fewest plane steps of a full wave, halo planes included
    const int slots = sm_count() * (P <= 3 ? 2 : 1);
    int best = 1;
    long long cost = -1;
    for (int c = 1; c <= 32 && c <= q.nel[2]; ++c) {
        const int z = (q.nel[2] + c - 1) / c;
        const long long t = ((long long)tiles * ((q.nel[2] + z - 1) / z) + slots - 1) / slots * (z + 2 * P + 1);
        if (cost < 0 || t < cost) { cost = t; best = c; }
    }
    const int zchunk = (q.nel[2] + best - 1) / best;
    k_quad3_cols<P><<<dim3(tiles, (q.nel[2] + zchunk - 1) / zchunk), S::NT, 0, st>>>(prm, zchunk);
}

template <class A, int P>
void launch_q3s(const QuadTerm &q, const QuadParams<typename QArith<A>::TT> &prm, cudaStream_t st) {
    constexpr int TE = qs_te<A, P>();
    using S = QStream<A, P, TE>;
    auto kern = k_quad3_stream<A, P, TE>;
    static_assert(S::smem <= 200 * 1024, "quadrature rings larger than the shared memory");
    static std::atomic<unsigned long long> done{0};
    once_per_device(done, [&] { allow_smem(kern, S::smem); });
    const int tiles = ((q.nel[0] + TE - 1) / TE) * ((q.nel[1] + TE - 1) / TE);
    // about two CTAs per SM in total, z chunks no shorter than 4 (p + 1) elements
    int chunks = std::max(1, (2 * sm_count() + tiles - 1) / tiles);
    chunks = std::max(1, std::min(chunks, q.nel[2] / (4 * (P + 1))));
    const int zchunk = (q.nel[2] + chunks - 1) / chunks;
    kern<<<dim3(tiles, (q.nel[2] + zchunk - 1) / zchunk), kQsThreads, S::smem, st>>>(prm, zchunk);
}

template <class T>
QuadParams<T> make_qparams(const QuadTerm &q, cd coef, const void *x, void *y) {
    QuadParams<T> prm{};
    const bool dbl = sizeof(T) == 8;
    prm.x = x;
    prm.y = y;
    prm.nq = q.nq;
    for (int d = 0; d < 3; ++d) {
        prm.n[d] = q.n[d];
        prm.nel[d] = q.nel[d];
        if (d < q.dim) {
            prm.off[d] = q.off[d].as<int>();
            prm.N[d] = static_cast<const T *>((dbl ? q.N64[d] : q.N32[d]).ptr);
            prm.w[d] = static_cast<const T *>((dbl ? q.w64[d] : q.w32[d]).ptr);
            prm.xq[d] = static_cast<const T *>((dbl ? q.x64[d] : q.x32[d]).ptr);
        }
    }
    prm.nsoft = q.nsoft;
    for (int c = 0; c < q.nsoft; ++c)
        for (int k = 0; k < 5; ++k) prm.soft[c][k] = (T)q.soft[c][k];
    prm.cre = (T)coef.real();
    prm.cim = (T)coef.imag();
    prm.cre_d = coef.real();
    prm.cim_d = coef.imag();
    return prm;
}

template <class T, int P>
void launch_q(const QuadTerm &q, const QuadParams<T> &prm, cudaStream_t st) {
    const long long nel = (long long)q.nel[0] * q.nel[1] * (q.dim == 3 ? q.nel[2] : 1);
    TDZ_CHECK(nel < (1LL << 31), TDZ_ERR_UNSUPPORTED, "too many elements for the quadrature term");
    if (q.dim == 3) k_quad<T, P><<<(unsigned)nel, kQThreads, 0, st>>>(prm);
    else k_quad2<T, P><<<(unsigned)nel, kQThreads, 0, st>>>(prm);
}

template <class T>
void dispatch_q(const QuadTerm &q, cd coef, const void *x, void *y, cudaStream_t st) {
    if (q.dim == 2 && (sizeof(T) == 8 ? q.st64 : q.st32).ptr) {
        switch (q.p) {
        case 2: launch_stencil2<T, 2>(q, coef, x, y, st); return;
        case 3: launch_stencil2<T, 3>(q, coef, x, y, st); return;
        case 4: launch_stencil2<T, 4>(q, coef, x, y, st); return;
        case 5: launch_stencil2<T, 5>(q, coef, x, y, st); return;
        default: throw Error(TDZ_ERR_UNSUPPORTED, "quadrature term supports degrees 2..5");
        }
    }
    const QuadParams<T> prm = make_qparams<T>(q, coef, x, y);
    if (stream_ok(q)) {   // FP32: FP32 arithmetic; FP64 vectors: double-float arithmetic
        auto stream = [&](auto deg) {
            constexpr int P = decltype(deg)::value;
            if constexpr (std::is_same<T, float>::value) launch_q3c<P>(q, prm, st);
            else launch_q3s<dff, P>(q, prm, st);
        };
        switch (q.p) {
        case 2: stream(std::integral_constant<int, 2>{}); return;
        case 3: stream(std::integral_constant<int, 3>{}); return;
        case 4: stream(std::integral_constant<int, 4>{}); return;
        case 5: stream(std::integral_constant<int, 5>{}); return;
        default: break;
        }
    }
    switch (q.p) {
    case 2: launch_q<T, 2>(q, prm, st); break;
    case 3: launch_q<T, 3>(q, prm, st); break;
    case 4: launch_q<T, 4>(q, prm, st); break;
    case 5: launch_q<T, 5>(q, prm, st); break;
    default: throw Error(TDZ_ERR_UNSUPPORTED, "quadrature term supports degrees 2..5");
    }
}

void assemble2(QuadTerm &q, const Space &s, int precs) {
    Asm2Params prm{};
    prm.n0 = q.n[0];
    prm.n1 = q.n[1];
    prm.Q = q.nq;
    prm.p = q.p;
    prm.nel0 = q.nel[0];
    prm.nel1 = q.nel[1];
    DevBuf lo[2], hi[2], wv;
    for (int d = 0; d < 2; ++d) {
        const Axis1D &a = s.ax[d];
        std::vector<int> l(a.n, a.nel), h(a.n, -1);
        for (int e = 0; e < a.nel; ++e)
            for (int k = a.offset[e]; k <= a.offset[e] + a.p; ++k) {
                l[k] = std::min(l[k], e);
                h[k] = std::max(h[k], e);
            }
        upload(lo[d], l);
        upload(hi[d], h);
        prm.off[d] = q.off[d].as<int>();
        prm.elo[d] = lo[d].as<int>();
        prm.ehi[d] = hi[d].as<int>();
        prm.N[d] = q.N64[d].as<double>();
        prm.w[d] = q.w64[d].as<double>();
        prm.xq[d] = q.x64[d].as<double>();
    }
    prm.nsoft = q.nsoft;
    for (int c = 0; c < q.nsoft; ++c)
        for (int k = 0; k < 5; ++k) prm.soft[c][k] = q.soft[c][k];
    const size_t N = (size_t)q.n[0] * q.n[1], pts = (size_t)q.nel[0] * q.nel[1] * q.nq * q.nq;
    const int ne = quad2_entries(q.p);
    wv.alloc(pts * sizeof(double));
    if (precs & kQuad64) q.st64.alloc(N * ne * sizeof(double));
    if (precs & kQuad32) q.st32.alloc(N * ne * sizeof(float));
    prm.wv = wv.as<double>();
    prm.st64 = q.st64.as<double>();
    prm.st32 = q.st32.as<float>();
    const size_t blocks = (N + 127) / 128;
    TDZ_CHECK(blocks < (1ull << 31), TDZ_ERR_UNSUPPORTED, "too many coefficients for the quadrature term");
    k_wv2<<<(int)std::min<size_t>((pts + 255) / 256, (size_t)16 * sm_count()), 256>>>(prm);
    k_assemble2<<<dim3((unsigned)blocks, ne), 128>>>(prm);
    TDZ_CUDA(cudaGetLastError());
    count_launch(2);
    TDZ_CUDA(cudaStreamSynchronize(nullptr));   // the stencil is used on any stream
}

}  // namespace

void QuadTerm::build(const Space &s, int nsoft_, const double *soft_, int precs, size_t table) {
    on = nsoft_ > 0;
    if (!on) return;
    TDZ_CHECK(s.dim >= 2, TDZ_ERR_UNSUPPORTED, "soft-core centres need a 2D or 3D space");
    TDZ_CHECK(nsoft_ <= kMaxSoft, TDZ_ERR_UNSUPPORTED, "at most 8 soft-core centres");
    TDZ_CHECK(soft_ != nullptr, TDZ_ERR_ARG, "soft-core parameters missing");
    TDZ_CHECK(s.nquad >= 1 && s.nquad <= kMaxQ, TDZ_ERR_UNSUPPORTED, "quadrature term supports 1..10 Gauss points");
    nsoft = nsoft_;
    for (int c = 0; c < nsoft; ++c) {
        for (int k = 0; k < 5; ++k) soft[c][k] = soft_[5 * c + k];
        TDZ_CHECK(soft[c][4] > 0.0, TDZ_ERR_ARG, "soft-core parameter a must be positive");
    }
    dim = s.dim;
    p = s.ax[0].p;
    nq = s.nquad;
    consecutive = true;
    for (int d = 0; d < dim; ++d) {
        const Axis1D &a = s.ax[d];
        TDZ_CHECK(a.nq == nq && a.p == p, TDZ_ERR_INTERNAL, "axis tables disagree");
        for (int e = 0; e + 1 < a.nel; ++e)
            if (a.offset[e + 1] != a.offset[e] + 1) consecutive = false;
        nel[d] = a.nel;
        n[d] = a.n;
        std::vector<int> o(a.offset.begin(), a.offset.end());
        upload(off[d], o);
        upload(N64[d], a.N);
        upload(w64[d], a.wq);
        upload(x64[d], a.xq);
        upload(N32[d], std::vector<float>(a.N.begin(), a.N.end()));
        upload(w32[d], std::vector<float>(a.wq.begin(), a.wq.end()));
        upload(x32[d], std::vector<float>(a.xq.begin(), a.xq.end()));
    }
    if (dim == 2 && (size_t)n[0] * n[1] * quad2_entries(p) * sizeof(double) <= table) assemble2(*this, s, precs);
}

void QuadTerm::apply(cd coef, int prec, const void *x, void *y, cudaStream_t st) const {
    if (!on || coef == cd(0.0)) return;
    if (prec == TDZ_FP32) dispatch_q<float>(*this, coef, x, y, st);
    else dispatch_q<double>(*this, coef, x, y, st);
    TDZ_CUDA(cudaGetLastError());
    count_launch();
}

}  // namespace tdz
