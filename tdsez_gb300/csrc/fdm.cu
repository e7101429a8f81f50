// Fast-diagonalisation preconditioner (Lynch-Rice-Thomas) for the z-layered
// operator family: dense eigenvector transforms along x and y and one banded
// complex LU solve per (x, y) line along z with the live stage coefficients.
// Exact inverse (up to FP32 rounding) when the inner axes carry only mass and
// stiffness, which is the heterostructure's case. 3D with n_x, n_y <= 256:
// the transforms run on the tensor cores (tgemm.cu) over row-planar FP32
// buffers; otherwise (2D, wider axes) on the smem-tiled FP32 GEMMs below.
#include "fdm.h"

#include <cmath>

#include "apply_kernels.cuh"

namespace tdz {

// ---------------------------------------------------------------- host eigen
void gen_eig(const BandD &S, const BandD &M, std::vector<double> &V, std::vector<double> &lam) {
    const int n = S.n, p = S.p;
    std::vector<double> L((size_t)n * n, 0.0), C((size_t)n * n, 0.0);
    auto m = [&](int i, int j) { return std::abs(i - j) <= p ? M.at(i, j) : 0.0; };
    auto s = [&](int i, int j) { return std::abs(i - j) <= p ? S.at(i, j) : 0.0; };
    // Cholesky M = L L^T (banded)
    for (int i = 0; i < n; ++i)
        for (int j = std::max(0, i - p); j <= i; ++j) {
            double v = m(i, j);
            for (int k = std::max(0, i - p); k < j; ++k) v -= L[(size_t)i * n + k] * L[(size_t)j * n + k];
            if (i == j) {
                TDZ_CHECK(v > 0, TDZ_ERR_INTERNAL, "mass band not positive definite");
                L[(size_t)i * n + i] = std::sqrt(v);
            } else L[(size_t)i * n + j] = v / L[(size_t)j * n + j];
        }
    // C = L^-1 S L^-T : first W = L^-1 S (columns), then C = W L^-T
    std::vector<double> W((size_t)n * n, 0.0);
    for (int c = 0; c < n; ++c)
        for (int i = 0; i < n; ++i) {
            double v = s(i, c);
            for (int k = std::max(0, i - p); k < i; ++k) v -= L[(size_t)i * n + k] * W[(size_t)k * n + c];
            W[(size_t)i * n + c] = v / L[(size_t)i * n + i];
        }
    for (int r = 0; r < n; ++r)
        for (int i = 0; i < n; ++i) {
            double v = W[(size_t)r * n + i];
            for (int k = std::max(0, i - p); k < i; ++k) v -= L[(size_t)i * n + k] * C[(size_t)r * n + k];
            C[(size_t)r * n + i] = v / L[(size_t)i * n + i];
        }
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < i; ++j) {
            const double a = 0.5 * (C[(size_t)i * n + j] + C[(size_t)j * n + i]);
            C[(size_t)i * n + j] = C[(size_t)j * n + i] = a;
        }
    // cyclic Jacobi on C, accumulate Q
    std::vector<double> Q((size_t)n * n, 0.0);
    for (int i = 0; i < n; ++i) Q[(size_t)i * n + i] = 1.0;
    for (int sweep = 0; sweep < 60; ++sweep) {
        double off = 0.0, tot = 0.0;
        for (int i = 0; i < n; ++i)
            for (int j = 0; j < n; ++j) {
                const double v = C[(size_t)i * n + j] * C[(size_t)i * n + j];
                tot += v;
                if (i != j) off += v;
            }
        if (off <= 1e-30 * tot) break;
        for (int pi = 0; pi < n - 1; ++pi)
            for (int qi = pi + 1; qi < n; ++qi) {
                const double apq = C[(size_t)pi * n + qi];
                if (std::abs(apq) < 1e-300) continue;
                const double app = C[(size_t)pi * n + pi], aqq = C[(size_t)qi * n + qi];
                const double theta = 0.5 * (aqq - app) / apq;
                const double t = (theta >= 0 ? 1.0 : -1.0) / (std::abs(theta) + std::sqrt(theta * theta + 1.0));
                const double c = 1.0 / std::sqrt(t * t + 1.0), sn = t * c;
                for (int k = 0; k < n; ++k) {
                    const double akp = C[(size_t)k * n + pi], akq = C[(size_t)k * n + qi];
                    C[(size_t)k * n + pi] = c * akp - sn * akq;
                    C[(size_t)k * n + qi] = sn * akp + c * akq;
                }
                for (int k = 0; k < n; ++k) {
                    const double apk = C[(size_t)pi * n + k], aqk = C[(size_t)qi * n + k];
                    C[(size_t)pi * n + k] = c * apk - sn * aqk;
                    C[(size_t)qi * n + k] = sn * apk + c * aqk;
                }
                for (int k = 0; k < n; ++k) {
                    const double qkp = Q[(size_t)k * n + pi], qkq = Q[(size_t)k * n + qi];
                    Q[(size_t)k * n + pi] = c * qkp - sn * qkq;
                    Q[(size_t)k * n + qi] = sn * qkp + c * qkq;
                }
            }
    }
    lam.assign(n, 0.0);
    for (int i = 0; i < n; ++i) lam[i] = C[(size_t)i * n + i];
    // V = L^-T Q (back substitution with L^T, column by column)
    V.assign((size_t)n * n, 0.0);
    for (int c = 0; c < n; ++c)
        for (int i = n - 1; i >= 0; --i) {
            double v = Q[(size_t)i * n + c];
            for (int k = i + 1; k <= std::min(n - 1, i + p); ++k) v -= L[(size_t)k * n + i] * V[(size_t)k * n + c];
            V[(size_t)i * n + c] = v / L[(size_t)i * n + i];
        }
}

namespace {

// multiply-accumulate of the transforms: complex data times a real or complex
// matrix entry (FP32, or FP64 for the FP64 preconditioner)
template <class C, class R> __device__ __forceinline__ void gmac(C &acc, C a, R b) {
    acc.x = fma(a.x, b, acc.x);
    acc.y = fma(a.y, b, acc.y);
}
template <class C, class R> __device__ __forceinline__ void gmac_r(C &acc, R a, C b) {
    acc.x = fma(a, b.x, acc.x);
    acc.y = fma(a, b.y, acc.y);
}
template <class C> __device__ __forceinline__ void gmac_c(C &acc, C a, C b) {
    acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
    acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}
__device__ __forceinline__ void gmac2(float2 &acc, float2 a, float b) { gmac(acc, a, b); }
__device__ __forceinline__ void gmac2(float2 &acc, float a, float2 b) { gmac_r(acc, a, b); }
__device__ __forceinline__ void gmac2(float2 &acc, float2 a, float2 b) { gmac_c(acc, a, b); }
__device__ __forceinline__ void gmac2(double2 &acc, double2 a, double b) { gmac(acc, a, b); }
__device__ __forceinline__ void gmac2(double2 &acc, double a, double2 b) { gmac_r(acc, a, b); }
__device__ __forceinline__ void gmac2(double2 &acc, double2 a, double2 b) { gmac_c(acc, a, b); }
template <class T> __device__ __forceinline__ T gzero();
template <> __device__ __forceinline__ float gzero<float>() { return 0.f; }
template <> __device__ __forceinline__ float2 gzero<float2>() { return make_float2(0.f, 0.f); }
template <> __device__ __forceinline__ double gzero<double>() { return 0.0; }
template <> __device__ __forceinline__ double2 gzero<double2>() { return make_double2(0.0, 0.0); }

// Transform along x: C[M][N] = A[M][K] . B[K][N] (A the complex data, B real or
// complex); along y, per plane z: C_z = A . B_z (A the real or complex matrix,
// B_z complex). Row-major, FP32 or FP64 FMAs; a CTA of 256 threads computes a
// (16 TT)^2 tile, TT x TT outputs per thread. The next K chunk is requested
// into registers before the current one is used and shared memory is double
// buffered, so a chunk costs one barrier and its load latency overlaps the
// products. TT = 2 where TT = 4 would leave SMs idle, in FP32 with KS = 2 groups
// of 256 threads that take every other K chunk and add up at the end. MA and MC
// are the types in memory: the first and the last transform of an FP32
// application read and write the FP64 vectors themselves. A 260 x 260 x 260
// complex transform (the 2D runs) has 25 tiles of 64 x 64 and 81 of 32 x 32: 79
// us with one buffer and 25 tiles, 21 us with 81 and 3 us for the cast beside
// it; with two groups 24 us from FP64 and 15 us to FP64, no cast.
// K chunk: half as long for the FP64 64 x 64 tiles, whose buffers would pass 48 KB
template <class C2, int TT> constexpr int kGemmK = sizeof(C2) == 16 && TT == 4 ? 8 : 16;
template <class D, class S> __device__ __forceinline__ D gconv(const S &v) { return v; }
template <> __device__ __forceinline__ float2 gconv<float2, double2>(const double2 &v) {
    return make_float2(dff_split(v.x).hi, dff_split(v.y).hi);
}
template <> __device__ __forceinline__ double2 gconv<double2, float2>(const float2 &v) {
    return make_double2(f2d_exact(v.x), f2d_exact(v.y));
}
template <class MA, class TA, class TB, class C2, class MC, int TT, int KS>
__global__ void __launch_bounds__(256 * KS) k_gemm(const MA *__restrict__ A, const TB *__restrict__ B,
                                                   MC *__restrict__ Cm, int M, int N, int K, size_t bplane,
                                                   size_t cplane) {
    constexpr int BT = 16 * TT, BK = kGemmK<C2, TT>, L = BT * BK / 256;
    __shared__ TA As[KS][2][BK][BT + 1];
    __shared__ TB Bs[KS][2][BK][BT + 1];
    const int tid = threadIdx.x % 256, grp = threadIdx.x / 256, tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BT, n0 = blockIdx.x * BT;
    B += blockIdx.z * bplane;
    Cm += blockIdx.z * cplane;
    C2 acc[TT][TT];
#pragma unroll
    for (int r = 0; r < TT; ++r)
#pragma unroll
        for (int c = 0; c < TT; ++c) acc[r][c] = gzero<C2>();
    TA pa[L];
    TB pb[L];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int q = 0; q < L; ++q) {
            const int i = tid + 256 * q;
            const int gm = m0 + i / BK, ka = k0 + i % BK, kb = k0 + i / BT, gn = n0 + i % BT;
            pa[q] = gm < M && ka < K ? gconv<TA, MA>(A[(size_t)gm * K + ka]) : gzero<TA>();
            pb[q] = kb < K && gn < N ? B[(size_t)kb * N + gn] : gzero<TB>();
        }
    };
    auto put = [&](int s) {
#pragma unroll
        for (int q = 0; q < L; ++q) {
            const int i = tid + 256 * q;
            As[grp][s][i % BK][i / BK] = pa[q];
            Bs[grp][s][i / BT][i % BT] = pb[q];
        }
    };
    fetch(grp * BK);
    put(0);
    __syncthreads();
    int s = 0;
    for (int k0 = 0; k0 < K; k0 += KS * BK, s ^= 1) {   // chunk k0 + grp BK of each group
        const bool more = k0 + KS * BK < K;
        if (more) fetch(k0 + (KS + grp) * BK);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            TA a[TT];
            TB b[TT];
#pragma unroll
            for (int r = 0; r < TT; ++r) a[r] = As[grp][s][k][ty * TT + r];
#pragma unroll
            for (int c = 0; c < TT; ++c) b[c] = Bs[grp][s][k][tx + 16 * c];
#pragma unroll
            for (int r = 0; r < TT; ++r)
#pragma unroll
                for (int c = 0; c < TT; ++c) gmac2(acc[r][c], a[r], b[c]);
        }
        if (more) put(s ^ 1);   // last read before the previous barrier
        __syncthreads();
    }
    if constexpr (KS == 2) {
        __shared__ C2 part[TT * TT][256];
        if (grp == 1)
#pragma unroll
            for (int r = 0; r < TT; ++r)
#pragma unroll
                for (int c = 0; c < TT; ++c) part[r * TT + c][tid] = acc[r][c];
        __syncthreads();
        if (grp == 1) return;
#pragma unroll
        for (int r = 0; r < TT; ++r)
#pragma unroll
            for (int c = 0; c < TT; ++c) {
                const C2 v = part[r * TT + c][tid];
                acc[r][c].x += v.x;
                acc[r][c].y += v.y;
            }
    }
#pragma unroll
    for (int r = 0; r < TT; ++r)
#pragma unroll
        for (int c = 0; c < TT; ++c) {
            const int gm = m0 + ty * TT + r, gn = n0 + tx + 16 * c;
            if (gm < M && gn < N) Cm[(size_t)gm * N + gn] = gconv<MC, C2>(acc[r][c]);
        }
}

template <class MA, class TA, class TB, class C2, class MC>
void gemm(const MA *A, const TB *B, MC *Cm, int M, int N, int K, int planes, size_t bplane, size_t cplane,
          cudaStream_t st) {
    constexpr int KS = sizeof(C2) == 8 ? 2 : 1;
    const long long big = (long long)((M + 63) / 64) * ((N + 63) / 64) * planes;
    if (big >= 2LL * sm_count())
        k_gemm<MA, TA, TB, C2, MC, 4, 1>
            <<<dim3((N + 63) / 64, (M + 63) / 64, planes), 256, 0, st>>>(A, B, Cm, M, N, K, bplane, cplane);
    else
        k_gemm<MA, TA, TB, C2, MC, 2, KS>
            <<<dim3((N + 31) / 32, (M + 31) / 32, planes), 256 * KS, 0, st>>>(A, B, Cm, M, N, K, bplane, cplane);
}
// along x: rows of n0 entries times an n0 x n0 matrix
template <class TM, class C2, class MI, class MO>
void gemm_x(const DevBuf &Mx, const MI *in, MO *out, int rows, int n0, cudaStream_t st) {
    gemm<MI, C2, TM, C2, MO>(in, Mx.as<TM>(), out, rows, n0, n0, 1, 0, 0, st);
}
// along y: an n1 x n1 matrix times every n1 x n0 plane
template <class TM, class C2>
void gemm_y(const DevBuf &My, const C2 *in, C2 *out, int n0, int n1, int planes, cudaStream_t st) {
    const size_t plane = (size_t)n0 * n1;
    gemm<TM, TM, C2, C2, C2>(My.as<TM>(), in, out, n1, n0, n1, planes, plane, plane, st);
}

__device__ __forceinline__ float2 cmulf(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 crecf(float2 a) {
    const float d = 1.f / (a.x * a.x + a.y * a.y);
    return make_float2(a.x * d, -a.y * d);
}

// natural-order complex FP64 -> row-planar FP32 [z][y][c][x] (row pitch ld)
__global__ void k_to_planar(const double2 *__restrict__ r, float *__restrict__ a, int n0, size_t rows, int ld) {
    const size_t total = rows * (size_t)n0;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t row = e / n0;
        const int x = (int)(e % n0);
        const double2 v = r[e];   // FP64 -> FP32 without the (slow) FP64 pipe
        a[(row * 2) * ld + x] = dff_split(v.x).hi;
        a[(row * 2 + 1) * ld + x] = dff_split(v.y).hi;
    }
}

// the same with ||z||^2: FP32 sums per thread (a few dozen squares of FP32
// values), FP64 per block into part[block]
__global__ void __launch_bounds__(256) k_from_planar_norm(const float *__restrict__ a, double2 *__restrict__ z, int n0,
                                                          size_t rows, int ld, double *__restrict__ part) {
    const size_t total = rows * (size_t)n0;
    float acc = 0.f;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t row = e / n0;
        const int x = (int)(e % n0);
        const float re = a[(row * 2) * ld + x], im = a[(row * 2 + 1) * ld + x];
        z[e] = make_double2(f2d_exact(re), f2d_exact(im));
        acc = fmaf(re, re, fmaf(im, im, acc));
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    __shared__ double ws[8];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = (double)acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ws[w];
        part[blockIdx.x] = t;
    }
}

// *out = sum of part[0 .. n) in a fixed order (one CTA)
__global__ void __launch_bounds__(512) k_sum_parts(const double *__restrict__ part, int n, double *out) {
    double t = 0.0;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += 512) t += part[i];
    t = block_sum<512>(t, 0.0).x;
    if (threadIdx.x == 0) *out = t;
}

__global__ void k_from_planar(const float *__restrict__ a, double2 *__restrict__ z, int n0, size_t rows, int ld) {
    const size_t total = rows * (size_t)n0;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t row = e / n0;
        const int x = (int)(e % n0);
        z[e] = make_double2(f2d_exact(a[(row * 2) * ld + x]), f2d_exact(a[(row * 2 + 1) * ld + x]));
    }
}

struct ZSolveParams {
    float *x;               // in/out: real part of (line (i, j), row k) at x[k ks + j js + i is], imaginary at + cs
    size_t ks;
    int js, is, cs;
    float2 *ck;             // scratch: elimination state at the start of each row block, [half][b][e][line]
    float4 *zb;             // scratch: upper band rows of (Bc, Cc) in elimination order, [half][row][P+1]
    const float *bands;     // outer base bands [nb][n2][bw]
    const float *lx, *ly;   // inner eigenvalues
    const float *lxi, *lyi; // their imaginary parts (complex axis pencils), else null
    int n0, n1, n2;
    CombP<float> Bc, Cc;    // A_z(s) = Bc + s Cc
    float4 *fac;            // stored factor (k_zfac): [half][row][line][pairs of entries], or null
};

// ---- line solves along the outer axis: banded complex L D L^T (no pivoting),
// two threads per line, lines contiguous in memory (coalesced across the warp).
//
// The line matrices are complex symmetric (combinations of the mass,
// stiffness, potential and absorbing bands with complex scalars), so one
// triangle carries everything: row k needs its P+1 upper band entries, and
// the multiplier of row k-d is u(k-d, k) / u(k-d, k-d).
//
// Twisted factorisation: one thread eliminates the first half of the rows from
// the top, its partner the rest from the bottom (the line read backwards).
// Each half's elimination keeps the band's columns past its end, so its last P
// rows carry the coupling to the other half. The two final states meet in
// shared memory, where both threads solve the same 2P x 2P system for the P
// unknowns on either side of the cut: with the tail rows scaled by the
// reciprocal pivots, U1 T1 + W1 T2 = c1 and U2 T2 + W2 T1 = c2 (U unit upper
// triangular), so S T2 = c2 - W2 U1^-1 c1 with S = U2 - W2 U1^-1 W1, and
// T1 = U1^-1 (c1 - W1 T2). Each thread then back-substitutes its half from the
// partner's tail values.
//
// No factor is stored: the forward pass saves the elimination state (the live
// parts of the last P rows) at the start of every block of B rows; the
// backward pass redoes a block's elimination from it (u rows into shared
// memory, L^-1 r into registers), back-substitutes and writes the solution in
// place. Rows and states are fetched into registers one block ahead. Both
// halves run the same number of full blocks (identity rows in front of the
// first real row), so the row loop is fully unrolled with static ring slots
// and a body short enough for the instruction cache.
//
// Bound by issue slots and the latency of the recursion (about 12 complex
// multiply-subtracts per row and pass for P = 3). The former unsymmetric
// elimination with a 32-row unrolled ring took 257 us per solve on 163 x 163
// lines of 343 rows (P = 3) and 293 us on 260 lines of 260 rows (P = 4,
// complex pencils); this one 97 us and 55 us.
constexpr int kZLines = 64;                      // lines per CTA (two threads each)
template <int P> struct ZBlk {
    static constexpr int B = P == 3 ? 9 : (P == 5 ? 10 : 8);   // rows per block (a multiple of P)
    static constexpr int NS = P * (P + 1) / 2 + 2 * P;         // complex entries of the saved state
    static constexpr int NX = P * (P + 1) + P;                 // complex entries exchanged at the cut
    static_assert(B % P == 0, "ring slots are static within a block");
    static_assert(NX <= B * (P + 1), "the u block doubles as the exchange buffer");
};
// rows of the upper half, blocks per half
__host__ __device__ inline int z_half(int n) { return (n + 1) / 2; }
__host__ __device__ inline int z_blocks(int n, int B) { return (z_half(n) + B - 1) / B; }

template <int P> size_t zsolve_smem(int n2) {
    return (size_t)2 * z_blocks(n2, ZBlk<P>::B) * ZBlk<P>::B * (P + 1) * sizeof(float4) +
           (size_t)ZBlk<P>::B * (P + 1) * 2 * kZLines * sizeof(float2);
}

// the upper band rows of A_z(s) = Bc + s Cc for the current stage, in the
// elimination order of each half: entry q of local row k couples it to local
// row k + q; identity rows in front
template <int P> __global__ void k_zbands(const ZSolveParams prm) {
    constexpr int B = ZBlk<P>::B, bw = 2 * P + 1;
    const int n = prm.n2, rows = z_blocks(n, B) * B, h0 = z_half(n);
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 2 * rows * (P + 1)) return;
    const int q = e % (P + 1), k = (e / (P + 1)) % rows, half = e / ((P + 1) * rows);
    const int pad = rows - (half ? n - h0 : h0);
    float2 b = make_float2(k < pad && q == 0 ? 1.f : 0.f, 0.f), c = make_float2(0.f, 0.f);
    if (k >= pad) {
        const int row = half ? n - 1 - (k - pad) : k - pad, col = half ? row - q : row + q;
        if (col >= 0 && col < n) {
            b = comb_at<float, float2>(prm.Bc, prm.bands, n, bw, row, col - row + P);
            c = comb_at<float, float2>(prm.Cc, prm.bands, n, bw, row, col - row + P);
        }
    }
    prm.zb[e] = make_float4(b.x, b.y, c.x, c.y);
}

__device__ __forceinline__ float2 csubf(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// acc -= a b
__device__ __forceinline__ void csubmul(float2 &acc, float2 a, float2 b) {
    acc.x = fmaf(a.y, b.y, fmaf(-a.x, b.x, acc.x));
    acc.y = fmaf(-a.y, b.x, fmaf(-a.x, b.y, acc.y));
}

// the 2P x 2P system at the cut: U1 T1 + W1 T2 = c1, U2 T2 + W2 T1 = c2 (U unit
// upper triangular, its diagonal not stored)
template <int P>
__device__ __forceinline__ void twist_solve(const float2 (&U1)[P][P], const float2 (&W1)[P][P], const float2 (&c1)[P],
                                            const float2 (&U2)[P][P], const float2 (&W2)[P][P], const float2 (&c2)[P],
                                            float2 (&T1)[P], float2 (&T2)[P]) {
    // z1 = U1^-1 c1, M1 = U1^-1 W1 (unit upper triangular)
    float2 z1[P], M1[P][P];
#pragma unroll
    for (int r = P - 1; r >= 0; --r) {
        z1[r] = c1[r];
#pragma unroll
        for (int k = 0; k < P; ++k) M1[r][k] = W1[r][k];
#pragma unroll
        for (int q = r + 1; q < P; ++q) {
            z1[r] = csubf(z1[r], cmulf(U1[r][q], z1[q]));
#pragma unroll
            for (int k = 0; k < P; ++k) M1[r][k] = csubf(M1[r][k], cmulf(U1[r][q], M1[q][k]));
        }
    }
    // S = U2 + I - W2 M1 (U2 holds the strict upper part), g = c2 - W2 z1
    float2 S[P][P], g[P];
#pragma unroll
    for (int r = 0; r < P; ++r) {
        g[r] = c2[r];
#pragma unroll
        for (int k = 0; k < P; ++k) S[r][k] = k == r ? make_float2(1.f, 0.f) : U2[r][k];
#pragma unroll
        for (int q = 0; q < P; ++q) {
            g[r] = csubf(g[r], cmulf(W2[r][q], z1[q]));
#pragma unroll
            for (int k = 0; k < P; ++k) S[r][k] = csubf(S[r][k], cmulf(W2[r][q], M1[q][k]));
        }
    }
    // S T2 = g: Gaussian elimination without pivoting, then T1 = z1 - M1 T2
#pragma unroll
    for (int c = 0; c < P; ++c) {
        const float2 inv = crecf(S[c][c]);
#pragma unroll
        for (int r = c + 1; r < P; ++r) {
            const float2 f = cmulf(S[r][c], inv);
#pragma unroll
            for (int k = c + 1; k < P; ++k) S[r][k] = csubf(S[r][k], cmulf(f, S[c][k]));
            g[r] = csubf(g[r], cmulf(f, g[c]));
        }
        S[c][c] = inv;
    }
#pragma unroll
    for (int r = P - 1; r >= 0; --r) {
        float2 v = g[r];
#pragma unroll
        for (int k = r + 1; k < P; ++k) v = csubf(v, cmulf(S[r][k], T2[k]));
        T2[r] = cmulf(v, S[r][r]);
    }
#pragma unroll
    for (int r = 0; r < P; ++r) {
        T1[r] = z1[r];
#pragma unroll
        for (int k = 0; k < P; ++k) T1[r] = csubf(T1[r], cmulf(M1[r][k], T2[k]));
    }
}

template <int P, bool CI>
__global__ void __launch_bounds__(2 * kZLines, P <= 3 ? 3 : 2) k_zsolve(const ZSolveParams prm) {
    constexpr int B = ZBlk<P>::B, NS = ZBlk<P>::NS, T = 2 * kZLines;
    extern __shared__ float4 zs_smem[];
    const int n = prm.n2, nb = z_blocks(n, B), rows = nb * B;
    float4 *sZ = zs_smem;                                                   // [half][row][P+1]
    float2 *sU = reinterpret_cast<float2 *>(zs_smem + (size_t)2 * rows * (P + 1));   // [slot][thread]
    for (int e = threadIdx.x; e < 2 * rows * (P + 1); e += blockDim.x) sZ[e] = prm.zb[e];
    __syncthreads();
    const int half = threadIdx.x / kZLines;        // 0: from the top, 1: from the bottom
    const int li = threadIdx.x % kZLines;
    const int nl = prm.n0 * prm.n1;
    const int lraw = blockIdx.x * kZLines + li;
    const bool valid = lraw < nl;
    const int l = valid ? lraw : nl - 1;           // idle threads shadow a real line, store nothing
    const int h0 = z_half(n), pad = rows - (half ? n - h0 : h0);
    const int i = l % prm.n0, j = l / prm.n0;
    const float s = prm.lx[i] + (prm.ly ? prm.ly[j] : 0.f);
    const float si = CI ? prm.lxi[i] + (prm.lyi ? prm.lyi[j] : 0.f) : 0.f;
    const int cs = prm.cs;
    // local row k at xl + k ks (rows below pad are identity rows, not in memory)
    const long long ks = half ? -(long long)prm.ks : (long long)prm.ks;
    float *xl = prm.x + (size_t)j * prm.js + (size_t)i * prm.is + (half ? (long long)(n - 1) * (long long)prm.ks : 0) -
                (long long)pad * ks;
    const size_t cst = (size_t)nl;
    float2 *ck = prm.ck + (size_t)half * nb * NS * cst + l;
    const float4 *zt = sZ + (size_t)half * rows * (P + 1);
    float2 *su = sU + threadIdx.x;

    // ring of the last P rows: u(k, k+1 .. k+P), the reciprocal pivot, L^-1 r
    float2 U[P][P], iv[P], y[P];
    auto reset = [&]() {
#pragma unroll
        for (int d = 0; d < P; ++d) {
            iv[d] = make_float2(1.f, 0.f);
            y[d] = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < P; ++q) U[d][q] = make_float2(0.f, 0.f);
        }
    };
    // local row b B + r into ring slot r % P
    auto eliminate = [&](const float4 *zr, int r, float2 rhs) {
        float2 a[P + 1];
#pragma unroll
        for (int q = 0; q <= P; ++q) {
            const float4 z = zr[r * (P + 1) + q];
            a[q] = CI ? make_float2(fmaf(-si, z.w, fmaf(s, z.z, z.x)), fmaf(si, z.z, fmaf(s, z.w, z.y)))
                      : make_float2(fmaf(s, z.z, z.x), fmaf(s, z.w, z.y));
        }
#pragma unroll
        for (int d = P; d >= 1; --d) {
            const int o = (r + P - d) % P;          // slot of row k - d
            const float2 f = cmulf(U[o][d - 1], iv[o]);
#pragma unroll
            for (int q = 0; q + d <= P; ++q) csubmul(a[q], f, U[o][d + q - 1]);
            csubmul(rhs, f, y[o]);
        }
        const int o = r % P;
        iv[o] = crecf(a[0]);
        y[o] = rhs;
#pragma unroll
        for (int q = 0; q < P; ++q) U[o][q] = a[q + 1];
    };
    // rows of block b (only block 0 has identity rows)
    float2 nr[B];
    auto fetch = [&](int b) {
#pragma unroll
        for (int r = 0; r < B; ++r) {
            const int k = b * B + r;
            nr[r] = make_float2(0.f, 0.f);
            if (k >= pad) {
                const float *q = xl + (long long)k * ks;
                nr[r] = make_float2(q[0], q[cs]);
            }
        }
    };
    // the live part of the state at the start of a block: row k-d (slot P-d)
    // still needs u(k-d, k .. k-d+P), its pivot and L^-1 r
    auto save = [&](int b) {
        float2 *c = ck + (size_t)b * NS * cst;
        int e = 0;
#pragma unroll
        for (int d = 1; d <= P; ++d) {
#pragma unroll
            for (int q = d; q <= P; ++q) c[(size_t)(e++) * cst] = U[P - d][q - 1];
            c[(size_t)(e++) * cst] = iv[P - d];
            c[(size_t)(e++) * cst] = y[P - d];
        }
    };

    // forward pass of this half
    reset();
    fetch(0);
    for (int b = 0; b < nb; ++b) {
        float2 rr[B];
#pragma unroll
        for (int r = 0; r < B; ++r) rr[r] = nr[r];
        if (b + 1 < nb) fetch(b + 1);
        if (b > 0 && valid) save(b);
        const float4 *zr = zt + (size_t)b * B * (P + 1);
#pragma unroll
        for (int r = 0; r < B; ++r) eliminate(zr, r, rr[r]);
    }

    // exchange the final states ([d-1]: the row d places from the end) and
    // solve the twist system (same arithmetic in both threads)
    float2 *ex = sU;   // [e][thread]
#pragma unroll
    for (int d = 0; d < P; ++d) {
        const int o = P - 1 - d;
        ex[(size_t)(d * (P + 1)) * T + threadIdx.x] = iv[o];
#pragma unroll
        for (int q = 1; q <= P; ++q) ex[(size_t)(d * (P + 1) + q) * T + threadIdx.x] = U[o][q - 1];
        ex[(size_t)(P * (P + 1) + d) * T + threadIdx.x] = y[o];
    }
    __syncthreads();
    float2 T1[P], T2[P];
    {
        float2 U1[P][P], W1[P][P], c1[P], U2[P][P], W2[P][P], c2[P];
        auto tail = [&](int col, float2 (&Um)[P][P], float2 (&W)[P][P], float2 (&c)[P]) {
            auto st = [&](int e) { return ex[(size_t)e * T + col]; };
#pragma unroll
            for (int r = 0; r < P; ++r) {
                const int d = P - 1 - r;
                const float2 rp = st(d * (P + 1));
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    Um[r][k] = k > r ? cmulf(rp, st(d * (P + 1) + (k - r))) : make_float2(0.f, 0.f);
                    W[r][k] = k >= P - 1 - r ? cmulf(rp, st(d * (P + 1) + (2 * P - 1 - r - k))) : make_float2(0.f, 0.f);
                }
                c[r] = cmulf(rp, st(P * (P + 1) + d));
            }
        };
        tail(li, U1, W1, c1);
        tail(li + kZLines, U2, W2, c2);
        __syncthreads();   // the exchange buffer is this thread's u block from here on
        twist_solve<P>(U1, W1, c1, U2, W2, c2, T1, T2);
    }

    // backward pass of this half; local row rows + c is the partner's tail row P-1-c
    float2 nst[NS];
    auto fetch_state = [&](int b) {
        const float2 *c = ck + (size_t)b * NS * cst;
#pragma unroll
        for (int e = 0; e < NS; ++e) nst[e] = c[(size_t)e * cst];
    };
    float2 xw[P];
#pragma unroll
    for (int c = 0; c < P; ++c) xw[c] = half ? T1[P - 1 - c] : T2[P - 1 - c];
    fetch(nb - 1);
    if (nb > 1) fetch_state(nb - 1);
    for (int b = nb - 1; b >= 0; --b) {
        float2 yb[B];
#pragma unroll
        for (int r = 0; r < B; ++r) yb[r] = nr[r];
        reset();
        if (b > 0) {
            int e = 0;
#pragma unroll
            for (int d = 1; d <= P; ++d) {
#pragma unroll
                for (int q = d; q <= P; ++q) U[P - d][q - 1] = nst[e++];
                iv[P - d] = nst[e++];
                y[P - d] = nst[e++];
            }
            fetch(b - 1);
            if (b > 1) fetch_state(b - 1);
        }
        // redo the block's elimination
        const float4 *zr = zt + (size_t)b * B * (P + 1);
#pragma unroll
        for (int r = 0; r < B; ++r) {
            eliminate(zr, r, yb[r]);
            yb[r] = y[r % P];
            su[(size_t)(r * (P + 1)) * T] = iv[r % P];
#pragma unroll
            for (int q = 1; q <= P; ++q) su[(size_t)(r * (P + 1) + q) * T] = U[r % P][q - 1];
        }
#pragma unroll
        for (int r = B - 1; r >= 0; --r) {
            float2 v = yb[r];
#pragma unroll
            for (int q = P; q >= 1; --q) csubmul(v, su[(size_t)(r * (P + 1) + q) * T], xw[q - 1]);
            v = cmulf(v, su[(size_t)(r * (P + 1)) * T]);
#pragma unroll
            for (int d = P - 1; d > 0; --d) xw[d] = xw[d - 1];
            xw[0] = v;
            const int k = b * B + r;
            if (valid && k >= pad) {
                float *q = xl + (long long)k * ks;
                q[0] = v.x;
                q[cs] = v.y;
            }
        }
    }
}

// ---- stored factor, for small problems
// The line matrices change only with the stage coefficients, and a stage solve
// applies the preconditioner several times. Where the whole factor stays in
// L2, k_zfac stores the reciprocal pivot and the unit factor row of every row
// once per stage, and k_zsub only substitutes: P complex multiply-subtracts per
// row and pass against the 14 (P = 4) of an elimination plus its repetition.
// With few lines both are bound by one warp's issue rate and dependent
// products, so a row's instructions are what counts: its factor is one padded
// record per line, fetched by 16-byte asynchronous copies into a ring of
// kRing rows with static slots, and L^-1 r stays in shared memory. 260 lines of
// 260 rows, P = 4: 59 us per application (k_zbands and k_zsolve) before,
// 30 us now; with one 8-byte copy per entry and computed addresses 65 us.
constexpr int kZSubLines = 32;
template <int P> struct ZFac {
    static constexpr int FP = (P + 2) / 2;                      // float4 per record (1/u(k,k), unit row, padding)
    static constexpr int kRing = P == 3 || P == 5 ? 15 : 16;    // a multiple of P
    static_assert(kRing % P == 0, "static ring slots");
    static_assert(P * (P + 1) <= kRing * 2 * FP, "the ring doubles as the exchange buffer");
};
template <int P> size_t zsub_smem(int n2) {
    const size_t rows = (size_t)z_blocks(n2, ZBlk<P>::B) * ZBlk<P>::B;
    return (ZFac<P>::kRing * (2 * ZFac<P>::FP + 1) + rows) * 2 * kZSubLines * sizeof(float2);
}
__device__ __forceinline__ void cp_async16(float4 *dst, const float4 *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int P, bool CI> __global__ void __launch_bounds__(2 * kZSubLines) k_zfac(const ZSolveParams prm) {
    constexpr int B = ZBlk<P>::B;
    const int n = prm.n2, rows = z_blocks(n, B) * B;
    const int half = threadIdx.x / kZSubLines, nl = prm.n0 * prm.n1;
    const int l = blockIdx.x * kZSubLines + threadIdx.x % kZSubLines;
    if (l >= nl) return;
    const int i = l % prm.n0, j = l / prm.n0;
    const float s = prm.lx[i] + (prm.ly ? prm.ly[j] : 0.f);
    const float si = CI ? prm.lxi[i] + (prm.lyi ? prm.lyi[j] : 0.f) : 0.f;
    const float4 *zt = prm.zb + (size_t)half * rows * (P + 1);
    constexpr int FP = ZFac<P>::FP;
    float4 *out = prm.fac + ((size_t)half * rows * nl + l) * FP;
    float2 U[P][P], F[P][P];   // u(k, k+q) and u(k, k+q) / u(k, k) of the last P rows
#pragma unroll
    for (int d = 0; d < P; ++d)
#pragma unroll
        for (int q = 0; q < P; ++q) U[d][q] = F[d][q] = make_float2(0.f, 0.f);
    float4 z[P + 1];
#pragma unroll
    for (int q = 0; q <= P; ++q) z[q] = zt[q];
    for (int k0 = 0; k0 < rows; k0 += P) {
#pragma unroll
        for (int r = 0; r < P; ++r) {
            const int k = k0 + r;
            float2 a[P + 1];
#pragma unroll
            for (int q = 0; q <= P; ++q) {
                a[q] = CI ? make_float2(fmaf(-si, z[q].w, fmaf(s, z[q].z, z[q].x)), fmaf(si, z[q].z, fmaf(s, z[q].w, z[q].y)))
                          : make_float2(fmaf(s, z[q].z, z[q].x), fmaf(s, z[q].w, z[q].y));
                if (k + 1 < rows) z[q] = zt[(size_t)(k + 1) * (P + 1) + q];
            }
#pragma unroll
            for (int d = P; d >= 1; --d) {
                const int o = (r + P - d) % P;
#pragma unroll
                for (int q = 0; q + d <= P; ++q) csubmul(a[q], F[o][d - 1], U[o][d + q - 1]);
            }
            float2 rec[2 * FP];
            rec[0] = crecf(a[0]);
            rec[2 * FP - 1] = make_float2(0.f, 0.f);
#pragma unroll
            for (int q = 0; q < P; ++q) {
                U[r][q] = a[q + 1];
                rec[q + 1] = F[r][q] = cmulf(a[q + 1], rec[0]);
            }
#pragma unroll
            for (int h = 0; h < FP; ++h)
                out[(size_t)k * nl * FP + h] = make_float4(rec[2 * h].x, rec[2 * h].y, rec[2 * h + 1].x, rec[2 * h + 1].y);
        }
    }
}

// IL: the lines' real and imaginary parts are neighbours (cs = 1)
template <int P, bool IL> __global__ void __launch_bounds__(2 * kZSubLines) k_zsub(const ZSolveParams prm) {
    constexpr int B = ZBlk<P>::B, T = 2 * kZSubLines, FP = ZFac<P>::FP, D = ZFac<P>::kRing;
    extern __shared__ float4 zs_smem[];
    const int n = prm.n2, rows = z_blocks(n, B) * B;
    float4 *rf = zs_smem + threadIdx.x;                                           // [slot][FP][thread]
    float2 *rx = reinterpret_cast<float2 *>(zs_smem + D * FP * T) + threadIdx.x;  // [slot][thread]
    float2 *sy = rx + D * T;                                                      // [row][thread]: L^-1 r
    const int half = threadIdx.x / kZSubLines, li = threadIdx.x % kZSubLines, nl = prm.n0 * prm.n1;
    const int lraw = blockIdx.x * kZSubLines + li;
    const bool valid = lraw < nl;
    const int l = valid ? lraw : nl - 1;
    const int h0 = z_half(n), pad = rows - (half ? n - h0 : h0);
    const int i = l % prm.n0, j = l / prm.n0, cs = prm.cs;
    const long long ks = half ? -(long long)prm.ks : (long long)prm.ks;
    float *xl = prm.x + (size_t)j * prm.js + (size_t)i * prm.is + (half ? (long long)(n - 1) * (long long)prm.ks : 0) -
                (long long)pad * ks;
    const float4 *fac = prm.fac + ((size_t)half * rows * nl + l) * FP;
    const long long fs = (long long)nl * FP;
    // the next row's record into a slot (past the last row only the group is counted)
    const float4 *pf = fac;
    const float *px = xl;
    int left = rows;
    auto issue = [&](int slot) {
        if (left > 0) {
#pragma unroll
            for (int h = 0; h < FP; ++h) cp_async16(rf + (slot * FP + h) * T, pf + h);
            if (left <= rows - pad) {
                if constexpr (IL) {
                    cp_async8(rx + slot * T, px);
                } else {
                    cp_async4(&rx[slot * T].x, px);
                    cp_async4(&rx[slot * T].y, px + cs);
                }
            } else {
                rx[slot * T] = make_float2(0.f, 0.f);   // identity row
            }
            pf += fs;
            px += ks;
            --left;
        }
        cp_async_commit();
    };
    auto record = [&](int slot, float2 (&f)[2 * FP]) {
#pragma unroll
        for (int h = 0; h < FP; ++h) {
            const float4 v = rf[(slot * FP + h) * T];
            f[2 * h] = make_float2(v.x, v.y);
            f[2 * h + 1] = make_float2(v.z, v.w);
        }
    };
    // forward: t holds what the last P rows subtract from the next ones
    float2 t[P], fl[P][2 * FP], yl[P];   // and the last P rows' records and results
#pragma unroll
    for (int d = 0; d < P; ++d) t[d] = make_float2(0.f, 0.f);
#pragma unroll
    for (int u = 0; u < D; ++u) issue(u);
    for (int k0 = 0, s0 = 0; k0 < rows; k0 += P, s0 = s0 + P == D ? 0 : s0 + P) {
#pragma unroll
        for (int r = 0; r < P; ++r) {
            cp_async_wait<D - 1>();
            record(s0 + r, fl[r]);
            const float2 y = csubf(rx[(s0 + r) * T], t[r]);
            issue(s0 + r);
            yl[r] = y;
            sy[(size_t)(k0 + r) * T] = y;
            const float2 ny = make_float2(-y.x, -y.y);
#pragma unroll
            for (int d = 1; d < P; ++d) csubmul(t[(r + d) % P], fl[r][d], ny);
            t[r] = cmulf(fl[r][P], y);
        }
    }
    cp_async_wait<0>();
    // the system at the cut (see k_zsolve), here with unit rows as stored
    __syncthreads();
    float2 *ex = reinterpret_cast<float2 *>(zs_smem);   // the ring is free: [e][thread]
#pragma unroll
    for (int d = 0; d < P; ++d) {
        const int o = P - 1 - d;
#pragma unroll
        for (int q = 1; q <= P; ++q) ex[(size_t)(d * P + q - 1) * T + threadIdx.x] = fl[o][q];
        ex[(size_t)(P * P + d) * T + threadIdx.x] = cmulf(fl[o][0], yl[o]);
    }
    __syncthreads();
    float2 T1[P], T2[P];
    {
        float2 U1[P][P], W1[P][P], c1[P], U2[P][P], W2[P][P], c2[P];
        auto tail = [&](int col, float2 (&Um)[P][P], float2 (&W)[P][P], float2 (&c)[P]) {
#pragma unroll
            for (int r = 0; r < P; ++r) {
                const int d = P - 1 - r;
                auto st = [&](int q) { return ex[(size_t)(d * P + q - 1) * T + col]; };
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    Um[r][k] = k > r ? st(k - r) : make_float2(0.f, 0.f);
                    W[r][k] = k >= P - 1 - r ? st(2 * P - 1 - r - k) : make_float2(0.f, 0.f);
                }
                c[r] = ex[(size_t)(P * P + d) * T + col];
            }
        };
        tail(li, U1, W1, c1);
        tail(li + kZSubLines, U2, W2, c2);
        twist_solve<P>(U1, W1, c1, U2, W2, c2, T1, T2);
    }
    __syncthreads();   // the ring is in use again from here on
    // backward: local row rows + c is the partner's tail row P-1-c
    float2 xw[P];      // x of row k+1 .. k+P, row k+q in slot (k+q) % P; row rows + c in slot c (P divides rows)
#pragma unroll
    for (int c = 0; c < P; ++c) xw[c] = half ? T1[P - 1 - c] : T2[P - 1 - c];
    pf = fac + (size_t)(rows - 1) * fs;
    left = rows;
    auto issue_back = [&](int slot) {
        if (left > 0) {
#pragma unroll
            for (int h = 0; h < FP; ++h) cp_async16(rf + (slot * FP + h) * T, pf + h);
            pf -= fs;
            --left;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int u = 0; u < D; ++u) issue_back(u);
    float *out = xl + (long long)(rows - 1) * ks;
    for (int k0 = rows - P, s0 = 0; k0 >= 0; k0 -= P, s0 = s0 + P == D ? 0 : s0 + P) {
#pragma unroll
        for (int r = P - 1; r >= 0; --r) {
            const int slot = s0 + P - 1 - r;
            cp_async_wait<D - 1>();
            float2 f[2 * FP];
            record(slot, f);
            issue_back(slot);
            float2 v = cmulf(sy[(size_t)(k0 + r) * T], f[0]);
#pragma unroll
            for (int q = P; q >= 1; --q) csubmul(v, f[q], xw[(r + q) % P]);
            xw[r] = v;
            if (valid && k0 + r >= pad) {
                if constexpr (IL) {
                    *reinterpret_cast<float2 *>(out) = v;
                } else {
                    out[0] = v.x;
                    out[cs] = v.y;
                }
            }
            out -= ks;
        }
    }
    cp_async_wait<0>();
}

// fresh: the stored factor is not the current stage's
template <int P, bool CI> void launch_zsolve_t(const ZSolveParams &zp, bool fresh, cudaStream_t st) {
    constexpr size_t kMax = 220 * 1024;
    static std::atomic<unsigned long long> done{0};
    once_per_device(done, [] {
        allow_smem(k_zsolve<P, CI>, kMax);
        allow_smem(k_zsub<P, true>, kMax);
        allow_smem(k_zsub<P, false>, kMax);
    });
    const int nl = zp.n0 * zp.n1;
    if (zp.fac) {
        const int blocks = (nl + kZSubLines - 1) / kZSubLines;
        if (fresh) {
            const int entries = 2 * z_blocks(zp.n2, ZBlk<P>::B) * ZBlk<P>::B * (P + 1);
            k_zbands<P><<<(entries + 127) / 128, 128, 0, st>>>(zp);
            k_zfac<P, CI><<<blocks, 2 * kZSubLines, 0, st>>>(zp);
            count_launch(2);
        }
        (zp.cs == 1 ? k_zsub<P, true> : k_zsub<P, false>)<<<blocks, 2 * kZSubLines, zsub_smem<P>(zp.n2), st>>>(zp);
        count_launch();
        return;
    }
    const size_t smem = zsolve_smem<P>(zp.n2);
    TDZ_CHECK(smem <= kMax, TDZ_ERR_UNSUPPORTED, "outer axis too long for the FDM line solve");
    const int entries = 2 * z_blocks(zp.n2, ZBlk<P>::B) * ZBlk<P>::B * (P + 1);
    k_zbands<P><<<(entries + 127) / 128, 128, 0, st>>>(zp);
    k_zsolve<P, CI><<<(nl + kZLines - 1) / kZLines, 2 * kZLines, smem, st>>>(zp);
    count_launch(2);
}

// complex eigenvalues (complex axis pencils) take the variant with the
// imaginary part of the line shift
template <int P> void launch_zsolve(const ZSolveParams &zp, bool fresh, cudaStream_t st) {
    if (zp.lxi) launch_zsolve_t<P, true>(zp, fresh, st);
    else launch_zsolve_t<P, false>(zp, fresh, st);
}

// scratch of the line solves: saved states (float2 entries) and band rows (float4 entries)
template <int P> size_t state_entries(int n2, size_t lines) {
    return (size_t)2 * z_blocks(n2, ZBlk<P>::B) * ZBlk<P>::NS * lines;
}
size_t zsolve_state_size(int P, int n2, size_t lines) {
    switch (P) {
    case 2: return state_entries<2>(n2, lines);
    case 3: return state_entries<3>(n2, lines);
    case 4: return state_entries<4>(n2, lines);
    default: return state_entries<5>(n2, lines);
    }
}
// Stored factor (float4 entries), 0 where it is not used: beyond 64 MB it would not
// stay in L2, and with more lines than one CTA of k_zsub per SM (two at degree 5,
// whose elimination is the longest) the substitution is no longer the shorter chain.
// Applications of the whole inverse, us, elimination and stored factor; then two
// applications with a factorisation before them, as a step with new field values
// takes them (degree 3, lines x rows):
//   4489 x 69: 66 and 56, 128 and 128       5041 x 69: 66 and 62, 129 and 142
//   10609 x 59: 72 and 70, 140 and 148      17689 x 69: 88 and 97, 169 and 201
//   degree 5: 9409 x 65: 93 and 77, 171 and 165
template <int P> size_t factor_entries(int n2, size_t lines) {
    const size_t e = (size_t)2 * z_blocks(n2, ZBlk<P>::B) * ZBlk<P>::B * ZFac<P>::FP * lines;
    const size_t most = (size_t)(P == 5 ? 2 : 1) * kZSubLines * sm_count();
    return lines <= most && e * sizeof(float4) <= ((size_t)64 << 20) && zsub_smem<P>(n2) <= 220 * 1024 ? e : 0;
}
size_t zsolve_factor_size(int P, int n2, size_t lines) {
    switch (P) {
    case 2: return factor_entries<2>(n2, lines);
    case 3: return factor_entries<3>(n2, lines);
    case 4: return factor_entries<4>(n2, lines);
    default: return factor_entries<5>(n2, lines);
    }
}
size_t zsolve_band_size(int P, int n2) {
    const int B = P == 2 ? ZBlk<2>::B : P == 3 ? ZBlk<3>::B : P == 4 ? ZBlk<4>::B : ZBlk<5>::B;
    return (size_t)2 * z_blocks(n2, B) * B * (P + 1);
}

}  // namespace

void PcFDM::setup(Operator *op_, int prec) {
    op = op_;
    TDZ_CHECK(prec == TDZ_FP32 || prec == TDZ_FP64, TDZ_ERR_ARG, "FDM precision must be FP32 or FP64");
    f64 = prec == TDZ_FP64;
    const Space &s = *op->sp;
    dim = s.dim;
    TDZ_CHECK(dim >= 2, TDZ_ERR_UNSUPPORTED, "the FDM preconditioner needs 2D or 3D");
    P = s.ax[0].p;
    TDZ_CHECK(P >= 2 && P <= 5, TDZ_ERR_UNSUPPORTED, "the FDM preconditioner supports degrees 2..5");
    const Plan &pl = op->plan(TDZ_STAGE);
    // Inner-axis pencils. With only stiffness on the inner axes the
    // eigenvectors are those of (S_d, M_d) and the stage factor comes from
    // the stiffness terms (this also diagonalises stream C). Otherwise, with
    // no stream C, the pencil is S_d = sum_t f_t B_t over the inner one-axis
    // terms on the stiffness's stage scalar g (kinetic, potential and
    // absorbing layer of axis d), with stage factor g: complex symmetric when
    // the axis has an absorbing layer. Inner terms on other scalars (a field
    // along an inner axis) are left out of the fast inverse.
    exact = true;
    pencil = 0;
    cplx = false;
    dropped.clear();
    auto pure_s = [&](const Comb &c) {
        for (int i = 0; i < c.n; ++i)
            if (c.base[i] != kS) return false;
        return true;
    };
    const Comb *inner[2] = {&pl.xT, &pl.yT};
    if (pl.hasB && (!pure_s(pl.xT) || (dim == 3 && !pure_s(pl.yT)))) {
        if (pl.hasC) {
            exact = false;
        } else {
            pencil = 1;
            pencil_scalar = -1;
            for (int t = 0; t < pl.xT.n; ++t)
                if (pl.xT.base[t] == kS) pencil_scalar = pl.xT.scalar[t];
            TDZ_CHECK(pencil_scalar >= 0, TDZ_ERR_INTERNAL, "inner axis without a stiffness term");
            for (int d = 0; d < dim - 1; ++d)
                for (int t = 0; t < inner[d]->n; ++t)
                    if (inner[d]->scalar[t] != pencil_scalar) {
                        exact = false;
                        dropped.push_back(inner[d]->scalar[t]);
                    }
        }
    }
    if (op->quad.on) exact = false;   // the non-separable term is left out of the fast inverse
    for (int d = 0; d < 3; ++d) n[d] = d < dim ? s.ax[d].n : 1;
    N = (size_t)s.ndof();
    // axis pencils: real (S_d, M_d) eigenvectors, or complex ones
    std::vector<double> Vr[2], lr[2];
    std::vector<cd> Vc[2], lc[2];
    bool is_c[2] = {false, false};
    for (int d = 0; d < dim - 1; ++d) {
        if (pencil == 0) {
            gen_eig(op->bases[d][kS], op->bases[d][kM], Vr[d], lr[d]);
            continue;
        }
        const int bw = 2 * P + 1;
        std::vector<cd> band((size_t)n[d] * bw, cd(0.0));
        for (int t = 0; t < inner[d]->n; ++t) {
            if (inner[d]->scalar[t] != pencil_scalar) continue;
            const BandD &B = op->bases[d][inner[d]->base[t]];
            for (size_t e = 0; e < band.size(); ++e) band[e] += inner[d]->factor[t] * B.v[e];
        }
        bool imag = false;
        for (const cd &v : band) imag = imag || v.imag() != 0.0;
        if (!imag) {
            BandD re(n[d], P);
            for (size_t e = 0; e < band.size(); ++e) re.v[e] = band[e].real();
            gen_eig(re, op->bases[d][kM], Vr[d], lr[d]);
        } else if (gen_eig_complex(band, P, op->bases[d][kM], Vc[d], lc[d])) {
            is_c[d] = true;
        } else {
            // no complex-orthogonal eigenbasis: fall back to the stiffness pencil
            pencil = 0;
            exact = false;
            dropped.clear();
            for (int e = 0; e < dim - 1; ++e) {
                is_c[e] = false;
                gen_eig(op->bases[e][kS], op->bases[e][kM], Vr[e], lr[e]);
            }
            break;
        }
    }
    cplx = is_c[0] || is_c[1];
    tensor = !f64 && !cplx && dim == 3 && transform_supported(n[0]) && transform_supported(n[1]);
    // transform matrices and eigenvalues in the preconditioner's precision
    auto up = [&](DevBuf &b, const std::vector<double> &v) {
        if (f64) upload(b, v);
        else upload(b, std::vector<float>(v.begin(), v.end()));
    };
    auto upc = [&](DevBuf &b, const std::vector<cd> &v) {
        if (f64) {
            std::vector<double2> h(v.size());
            for (size_t e = 0; e < v.size(); ++e) h[e] = make_double2(v[e].real(), v[e].imag());
            upload(b, h);
        } else {
            std::vector<float2> h(v.size());
            for (size_t e = 0; e < v.size(); ++e) h[e] = make_float2((float)v[e].real(), (float)v[e].imag());
            upload(b, h);
        }
    };
    for (int d = 0; d < dim - 1; ++d) {
        const int nd = n[d];
        if (cplx) {
            // complex transforms (SIMT): V and V^T complex, eigenvalues split into parts
            const std::vector<cd> vc = is_c[d] ? Vc[d] : std::vector<cd>(Vr[d].begin(), Vr[d].end());
            const std::vector<cd> l = is_c[d] ? lc[d] : std::vector<cd>(lr[d].begin(), lr[d].end());
            std::vector<cd> vt((size_t)nd * nd);
            for (int i = 0; i < nd; ++i)
                for (int j = 0; j < nd; ++j) vt[(size_t)j * nd + i] = vc[(size_t)i * nd + j];
            std::vector<double> lre(nd), lim(nd);
            for (int i = 0; i < nd; ++i) { lre[i] = l[i].real(); lim[i] = l[i].imag(); }
            upc(V[d], vc);
            upc(VT[d], vt);
            up(lam[d], lre);
            up(lami[d], lim);
            continue;
        }
        const std::vector<double> &Vd = Vr[d], &ld = lr[d];
        std::vector<double> VTd((size_t)nd * nd);
        for (int i = 0; i < nd; ++i)
            for (int j = 0; j < nd; ++j) VTd[(size_t)j * nd + i] = Vd[(size_t)i * nd + j];
        up(lam[d], ld);
        if (tensor) {
            // 3D: eigenvector transforms on the tensor cores (forward with V, inverse with V^T)
            Tf[d].build(Vd, nd, nd);
            Ti[d].build(VTd, nd, nd);
        } else {
            up(V[d], Vd);
            up(VT[d], VTd);
        }
    }
    if (f64) {
        ufac.alloc(N * (3 * P + 1) * sizeof(double2));
        piv64.alloc(N * sizeof(int));
        b1.alloc(N * sizeof(double2));
        b2.alloc(N * sizeof(double2));
        return;
    }
    ufac.alloc(zsolve_state_size(P, n[dim - 1], N / n[dim - 1]) * sizeof(float2));
    zb.alloc(zsolve_band_size(P, n[dim - 1]) * sizeof(float4));
    zfac.alloc(zsolve_factor_size(P, n[dim - 1], N / n[dim - 1]) * sizeof(float4));
    zfac_valid = false;
    if (tensor) {
        npart.alloc((size_t)16 * sm_count() * sizeof(double));
        ldx = (n[0] + 3) / 4 * 4;
        ldy = (n[1] + 3) / 4 * 4;
        pa.alloc((size_t)n[2] * n[1] * 2 * ldx * sizeof(float));
        pb.alloc((size_t)n[2] * n[0] * 2 * ldy * sizeof(float));
    } else {
        b1.alloc(N * sizeof(float2));
        b2.alloc(N * sizeof(float2));
    }
}

bool PcFDM::exact_now() const {
    if (op->quad.on) return false;
    if (pencil == 0) return exact;
    for (int sc : dropped)
        if (op->sigma[sc] != cd(0.0)) return false;
    return true;
}

namespace {

// line solve parameters of the current stage (bands and eigenvalues; the
// caller sets the data layout)
// stage coefficients of the line matrices A_z(s) = Bc + s Cc of the current
// (or pole) stage, as CombP of the precision T
template <class T> void line_combs(const PcFDM &f, CombP<T> &Bc, CombP<T> &Cc) {
    const Operator *op = f.op;
    const Plan &pl = const_cast<Operator *>(op)->plan(TDZ_STAGE);
    const std::array<cd, 5> &sg = f.pole ? f.pole_sigma : op->sigma;
    auto eval = [&](const Comb &c) {
        CombP<T> out{};
        out.n = c.n;
        for (int i = 0; i < c.n; ++i) {
            const cd v = c.factor[i] * sg[c.scalar[i]];
            out.base[i] = c.base[i];
            out.re[i] = (T)v.real();
            out.im[i] = (T)v.imag();
        }
        return out;
    };
    Bc = eval(pl.zA);
    Comb cc = pl.zC;
    if (f.pencil == 1) {
        // stream B in the eigenbasis: g (lam_x + lam_y) M_out (no stream C)
        Comb gm;
        gm.add(kM, f.pencil_scalar, 1.0);
        Cc = eval(gm);
    } else if (pl.hasB && pl.xT.n > 0) {
        // stream B: M_out (x) (M_y (x) beta S_x + beta S_y (x) M_x) -> beta M_out
        cd beta = 0.0;
        for (int t = 0; t < pl.xT.n; ++t)
            if (pl.xT.base[t] == kS) beta += pl.xT.factor[t] * sg[pl.xT.scalar[t]];
        cc.add(kM, 0, 0.0);
        CombP<T> c = eval(cc);
        for (int t = 0; t < c.n; ++t)
            if (c.base[t] == kM) { c.re[t] += (T)beta.real(); c.im[t] += (T)beta.imag(); }
        Cc = c;
    } else {
        Cc = eval(cc);
    }
}

ZSolveParams line_params(const PcFDM &f) {
    const Operator *op = f.op;
    const int dim = f.dim;
    const int *n = f.n;
    const int outer = dim - 1;
    ZSolveParams zp{};
    zp.ck = f.ufac.as<float2>();
    zp.zb = f.zb.as<float4>();
    zp.bands = op->dev32[outer].as<float>();
    zp.lx = f.lam[0].as<float>();
    zp.ly = dim == 3 ? f.lam[1].as<float>() : nullptr;
    if (f.cplx) {
        zp.lxi = f.lami[0].as<float>();
        zp.lyi = dim == 3 ? f.lami[1].as<float>() : nullptr;
    }
    zp.n0 = n[0];
    zp.n1 = dim == 3 ? n[1] : 1;
    zp.n2 = n[outer];
    line_combs<float>(f, zp.Bc, zp.Cc);
    return zp;
}

// FP64 line solves (the FP64 preconditioner): one thread per line, banded LU
// with partial pivoting (the lines of the end term's indefinite stages need
// it), the line matrix evaluated from the FP64 bands into a global scratch
// whose row r holds columns r - P .. r + 2P, lines interleaved (coalesced)
struct Line64Params {
    double2 *x;               // line (i, j), row k at x[k ks + j js + i]
    size_t ks;
    int js;
    int n0, n1, n2;
    const double *bands;      // outer base bands [nb][n2][2P+1] (FP64)
    const double *lx, *ly, *lxi, *lyi;
    CombP<double> Bc, Cc;
    double2 *U;               // [n2][3P + 1][lines]: the line's LU factors
    int *piv;                 // [n2][lines]: row interchanged with row k at step k
};

template <int P> __global__ void __launch_bounds__(128) k_line64(const Line64Params prm) {
    constexpr int BW = 2 * P + 1, W = 3 * P + 1;
    const int nl = prm.n0 * prm.n1;
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= nl) return;
    const int i = l % prm.n0, j = l / prm.n0;
    const double sr = prm.lx[i] + (prm.ly ? prm.ly[j] : 0.0);
    const double si = (prm.lxi ? prm.lxi[i] : 0.0) + (prm.lyi ? prm.lyi[j] : 0.0);
    double2 *xl = prm.x + (size_t)j * prm.js + i;
    const int n = prm.n2;
    const size_t ks = prm.ks;
    // entry (r, c) of the line matrix, |c - r| within the widened band
    auto A = [&](int r, int c) -> double2 & { return prm.U[((size_t)r * W + (c - r + P)) * nl + l]; };
    auto cm = [](double2 a, double2 b) { return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); };
    for (int r = 0; r < n; ++r)
        for (int o = 0; o < W; ++o) {
            double2 v = make_double2(0.0, 0.0);
            if (o < BW) {
                const double2 b = comb_at<double, double2>(prm.Bc, prm.bands, n, BW, r, o);
                const double2 c = comb_at<double, double2>(prm.Cc, prm.bands, n, BW, r, o);
                v = make_double2(b.x + sr * c.x - si * c.y, b.y + sr * c.y + si * c.x);
            }
            prm.U[((size_t)r * W + o) * nl + l] = v;
        }
    for (int k = 0; k < n; ++k) {
        const int rmax = min(k + P, n - 1), cmax = min(k + 2 * P, n - 1);
        int bi = k;
        double best = fabs(A(k, k).x) + fabs(A(k, k).y);
        for (int r = k + 1; r <= rmax; ++r) {
            const double m = fabs(A(r, k).x) + fabs(A(r, k).y);
            if (m > best) { best = m; bi = r; }
        }
        prm.piv[(size_t)k * nl + l] = bi;
        if (!(best > 0.0)) continue;   // singular column: the solve returns non-finite values
        if (bi != k)
            for (int c = k; c <= cmax; ++c) {
                const double2 t = A(k, c);
                A(k, c) = A(bi, c);
                A(bi, c) = t;
            }
        const double2 d = A(k, k);
        const double dd = 1.0 / (d.x * d.x + d.y * d.y);
        const double2 inv = make_double2(d.x * dd, -d.y * dd);
        for (int r = k + 1; r <= rmax; ++r) {
            const double2 f = cm(A(r, k), inv);
            A(r, k) = f;
            for (int c = k + 1; c <= cmax; ++c) {
                const double2 u = cm(f, A(k, c));
                double2 &t = A(r, c);
                t.x -= u.x;
                t.y -= u.y;
            }
        }
    }
    for (int k = 0; k < n; ++k) {
        const int q = prm.piv[(size_t)k * nl + l];
        if (q != k) {
            const double2 t = xl[(size_t)k * ks];
            xl[(size_t)k * ks] = xl[(size_t)q * ks];
            xl[(size_t)q * ks] = t;
        }
        const double2 xk = xl[(size_t)k * ks];
        for (int r = k + 1; r <= min(k + P, n - 1); ++r) {
            const double2 u = cm(A(r, k), xk);
            xl[(size_t)r * ks].x -= u.x;
            xl[(size_t)r * ks].y -= u.y;
        }
    }
    for (int k = n - 1; k >= 0; --k) {
        double2 v = xl[(size_t)k * ks];
        for (int c = k + 1; c <= min(k + 2 * P, n - 1); ++c) {
            const double2 u = cm(A(k, c), xl[(size_t)c * ks]);
            v.x -= u.x;
            v.y -= u.y;
        }
        const double2 d = A(k, k);
        const double dd = 1.0 / (d.x * d.x + d.y * d.y);
        xl[(size_t)k * ks] = make_double2((v.x * d.x + v.y * d.y) * dd, (v.y * d.x - v.x * d.y) * dd);
    }
}

void line_solve64(const PcFDM &f, double2 *x, cudaStream_t st) {
    const int dim = f.dim, outer = dim - 1;
    Line64Params lp{};
    lp.x = x;
    lp.n0 = f.n[0];
    lp.n1 = dim == 3 ? f.n[1] : 1;
    lp.n2 = f.n[outer];
    lp.ks = (size_t)lp.n0 * lp.n1;
    lp.js = lp.n0;
    lp.bands = f.op->dev64[outer].as<double>();
    lp.lx = f.lam[0].as<double>();
    lp.ly = dim == 3 ? f.lam[1].as<double>() : nullptr;
    if (f.cplx) {
        lp.lxi = f.lami[0].as<double>();
        lp.lyi = dim == 3 ? f.lami[1].as<double>() : nullptr;
    }
    line_combs<double>(f, lp.Bc, lp.Cc);
    lp.U = f.ufac.as<double2>();
    lp.piv = f.piv64.as<int>();
    const int nl = lp.n0 * lp.n1, blocks = (nl + 127) / 128;
    switch (f.P) {
    case 2: k_line64<2><<<blocks, 128, 0, st>>>(lp); break;
    case 3: k_line64<3><<<blocks, 128, 0, st>>>(lp); break;
    case 4: k_line64<4><<<blocks, 128, 0, st>>>(lp); break;
    case 5: k_line64<5><<<blocks, 128, 0, st>>>(lp); break;
    }
    TDZ_CUDA(cudaGetLastError());
    count_launch();
}

// The stored factor is kept while the stage coefficients of the line matrices
// stay the same values. A captured call must stand on its own at every replay
// and must not overwrite it: it takes the kernel without a stored factor.
void line_solve(PcFDM &f, ZSolveParams &zp, cudaStream_t st) {
    bool fresh = false;
    if (f.zfac.ptr) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        const bool plain = cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
        if (!plain) {
            cudaGetLastError();
        } else {
            zp.fac = f.zfac.as<float4>();
            auto key = [](const CombP<float> &c, std::vector<float> &out) {
                out.push_back((float)c.n);
                for (int i = 0; i < c.n; ++i) {
                    out.push_back((float)c.base[i]);
                    out.push_back(c.re[i]);
                    out.push_back(c.im[i]);
                }
            };
            std::vector<float> now;
            key(zp.Bc, now);
            key(zp.Cc, now);
            fresh = !f.zfac_valid || now != f.zfac_key;
            if (fresh) f.zfac_valid = false;   // until its launches have gone out
            f.zfac_key = std::move(now);
        }
    }
    switch (f.P) {
    case 2: launch_zsolve<2>(zp, fresh, st); break;
    case 3: launch_zsolve<3>(zp, fresh, st); break;
    case 4: launch_zsolve<4>(zp, fresh, st); break;
    case 5: launch_zsolve<5>(zp, fresh, st); break;
    }
    TDZ_CUDA(cudaGetLastError());
    if (zp.fac) f.zfac_valid = true;
}

}  // namespace

void PcFDM::apply_norm(const double2 *r, double2 *z, double *norm2, cudaStream_t st) {
    TDZ_CHECK(tensor, TDZ_ERR_INTERNAL, "fused norm only on the tensor-core path");
    norm_out = norm2;
    apply(r, z, st);
    norm_out = nullptr;
}

void PcFDM::apply(const double2 *r, double2 *z, cudaStream_t st) {
    const size_t rows = (size_t)n[1] * n[2];
    if (tensor) {
        // [z][y][c][x] -> [z][x'][c][y] -> [z][y'][c][x'] -> line solves -> [z][x][c][y'] -> [z][y][c][x]
        float *a = pa.as<float>(), *b = pb.as<float>();
        const int blocks = (int)std::min<size_t>((N + 255) / 256, (size_t)16 * sm_count());
        // the first and last transforms read and write the natural-order FP64
        // vectors themselves where their kernel can
        if (transform_natural(Tf[0])) {
            transform_from64(Tf[0], r, n[2], n[1], b, ldy, st);
        } else {
            k_to_planar<<<blocks, 256, 0, st>>>(r, a, n[0], rows, ldx);
            count_launch();
            transform(Tf[0], a, n[2], n[1], ldx, b, ldy, st);
        }
        transform(Tf[1], b, n[2], n[0], ldy, a, ldx, st);
        ZSolveParams zp = line_params(*this);
        zp.x = a;
        zp.ks = (size_t)2 * n[1] * ldx;
        zp.js = 2 * ldx;
        zp.is = 1;
        zp.cs = ldx;
        line_solve(*this, zp, st);
        transform(Ti[0], a, n[2], n[1], ldx, b, ldy, st);
        int parts = blocks;
        if (transform_natural(Ti[1])) {
            transform_to64(Ti[1], b, n[2], n[0], ldy, z, norm_out ? npart.as<double>() : nullptr, st);
            parts = transform_norm_parts(n[2], n[0]);
        } else {
            transform(Ti[1], b, n[2], n[0], ldy, a, ldx, st);
            if (norm_out) k_from_planar_norm<<<blocks, 256, 0, st>>>(a, z, n[0], rows, ldx, npart.as<double>());
            else k_from_planar<<<blocks, 256, 0, st>>>(a, z, n[0], rows, ldx);
            count_launch();
        }
        if (norm_out) {
            k_sum_parts<<<1, 512, 0, st>>>(npart.as<double>(), parts, norm_out);
            count_launch();
        }
        TDZ_CUDA(cudaGetLastError());
        ++applies;
        return;
    }
    const int grows = (int)rows;
    if (f64) {
        // FP64 preconditioner (SIMT transforms, FP64 line solves)
        double2 *y1 = b1.as<double2>(), *y2 = b2.as<double2>();
        auto x64 = [&](const DevBuf &Mx, const double2 *in, double2 *out) {
            if (cplx) gemm_x<double2, double2>(Mx, in, out, grows, n[0], st);
            else gemm_x<double, double2>(Mx, in, out, grows, n[0], st);
        };
        auto y64 = [&](const DevBuf &My, const double2 *in, double2 *out) {
            if (cplx) gemm_y<double2>(My, in, out, n[0], n[1], n[2], st);
            else gemm_y<double>(My, in, out, n[0], n[1], n[2], st);
        };
        x64(V[0], r, y2);
        double2 *cur = y2, *oth = y1;
        if (dim == 3) {
            y64(VT[1], y2, y1);
            std::swap(cur, oth);
        }
        TDZ_CUDA(cudaGetLastError());
        line_solve64(*this, cur, st);
        if (dim == 3) {
            y64(V[1], cur, oth);
            std::swap(cur, oth);
        }
        x64(VT[0], cur, z);
        TDZ_CUDA(cudaGetLastError());
        count_launch(dim == 3 ? 4 : 2);
        ++applies;
        return;
    }
    float2 *x1 = b1.as<float2>(), *x2 = b2.as<float2>();
    // transforms along x (rows of n0) and along y (planes of n1 x n0) with a
    // real or complex FP32 matrix
    auto along_x = [&](const DevBuf &Mx, const auto *in, auto *out) {
        if (cplx) gemm_x<float2, float2>(Mx, in, out, grows, n[0], st);
        else gemm_x<float, float2>(Mx, in, out, grows, n[0], st);
    };
    auto along_y = [&](const DevBuf &My, const float2 *in, float2 *out) {
        if (cplx) gemm_y<float2>(My, in, out, n[0], n[1], n[2], st);
        else gemm_y<float>(My, in, out, n[0], n[1], n[2], st);
    };
    // forward transforms: along x with V (t_i = sum_i' V[i'][i] r_i'), along y with V^T
    along_x(V[0], r, x2);   // FP64 in
    float2 *cur = x2, *oth = x1;
    if (dim == 3) {
        along_y(VT[1], x2, x1);
        cur = x1;
        oth = x2;
    }
    TDZ_CUDA(cudaGetLastError());
    // line solves along the outer axis: A_z(s) = zA + s (beta M + zC), interleaved complex
    ZSolveParams zp = line_params(*this);
    zp.x = reinterpret_cast<float *>(cur);
    zp.ks = (size_t)2 * n[0] * (dim == 3 ? n[1] : 1);
    zp.js = 2 * n[0];
    zp.is = 2;
    zp.cs = 1;
    line_solve(*this, zp, st);
    // inverse transforms: along y with V, along x with V^T
    if (dim == 3) {
        along_y(V[1], cur, oth);
        std::swap(cur, oth);
    }
    along_x(VT[0], cur, z);   // FP64 out
    TDZ_CUDA(cudaGetLastError());
    count_launch(dim == 3 ? 4 : 2);
    ++applies;
}

}  // namespace tdz
