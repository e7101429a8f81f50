// Dense-axis Chebyshev steps of small multigrid levels.
//
// With A = alpha M + g H_E and every term of H_E a Kronecker product of 1D
// bands,
//   M^-1 A = alpha I + g [ R_z + C_z (R_x + R_y) ],
//   R_z = M_z^-1 (one-axis bands of z),  R_x, R_y = M^-1 (inner bands),
//   C_z = M_z^-1 Mm_z for a mass layered along z, else I,
// with R_z along z, R_x along x and so on. The matrices are dense but small
// (n_d x n_d), and a Chebyshev step in the preconditioned residual z = M^-1 r
// needs two kernels of independent dot products instead of a banded apply and
// three recurrences along whole axes, whose latency is all that a small level
// spends its time on:
//   k_dense_xy   u = (R_x + R_y) d, one z plane per CTA
//   k_dense_z    z -= alpha d + g (R_z d + C_z u); d = a z + b d; x += d,
//                a few columns per CTA, their whole length in shared memory,
//                and the matrices streamed through it
// Products are packed FP32 on both components; the z matrices are stored as
// equal pairs, so a coefficient needs no move to become an operand. Used for
// 3D FP32 levels whose estimated step is shorter (pays) and whose stage
// has real ratios to g (no absorbing layer); checked per cycle, else the
// general step runs.
//
// 51 x 51 x 109 level, degree 3: a step of 4 launches and 57 us becomes 2
// launches and 35 us; on the small levels the launches count, 39 against 19 us
// (27 x 27 x 74) and 33 against 15 us (15 x 15 x 49).
#include <algorithm>
#include <cmath>

#include "cplx.cuh"
#include "mg.h"

namespace tdz {

namespace {

constexpr int kRows = 8;   // rows per thread
inline int up8(int n) { return (n + 7) / 8 * 8; }

struct CombineParams {
    // out[k][i] = sum_t w_t base[t][i][k] (rows padded to `pitch`), as pairs (dup) or single
    const float *base;       // [bands][n][n]
    int n, pitch, nt, dup;
    int band[kMaxComb];
    float w[kMaxComb];
    float *out;
};
struct CombineSet {
    CombineParams m[4];
};

__global__ void k_dense_combine(const CombineSet set) {
    const CombineParams &c = set.m[blockIdx.y];
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < c.n * c.pitch; e += gridDim.x * blockDim.x) {
        const int k = e / c.pitch, i = e % c.pitch;
        float v = 0.f;
        if (i < c.n)
            for (int t = 0; t < c.nt; ++t) v = fmaf(c.w[t], c.base[((size_t)c.band[t] * c.n + i) * c.n + k], v);
        if (c.dup) reinterpret_cast<float2 *>(c.out)[e] = make_float2(v, v);
        else c.out[e] = v;
    }
}

__device__ __forceinline__ float2 pmac(float a, float2 v, float2 acc) { return __ffma2_rn(make_float2(a, a), v, acc); }

// u[y][x] = sum_k Rx[x][k] d[y][k] + sum_k Ry[y][k] d[k][x] of plane blockIdx.x
__global__ void __launch_bounds__(512) k_dense_xy(const float *__restrict__ rx, const float *__restrict__ ry, int n0,
                                                  int n1, int px, int pd, int py, const float2 *__restrict__ d,
                                                  float2 *__restrict__ u) {
    extern __shared__ __align__(16) unsigned char dx_raw[];
    float2 *sP = reinterpret_cast<float2 *>(dx_raw);             // [n1][pd] (pd even, zero padded)
    float *sX = reinterpret_cast<float *>(sP + (size_t)n1 * pd);   // [pd][px]: Rx transposed, zero rows past n0
    float *sY = sX + ((size_t)pd * px + 3) / 4 * 4;              // [n1][py]: Ry transposed (16-byte rows)
    const size_t plane = (size_t)blockIdx.x * n0 * n1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, nt = blockDim.x;
    for (int y = warp; y < n1; y += nw)   // a row per warp: no division
        for (int x = lane; x < pd; x += 32)
            sP[y * pd + x] = x < n0 ? d[plane + (size_t)y * n0 + x] : make_float2(0.f, 0.f);
    for (int e = threadIdx.x; e < pd * px; e += nt) sX[e] = e < n0 * px ? rx[e] : 0.f;
    for (int e = threadIdx.x; e < n1 * py; e += nt) sY[e] = ry[e];
    __syncthreads();
    const int tx = (n0 + 31) / 32, ty = py / kRows;
    for (int t = warp; t < tx * ty; t += nw) {
        const int x = (t % tx) * 32 + lane, xc = min(x, n0 - 1), y0 = (t / tx) * kRows;
        float2 acc[kRows];
        const float2 *row[kRows];
#pragma unroll
        for (int j = 0; j < kRows; ++j) {
            acc[j] = make_float2(0.f, 0.f);
            row[j] = sP + (size_t)min(y0 + j, n1 - 1) * pd;
        }
        for (int k = 0; k < pd; k += 2) {
            const float a0 = sX[k * px + xc], a1 = sX[(k + 1) * px + xc];
#pragma unroll
            for (int j = 0; j < kRows; ++j) {
                const float4 p = *reinterpret_cast<const float4 *>(row[j] + k);
                acc[j] = pmac(a0, make_float2(p.x, p.y), acc[j]);
                acc[j] = pmac(a1, make_float2(p.z, p.w), acc[j]);
            }
        }
#pragma unroll 2
        for (int k = 0; k < n1; ++k) {
            const float4 c0 = *reinterpret_cast<const float4 *>(sY + k * py + y0);
            const float4 c1 = *reinterpret_cast<const float4 *>(sY + k * py + y0 + 4);
            const float2 v = sP[(size_t)k * pd + xc];
            const float c[kRows] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
            for (int j = 0; j < kRows; ++j) acc[j] = pmac(c[j], v, acc[j]);
        }
        if (x < n0)
#pragma unroll
            for (int j = 0; j < kRows; ++j)
                if (y0 + j < n1) u[plane + (size_t)(y0 + j) * n0 + x] = acc[j];
    }
}

struct DenseStep {
    const float2 *rz, *cz;      // [n2][pz] equal pairs, transposed; cz null: identity
    int n2, pz, zc, chunk;
    size_t cols;                // n0 n1
    const float2 *u;
    float2 *z, *d, *x;
    float2 alpha, g, a, b;
};

// s.zc columns per CTA, KR rows per thread, the matrices in stages of s.chunk
// rows. Where they make a CTA for each SM: 8 rows, stages of 16 rows, and as many
// columns as give every SM the same number of CTAs (51 x 51 x 109: 16 columns, 163
// CTAs, 26.5 us; 18 columns, 145 CTAs, 19.8 us), an even number of them (61 x 61 x
// 131, both kernels: 13 columns 63 us, 14 columns 51 us). Else 8 columns, 4 rows and both
// matrices requested whole at the start, since there a thread's chain of stages
// and products is all the time (with 16 columns, 8 rows and stages: 27 x 27 x 64
// 15.6 us, now 7.2 us; 15 x 15 x 39 12.4 and 6.0 us; 9 x 9 x 28 9.9 and 5.0 us).
// More warps with fewer rows hide no more (4 rows: 27.6 us), and larger tiles per
// thread (4 x 4) leave too few warps (35 us).
template <int KR> __global__ void k_dense_z(const DenseStep s) {
    extern __shared__ __align__(16) unsigned char dz_raw[];
    const int nm = s.cz ? 2 : 1, zc = s.zc;
    float2 *sD = reinterpret_cast<float2 *>(dz_raw);   // [n2][zc]
    float2 *sU = sD + (size_t)s.n2 * zc;
    float2 *sM = sU + (size_t)s.n2 * zc;           // stages of [matrix][chunk][pz]
    const size_t c0 = (size_t)blockIdx.x * zc;
    const int nc = (int)min((size_t)zc, s.cols - c0);
    // rows k0 .. k0 + chunk - 1 of both matrices into stage (k0 / chunk) & 1
    auto issue = [&](int k0) {
        const int per = min(s.chunk, s.n2 - k0) * s.pz / 2;   // 16-byte pieces per matrix
        for (int m = 0; m < nm; ++m) {
            const float4 *src = reinterpret_cast<const float4 *>((m ? s.cz : s.rz) + (size_t)k0 * s.pz);
            float4 *dst = reinterpret_cast<float4 *>(sM + ((size_t)(k0 / s.chunk & 1) * nm + m) * s.chunk * s.pz);
            for (int p = threadIdx.x; p < per; p += blockDim.x)
                asm volatile(
                    "cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst + p)),
                    "l"(src + p)
                    : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    issue(0);
    const int c = threadIdx.x % zc, g = threadIdx.x / zc, z0 = g * KR;
    for (int k = g; k < s.n2; k += s.pz / KR) {
        const size_t i = (size_t)k * s.cols + c0 + min(c, nc - 1);
        sD[k * zc + c] = s.d[i];
        sU[k * zc + c] = s.u[i];
    }
    // the vectors of this thread's rows, requested before the products
    float2 zv[KR], xv[KR];
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        const size_t i = (size_t)min(z0 + j, s.n2 - 1) * s.cols + c0 + min(c, nc - 1);
        zv[j] = s.z[i];
        xv[j] = s.x[i];
    }
    float2 acc[KR];
#pragma unroll
    for (int j = 0; j < KR; ++j) acc[j] = make_float2(0.f, 0.f);
    for (int k0 = 0; k0 < s.n2; k0 += s.chunk) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();   // this stage has arrived; the other one is no longer read
        if (k0 + s.chunk < s.n2) issue(k0 + s.chunk);
        const int rows = min(s.chunk, s.n2 - k0);
        for (int m = 0; m < nm; ++m) {
            const float2 *mat = sM + ((size_t)((k0 / s.chunk) & 1) * nm + m) * s.chunk * s.pz + z0;
            const float2 *v = (m ? sU : sD) + (size_t)k0 * zc + c;
#pragma unroll 4
            for (int k = 0; k < rows; ++k) {
                const float4 *q = reinterpret_cast<const float4 *>(mat + (size_t)k * s.pz);
                const float2 w = v[k * zc];
#pragma unroll
                for (int j = 0; j < KR / 2; ++j) {
                    const float4 p = q[j];
                    acc[2 * j] = __ffma2_rn(make_float2(p.x, p.y), w, acc[2 * j]);
                    acc[2 * j + 1] = __ffma2_rn(make_float2(p.z, p.w), w, acc[2 * j + 1]);
                }
            }
        }
    }
    if (c >= nc) return;
#pragma unroll
    for (int j = 0; j < KR; ++j) {
        const int k = z0 + j;
        if (k >= s.n2) break;
        const size_t i = (size_t)k * s.cols + c0 + c;
        if (!s.cz) acc[j] = __fadd2_rn(acc[j], sU[k * zc + c]);
        const float2 dv = sD[k * zc + c];
        float2 t = zv[j];   // z - alpha d - g acc
        cfma(t, make_float2(-s.alpha.x, -s.alpha.y), dv);
        cfma(t, make_float2(-s.g.x, -s.g.y), acc[j]);
        float2 nd = make_float2(0.f, 0.f);
        cfma(nd, s.a, t);
        cfma(nd, s.b, dv);
        s.z[i] = t;
        s.d[i] = nd;
        s.x[i] = __fadd2_rn(xv[j], nd);
    }
}

constexpr size_t kDenseSmem = 200 * 1024;
size_t xy_smem(int n0, int n1) {
    const size_t pd = (n0 + 1) / 2 * 2, px = n0, py = up8(n1);
    return (size_t)n1 * pd * 8 + (pd * px + 3) / 4 * 16 + (size_t)n1 * py * 4;
}
size_t z_smem(int n2, int zc, int chunk) {
    return (size_t)2 * n2 * zc * 8 + (size_t)(chunk == n2 ? 2 : 4) * chunk * up8(n2) * 8;
}

}  // namespace

// Estimated step times (us). Dense: latency; the products of a plane, n_x n_y (n_x +
// n_y), on one SM, which a second one shares where there are more planes than SMs;
// the 2 n_z^2 products of an SM's share of the columns, two CTAs of which overlap.
// General: four launches of kernels bound by the latency of their lines. Measured
// (coefficients, degree 3 but for the last; dense and general):
//   27 x 27 x 74   21 and 45      66 x 66 x 133   61 and 65
//   53 x 53 x 113  37 and 57      75 x 75 x 153  117 and 75
//   33 x 33 x 193  43 and 61      88 x 88 x 113   92 and 71
//   83 x 83 x 43   49 and 53      98 x 98 x 53    77 and 61
//   73 x 73 x 155 of degree 5: 110 and 116
bool DenseLevel::pays(const int *n, int p, size_t ndof) {
    if (xy_smem(n[0], n[1]) > kDenseSmem || z_smem(n[2], 16, 16) > kDenseSmem) return false;
    const double cols = std::max(8.0, std::ceil((double)n[0] * n[1] / sm_count()));
    const double xy = (double)n[0] * n[1] * (n[0] + n[1]) / 32e3 * (n[2] <= sm_count() ? 1.0 : 1.6);
    const double z = cols * 2.0 * n[2] * n[2] / 26e3 * (cols > 20 ? 0.8 : 1.0);
    const double general = (22.0 + 0.13 * (n[0] + n[1] + n[2]) + 15e-6 * ndof) * (p == 5 ? 1.5 : 0.55 + 0.15 * p);
    return 8.0 + xy + z < general;
}

void DenseLevel::build(const Operator &op, const int *n_) {
    ok = false;
    if (op.sp->dim != 3 || op.quad.on || op.wall1d) return;
    const Plan &pl = const_cast<Operator &>(op).plan(TDZ_STAGE);
    if (pl.hasB && pl.hasC) return;
    for (int d = 0; d < 3; ++d) {
        n[d] = n_[d];
        BandChol f;
        f.factor(op.bases[d][kM]);
        const int nb = (int)op.bases[d].size(), N = n[d], p = f.p;
        std::vector<float> h((size_t)nb * N * N);
        std::vector<double> col(N);
        for (int b = 0; b < nb; ++b)
            for (int c = 0; c < N; ++c) {   // column c of M^-1 B
                const BandD &B = op.bases[d][b];
                for (int i = 0; i < N; ++i) col[i] = std::abs(i - c) <= p ? B.at(i, c) : 0.0;
                for (int i = 0; i < N; ++i) {
                    double v = col[i];
                    for (int k = 1; k <= p && i - k >= 0; ++k) v -= f.L[(size_t)i * (p + 1) + p - k] * col[i - k];
                    col[i] = v * f.L[(size_t)i * (p + 1) + p];
                }
                for (int i = N - 1; i >= 0; --i) {
                    double v = col[i];
                    for (int k = 1; k <= p && i + k < N; ++k) v -= f.L[(size_t)(i + k) * (p + 1) + p - k] * col[i + k];
                    col[i] = v * f.L[(size_t)i * (p + 1) + p];
                }
                for (int i = 0; i < N; ++i) h[((size_t)b * N + i) * N + c] = (float)col[i];
            }
        upload(base[d], h);
    }
    pd = (n[0] + 1) / 2 * 2;
    py = up8(n[1]);
    pz = up8(n[2]);
    rx.alloc((size_t)n[0] * n[0] * sizeof(float));
    ry.alloc((size_t)n[1] * py * sizeof(float));
    rz.alloc((size_t)n[2] * pz * sizeof(float2));
    cz.alloc((size_t)n[2] * pz * sizeof(float2));
    ok = true;
}

bool DenseLevel::prepare(const Operator &op, cudaStream_t st) {
    ready = false;
    if (!ok) return false;
    const Plan &pl = const_cast<Operator &>(op).plan(TDZ_STAGE);
    const cd g = op.sigma[1];
    if (g == cd(0.0)) return false;
    bool real = true;
    auto weights = [&](const Comb &c, CombineParams &o, bool skip_mass) {
        for (int i = 0; i < c.n; ++i) {
            if (skip_mass && c.scalar[i] == 0) {
                if (c.base[i] != kM) real = false;   // alpha multiplies the overlap only
                continue;
            }
            const cd w = c.factor[i] * op.sigma[c.scalar[i]] / g;
            if (std::abs(w.imag()) > 1e-12 * std::abs(w.real())) real = false;
            o.band[o.nt] = c.base[i];
            o.w[o.nt++] = (float)w.real();
        }
    };
    CombineSet set{};
    auto target = [&](int m, int d, int pitch, int dup, DevBuf &out) {
        set.m[m].base = base[d].as<float>();
        set.m[m].n = n[d];
        set.m[m].pitch = pitch;
        set.m[m].dup = dup;
        set.m[m].out = out.as<float>();
    };
    target(0, 2, pz, 1, rz);
    target(1, 0, n[0], 0, rx);
    target(2, 1, py, 0, ry);
    target(3, 2, pz, 1, cz);
    weights(pl.zA, set.m[0], true);
    has_c = pl.hasC;
    if (pl.hasC) {   // stream C: the stiffness of x and y under the layered mass
        for (int m = 1; m <= 2; ++m) {
            set.m[m].nt = 1;
            set.m[m].band[0] = kS;
            set.m[m].w[0] = 1.f;
        }
        weights(pl.zC, set.m[3], false);
    } else {
        weights(pl.xT, set.m[1], false);
        weights(pl.yT, set.m[2], false);
    }
    if (!real) return false;
    k_dense_combine<<<dim3(32, has_c ? 4 : 3), 256, 0, st>>>(set);
    TDZ_CUDA(cudaGetLastError());
    count_launch();
    ready = true;
    return true;
}

void DenseLevel::step(const Operator &op, void *z, void *d, void *x, void *u, cd a, cd b, cudaStream_t st) const {
    static std::atomic<unsigned long long> done{0};
    once_per_device(done, [] {
        allow_smem(k_dense_xy, kDenseSmem);
        allow_smem(k_dense_z<8>, kDenseSmem);
        allow_smem(k_dense_z<4>, kDenseSmem);
    });
    const int tasks = (n[0] + 31) / 32 * (py / kRows), rounds = (tasks + 15) / 16;   // one per warp and round
    k_dense_xy<<<n[2], 32 * std::max(8, (tasks + rounds - 1) / rounds), xy_smem(n[0], n[1]), st>>>(
        rx.as<float>(), ry.as<float>(), n[0], n[1], n[0], pd, py, static_cast<const float2 *>(d),
        static_cast<float2 *>(u));
    auto f2 = [](cd v) { return make_float2((float)v.real(), (float)v.imag()); };
    DenseStep s{};
    s.rz = rz.as<float2>();
    s.cz = has_c ? cz.as<float2>() : nullptr;
    s.n2 = n[2];
    s.pz = pz;
    s.cols = (size_t)n[0] * n[1];
    s.u = static_cast<const float2 *>(u);
    s.z = static_cast<float2 *>(z);
    s.d = static_cast<float2 *>(d);
    s.x = static_cast<float2 *>(x);
    s.alpha = f2(op.sigma[0]);
    s.g = f2(op.sigma[1]);
    s.a = f2(a);
    s.b = f2(b);
    if (s.cols > (size_t)8 * sm_count() || z_smem(n[2], 8, n[2]) > kDenseSmem) {
        const size_t most = z_smem(n[2], 20, 16) <= kDenseSmem ? 20 : 16, sms = sm_count();
        const size_t ctas = (s.cols + sms * most - 1) / (sms * most) * sms;
        s.zc = (int)std::max<size_t>(8, ((s.cols + ctas - 1) / ctas + 1) / 2 * 2);
        s.chunk = 16;
        k_dense_z<8><<<(unsigned)((s.cols + s.zc - 1) / s.zc), s.zc * (pz / 8), z_smem(n[2], s.zc, 16), st>>>(s);
    } else {
        s.zc = 8;
        s.chunk = n[2];
        k_dense_z<4><<<(unsigned)((s.cols + 7) / 8), 8 * (pz / 4), z_smem(n[2], 8, n[2]), st>>>(s);
    }
    TDZ_CUDA(cudaGetLastError());
    count_launch(2);
}

}  // namespace tdz
