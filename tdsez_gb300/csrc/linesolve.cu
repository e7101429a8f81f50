// Banded Cholesky line solves (the exact Kronecker inverse of the overlap).
//
// The factors are real, so a complex line is two real lines side by side. A
// warp owns a tile of 16 complex (32 real) lines, the whole length of them:
// every row of the tile is requested at once by asynchronous copies into
// shared memory, one lane runs the recurrence of one real line there, and the
// result leaves with coalesced stores. One read and one write of HBM per axis,
// and no global load inside the recurrence, whose dependent chain is one FMA
// per row (the rows are scaled by their reciprocal pivots beforehand). Lines
// along x are transposed on the way into shared memory (pitch 34: no bank
// conflicts either way).
//
// Axes too long for shared memory keep the first design: one thread per
// line, every step of the recurrence a load and a store.
//
// Measured, FP32, degree 3, 123 x 123 x 253: 99 us for the three axes
// (1.9 TB/s of one read and one write per axis) against 240 us with the
// recurrence loading from global memory (y, z) or run by one thread per
// unpadded row (x).
#include "linesolve.h"

#include <cmath>
#include <cstring>

#include "blas.h"
#include "cplx.cuh"

namespace tdz {

void BandChol::factor(const BandD &A) {
    n = A.n;
    p = A.p;
    L.assign((size_t)n * (p + 1), 0.0);
    auto Lat = [&](int i, int j) -> double & { return L[(size_t)i * (p + 1) + (j - i + p)]; };
    for (int i = 0; i < n; ++i) {
        for (int j = std::max(0, i - p); j <= i; ++j) {
            double s = A.at(i, j);
            for (int k = std::max(std::max(0, i - p), j - p); k < j; ++k) s -= Lat(i, k) * Lat(j, k);
            if (i == j) {
                TDZ_CHECK(s > 0.0, TDZ_ERR_INTERNAL, "band is not positive definite");
                Lat(i, i) = std::sqrt(s);
            } else {
                Lat(i, j) = s / Lat(j, j);
            }
        }
    }
    for (int i = 0; i < n; ++i) Lat(i, i) = 1.0 / Lat(i, i);
}

// entries of one row of the recurrence table: forward (1 / L(i, i), then
// L(i, i-k) / L(i, i)), backward (1 / L(i, i), then L(i+k, i) / L(i, i)), each
// padded to whole 16-byte words of either precision
static int rec_width(int p) { return (p + 1 + 3) / 4 * 4; }

void BandChol::upload() {
    std::vector<float> l32(L.begin(), L.end());
    tdz::upload(L64, L);
    tdz::upload(L32, l32);
    const int w = rec_width(p);
    std::vector<double> r((size_t)n * 2 * w, 0.0);
    for (int i = 0; i < n; ++i) {
        double *f = &r[(size_t)i * 2 * w], *g = f + w;
        const double d = L[(size_t)i * (p + 1) + p];   // 1 / L(i, i)
        f[0] = g[0] = d;
        for (int k = 1; k <= p; ++k) {
            if (i - k >= 0) f[k] = L[(size_t)i * (p + 1) + p - k] * d;
            if (i + k < n) g[k] = L[(size_t)(i + k) * (p + 1) + p - k] * d;
        }
    }
    tdz::upload(R64, r);
    tdz::upload(R32, std::vector<float>(r.begin(), r.end()));
}

namespace {

constexpr int kTileC = 16;         // complex lines per warp
template <bool X> constexpr int kTilePitch = X ? 34 : 32;   // reals per row of a tile in shared memory
constexpr size_t kTileSmem = 224 * 1024, kLineSmem = 200 * 1024;

template <class T> struct TileArgs {
    const typename CT<T>::type *src;
    typename CT<T>::type *dst;
    const T *rec;                  // recurrence table [n][2][width]
    int n;                         // line length
    int lines;                     // lines per group (x: all rows; else the contiguous extent)
    long long tiles, tiles_per_group;
    long long stride, gstride;     // complex steps along a line and between groups (x: 1, 0)
    // epilogue of a Chebyshev step (ch_x set): d = a z + b d, x = (set ? d : x + d)
    typename CT<T>::type *ch_d, *ch_x;
    T ar, ai, br, bi;
    int ch_set, ch_keep;
};

template <class T> __device__ __forceinline__ void cp_async_c(void *dst, const void *src) {
    constexpr int B = 2 * sizeof(T);
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (B == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
    else asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}

// W table entries by 16-byte shared-memory loads
template <int W, class T> __device__ __forceinline__ void row16(T (&f)[W], const T *src) {
    constexpr int K = 16 / sizeof(T);
#pragma unroll
    for (int j = 0; j < W / K; ++j) {
        const uint4 v = reinterpret_cast<const uint4 *>(src)[j];
        memcpy(f + j * K, &v, 16);
    }
}

// one sweep of the recurrence over the rows row(0), row(1), ...: the values
// and table rows of the next U rows are requested before the current ones are
// stored, so a row costs its dependent FMA, not a shared-memory round trip
template <class T, int P, int PITCH, class Row>
__device__ __forceinline__ void line_sweep(T *line, const T *tab, int n, Row row) {
    constexpr int W = (P + 1 + 3) / 4 * 4, U = 4;
    T w[P], f[2][U][W], v[2][U];
#pragma unroll
    for (int k = 0; k < P; ++k) w[k] = T(0);
    auto fetch = [&](int i0, T (&ff)[U][W], T (&vv)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = row(min(i0 + u, n - 1));
            row16<W>(ff[u], tab + (size_t)i * 2 * W);
            vv[u] = line[(size_t)i * PITCH];
        }
    };
    auto work = [&](int i0, const T (&ff)[U][W], const T (&vv)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u >= n) break;
            T a = ff[u][0] * vv[u];
#pragma unroll
            for (int k = P; k >= 1; --k) a = tfma(-ff[u][k], w[k - 1], a);
#pragma unroll
            for (int k = P - 1; k > 0; --k) w[k] = w[k - 1];
            w[0] = a;
            line[(size_t)row(i0 + u) * PITCH] = a;
        }
    };
    fetch(0, f[0], v[0]);
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 2 * U) {
        fetch(i0 + U, f[1], v[1]);
        work(i0, f[0], v[0]);
        fetch(i0 + 2 * U, f[0], v[0]);
        work(i0 + U, f[1], v[1]);
    }
}

// X: lines along the contiguous axis (line r is row r); else lines at `stride`
// (512 threads at most in FP32, 256 in FP64, whose sweeps hold more registers)
template <class T> constexpr int kTileWarps = sizeof(T) == 4 ? 16 : 8;
template <class T, int P, bool X>
__global__ void __launch_bounds__(32 * kTileWarps<T>) k_line_tile(const TileArgs<T> g) {
    using C = typename CT<T>::type;
    constexpr int W = (P + 1 + 3) / 4 * 4, PITCH = kTilePitch<X>;
    extern __shared__ __align__(16) unsigned char ls_raw[];
    const int n = g.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T *tab = reinterpret_cast<T *>(ls_raw);
    T *buf = tab + (size_t)n * 2 * W + (size_t)warp * n * PITCH;
    for (int e = threadIdx.x; e < n * 2 * W * (int)sizeof(T) / 16; e += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (unsigned)__cvta_generic_to_shared(reinterpret_cast<uint4 *>(tab) + e)),
                     "l"(reinterpret_cast<const uint4 *>(g.rec) + e)
                     : "memory");
    const long long tile = blockIdx.x * (long long)(blockDim.x >> 5) + warp;
    const bool live = tile < g.tiles;
    long long base = 0;   // first complex element of the tile
    int nl = 0;           // its lines
    if (live) {
        const long long grp = tile / g.tiles_per_group, t = tile % g.tiles_per_group;
        base = X ? t * kTileC * (long long)n : grp * g.gstride + t * kTileC;
        nl = (int)min((long long)kTileC, (long long)g.lines - t * kTileC);
    }
    // this lane's elements: X: every 32nd of the tile's nl n contiguous ones;
    // else column lane % 16 of every second row
    const int c0 = lane & 15, half = lane >> 4;
    const int cnt = X ? (nl * n - lane + 31) / 32 : (c0 < nl ? (n - half + 1) / 2 : 0);
    int r = 0, i = X ? lane : 0;   // X: (row, position) of the lane's current element
    auto wrap = [&]() {
        while (i >= n) { i -= n; ++r; }
    };
    if constexpr (X) {
        wrap();
        for (int j = 0; j < cnt; ++j) {
            cp_async_c<T>(buf + (size_t)i * PITCH + 2 * r, g.src + base + lane + 32LL * j);
            i += 32;
            wrap();
        }
    } else {
        for (int j = 0; j < cnt; ++j)
            cp_async_c<T>(buf + (size_t)(half + 2 * j) * PITCH + 2 * c0, g.src + base + (half + 2LL * j) * g.stride + c0);
    }
    asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (!live) return;

    line_sweep<T, P, PITCH>(buf + lane, tab, n, [](int k) { return k; });
    line_sweep<T, P, PITCH>(buf + lane, tab + W, n, [n](int k) { return n - 1 - k; });
    __syncwarp();

    // store, or the Chebyshev epilogue; E elements of d and x in flight at a time
    constexpr int E = 8;
    if constexpr (X) { r = 0; i = lane; wrap(); }
    for (int j0 = 0; j0 < cnt; j0 += E) {
        C d[E], x[E];
        if (g.ch_x) {
#pragma unroll
            for (int u = 0; u < E; ++u) {
                const int j = j0 + u;
                if (j >= cnt) break;
                const long long e = X ? base + lane + 32LL * j : base + (half + 2LL * j) * g.stride + c0;
                if (g.br != T(0) || g.bi != T(0)) d[u] = g.ch_d[e];
                if (!g.ch_set) x[u] = g.ch_x[e];
            }
        }
#pragma unroll
        for (int u = 0; u < E; ++u) {
            const int j = j0 + u;
            if (j >= cnt) break;
            const long long e = X ? base + lane + 32LL * j : base + (half + 2LL * j) * g.stride + c0;
            const C z = *reinterpret_cast<const C *>(X ? buf + (size_t)i * PITCH + 2 * r
                                                       : buf + (size_t)(half + 2 * j) * PITCH + 2 * c0);
            if constexpr (X) {
                i += 32;
                wrap();
            }
            if (!g.ch_x) {
                g.dst[e] = z;
                continue;
            }
            if (g.ch_keep) g.dst[e] = z;
            C o;
            o.x = g.ar * z.x - g.ai * z.y;
            o.y = g.ar * z.y + g.ai * z.x;
            if (g.br != T(0) || g.bi != T(0)) {
                o.x += g.br * d[u].x - g.bi * d[u].y;
                o.y += g.br * d[u].y + g.bi * d[u].x;
            }
            g.ch_d[e] = o;
            if (!g.ch_set) {
                o.x += x[u].x;
                o.y += x[u].y;
            }
            g.ch_x[e] = o;
        }
    }
}

// v -= l w by scalar products: in a row's chain of dependent products what
// counts is the latency, which is longer for a packed pair (one FP32 line of 1703
// rows of degree 3: 481 us packed, 388 us scalar; 20 003 rows: 6.8 and 5.6 ms)
template <class C, class T> __device__ __forceinline__ void chain_sub(C &v, T l, const C &w) {
    v.x = tfma(-l, w.x, v.x);
    v.y = tfma(-l, w.y, v.y);
}

// strided lines: element k of line (a, b) at base + k*stride
template <class T, int P>
__global__ void k_line_strided(const T *__restrict__ L, int n, typename CT<T>::type *x, int nx_lines, int nb,
                               size_t stride, size_t bstride) {
    using C = typename CT<T>::type;
    const int a = blockIdx.x * blockDim.x + threadIdx.x;
    const int b = blockIdx.y;
    if (a >= nx_lines || b >= nb) return;
    C *line = x + (size_t)b * bstride + a;
    C win[P + 1];
#pragma unroll
    for (int k = 0; k <= P; ++k) win[k] = czero<C>();
    // forward: y_i = (b_i - sum_k L(i, i-k) y_{i-k}) / L(i, i); win[0] is y_{i-1}
    for (int i = 0; i < n; ++i) {
        C v = line[(size_t)i * stride];
        const T *Li = L + (size_t)i * (P + 1);
#pragma unroll
        for (int k = 1; k <= P; ++k)
            if (i - k >= 0) chain_sub(v, Li[P - k], win[k - 1]);
        const T d = Li[P];
        v.x *= d;
        v.y *= d;
#pragma unroll
        for (int k = P; k > 0; --k) win[k] = win[k - 1];
        win[0] = v;
        line[(size_t)i * stride] = v;
    }
    // backward: x_i = (y_i - sum_k L(i+k, i) x_{i+k}) / L(i, i)
#pragma unroll
    for (int k = 0; k <= P; ++k) win[k] = czero<C>();
    for (int i = n - 1; i >= 0; --i) {
        C v = line[(size_t)i * stride];
#pragma unroll
        for (int k = 1; k <= P; ++k)
            if (i + k < n) chain_sub(v, L[(size_t)(i + k) * (P + 1) + (P - k)], win[k - 1]);
        const T d = L[(size_t)i * (P + 1) + P];
        v.x *= d;
        v.y *= d;
#pragma unroll
        for (int k = P; k > 0; --k) win[k] = win[k - 1];
        win[0] = v;
        line[(size_t)i * stride] = v;
    }
}

// contiguous rows of length n (axis x): stage ROWS rows in shared memory
template <class T, int P>
__global__ void k_line_rows(const T *__restrict__ L, int n, typename CT<T>::type *x, int nrows) {
    using C = typename CT<T>::type;
    extern __shared__ unsigned char smem_raw[];
    C *tile = reinterpret_cast<C *>(smem_raw);
    const int rows = blockDim.x;
    const int r0 = blockIdx.x * rows;
    const int nr = min(rows, nrows - r0);
    // coalesced load of nr rows
    for (int e = threadIdx.x; e < nr * n; e += blockDim.x) tile[e] = x[(size_t)r0 * n + e];
    __syncthreads();
    if (threadIdx.x < nr) {
        C *line = tile + (size_t)threadIdx.x * n;
        C win[P + 1];
#pragma unroll
        for (int k = 0; k <= P; ++k) win[k] = czero<C>();
        for (int i = 0; i < n; ++i) {
            C v = line[i];
            const T *Li = L + (size_t)i * (P + 1);
#pragma unroll
            for (int k = 1; k <= P; ++k)
                if (i - k >= 0) chain_sub(v, Li[P - k], win[k - 1]);
            const T d = Li[P];
            v.x *= d;
            v.y *= d;
#pragma unroll
            for (int k = P; k > 0; --k) win[k] = win[k - 1];
            win[0] = v;
            line[i] = v;
        }
#pragma unroll
        for (int k = 0; k <= P; ++k) win[k] = czero<C>();
        for (int i = n - 1; i >= 0; --i) {
            C v = line[i];
#pragma unroll
            for (int k = 1; k <= P; ++k)
                if (i + k < n) chain_sub(v, L[(size_t)(i + k) * (P + 1) + (P - k)], win[k - 1]);
            const T d = L[(size_t)i * (P + 1) + P];
            v.x *= d;
            v.y *= d;
#pragma unroll
            for (int k = P; k > 0; --k) win[k] = win[k - 1];
            win[0] = v;
            line[i] = v;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nr * n; e += blockDim.x) x[(size_t)r0 * n + e] = tile[e];
}

// lines too long for a tile in shared memory: in place, one thread per line
template <class T, int P>
void run_axis_long(const T *L, int axis, typename CT<T>::type *x, int n0, int n1, int n2, cudaStream_t st) {
    using C = typename CT<T>::type;
    if (axis == 0) {
        int rows = 32;
        while (rows > 1 && (size_t)rows * n0 * sizeof(C) > 96 * 1024) rows /= 2;
        const size_t smem = (size_t)rows * n0 * sizeof(C);
        TDZ_CHECK(smem <= kLineSmem, TDZ_ERR_UNSUPPORTED, "axis too long for the row line solve");
        static std::atomic<unsigned long long> done{0};
        once_per_device(done, [] { allow_smem(k_line_rows<T, P>, kLineSmem); });
        const int nrows = n1 * n2;
        k_line_rows<T, P><<<(nrows + rows - 1) / rows, rows, smem, st>>>(L, n0, x, nrows);
    } else if (axis == 1) {
        // lines along y: a = x index, b = z index; stride n0, line base b*n0*n1 + a
        dim3 grid((n0 + 127) / 128, n2);
        k_line_strided<T, P><<<grid, 128, 0, st>>>(L, n1, x, n0, n2, (size_t)n0, (size_t)n0 * n1);
    } else {
        // lines along z: a = x + n0 y, stride n0 n1
        const int nl = n0 * n1;
        dim3 grid((nl + 127) / 128, 1);
        k_line_strided<T, P><<<grid, 128, 0, st>>>(L, n2, x, nl, 1, (size_t)n0 * n1, 0);
    }
}

// d = a z + b d, x = (set ? d : x + d) on the solution z (see TileArgs)
template <class T, int P>
bool run_axis(const BandChol &F, int axis, const typename CT<T>::type *src, typename CT<T>::type *dst, int n0, int n1,
              int n2, const ChebStep *ch, cudaStream_t st) {
    using C = typename CT<T>::type;
    constexpr int W = (P + 1 + 3) / 4 * 4;
    const int n = F.n;
    const size_t tab = (size_t)n * 2 * W * sizeof(T);
    const size_t per_warp = (size_t)n * (axis == 0 ? kTilePitch<true> : kTilePitch<false>) * sizeof(T);
    bool fused = false;
    if (tab + per_warp > kTileSmem) {
        if (src != dst) blas::copy(src, dst, (size_t)n0 * n1 * n2, sizeof(T) == 8 ? TDZ_FP64 : TDZ_FP32, st);
        run_axis_long<T, P>(sizeof(T) == 8 ? reinterpret_cast<const T *>(F.L64.ptr) : reinterpret_cast<const T *>(F.L32.ptr),
                            axis, dst, n0, n1, n2, st);
    } else {
        TileArgs<T> g{};
        g.src = src;
        g.dst = dst;
        g.rec = reinterpret_cast<const T *>(sizeof(T) == 8 ? F.R64.ptr : F.R32.ptr);
        g.n = n;
        g.lines = axis == 0 ? n1 * n2 : axis == 1 ? n0 : n0 * n1;
        g.tiles_per_group = (g.lines + kTileC - 1) / kTileC;
        g.tiles = g.tiles_per_group * (axis == 1 ? n2 : 1);
        g.stride = axis == 1 ? n0 : (long long)n0 * n1;
        g.gstride = axis == 1 ? (long long)n0 * n1 : 0;
        if (ch) {
            g.ch_d = static_cast<C *>(ch->d);
            g.ch_x = static_cast<C *>(ch->x);
            g.ar = (T)ch->a.real();
            g.ai = (T)ch->a.imag();
            g.br = (T)ch->b.real();
            g.bi = (T)ch->b.imag();
            g.ch_set = ch->set ? 1 : 0;
            g.ch_keep = ch->keep ? 1 : 0;
            fused = true;
        }
        // warps per CTA: the fewest waves of tiles (shared memory decides how many
        // are resident), the smallest CTAs among equals (they spread over the SMs)
        int warps = 1;
        long long waves = -1;
        for (int w = 1; w <= kTileWarps<T>; ++w) {
            const size_t cta = tab + w * per_warp;
            if (cta > kTileSmem) break;
            const long long res = (long long)std::min<size_t>(227 * 1024 / (cta + 1024), 32) * w * sm_count();
            const long long k = (g.tiles + res - 1) / res;
            if (waves < 0 || k < waves) { waves = k; warps = w; }
        }
        auto kern = axis == 0 ? k_line_tile<T, P, true> : k_line_tile<T, P, false>;
        static std::atomic<unsigned long long> done{0};
        once_per_device(done, [] {
            allow_smem(k_line_tile<T, P, true>, kTileSmem);
            allow_smem(k_line_tile<T, P, false>, kTileSmem);
        });
        const long long grid = (g.tiles + warps - 1) / warps;
        TDZ_CHECK(grid < (1LL << 31), TDZ_ERR_UNSUPPORTED, "too many lines");
        kern<<<(unsigned)grid, 32 * warps, tab + warps * per_warp, st>>>(g);
    }
    TDZ_CUDA(cudaGetLastError());
    count_launch();
    return fused;
}

template <class T>
bool run_axis_p(const BandChol &F, int axis, const void *src, void *dst, int n0, int n1, int n2, const ChebStep *ch,
                cudaStream_t st) {
    using C = typename CT<T>::type;
    const C *s = static_cast<const C *>(src);
    C *d = static_cast<C *>(dst);
    switch (F.p) {
    case 1: return run_axis<T, 1>(F, axis, s, d, n0, n1, n2, ch, st);
    case 2: return run_axis<T, 2>(F, axis, s, d, n0, n1, n2, ch, st);
    case 3: return run_axis<T, 3>(F, axis, s, d, n0, n1, n2, ch, st);
    case 4: return run_axis<T, 4>(F, axis, s, d, n0, n1, n2, ch, st);
    case 5: return run_axis<T, 5>(F, axis, s, d, n0, n1, n2, ch, st);
    case 6: return run_axis<T, 6>(F, axis, s, d, n0, n1, n2, ch, st);
    case 7: return run_axis<T, 7>(F, axis, s, d, n0, n1, n2, ch, st);
    default: throw Error(TDZ_ERR_UNSUPPORTED, "line solves support degrees 1..7");
    }
}

}  // namespace

bool line_solve(const BandChol &F, int axis, const void *src, void *dst, int n0, int n1, int n2, int prec,
                cudaStream_t st, const ChebStep *ch) {
    return prec == TDZ_FP64 ? run_axis_p<double>(F, axis, src, dst, n0, n1, n2, ch, st)
                            : run_axis_p<float>(F, axis, src, dst, n0, n1, n2, ch, st);
}

void KronSolve::setup(const std::array<const BandD *, 3> &bands, int dim_) {
    dim = dim_;
    for (int d = 0; d < 3; ++d) n[d] = 1;
    for (int d = 0; d < dim; ++d) {
        f[d].factor(*bands[d]);
        f[d].upload();
        n[d] = bands[d]->n;
    }
}

void KronSolve::apply(const void *src, void *x, int prec, cudaStream_t st, const ChebStep *ch) const {
    bool fused = false;
    for (int d = 0; d < dim; ++d) {
        fused = line_solve(f[d], d, src, x, n[0], n[1], n[2], prec, st, d == dim - 1 ? ch : nullptr);
        src = x;
    }
    if (ch && !fused) {
        const size_t N = (size_t)n[0] * n[1] * n[2];
        blas::axpby(ch->d, ch->a, x, ch->b, N, prec, st);
        if (ch->set) blas::copy(ch->d, ch->x, N, prec, st);
        else blas::axpby(ch->x, 1.0, ch->d, 1.0, N, prec, st);
    }
}

}  // namespace tdz
