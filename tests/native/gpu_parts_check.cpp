// Internal parts of the library that whole solves reach only indirectly, on the
// GPU, against FP64 sums on the host. Reads lines from stdin:
//   from64 K N planes R     the transform that reads natural-order FP64 vectors
//   to64 K N planes R       the one that writes them, with its fused norm
//   quad2 p nq nx ny prec   the 2D soft-core term with its table against the one
//                           without (prec 0: FP32, 1: FP64)
// and prints one line each: the largest error over the largest result, then for
// to64 the relative error of the norm, for quad2 which tables either holds.
// Linked against libtdz.so; run by tests/test_gpu_native_parts.py.
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "quad.h"
#include "space.h"
#include "tgemm.h"

using tdz::DevBuf;
using cd = std::complex<double>;

static std::mt19937_64 rng(7);
static double normal() { return std::normal_distribution<double>()(rng); }
template <class T> static std::vector<T> fetch(const DevBuf &b, size_t n) {
    std::vector<T> h(n);
    TDZ_CUDA(cudaMemcpy(h.data(), b.ptr, n * sizeof(T), cudaMemcpyDeviceToHost));
    return h;
}

static void transform(bool to, int K, int N, int planes, int R) {
    std::vector<double> B((size_t)K * N);
    for (double &v : B) v = normal();
    tdz::TransformMat T;
    T.build(B, K, N);
    if (!tdz::transform_natural(T)) throw std::runtime_error("not a resident matrix");
    const size_t rows = (size_t)planes * R;
    std::vector<cd> x(rows * K);
    for (cd &v : x) v = to ? cd((float)normal(), (float)normal()) : cd(normal(), normal());
    const int ldi = (K + 3) / 4 * 4 + 4, ldo = (R + 3) / 4 * 4;
    std::vector<cd> got(rows * N);
    double normerr = 0.0;
    DevBuf in, out;
    if (to) {
        std::vector<float> h(rows * 2 * ldi, NAN);   // the pitch's padding is never taken for data
        for (size_t r = 0; r < rows; ++r)
            for (int k = 0; k < K; ++k) {
                h[(2 * r) * ldi + k] = (float)x[r * K + k].real();
                h[(2 * r + 1) * ldi + k] = (float)x[r * K + k].imag();
            }
        tdz::upload(in, h);
        const int parts = tdz::transform_norm_parts(planes, R);
        std::vector<double> nan(parts, NAN);
        DevBuf norm;
        tdz::upload(norm, nan);
        out.alloc(rows * N * sizeof(double2));
        tdz::transform_to64(T, in.as<float>(), planes, R, ldi, out.as<double2>(), norm.as<double>(), nullptr);
        TDZ_CUDA(cudaDeviceSynchronize());
        got = fetch<cd>(out, rows * N);   // [p][n][r]
        double sum = 0.0, want = 0.0;
        for (double v : fetch<double>(norm, parts)) sum += v;
        for (const cd &v : got) want += std::norm(v);
        normerr = std::abs(sum - want) / want;
    } else {
        tdz::upload(in, x);
        std::vector<float> nan((size_t)planes * N * 2 * ldo, NAN);
        tdz::upload(out, nan);
        tdz::transform_from64(T, in.as<double2>(), planes, R, out.as<float>(), ldo, nullptr);
        TDZ_CUDA(cudaDeviceSynchronize());
        const auto h = fetch<float>(out, nan.size());
        for (int p = 0; p < planes; ++p)
            for (int n = 0; n < N; ++n)
                for (int r = 0; r < R; ++r)
                    got[((size_t)p * N + n) * R + r] = cd(h[(((size_t)p * N + n) * 2) * ldo + r], h[(((size_t)p * N + n) * 2 + 1) * ldo + r]);
    }
    double err = 0.0, top = 0.0;
    for (int p = 0; p < planes; ++p)
        for (int r = 0; r < R; ++r) {
            std::vector<cd> sum(N, cd(0.0));
            const cd *row = &x[((size_t)p * R + r) * K];
            for (int k = 0; k < K; ++k)
                for (int n = 0; n < N; ++n) sum[n] += row[k] * B[(size_t)k * N + n];
            for (int n = 0; n < N; ++n) {
                const double e = std::abs(got[((size_t)p * N + n) * R + r] - sum[n]);
                err = e <= err ? err : e;   // a NaN stays
                top = std::max(top, std::abs(sum[n]));
            }
        }
    std::printf("%.3e %.3e %d\n", err / top, normerr, tdz::take_transform_error());
}

static void quad2(int p, int nq, int nx, int ny, int prec) {
    tdz::Space s;
    s.dim = 2;
    s.nquad = nq;
    for (int d = 0; d < 2; ++d) {
        const int nel = d ? ny : nx;
        std::vector<double> U(p, -8.0);
        for (int i = 0; i <= nel; ++i) U.push_back(-8.0 + 16.0 * i / nel);
        U.insert(U.end(), p, 8.0);
        s.ax[d].setup(U.data(), (int)U.size(), p, nq);
    }
    const double soft[2][5] = {{1.0, 0.3, -0.4, 0.0, 0.7}, {0.5, -2.0, 1.0, 0.0, 1.5}};
    tdz::QuadTerm with, without;
    with.build(s, 2, &soft[0][0], prec ? tdz::kQuad64 : tdz::kQuad32);
    without.build(s, 2, &soft[0][0], tdz::kQuad64 | tdz::kQuad32, 0);
    const size_t n = (size_t)s.ax[0].n * s.ax[1].n, es = prec ? sizeof(cd) : sizeof(std::complex<float>);
    std::vector<cd> x(n), y[2];
    for (cd &v : x) v = cd(normal(), normal());
    const std::vector<std::complex<float>> xf(x.begin(), x.end());
    DevBuf dx, dy;
    if (prec) tdz::upload(dx, x);
    else tdz::upload(dx, xf);
    for (int k = 0; k < 2; ++k) {
        dy.alloc(n * es);
        TDZ_CUDA(cudaMemset(dy.ptr, 0, n * es));
        (k ? without : with).apply(cd(0.3, 0.7), prec ? TDZ_FP64 : TDZ_FP32, dx.ptr, dy.ptr, nullptr);
        TDZ_CUDA(cudaDeviceSynchronize());
        if (prec) y[k] = fetch<cd>(dy, n);
        else {
            const auto h = fetch<std::complex<float>>(dy, n);
            y[k].assign(h.begin(), h.end());
        }
    }
    double err = 0.0, top = 0.0;
    for (size_t i = 0; i < n; ++i) {
        const double e = std::abs(y[0][i] - y[1][i]);
        err = e <= err ? err : e;
        top = std::max(top, std::abs(y[1][i]));
    }
    std::printf("%.3e %d%d%d%d\n", err / top, with.st64.ptr != nullptr, with.st32.ptr != nullptr,
                without.st64.ptr != nullptr, without.st32.ptr != nullptr);
}

int main() {
    char cmd[16];
    int a, b, c, d, e;
    try {
        while (std::scanf("%15s %d %d %d %d", cmd, &a, &b, &c, &d) == 5) {
            if (!std::strcmp(cmd, "quad2")) {
                if (std::scanf("%d", &e) != 1) return 2;
                quad2(a, b, c, d, e);
            } else {
                transform(!std::strcmp(cmd, "to64"), a, b, c, d);
            }
        }
    } catch (const std::exception &ex) {
        std::fprintf(stderr, "%s\n", ex.what());
        return 1;
    }
    return 0;
}
