// Runs the library's host code against a fake CUDA runtime defined here (device
// memory is host memory, kernels do nothing) on two devices in turn and checks
// at every launch that the kernel was allowed its dynamic shared memory on the
// device it is launched on. Prints "launches N large L refused R" and one line
// per refused launch. Linked against libtdz.so; run by tests/test_smem_opt_in.py.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <vector>

#include "tdz.h"

static int g_dev = 0;
static std::map<std::pair<int, const void *>, size_t> g_allowed;
static long long g_launches = 0, g_large = 0, g_refused = 0;

static struct {
    dim3 grid, block;
    size_t smem;
    cudaStream_t st;
} g_cfg;

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = g_dev; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { *p = std::calloc(n + 256, 1); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void *p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) g_allowed[{g_dev, f}] = (size_t)v;
    return cudaSuccess;
}
// an encoder that accepts every tensor map
static int fake_encode() { return 0; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **p, unsigned, unsigned long long, cudaDriverEntryPointQueryResult *q) {
    *p = reinterpret_cast<void *>(&fake_encode);
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t s, struct CUstream_st *st) {
    g_cfg = {g, b, s, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st) {
    *g = g_cfg.grid;
    *b = g_cfg.block;
    *s = g_cfg.smem;
    *static_cast<cudaStream_t *>(st) = g_cfg.st;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void *>(f));
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3 block, void **, size_t smem, cudaStream_t) {
    ++g_launches;
    if (smem > 48 * 1024) {
        ++g_large;
        auto it = g_allowed.find({g_dev, f});
        if (it == g_allowed.end() || it->second < smem) {
            ++g_refused;
            std::printf("device %d: a kernel of %u threads with %zu bytes of dynamic shared memory\n", g_dev,
                        block.x * block.y, smem);
        }
    }
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void **a, size_t s, cudaStream_t st) {
    return cudaLaunchKernel(reinterpret_cast<const void *>(k), g, b, a, s, st);
}
}

static void ok(tdz_status s, const char *what) {
    if (s != TDZ_OK) {
        std::printf("%s: %s\n", what, tdz_last_error());
        std::exit(2);
    }
}

static tdz_space *space(int p, const std::vector<int> &nel) {
    std::vector<std::vector<double>> k(nel.size());
    std::vector<const double *> kp;
    std::vector<int> deg(nel.size(), p), nk;
    for (size_t d = 0; d < nel.size(); ++d) {
        for (int i = 0; i < p; ++i) k[d].push_back(-10.0);
        for (int i = 0; i <= nel[d]; ++i) k[d].push_back(-10.0 + 20.0 * i / nel[d]);
        for (int i = 0; i < p; ++i) k[d].push_back(10.0);
        kp.push_back(k[d].data());
        nk.push_back((int)k[d].size());
    }
    tdz_space *s = nullptr;
    ok(tdz_space_create((int)nel.size(), deg.data(), nk.data(), kp.data(), p + 1, &s), "space");
    return s;
}

// one operator's applies, mass solves and preconditioners
static void use(int p, const std::vector<int> &nel, bool soft, const std::vector<int> &pcs) {
    tdz_space *s = space(p, nel);
    tdz_physics ph;
    std::memset(&ph, 0, sizeof(ph));
    ph.charge = -1.0;
    ph.inv_mass = 1.0;
    ph.mass_axis = -1;
    ph.coupled[nel.size() - 1] = 1;
    const double centre[5] = {1.0, 0.0, 0.0, 0.0, 0.5};
    if (soft) { ph.nsoft = 1; ph.soft = centre; }
    tdz_op *op = nullptr;
    ok(tdz_operator_create(s, &ph, &op), "operator");
    const double c[2] = {0.01, 0.0};
    ok(tdz_operator_set_stage(op, 1.0, 0.0, 0.0, 0.1, 1, c), "stage");
    long long n = 0;
    ok(tdz_space_ndof(s, &n), "ndof");
    std::vector<double> x(2 * n + 32, 0.5), y(2 * n + 32);
    auto al = [](std::vector<double> &v) { return reinterpret_cast<double *>((reinterpret_cast<size_t>(v.data()) + 127) & ~(size_t)127); };
    for (int which : {TDZ_MASS, TDZ_HAMILTONIAN, TDZ_STAGE})
        for (int prec : {TDZ_FP32, TDZ_FP64, TDZ_FP64_DF})
            if (nel.size() > 1 || prec != TDZ_FP64_DF) ok(tdz_operator_apply(op, which, prec, al(x), al(y), nullptr), "apply");
    for (int prec : {TDZ_FP32, TDZ_FP64}) ok(tdz_operator_mass_solve(op, prec, al(x), nullptr), "mass solve");
    for (int pc : pcs) {
        tdz_solver_opts o;
        std::memset(&o, 0, sizeof(o));
        o.pc = pc;
        o.pc_precision = pc == TDZ_PC_BAND ? TDZ_FP64 : TDZ_FP32;
        tdz_solver *sv = nullptr;
        ok(tdz_solver_create(op, &o, nullptr, &sv), "solver");
        ok(tdz_solver_precondition(sv, al(x), al(y), nullptr), "precondition");
        tdz_solver_destroy(sv);
    }
    tdz_operator_destroy(op);
    tdz_space_destroy(s);
}

int main() {
    tdz_set_autotune(0);
    for (g_dev = 0; g_dev < 2; ++g_dev) {
        for (int p = 2; p <= 5; ++p) {
            use(p, {30, 40}, true, {TDZ_PC_FDM, TDZ_PC_MG});
            use(p, {12, 14, 200}, false, {TDZ_PC_FDM});
            use(p, {24, 24, 48}, p == 3, {TDZ_PC_FDM, TDZ_PC_MG});
        }
        use(3, {180, 20, 24}, false, {TDZ_PC_FDM});   // beyond the resident transforms
        use(3, {3000}, false, {TDZ_PC_BAND});
        use(3, {40, 1700}, false, {TDZ_PC_MASS});
    }
    std::printf("launches %lld large %lld refused %lld\n", g_launches, g_large, g_refused);
    return 0;
}
