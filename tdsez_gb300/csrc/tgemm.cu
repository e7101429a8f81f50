// tcgen05 transform kernel (see tgemm.h).
//
// Persistent CTAs (one per SM, 160 threads) walk 256 x Np output tiles (two
// 128-row sub-tiles), 64 complex rows per sub-tile with real and imaginary
// part rows interleaved; the accumulators live in tensor memory (TMEM,
// columns 0 and 256). K runs in chunks of 16 (one 64-byte swizzled row per
// operand row) through an NS-stage ring (as many stages as fit, 5 for
// Np = 176) that warp 4 fills with TMA (cp.async.bulk.tensor, 64-byte
// swizzle) up to NS chunks ahead, across tile boundaries:
//   stage = A (256 x 16 FP32, split by warps 0-3 in place into TF32 hi, with
//           the lo part in one of two extra buffers; both rounded to nearest)
//         + B hi, B lo (Np x 16 each, split on the host).
// Short chunks and a deep ring keep several chunks of loads in flight behind
// the MMAs (with two 32-wide stages the loads of a chunk could only start
// when the MMAs two chunks back had finished, which left the tensor pipe idle
// most of the time).
// Per 8-wide K step thread 0 issues four MMAs,
//   D += A_hi B_hi + A_hi B_lo + A_lo B_hi + A_lo B_lo,
// the full product of the hi/lo splits (each part rounded to TF32), so the
// result has FP32 accuracy at TF32 tensor-core rates. At the end
// of a tile warps 0-3 read TMEM with tcgen05.ld (warp w owns lanes
// 32w..32w+31, lane = tile row) and store the tile transposed per plane.
// Every wait on an mbarrier is bounded (clock64): on time-out the kernel sets
// the error word, the consumers leave together, and TMEM is still freed.
#include "tgemm.h"

#include "cplx.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <set>

namespace tdz {

namespace {

constexpr int TM = 128;        // tile rows (GEMM rows)
constexpr int KC = 16;         // K per stage (64 bytes of FP32: one 64-byte swizzled row)
constexpr int A_BYTES = TM * KC * 4;   // 8 KB
constexpr long long kWaitCycles = 4000000000LL;   // about 2 s at 2 GHz

// pinned host word that a wait which ran out sets (the same for every device)
__device__ int *g_tgemm_error = nullptr;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait for the completion of the phase with the given parity
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    if (mbar_try(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_try(bar, parity)) {
        if (clock64() - t0 > kWaitCycles) {
            if (g_tgemm_error) *reinterpret_cast<volatile int *>(g_tgemm_error) = 1;
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// shared-memory matrix descriptor: K-major operand in the canonical 64-byte
// swizzled layout (8-row groups 512 bytes apart), start address addr
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);          // start address >> 4      bits  0-13
    d |= (uint64_t)1 << 16;                          // leading offset (unused) bits 16-29
    d |= (uint64_t)((8 * KC * 4) >> 4) << 32;        // stride offset 512 B     bits 32-45
    d |= (uint64_t)1 << 46;                          // descriptor version      bits 46-47
    d |= (uint64_t)4 << 61;                          // 64-byte swizzle         bits 61-63
    return d;
}

// instruction descriptor: kind::tf32, FP32 accumulator, K-major A and B, M = 128
__host__ __device__ constexpr uint32_t instr_desc(int n) {
    return (1u << 4)                         // D format F32
           | (2u << 7)                       // A format TF32
           | (2u << 10)                      // B format TF32
           | ((uint32_t)(n >> 3) << 17)      // N >> 3
           | ((uint32_t)(TM >> 4) << 24);    // M >> 4
}

__device__ __forceinline__ void mma_tf32(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// nearest TF32 value (10 explicit mantissa bits; halfway cases away from zero)
__device__ __forceinline__ float tf32_round(float v) {
    return __uint_as_float((__float_as_uint(v) + 0x1000u) & 0xFFFFE000u);
}

struct TGParams {
    float *out;
    int rows;      // GEMM rows = 2 planes R
    int R, N, ldo, nchunks, tiles;
};

// barrier.sync + AND-reduction over `count` threads on named barrier `id`
__device__ __forceinline__ bool bar_and(int id, int count, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, %2, %3, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)v), "r"(id), "r"(count)
        : "memory");
    return r != 0;
}

__device__ __forceinline__ void bar_sync(int id, int count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// MS = 128-row sub-tiles per tile (1 or 2): with 2, each B chunk loaded by TMA
// serves 256 rows (two accumulators in TMEM at columns 0 and 256)
// Stages: as many as fit (up to 6), so that a stage's loads have several
// chunks of MMA time to land.
template <int NP, int MS> struct TGShape {
    static constexpr int B_BYTES = NP * KC * 4;
    static constexpr int A_T = MS * A_BYTES;
    static constexpr int STAGE = A_T + 2 * B_BYTES;          // A (FP32 -> TF32 hi in place), B hi, B lo
    static constexpr size_t smem_for(int ns) { return 1024 + (size_t)ns * STAGE + 2 * A_T + 2 * ns * 8 + 16; }
    static constexpr int NS = smem_for(6) <= 232448   ? 6
                              : smem_for(5) <= 232448 ? 5
                              : smem_for(4) <= 232448 ? 4
                              : smem_for(3) <= 232448 ? 3
                                                      : 2;
    static constexpr size_t SMEM = smem_for(NS);
    static constexpr bool fits = SMEM <= 232448;
};

// Persistent, warp-specialised: warps 0-3 split A, issue the MMAs (thread 0)
// and run the epilogue; warp 4 (one lane) is the TMA producer, running up to
// NS chunks ahead across tile boundaries, so loads overlap the epilogue.
template <int NP, int MS>
__global__ void __launch_bounds__(160, 1)
    k_transform(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap, const TGParams prm) {
    using S = TGShape<NP, MS>;
    constexpr int NS = S::NS, STAGE = S::STAGE, B_BYTES = S::B_BYTES, A_T = S::A_T, TMT = TM * MS;
    constexpr uint32_t TMEM_COLS = MS == 2 ? 512 : NP <= 32 ? 32 : NP <= 64 ? 64 : NP <= 128 ? 128 : 256;
    static_assert(NP % 16 == 0 && NP >= 16 && NP <= 256, "N tile");
    static_assert(S::fits, "shared memory");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *alo_base = base + NS * STAGE;
    uint64_t *bars = reinterpret_cast<uint64_t *>(alo_base + 2 * A_T);   // full[NS], done[NS]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 2 * NS);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nch = prm.nchunks;
    const int my_tiles = prm.tiles > (int)blockIdx.x ? (prm.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int G = my_tiles * nch;
    auto a_st = [&](int s) { return base + s * STAGE; };
    auto bh_st = [&](int s) { return base + s * STAGE + A_T; };
    auto bl_st = [&](int s) { return base + s * STAGE + A_T + B_BYTES; };
    auto a_lo = [&](int g) { return alo_base + (g & 1) * A_T; };
    const uint32_t full0 = smem_u32(&bars[0]), done0 = smem_u32(&bars[NS]);

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(done0 + 8 * s, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 4) {
        // ---- producer
        if (lane == 0) {
            constexpr uint32_t TX = A_T + 2 * B_BYTES;
            for (int g = 0; g < G; ++g) {
                const int s = g % NS;
                if (g >= NS && !mbar_wait(done0 + 8 * s, ((g - NS) / NS) & 1)) break;
                const int tile = (int)blockIdx.x + (g / nch) * (int)gridDim.x, c = g % nch;
                mbar_expect_tx(full0 + 8 * s, TX);
                tma_load_2d(smem_u32(a_st(s)), &amap, c * KC, tile * TMT, full0 + 8 * s);
                tma_load_2d(smem_u32(bh_st(s)), &bmap, c * KC, 0, full0 + 8 * s);
                tma_load_2d(smem_u32(bl_st(s)), &bmap, c * KC, NP, full0 + 8 * s);
            }
        }
    } else {
        // ---- consumers: 128 threads, named barrier 1
        const uint32_t idesc = instr_desc(NP);
        for (int g = 0; g < G; ++g) {
            const int s = g % NS, c = g % nch;
            bool ok = mbar_wait(full0 + 8 * s, (g / NS) & 1);
            if (ok && g >= 2) ok = mbar_wait(done0 + 8 * ((g - 2) % NS), ((g - 2) / NS) & 1);   // A_lo[g & 1] free
            if (!bar_and(1, 128, ok)) break;
            // split A into TF32 hi (in place) and lo, both rounded to nearest
            float4 *ah = reinterpret_cast<float4 *>(a_st(s));
            float4 *al = reinterpret_cast<float4 *>(a_lo(g));
#pragma unroll
            for (int q = 0; q < A_T / 16 / 128; ++q) {
                const int e = tid + q * 128;
                const float4 v = ah[e];
                const float4 h = make_float4(tf32_round(v.x), tf32_round(v.y), tf32_round(v.z), tf32_round(v.w));
                ah[e] = h;
                al[e] = make_float4(tf32_round(v.x - h.x), tf32_round(v.y - h.y), tf32_round(v.z - h.z),
                                    tf32_round(v.w - h.w));
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            bar_sync(1, 128);
            if (tid == 0) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ah_a = smem_u32(a_st(s)), al_a = smem_u32(a_lo(g));
                const uint32_t bh_a = smem_u32(bh_st(s)), bl_a = smem_u32(bl_st(s));
#pragma unroll
                for (int j = 0; j < KC / 8; ++j) {
                    const uint32_t off = j * 32;   // 8 TF32 = 32 bytes along the 64-byte swizzled row
                    const uint64_t dbh = smem_desc(bh_a + off), dbl = smem_desc(bl_a + off);
#pragma unroll
                    for (int t = 0; t < MS; ++t) {   // sub-tile t: A rows 128 t.., accumulator columns 256 t..
                        const uint64_t dah = smem_desc(ah_a + t * A_BYTES + off), dal = smem_desc(al_a + t * A_BYTES + off);
                        const uint32_t d = tmem + (uint32_t)(t * 256);
                        mma_tf32(d, dah, dbh, idesc, (c > 0 || j > 0) ? 1u : 0u);
                        mma_tf32(d, dah, dbl, idesc, 1u);
                        mma_tf32(d, dal, dbh, idesc, 1u);
                        mma_tf32(d, dal, dbl, idesc, 1u);
                    }
                }
                mma_commit(done0 + 8 * s);
            }
            if (c == nch - 1) {
                // tile complete: TMEM -> registers -> global (transposed per plane)
                const bool okd = mbar_wait(done0 + 8 * s, (g / NS) & 1);
                if (!bar_and(1, 128, okd)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int tile = (int)blockIdx.x + (g / nch) * (int)gridDim.x;
                const size_t nstride = (size_t)2 * prm.ldo;
#pragma unroll 1
                for (int t = 0; t < MS; ++t) {
                    const int row = tile * TMT + t * TM + warp * 32 + lane;
                    const bool row_ok = row < prm.rows;
                    const int cr = row >> 1, part = row & 1;
                    const int p = row_ok ? cr / prm.R : 0, r = row_ok ? cr % prm.R : 0;
                    float *orow = prm.out + ((size_t)p * prm.N * 2 + part) * prm.ldo + r;
#pragma unroll 1
                    for (int c0 = 0; c0 < NP; c0 += 16) {
                        uint32_t v[16];
                        const uint32_t taddr = tmem + (uint32_t)(t * 256) + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0;
                        asm volatile(
                            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
                            "%12, %13, %14, %15}, [%16];"
                            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                              "=r"(v[14]), "=r"(v[15])
                            : "r"(taddr));
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                        if (row_ok) {
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const int n = c0 + j;
                                if (n < prm.N) orow[(size_t)n * nstride] = __uint_as_float(v[j]);
                            }
                        }
                    }
                }
                // the next tile's first MMA overwrites the accumulator
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                bar_sync(1, 128);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

// Warp-specialised variant with double-buffered accumulators (320 threads,
// one CTA per SM, 128-row tiles):
//   warps 0-3  split each A chunk into TF32 hi (in place) and lo (a buffer of
//              the same stage), then arrive on the stage's `split` barrier;
//   warp 9     (one thread) issues the stage's MMAs into accumulator
//              tile & 1 (TMEM columns 0 or 256) and commits them to the
//              stage's `done` barrier, and at the end of a tile to `accf`;
//   warps 4-7  drain accumulator tile & 1 (warp w reads TMEM lanes
//              32 (w % 4)..) into the transposed output, then arrive on
//              `acce`, so the MMAs of the next tile run meanwhile;
//   warp 8     (one thread) keeps the stage ring full with TMA.
// The lo part lives in its stage, so the split of a chunk never waits for
// MMAs (the producer recycles a stage only after its MMAs completed).
template <int NP> struct WSShape {
    static constexpr int B_BYTES = NP * KC * 4;
    static constexpr int STAGE = 2 * A_BYTES + 2 * B_BYTES;   // A (hi in place), A lo, B hi, B lo
    static constexpr size_t smem_for(int ns) { return 1024 + (size_t)ns * STAGE + (3 * ns + 4) * 8 + 16; }
    static constexpr int NS = smem_for(6) <= 232448   ? 6
                              : smem_for(5) <= 232448 ? 5
                              : smem_for(4) <= 232448 ? 4
                              : smem_for(3) <= 232448 ? 3
                                                      : 2;
    static constexpr size_t SMEM = smem_for(NS);
    static constexpr bool fits = SMEM <= 232448;
};

template <int NP>
__global__ void __launch_bounds__(320, 1)
    k_transform_ws(const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap,
                   const TGParams prm) {
    using S = WSShape<NP>;
    constexpr int NS = S::NS, STAGE = S::STAGE, B_BYTES = S::B_BYTES;
    constexpr uint32_t TMEM_COLS = 512;   // two accumulators, columns 0 and 256
    static_assert(NP % 16 == 0 && NP >= 16 && NP <= 256, "N tile");
    static_assert(S::fits, "shared memory");
    static_assert(STAGE % 1024 == 0 && A_BYTES % 1024 == 0 && B_BYTES % 512 == 0, "swizzle alignment");
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *bars = reinterpret_cast<uint64_t *>(base + NS * STAGE);   // full, split, done [NS]; accf, acce [2]
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 3 * NS + 4);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nch = prm.nchunks;
    const int my_tiles = prm.tiles > (int)blockIdx.x ? (prm.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int G = my_tiles * nch;
    auto a_st = [&](int s) { return base + s * STAGE; };
    auto alo_st = [&](int s) { return base + s * STAGE + A_BYTES; };
    auto bh_st = [&](int s) { return base + s * STAGE + 2 * A_BYTES; };
    auto bl_st = [&](int s) { return base + s * STAGE + 2 * A_BYTES + B_BYTES; };
    const uint32_t full0 = smem_u32(&bars[0]), split0 = smem_u32(&bars[NS]), done0 = smem_u32(&bars[2 * NS]);
    const uint32_t accf0 = smem_u32(&bars[3 * NS]), acce0 = smem_u32(&bars[3 * NS + 2]);

    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(split0 + 8 * s, 128);
            mbar_init(done0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(accf0 + 8 * b, 1);
            mbar_init(acce0 + 8 * b, 128);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 8) {
        // ---- producer
        if (lane == 0) {
            constexpr uint32_t TX = A_BYTES + 2 * B_BYTES;
            for (int g = 0; g < G; ++g) {
                const int s = g % NS;
                if (g >= NS && !mbar_wait(done0 + 8 * s, ((g - NS) / NS) & 1)) break;
                const int tile = (int)blockIdx.x + (g / nch) * (int)gridDim.x, c = g % nch;
                mbar_expect_tx(full0 + 8 * s, TX);
                tma_load_2d(smem_u32(a_st(s)), &amap, c * KC, tile * TM, full0 + 8 * s);
                tma_load_2d(smem_u32(bh_st(s)), &bmap, c * KC, 0, full0 + 8 * s);
                tma_load_2d(smem_u32(bl_st(s)), &bmap, c * KC, NP, full0 + 8 * s);
            }
        }
    } else if (warp == 9) {
        // ---- MMA issue
        if (lane == 0) {
            const uint32_t idesc = instr_desc(NP);
            for (int g = 0; g < G; ++g) {
                const int s = g % NS, c = g % nch, t = g / nch, b = t & 1;
                if (c == 0 && t >= 2 && !mbar_wait(acce0 + 8 * b, ((t - 2) >> 1) & 1)) break;
                if (!mbar_wait(split0 + 8 * s, (g / NS) & 1)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ah_a = smem_u32(a_st(s)), al_a = smem_u32(alo_st(s));
                const uint32_t bh_a = smem_u32(bh_st(s)), bl_a = smem_u32(bl_st(s));
                const uint32_t d = tmem + (uint32_t)(b * 256);
#pragma unroll
                for (int j = 0; j < KC / 8; ++j) {
                    const uint32_t off = j * 32;   // 8 TF32 = 32 bytes along the 64-byte swizzled row
                    const uint64_t dah = smem_desc(ah_a + off), dal = smem_desc(al_a + off);
                    const uint64_t dbh = smem_desc(bh_a + off), dbl = smem_desc(bl_a + off);
                    // the full product of the splits: without lo.lo (2^-22 of each
                    // product) the FDM guess of the CN step is a few times less
                    // accurate, and the certified FP32 Arnoldi cycle fails its bound
                    // on some steps (measured: 4.30 against 3.69 ms per step)
                    mma_tf32(d, dah, dbh, idesc, (c > 0 || j > 0) ? 1u : 0u);
                    mma_tf32(d, dah, dbl, idesc, 1u);
                    mma_tf32(d, dal, dbh, idesc, 1u);
                    mma_tf32(d, dal, dbl, idesc, 1u);
                }
                mma_commit(done0 + 8 * s);
                if (c == nch - 1) mma_commit(accf0 + 8 * b);
            }
        }
    } else if (warp < 4) {
        // ---- A split: TF32 hi in place, lo into the stage's lo buffer, both rounded to nearest
        for (int g = 0; g < G; ++g) {
            const int s = g % NS;
            if (!mbar_wait(full0 + 8 * s, (g / NS) & 1)) break;
            float4 *ah = reinterpret_cast<float4 *>(a_st(s));
            float4 *al = reinterpret_cast<float4 *>(alo_st(s));
#pragma unroll
            for (int q = 0; q < A_BYTES / 16 / 128; ++q) {
                const int e = tid + q * 128;
                const float4 v = ah[e];
                const float4 h = make_float4(tf32_round(v.x), tf32_round(v.y), tf32_round(v.z), tf32_round(v.w));
                ah[e] = h;
                al[e] = make_float4(tf32_round(v.x - h.x), tf32_round(v.y - h.y), tf32_round(v.z - h.z),
                                    tf32_round(v.w - h.w));
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(split0 + 8 * s);
        }
    } else {
        // ---- epilogue: TMEM -> registers -> global (transposed per plane)
        const int q = warp & 3;
        const size_t nstride = (size_t)2 * prm.ldo;
        for (int t = 0; t < my_tiles; ++t) {
            const int b = t & 1;
            if (!mbar_wait(accf0 + 8 * b, (t >> 1) & 1)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int tile = (int)blockIdx.x + t * (int)gridDim.x;
            const int row = tile * TM + q * 32 + lane;
            const bool row_ok = row < prm.rows;
            const int cr = row >> 1, part = row & 1;
            const int p = row_ok ? cr / prm.R : 0, r = row_ok ? cr % prm.R : 0;
            float *orow = prm.out + ((size_t)p * prm.N * 2 + part) * prm.ldo + r;
            const uint32_t tbase = tmem + (uint32_t)(b * 256) + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
            for (int c0 = 0; c0 < NP; c0 += 16) {
                uint32_t v[16];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
                    "%12, %13, %14, %15}, [%16];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                      "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                      "=r"(v[14]), "=r"(v[15])
                    : "r"(tbase + (uint32_t)c0));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (row_ok) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        const int n = c0 + j;
                        if (n < prm.N) orow[(size_t)n * nstride] = __uint_as_float(v[j]);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(acce0 + 8 * b);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

// ---- B-resident variant: BF16 x 3 slices
// Both operands as sums of three BF16 slices (v = h + m + l, 24 significant
// bits and FP32's exponent range); the product keeps the six slice pairs
// above 2^-24: h h, h m, m h, m m, h l, l h. BF16 MMAs run at twice the TF32
// rate, so this is three quarters of the TF32 hi/lo product's tensor time, and
// the slices take 6 bytes per entry instead of 8: all of B (186 KB for
// Np = Kp = 176) stays in shared memory for the whole launch. What bounded the
// streaming kernel was B: 248 KB per 128-row tile through L2 against 83 KB of
// A (57 us per transform at 111 818 rows of 163; this kernel 51 us).
//   warps 0-15  in groups of four, as many as there are stages (at most four),
//               the groups taking chunks in turn:
//               load an A chunk (128 rows x 16) into registers, split it and
//               store the slices to the stage ring. The proxy fence after the
//               stores waits for the thread's loads too, so a group has no
//               loads in flight across it; the other groups' cover the latency
//               (one set of warps with a register prefetch: 68 us)
//   warps 16-23 drain accumulator tile & 1 into the transposed output, two per
//               TMEM lane quarter with half of the columns each, the next 16
//               columns on their way while the last ones are stored (four warps
//               and nothing in flight: 69 us; 43 us with the stores left out)
//   warp 24     (one thread) loads B once by bulk copies, then issues the MMAs
// Operand tiles are K-major rows of 16 BF16 (32 bytes), 32-byte swizzle: the
// 16-byte halves of a row trade places when bit 2 of the row is set.
constexpr int kB3Slice = TM * 32;            // one slice of an A chunk
constexpr int kB3Stage = 3 * kB3Slice;       // 12 KB
constexpr int kB3Groups = 4;                 // loader groups of 128 threads
constexpr int kB3Epi = 8;                    // epilogue warps
constexpr int kB3Threads = (4 * kB3Groups + kB3Epi + 1) * 32;
constexpr size_t kB3Max = 232448;
inline size_t b3_bytes(int Kp, int Np) { return (size_t)6 * Kp * Np; }
// stages that fit beside B (0: B does not fit)
inline int b3_stages(int Kp, int Np) {
    const size_t fixed = 1024 + b3_bytes(Kp, Np) + 256;
    if (fixed + 2 * kB3Stage > kB3Max) return 0;
    return (int)std::min<size_t>(8, (kB3Max - fixed) / kB3Stage);
}
// byte offset of the 16-byte half h of row r in a K-major 32-byte-swizzled tile
__host__ __device__ inline int b3_off(int r, int h) { return r * 32 + ((h ^ ((r >> 2) & 1)) << 4); }

__device__ __forceinline__ uint64_t b3_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(256 >> 4) << 32;                 // 8-row groups 256 bytes apart
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)6 << 61;                          // 32-byte swizzle
    return d;
}
// kind::f16: BF16 operands, FP32 accumulator, K-major, M = 128
__host__ __device__ constexpr uint32_t b3_instr_desc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TM >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}
// two FP32 values to packed BF16 (first in the low half) and their remainders
__device__ __forceinline__ uint32_t bf16_split2(float &a, float &b) {
    uint32_t p;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p) : "f"(b), "f"(a));
    a -= __uint_as_float(p << 16);
    b -= __uint_as_float(p & 0xFFFF0000u);
    return p;
}

struct B3Params {
    const float *in;
    const double2 *in64;   // IN64: complex rows of K natural-order FP64 entries
    double *out64;         // OUT64: natural-order FP64, out64[((p N + n) R + r) 2 + part]
    double *norm;          // OUT64: per epilogue warp the sum of squares written (kB3Epi per CTA), or null
    const uint8_t *b;      // swizzled slices of B: [chunk][slice][Np x 32 bytes]
    float *out;
    int rows, R, K, N, Np, ldi, ldo, nch, tiles, ns;
};

template <bool IN64, bool OUT64>
__global__ void __launch_bounds__(kB3Threads, 1) k_transform_b3(const B3Params prm) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int nch = prm.nch, NS = prm.ns, Np = prm.Np;
    const int bchunk = 3 * Np * 32;
    uint8_t *sB = base, *sA = base + (size_t)nch * bchunk;
    uint64_t *bars = reinterpret_cast<uint64_t *>(sA + (size_t)NS * kB3Stage);   // full [8], done [8], accf [2], acce [2], B
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 21);
    const uint32_t full0 = smem_u32(&bars[0]), done0 = smem_u32(&bars[8]), accf0 = smem_u32(&bars[16]),
                   acce0 = smem_u32(&bars[18]), bbar = smem_u32(&bars[20]);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int my_tiles = prm.tiles > (int)blockIdx.x ? (prm.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int G = my_tiles * nch;
    if (tid == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(full0 + 8 * s, 128);
            mbar_init(done0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(accf0 + 8 * b, 1);
            mbar_init(acce0 + 8 * b, 32 * kB3Epi);
        }
        mbar_init(bbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp < 4 * kB3Groups) {
        const int lt = tid & 127;
        // no more groups than stages: a group then waits for the MMAs of its own
        // last chunk or an older one, never two phases of a barrier ahead
        const int ng = min(kB3Groups, NS);
        for (int g = (tid >> 7) < ng ? tid >> 7 : G; g < G; g += ng) {
            const int tile = (int)blockIdx.x + (g / nch) * (int)gridDim.x, k0 = (g % nch) * 16, s = g % NS;
            uint8_t *st = sA + (size_t)s * kB3Stage;
            if constexpr (IN64) {
                // complex rows lt / 4 and lt / 4 + 32, four entries each
                const int qt = lt & 3, k = k0 + 4 * qt;
                double2 v[2][4];
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const int row = tile * (TM / 2) + (lt >> 2) + 32 * m;
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        v[m][j] = 2 * row < prm.rows && k + j < prm.K ? prm.in64[(size_t)row * prm.K + k + j]
                                                                      : make_double2(0.0, 0.0);
                }
                if (g >= NS && !mbar_wait(done0 + 8 * s, ((g - NS) / NS) & 1)) break;
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const int r = (lt >> 2) + 32 * m;
                    float re[4], im[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        re[j] = dff_split(v[m][j].x).hi;   // rounded to FP32
                        im[j] = dff_split(v[m][j].y).hi;
                    }
                    uint8_t *sr = st + b3_off(2 * r, qt >> 1) + 8 * (qt & 1);
                    uint8_t *si = st + b3_off(2 * r + 1, qt >> 1) + 8 * (qt & 1);
#pragma unroll
                    for (int sl = 0; sl < 3; ++sl) {
                        uint2 a, b;
                        a.x = bf16_split2(re[0], re[1]);
                        a.y = bf16_split2(re[2], re[3]);
                        b.x = bf16_split2(im[0], im[1]);
                        b.y = bf16_split2(im[2], im[3]);
                        *reinterpret_cast<uint2 *>(sr + sl * kB3Slice) = a;
                        *reinterpret_cast<uint2 *>(si + sl * kB3Slice) = b;
                    }
                }
            } else {
                // rows lt / 4 + 32 m, 16 bytes each (a warp reads whole 64-byte row pieces)
                const int qt = lt & 3, k = k0 + 4 * qt;
                float4 v[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const int row = tile * TM + (lt >> 2) + 32 * m;
                    v[m] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (row < prm.rows && k < prm.K) {
                        v[m] = *reinterpret_cast<const float4 *>(prm.in + (size_t)row * prm.ldi + k);   // k + 3 < ldi
                        if (k + 1 >= prm.K) v[m].y = 0.f;
                        if (k + 2 >= prm.K) v[m].z = 0.f;
                        if (k + 3 >= prm.K) v[m].w = 0.f;
                    }
                }
                if (g >= NS && !mbar_wait(done0 + 8 * s, ((g - NS) / NS) & 1)) break;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    uint8_t *sr = st + b3_off((lt >> 2) + 32 * m, qt >> 1) + 8 * (qt & 1);
#pragma unroll
                    for (int sl = 0; sl < 3; ++sl) {
                        uint2 w;
                        w.x = bf16_split2(v[m].x, v[m].y);
                        w.y = bf16_split2(v[m].z, v[m].w);
                        *reinterpret_cast<uint2 *>(sr + sl * kB3Slice) = w;
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_arrive(full0 + 8 * s);
        }
    } else if (warp == 4 * kB3Groups + kB3Epi) {
        // tile t of this CTA's A rows (contiguous in memory) into L2: chunks are
        // 64-byte pieces of 128 rows, too small to fetch from HBM one at a time
        auto prefetch = [&](int t) {
            if (t >= my_tiles) return;
            const long long r0 = ((long long)blockIdx.x + (long long)t * gridDim.x) * TM;
            const int nr = (int)min((long long)TM, prm.rows - r0);
            const char *p = IN64 ? reinterpret_cast<const char *>(prm.in64 + r0 / 2 * prm.K)
                                 : reinterpret_cast<const char *>(prm.in + r0 * prm.ldi);
            const uint32_t bytes = IN64 ? (uint32_t)(nr / 2) * prm.K * 16
                                        : (uint32_t)((nr - 1) * prm.ldi + prm.K) * 4 / 16 * 16;
            if (bytes)
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
        };
        if (lane == 0 && G > 0) {
            prefetch(0);
            prefetch(1);
            mbar_expect_tx(bbar, (uint32_t)(nch * bchunk));
            for (int c = 0; c < nch; ++c)
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        smem_u32(sB + (size_t)c * bchunk)),
                    "l"(prm.b + (size_t)c * bchunk), "r"(bchunk), "r"(bbar)
                    : "memory");
            const uint32_t idesc = b3_instr_desc(Np);
            bool ok = mbar_wait(bbar, 0);
            int s = 0, ph = 0, c = 0, t = 0;
            for (int g = 0; g < G && ok; ++g) {
                const int b = t & 1;
                if (c == 0 && t >= 2 && !mbar_wait(acce0 + 8 * b, ((t - 2) >> 1) & 1)) break;
                if (!mbar_wait(full0 + 8 * s, ph)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t aa = smem_u32(sA + (size_t)s * kB3Stage), bb = smem_u32(sB + (size_t)c * bchunk);
                const uint64_t ah = b3_desc(aa), am = b3_desc(aa + kB3Slice), al = b3_desc(aa + 2 * kB3Slice);
                const uint64_t bh = b3_desc(bb), bm = b3_desc(bb + Np * 32), bl = b3_desc(bb + 2 * Np * 32);
                const uint32_t d = tmem + (uint32_t)(b * 256);
                mma_bf16(d, al, bh, idesc, c > 0 ? 1u : 0u);
                mma_bf16(d, ah, bl, idesc, 1u);
                mma_bf16(d, am, bm, idesc, 1u);
                mma_bf16(d, am, bh, idesc, 1u);
                mma_bf16(d, ah, bm, idesc, 1u);
                mma_bf16(d, ah, bh, idesc, 1u);
                mma_commit(done0 + 8 * s);
                if (++s == NS) { s = 0; ph ^= 1; }
                if (++c == nch) {
                    mma_commit(accf0 + 8 * b);
                    c = 0;
                    ++t;
                    prefetch(t + 1);
                }
            }
        }
    } else {
        // ---- epilogue: TMEM -> registers -> global (transposed per plane)
        const int q = warp & 3, hi = (warp - 4 * kB3Groups) >> 2;
        const int nc16 = Np / 16, c_lo = (hi ? (nc16 + 1) / 2 : 0) * 16, c_hi = (hi ? nc16 : (nc16 + 1) / 2) * 16;
        const size_t nstride = OUT64 ? (size_t)2 * prm.R : (size_t)2 * prm.ldo;
        double norm = 0.0;
        for (int t = 0; t < my_tiles; ++t) {
            const int b = t & 1;
            if (!mbar_wait(accf0 + 8 * b, (t >> 1) & 1)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int tile = (int)blockIdx.x + t * (int)gridDim.x;
            const int row = tile * TM + q * 32 + lane;
            const bool row_ok = row < prm.rows;
            const int cr = row >> 1, part = row & 1;
            const int p = row_ok ? cr / prm.R : 0, r = row_ok ? cr % prm.R : 0;
            float *orow = OUT64 ? nullptr : prm.out + ((size_t)p * prm.N * 2 + part) * prm.ldo + r;
            double *orow64 = OUT64 ? prm.out64 + ((size_t)p * prm.N * prm.R + r) * 2 + part : nullptr;
            float sq[2] = {0.f, 0.f};   // at most 48 squares each: relative error below 3e-6
            const uint32_t tbase = tmem + (uint32_t)(b * 256) + ((uint32_t)(q * 32) << 16);
            auto load = [&](uint32_t (&v)[16], int c0) {
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
                    "%12, %13, %14, %15}, [%16];"
                    : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
                      "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
                      "=r"(v[14]), "=r"(v[15])
                    : "r"(tbase + (uint32_t)c0));
            };
            // waits for the loads in flight, whose registers are not touched before
            auto arrived = [&](uint32_t (&v)[16]) {
                asm volatile("tcgen05.wait::ld.sync.aligned;"
                             : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]),
                               "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]),
                               "+r"(v[14]), "+r"(v[15])
                             :
                             : "memory");
            };
            auto store = [&](const uint32_t (&v)[16], int c0) {
                if (!row_ok) return;
                const int left = prm.N - c0;   // columns past N are padding
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (j >= left) break;
                    const float f = __uint_as_float(v[j]);
                    if constexpr (OUT64) {
                        orow64[(size_t)(c0 + j) * nstride] = f2d_exact(f);
                        sq[j & 1] = fmaf(f, f, sq[j & 1]);
                    } else {
                        orow[(size_t)(c0 + j) * nstride] = f;
                    }
                }
            };
            uint32_t v[2][16];
            if (c_lo < c_hi) load(v[0], c_lo);
#pragma unroll 1
            for (int c0 = c_lo; c0 < c_hi; c0 += 32) {
                arrived(v[0]);
                if (c0 + 16 < c_hi) load(v[1], c0 + 16);
                store(v[0], c0);
                if (c0 + 16 < c_hi) {
                    arrived(v[1]);
                    if (c0 + 32 < c_hi) load(v[0], c0 + 32);
                    store(v[1], c0 + 16);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(acce0 + 8 * b);
            if constexpr (OUT64)
                if (prm.norm) norm += (double)sq[0] + (double)sq[1];
        }
        if constexpr (OUT64)
            if (prm.norm) {
                for (int o = 16; o > 0; o >>= 1) norm += __shfl_down_sync(0xffffffffu, norm, o);
                if (lane == 0) prm.norm[kB3Epi * blockIdx.x + warp - 4 * kB3Groups] = norm;
            }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    TDZ_CHECK(fn != nullptr, TDZ_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
    return fn;
}

// 2D FP32 tensor map: inner extent `inner` (elements), `outer` rows of pitch
// `pitch` elements, box KC x box_rows, 64-byte swizzle, zero fill outside
void make_map(CUtensorMap *map, const void *ptr, uint64_t inner, uint64_t outer, uint64_t pitch, uint32_t box_rows) {
    TDZ_CHECK((reinterpret_cast<uintptr_t>(ptr) & 15) == 0, TDZ_ERR_ARG, "transform operand not 16-byte aligned");
    TDZ_CHECK((pitch * 4) % 16 == 0, TDZ_ERR_ARG, "transform row pitch not a multiple of 16 bytes");
    const cuuint64_t dims[2] = {inner, outer};
    const cuuint64_t strides[1] = {pitch * 4};
    const cuuint32_t box[2] = {(cuuint32_t)KC, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void *>(ptr), dims, strides,
                                   box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    TDZ_CHECK(r == CUDA_SUCCESS, TDZ_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
}

float tf32_round_host(double v) {
    float f = (float)v;
    uint32_t u;
    std::memcpy(&u, &f, 4);
    u = (u + 0x1000u) & 0xFFFFE000u;
    std::memcpy(&f, &u, 4);
    return f;
}

// 256-row tiles where two sub-tiles' stages fit in shared memory (Np <= 192), else 128
template <int NP> constexpr int sub_tiles() { return TGShape<NP, 2>::fits ? 2 : 1; }

// TDZ_TRANSFORM picks a kernel: "split" the single-accumulator-pair one, "ws"
// the streaming warp-specialised one; else the B-resident kernel where all of
// B fits in shared memory beside two stages (6 Kp Np bytes: up to 176 x 176)
// and the streaming one beyond
int variant() {
    static const int v = [] {
        const char *e = std::getenv("TDZ_TRANSFORM");
        return !e ? 0 : std::string(e) == "split" ? 2 : std::string(e) == "ws" ? 1 : 0;
    }();
    return v;
}

// the B-resident kernel: in / out FP32 planar, or in64 / out64 FP64 natural order
void launch_b3(const TransformMat &T, const float *in, const double2 *in64, int planes, int R, int ldi, float *out,
               int ldo, double2 *out64, double *norm, cudaStream_t st) {
    static std::atomic<unsigned long long> done{0};
    once_per_device(done, [] {
        for (auto k : {k_transform_b3<false, false>, k_transform_b3<true, false>, k_transform_b3<false, true>})
            allow_smem(k, kB3Max);
    });
    TDZ_CHECK((reinterpret_cast<uintptr_t>(in) & 15) == 0, TDZ_ERR_ARG, "transform operand not 16-byte aligned");
    TDZ_CHECK(ldi % 4 == 0, TDZ_ERR_ARG, "transform row pitch not a multiple of 16 bytes");
    const long long rows = 2LL * planes * R;
    TDZ_CHECK(rows < (1LL << 31), TDZ_ERR_ARG, "transform too large");
    B3Params prm{};
    prm.in = in;
    prm.in64 = in64;
    prm.b = T.slices.as<uint8_t>();
    prm.out = out;
    prm.out64 = reinterpret_cast<double *>(out64);
    prm.norm = norm;
    prm.rows = (int)rows;
    prm.R = R;
    prm.K = T.K;
    prm.N = T.N;
    prm.Np = T.Np;
    prm.ldi = ldi;
    prm.ldo = ldo;
    prm.nch = T.Kp / KC;
    prm.tiles = (prm.rows + TM - 1) / TM;
    prm.ns = b3_stages(T.Kp, T.Np);
    const size_t smem = 1024 + b3_bytes(T.Kp, T.Np) + (size_t)prm.ns * kB3Stage + 256;
    const int grid = std::min(prm.tiles, sm_count());
    if (in64) k_transform_b3<true, false><<<grid, kB3Threads, smem, st>>>(prm);
    else if (out64) k_transform_b3<false, true><<<grid, kB3Threads, smem, st>>>(prm);
    else k_transform_b3<false, false><<<grid, kB3Threads, smem, st>>>(prm);
    TDZ_CUDA(cudaGetLastError());
    count_launch();
}

template <int NP>
void launch(const TransformMat &T, const float *in, int ldi, TGParams prm, cudaStream_t st) {
    const bool ws = variant() != 2;
    constexpr int MS = sub_tiles<NP>();
    const size_t smem = ws ? WSShape<NP>::SMEM : TGShape<NP, MS>::SMEM;
    static std::atomic<unsigned long long> done{0};
    once_per_device(done, [] {
        allow_smem(k_transform<NP, MS>, TGShape<NP, MS>::SMEM);
        allow_smem(k_transform_ws<NP>, WSShape<NP>::SMEM);
    });
    CUtensorMap amap;
    const int rows_per_tile = ws ? TM : TM * MS;
    make_map(&amap, in, (uint64_t)T.K, (uint64_t)prm.rows, (uint64_t)ldi, (uint32_t)rows_per_tile);
    prm.tiles = (prm.rows + rows_per_tile - 1) / rows_per_tile;
    const int grid = std::min(prm.tiles, sm_count());
    if (ws) k_transform_ws<NP><<<grid, 320, smem, st>>>(amap, T.map, prm);
    else k_transform<NP, MS><<<grid, 160, smem, st>>>(amap, T.map, prm);
}

}  // namespace

namespace {
// the process's error word; its address goes to each device before its first transform
std::atomic<int> *error_word() {
    static std::atomic<int> *word = [] {
        void *p = nullptr;
        TDZ_CUDA(cudaHostAlloc(&p, sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
        return new (p) std::atomic<int>(0);
    }();
    static std::mutex mu;
    static std::set<int> done;
    int dev = 0;
    TDZ_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    if (!done.count(dev)) {
        TDZ_CUDA(cudaMemcpyToSymbol(g_tgemm_error, &word, sizeof(void *)));
        done.insert(dev);
    }
    return word;
}
}  // namespace

bool transform_supported(int N) { return N >= 1 && N <= 256; }

void TransformMat::build(const std::vector<double> &B, int K_, int N_) {
    K = K_;
    N = N_;
    TDZ_CHECK(transform_supported(N), TDZ_ERR_UNSUPPORTED, "tensor-core transform supports N <= 256");
    TDZ_CHECK((int)B.size() == K * N, TDZ_ERR_ARG, "transform matrix size");
    Kp = (K + KC - 1) / KC * KC;
    Np = (N + 15) / 16 * 16;
    error_word();
    std::vector<float> h((size_t)2 * Np * Kp, 0.f);
    for (int n = 0; n < N; ++n)
        for (int k = 0; k < K; ++k) {
            const double v = B[(size_t)k * N + n];
            const float hi = tf32_round_host(v);
            h[(size_t)n * Kp + k] = hi;
            h[(size_t)(Np + n) * Kp + k] = tf32_round_host(v - (double)hi);
        }
    upload(hilo, h);
    if (b3_stages(Kp, Np) > 0) {   // BF16 slices in the B-resident kernel's shared-memory order
        std::vector<uint16_t> b((size_t)3 * Kp * Np, 0);
        for (int n = 0; n < N; ++n)
            for (int k = 0; k < K; ++k) {
                double v = B[(size_t)k * N + n];
                for (int sl = 0; sl < 3; ++sl) {
                    float f = (float)v;
                    uint32_t u;
                    std::memcpy(&u, &f, 4);
                    u = (u + 0x7FFFu + ((u >> 16) & 1u)) & 0xFFFF0000u;   // nearest BF16, ties to even
                    std::memcpy(&f, &u, 4);
                    v -= (double)f;
                    const size_t off = ((size_t)(k / KC) * 3 + sl) * Np * 32 + b3_off(n, (k % KC) / 8) + (k % 8) * 2;
                    b[off / 2] = (uint16_t)(u >> 16);
                }
            }
        upload(slices, b);
    }
    make_map(&map, hilo.ptr, Kp, 2 * (uint64_t)Np, Kp, (uint32_t)Np);
}

int take_transform_error() { return error_word()->exchange(0); }

bool transform_natural(const TransformMat &T) { return variant() == 0 && T.slices.ptr; }
int transform_norm_parts(int planes, int R) {
    return kB3Epi * (int)std::min<long long>((2LL * planes * R + TM - 1) / TM, sm_count());
}
void transform_from64(const TransformMat &T, const double2 *in, int planes, int R, float *out, int ldo, cudaStream_t st) {
    TDZ_CHECK(transform_natural(T) && ldo >= R, TDZ_ERR_INTERNAL, "natural-order transform");
    launch_b3(T, nullptr, in, planes, R, 4, out, ldo, nullptr, nullptr, st);
}
void transform_to64(const TransformMat &T, const float *in, int planes, int R, int ldi, double2 *out, double *norm,
                    cudaStream_t st) {
    TDZ_CHECK(transform_natural(T) && ldi >= T.K, TDZ_ERR_INTERNAL, "natural-order transform");
    launch_b3(T, in, nullptr, planes, R, ldi, nullptr, 0, out, norm, st);
}

void transform(const TransformMat &T, const float *in, int planes, int R, int ldi, float *out, int ldo,
               cudaStream_t st) {
    TDZ_CHECK(ldi >= T.K && ldo >= R, TDZ_ERR_ARG, "transform pitches too small");
    const long long rows = 2LL * planes * R;
    TDZ_CHECK(rows < (1LL << 31), TDZ_ERR_ARG, "transform too large");
    TGParams prm{};
    prm.out = out;
    prm.rows = (int)rows;
    prm.R = R;
    prm.N = T.N;
    prm.ldo = ldo;
    prm.nchunks = T.Kp / KC;
    if (transform_natural(T)) {
        launch_b3(T, in, nullptr, planes, R, ldi, out, ldo, nullptr, nullptr, st);
        return;
    }
    switch (T.Np) {
    case 16: launch<16>(T, in, ldi, prm, st); break;
    case 32: launch<32>(T, in, ldi, prm, st); break;
    case 48: launch<48>(T, in, ldi, prm, st); break;
    case 64: launch<64>(T, in, ldi, prm, st); break;
    case 80: launch<80>(T, in, ldi, prm, st); break;
    case 96: launch<96>(T, in, ldi, prm, st); break;
    case 112: launch<112>(T, in, ldi, prm, st); break;
    case 128: launch<128>(T, in, ldi, prm, st); break;
    case 144: launch<144>(T, in, ldi, prm, st); break;
    case 160: launch<160>(T, in, ldi, prm, st); break;
    case 176: launch<176>(T, in, ldi, prm, st); break;
    case 192: launch<192>(T, in, ldi, prm, st); break;
    case 208: launch<208>(T, in, ldi, prm, st); break;
    case 224: launch<224>(T, in, ldi, prm, st); break;
    case 240: launch<240>(T, in, ldi, prm, st); break;
    case 256: launch<256>(T, in, ldi, prm, st); break;
    default: throw Error(TDZ_ERR_INTERNAL, "bad transform tile width");
    }
    TDZ_CUDA(cudaGetLastError());
    count_launch();
}

}  // namespace tdz
