// Complex helpers on float2 / double2 (device). Internal.
#pragma once
#include <cuda_runtime.h>

namespace tdz {

// Double-float: a value hi + lo carried as two FP32 numbers (about 48
// significant bits; Dekker 1971, as in the double-double arithmetic of Hida,
// Li and Bailey 2001 with single-precision halves). The product a.hi b.hi is
// split exactly with an fma residual, the sum uses Knuth's two-sum error term.
// Accumulations skip the per-term renormalisation: lo collects the product
// and rounding errors of a whole banded sum (a few dozen terms, so it stays
// far below hi's last bit times the term count) and renorm() folds it into
// hi once per stage result. Every step is an explicitly rounded intrinsic, so
// the compiler cannot contract or reorder it. Relative error near 1e-14 on
// the FP32 pipes, which on this GPU run at 64x the FP64 rate.
struct dff {
    float hi, lo;
    dff() = default;
    __host__ __device__ constexpr dff(float v) : hi(v), lo(0.f) {}
    __host__ __device__ constexpr dff(float h, float l) : hi(h), lo(l) {}
};
// complex double-float: the (re, im) pairs of the high and the low parts, so
// that one packed FP32 instruction (f32x2) works on both components. The
// pipes execute a packed instruction at the rate of its two halves, but it
// takes one issue slot instead of two, and the double-float kernels are bound
// by issue (3D stage apply of 8.8 M coefficients, degree 3: 925 us scalar, 816
// us packed; mass apply 533 and 436).
struct __align__(16) cdff {
    float2 hi, lo;
    __host__ __device__ dff re() const { return dff(hi.x, lo.x); }
    __host__ __device__ dff im() const { return dff(hi.y, lo.y); }
};
__host__ __device__ inline cdff make_cdff(dff re, dff im) {
    cdff c;
    c.hi = make_float2(re.hi, im.hi);
    c.lo = make_float2(re.lo, im.lo);
    return c;
}
__device__ __forceinline__ dff operator-(dff a) { return dff(-a.hi, -a.lo); }
// a * b + c in the arithmetic type of the operands
__device__ __forceinline__ float tfma(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double tfma(double a, double b, double c) { return ::fma(a, b, c); }
// double-float, unnormalised result (10 FP32 instructions). The error of
// s = c.hi + p by two-sum is (c.hi - (s - bv)) + (p - bv) with bv = s - c.hi, and
// the product's is a b - p: one fused a b - bv gives the two terms in p. Its
// rounding is 2^-24 of a term that is itself 2^-24 of the sum, as those of the
// cross products; together with dff_split's rounded high part the sums are no
// less accurate than with the errors taken one by one (12 instructions) and a
// truncated high part (products of 7 to 512 terms: rms 0.60 to 0.95 of it).
__device__ __forceinline__ dff tfma(dff a, dff b, dff c) {
    const float p = __fmul_rn(a.hi, b.hi);
    const float s = __fadd_rn(c.hi, p);
    const float nbv = __fsub_rn(c.hi, s);
    const float es = __fsub_rn(c.hi, __fadd_rn(s, nbv));
    float e = __fmaf_rn(a.hi, b.hi, nbv);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    return dff(s, __fadd_rn(__fadd_rn(c.lo, es), e));
}
// fold lo into hi (fast two-sum; |lo| <= |hi| for an accumulated value)
__device__ __forceinline__ dff renorm(dff a) {
    const float h = __fadd_rn(a.hi, a.lo);
    return dff(h, __fsub_rn(a.lo, __fsub_rn(h, a.hi)));
}
__host__ __device__ inline dff dff_from(double v) {
    const float h = (float)v;
    return dff(h, (float)(v - (double)h));
}

// FP64 -> double-float split off the FP64 pipe (GB300's FP64 pipe, which also
// executes FP64 <-> FP32 conversions, issues 2 instructions per clock per
// SM). hi = v rounded to 24 significant bits: its exponent is the FP64
// exponent's low 8 bits with the top one flipped (1023 - 127 = 0x380), so a
// funnel shift puts exponent and mantissa in place, and the first bit below
// rounds up. lo = the remaining 29 bits as a signed integer, converted (rounded
// to 24 bits) and scaled: hi + lo carries 49 bits or more. |v| < 2^-100 (and zero,
// subnormals) maps to 0; Inf/NaN and |v| that rounds to 2^128 or is beyond map
// to a non-finite hi. Selects, not branches: a kernel's other loads and splits
// are not held up by them (mass apply of 8.8 M coefficients 404 us with branches,
// 369 us without; stage apply 750 and 711; FP32 apply on FP64 vectors 275 and 253).
__device__ __forceinline__ dff dff_split(double v) {
    const unsigned int h32 = (unsigned int)__double2hiint(v), l32 = (unsigned int)__double2loint(v);
    const unsigned int sign = h32 & 0x80000000u;
    const unsigned int hb = ((__funnelshift_l(l32, h32, 3) ^ 0x40000000u) & 0x7FFFFFFFu) | sign;
    const unsigned int scale = (hb & 0xFF800000u) - (23u << 23);   // signed 2^(e - 23)
    const float lo = __fmul_rn(__fmul_rn(__int2float_rn((int)(l32 << 3)), 0x1p-32f), __uint_as_float(scale));
    const unsigned int above = (h32 & 0x7FFFFFFFu) - ((1023u - 100u) << 20);   // exponents -100 .. 127 stay below 228 << 20
    const bool normal = above < (228u << 20);
    const unsigned int other = (int)above < 0 ? sign : hb | 0x7F800000u;
    return dff(__uint_as_float(normal ? hb + ((l32 >> 28) & 1u) : other), normal ? lo : 0.f);
}
// exact FP32 -> FP64 widening with integer operations (normal values; zero and
// subnormals give signed zero, Inf/NaN stay non-finite)
__device__ __forceinline__ double f2d_exact(float f) {
    const unsigned int b = __float_as_uint(f), t = b & 0x7FFFFFFFu, sign = b & 0x80000000u;
    const bool normal = t - 0x00800000u < 0x7F000000u, big = t >= 0x7F800000u;
    const unsigned int h = normal ? (t >> 3) + 0x38000000u : big ? 0x7FF00000u | ((t & 0x7FFFFFu) >> 3) : 0u;
    return __hiloint2double((int)(sign | h), normal || big ? (int)(b << 29) : 0);
}
// hi + lo rounded to FP64: one FP64 add
__device__ __forceinline__ double dff_to_double(dff a) { return f2d_exact(a.hi) + f2d_exact(a.lo); }

template <class T> struct CT;
template <> struct CT<float> { using type = float2; };
template <> struct CT<double> { using type = double2; };
template <> struct CT<dff> { using type = cdff; };

// complex type in memory for each arithmetic type
template <class T> struct MemC { using type = typename CT<T>::type; };
template <> struct MemC<dff> { using type = double2; };
template <class C, class M> __device__ __forceinline__ C load_c(const M &m) { return m; }
template <> __device__ __forceinline__ cdff load_c<cdff, double2>(const double2 &m) {
    return make_cdff(dff_split(m.x), dff_split(m.y));
}
template <class M, class C> __device__ __forceinline__ M store_c(const C &c) { return c; }
template <> __device__ __forceinline__ double2 store_c<double2, cdff>(const cdff &c) {
    return make_double2(dff_to_double(c.re()), dff_to_double(c.im()));
}

template <class C> __device__ __forceinline__ C czero() { C c; c.x = 0; c.y = 0; return c; }
template <> __device__ __forceinline__ cdff czero<cdff>() { return make_cdff(dff(0.f), dff(0.f)); }
// a complex number from its parts, and the parts
template <class C, class T> __device__ __forceinline__ C cmake(T re, T im) {
    C c;
    c.x = re;
    c.y = im;
    return c;
}
template <> __device__ __forceinline__ cdff cmake<cdff, dff>(dff re, dff im) { return make_cdff(re, im); }
template <class C> __device__ __forceinline__ auto cre(const C &c) { return c.x; }
template <class C> __device__ __forceinline__ auto cim(const C &c) { return c.y; }
__device__ __forceinline__ dff cre(const cdff &c) { return c.re(); }
__device__ __forceinline__ dff cim(const cdff &c) { return c.im(); }

// packed pairs: a - b (one rounding, as a subtraction), renorm of both parts
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
// acc += a v for both components, a given per component (10 packed
// instructions, the arithmetic of the scalar tfma). With 12, and without mul2 for
// the first terms: 3D stage apply of 8.8 M coefficients, degree 3, 800 us, now
// 750 us; degree 4 with 1.4 M, 246 and 217 us
__device__ __forceinline__ void fma2(cdff &acc, float2 ahi, float2 alo, float2 vhi, float2 vlo) {
    // a fused + 0: a packed multiply with this addition as its only use gets
    // contracted with it, and the sum's error is then no longer bv's
    const float2 p = __ffma2_rn(ahi, vhi, make_float2(0.f, 0.f));
    const float2 s = __fadd2_rn(acc.hi, p);
    const float2 nbv = sub2(acc.hi, s);
    const float2 es = sub2(acc.hi, __fadd2_rn(s, nbv));
    float2 e = __ffma2_rn(ahi, vhi, nbv);
    e = __ffma2_rn(ahi, vlo, e);
    e = __ffma2_rn(alo, vhi, e);
    acc.hi = s;
    acc.lo = __fadd2_rn(__fadd2_rn(acc.lo, es), e);
}
// acc = a v (4 packed instructions): the first term of a sum
__device__ __forceinline__ void mul2(cdff &acc, float2 ahi, float2 alo, float2 vhi, float2 vlo) {
    const float2 p = __fmul2_rn(ahi, vhi);
    float2 e = __ffma2_rn(ahi, vhi, make_float2(-p.x, -p.y));
    e = __ffma2_rn(ahi, vlo, e);
    acc.hi = p;
    acc.lo = __ffma2_rn(alo, vhi, e);
}

// renormalise a stage result (identity for native types)
template <class C> __device__ __forceinline__ C cnorm(const C &c) { return c; }
template <> __device__ __forceinline__ cdff cnorm<cdff>(const cdff &c) {
    cdff r;
    r.hi = __fadd2_rn(c.hi, c.lo);
    r.lo = sub2(c.lo, sub2(r.hi, c.hi));
    return r;
}
template <class T, class C> __device__ __forceinline__ void rfma(C &acc, T a, C v) {
    acc.x = tfma(a, v.x, acc.x);
    acc.y = tfma(a, v.y, acc.y);
}
template <> __device__ __forceinline__ void rfma<dff, cdff>(cdff &acc, dff a, cdff v) {
    fma2(acc, make_float2(a.hi, a.hi), make_float2(a.lo, a.lo), v.hi, v.lo);
}
// acc += i b v (b real: the imaginary part of a purely imaginary coefficient)
template <class T, class C> __device__ __forceinline__ void ifma(C &acc, T b, C v) {
    acc.x = tfma(-b, v.y, acc.x);
    acc.y = tfma(b, v.x, acc.y);
}
template <> __device__ __forceinline__ void ifma<dff, cdff>(cdff &acc, dff b, cdff v) {
    // i v first: loops over b share it
    fma2(acc, make_float2(b.hi, b.hi), make_float2(b.lo, b.lo), make_float2(-v.hi.y, v.hi.x), make_float2(-v.lo.y, v.lo.x));
}
// acc = a v, acc = i b v: the first term of a sum. Double-float products skip the
// addition's six instructions; native types keep the fused form with zero.
template <class T, class C> __device__ __forceinline__ void rset(C &acc, T a, C v) {
    acc = czero<C>();
    rfma(acc, a, v);
}
template <> __device__ __forceinline__ void rset<dff, cdff>(cdff &acc, dff a, cdff v) {
    mul2(acc, make_float2(a.hi, a.hi), make_float2(a.lo, a.lo), v.hi, v.lo);
}
template <class T, class C> __device__ __forceinline__ void iset(C &acc, T b, C v) {
    acc = czero<C>();
    ifma(acc, b, v);
}
template <> __device__ __forceinline__ void iset<dff, cdff>(cdff &acc, dff b, cdff v) {
    mul2(acc, make_float2(b.hi, b.hi), make_float2(b.lo, b.lo), make_float2(-v.hi.y, v.hi.x), make_float2(-v.lo.y, v.lo.x));
}
// FP32 pairs packed as well (3D apply of 8.8 M FP32 coefficients, degree 3: 184 us
// scalar, 150 us packed)
template <> __device__ __forceinline__ void rfma<float, float2>(float2 &acc, float a, float2 v) {
    acc = __ffma2_rn(make_float2(a, a), v, acc);
}
template <> __device__ __forceinline__ void ifma<float, float2>(float2 &acc, float b, float2 v) {
    acc = __ffma2_rn(make_float2(b, b), make_float2(-v.y, v.x), acc);
}
template <class C> __device__ __forceinline__ void cfma(C &acc, C a, C v) {
    acc.x = tfma(a.x, v.x, acc.x);
    acc.x = tfma(-a.y, v.y, acc.x);
    acc.y = tfma(a.x, v.y, acc.y);
    acc.y = tfma(a.y, v.x, acc.y);
}
template <> __device__ __forceinline__ void cfma<float2>(float2 &acc, float2 a, float2 v) {
    rfma(acc, a.x, v);
    ifma(acc, a.y, v);
}
template <> __device__ __forceinline__ void cfma<cdff>(cdff &acc, cdff a, cdff v) {
    rfma(acc, a.re(), v);
    ifma(acc, a.im(), v);
}
// acc += a v with a of a known kind: 0 complex, 1 real, 2 imaginary
template <class C> __device__ __forceinline__ void kfma(C &acc, C a, C v, int kind) {
    if (kind == 1) rfma(acc, cre(a), v);
    else if (kind == 2) ifma(acc, cim(a), v);
    else cfma(acc, a, v);
}
// acc = a v (kset: a of a known kind)
template <class C> __device__ __forceinline__ void cset(C &acc, C a, C v) {
    acc = czero<C>();
    cfma(acc, a, v);
}
template <> __device__ __forceinline__ void cset<cdff>(cdff &acc, cdff a, cdff v) {
    rset(acc, a.re(), v);
    ifma(acc, a.im(), v);
}
template <class C> __device__ __forceinline__ void kset(C &acc, C a, C v, int kind) {
    if (kind == 1) rset(acc, cre(a), v);
    else if (kind == 2) iset(acc, cim(a), v);
    else cset(acc, a, v);
}
// acc += conj(a) v
template <class C> __device__ __forceinline__ void cfma_conj(C &acc, C a, C v) {
    acc.x = tfma(a.x, v.x, acc.x);
    acc.x = tfma(a.y, v.y, acc.x);
    acc.y = tfma(a.x, v.y, acc.y);
    acc.y = tfma(-a.y, v.x, acc.y);
}
template <> __device__ __forceinline__ void cfma_conj<cdff>(cdff &acc, cdff a, cdff v) {
    rfma(acc, a.re(), v);
    ifma(acc, -a.im(), v);
}

// sum of (re, im) over a CTA of NT threads, in a fixed order; valid in thread 0
template <int NT> __device__ __forceinline__ double2 block_sum(double re, double im) {
    __shared__ double2 ws[NT / 32];
    for (int o = 16; o > 0; o >>= 1) {
        re += __shfl_down_sync(0xffffffffu, re, o);
        im += __shfl_down_sync(0xffffffffu, im, o);
    }
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = make_double2(re, im);
    __syncthreads();
    double2 t = make_double2(0.0, 0.0);
    if (threadIdx.x == 0)
#pragma unroll
        for (int w = 0; w < NT / 32; ++w) {
            t.x += ws[w].x;
            t.y += ws[w].y;
        }
    return t;
}

}  // namespace tdz
