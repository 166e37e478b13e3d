// Device-side modular arithmetic on 64-bit residues (q < 2^62).
//
// The routines that name a formula of the reference's native backend
// reproduce it operation for operation, so results are bit-identical including
// the lazy representatives in [0, 2q) / [0, 4q).  64x64->128 products use
// __umul64hi / 64-bit mul.lo, no tensor cores.  Where only the residue
// matters (intermediate values of a transform whose output is reduced to
// [0, q)), the relaxed and FP64 forms below compute the same residues with
// other representatives; all of their arithmetic is exact.
#pragma once

#include <cstdint>

namespace axhel_dev {

// ConditionalSubtractNative (axhel/include/axhel/number-theory/modular-reduction.hpp:22-25)
__device__ __forceinline__ uint64_t csub(uint64_t x, uint64_t bound)
{
    return x >= bound ? x - bound : x;
}

// ReduceInputNative<F> (modular-reduction.hpp:48-67): cascade 8q -> 4q -> 2q -> q.
template <int F>
__device__ __forceinline__ uint64_t reduce_input(uint64_t x, uint64_t q)
{
    if constexpr (F == 8) x = csub(x, q << 2);
    if constexpr (F >= 4) x = csub(x, q << 1);
    if constexpr (F >= 2) x = csub(x, q);
    return x;
}

// Conditional subtract for the NTT's bounded ranges: the same function as
// csub() whenever bound <= 2^63 and x - bound < 2^63, which holds for every
// value a transform handles: x < 4q and bound <= 2q with q < 2^62 in the
// reference's butterflies, x < 32q and bound <= 16q with q < 2^59 in the relaxed
// ones.  Testing the sign of the difference takes one compare on its high word
// instead of a 64-bit compare.
__device__ __forceinline__ uint64_t csub_lazy(uint64_t x, uint64_t bound)
{
    const uint64_t d = x - bound;
    return static_cast<int64_t>(d) < 0 ? x : d;
}

// floor(a * b / 2^64) through a 32-bit multiply-add carry chain (seven
// integer multiply-adds and one add).
__device__ __forceinline__ uint64_t mul_hi64(uint64_t a, uint64_t b)
{
    uint64_t r;
    asm("{\n\t"
        ".reg .u32 a0, a1, b0, b1, t0, t1, t2, r0, r1;\n\t"
        "mov.b64 {a0, a1}, %1;\n\t"
        "mov.b64 {b0, b1}, %2;\n\t"
        "mul.hi.u32 t0, a0, b0;\n\t"
        "mad.lo.cc.u32 t0, a0, b1, t0;\n\t"
        "madc.hi.u32 t1, a0, b1, 0;\n\t"
        "mad.lo.cc.u32 t0, a1, b0, t0;\n\t"
        "madc.hi.cc.u32 t1, a1, b0, t1;\n\t"
        "addc.u32 t2, 0, 0;\n\t"
        "mad.lo.cc.u32 r0, a1, b1, t1;\n\t"
        "madc.hi.u32 r1, a1, b1, t2;\n\t"
        "mov.b64 %0, {r0, r1};\n\t"
        "}"
        : "=l"(r)
        : "l"(a), "l"(b));
    return r;
}

// (v * w + e * nq) mod 2^64 with 32-bit multiply-adds; nq = 2^64 - q turns
// the Shoup subtraction v*w - e*q into one accumulation chain.
__device__ __forceinline__ uint64_t mul_lo_acc(uint64_t v, uint64_t w, uint64_t e, uint64_t nq)
{
    uint64_t r;
    asm("{\n\t"
        ".reg .u32 v0, v1, w0, w1, e0, e1, n0, n1, r0, r1;\n\t"
        "mov.b64 {v0, v1}, %1;\n\t"
        "mov.b64 {w0, w1}, %2;\n\t"
        "mov.b64 {e0, e1}, %3;\n\t"
        "mov.b64 {n0, n1}, %4;\n\t"
        "mul.lo.u32 r0, v0, w0;\n\t"
        "mul.hi.u32 r1, v0, w0;\n\t"
        "mad.lo.u32 r1, v0, w1, r1;\n\t"
        "mad.lo.u32 r1, v1, w0, r1;\n\t"
        "mad.lo.u32 r1, e0, n1, r1;\n\t"
        "mad.lo.u32 r1, e1, n0, r1;\n\t"
        "mad.lo.cc.u32 r0, e0, n0, r0;\n\t"
        "madc.hi.u32 r1, e0, n0, r1;\n\t"
        "mov.b64 %0, {r0, r1};\n\t"
        "}"
        : "=l"(r)
        : "l"(v), "l"(w), "l"(e), "l"(nq));
    return r;
}

// MultiplyUIntModLazy (axhel/include/axhel/number-theory/uint-arith.hpp:48-52):
// value * w - floor(value * w' / 2^64) * q  (mod 2^64), in [0, 2q).
__device__ __forceinline__ uint64_t shoup_lazy(uint64_t v, uint64_t w, uint64_t wq, uint64_t q)
{
    return mul_lo_acc(v, w, mul_hi64(v, wq), 0 - q);
}

// Barrett product of EltwiseMulModNative (axhel/eltwise/eltwise-mul-mod.cpp:40-60),
// alpha = 62, beta = -2: x, y in [0, q); mu = floor(2^(k+62) / q); shift = k - 2.
__device__ __forceinline__ uint64_t barrett_mul(uint64_t x, uint64_t y, uint64_t q, uint64_t mu,
                                                uint32_t shift)
{
    const uint64_t lo = x * y;
    const uint64_t hi = __umul64hi(x, y);
    const uint64_t c1 = shift ? (lo >> shift) | (hi << (64 - shift)) : lo;
    const uint64_t qhat = __umul64hi(c1, mu);
    const uint64_t z = lo - qhat * q;
    return reduce_input<4>(z, q);
}

// BarrettReduceUInt64Native (axhel/eltwise/eltwise-reduce-mod.cpp:19-29).
__device__ __forceinline__ uint64_t barrett_reduce64(uint64_t x, uint64_t q, uint64_t mu, uint32_t shift)
{
    const uint64_t qhat = __umul64hi(x >> shift, mu);
    return reduce_input<4>(x - qhat * q, q);
}

// ForwardButterflyNative (axhel/ntt/ntt-internal.hpp:20-31).
__device__ __forceinline__ void fwd_butterfly(uint64_t& x, uint64_t& y, uint64_t w, uint64_t wq, uint64_t q,
                                              uint64_t q2)
{
    const uint64_t gx = csub_lazy(x, q2);
    const uint64_t t = shoup_lazy(y, w, wq, q);
    x = gx + t;
    y = gx + q2 - t;
}

// InverseButterflyNative (axhel/ntt/ntt-internal.hpp:37-49).
__device__ __forceinline__ void inv_butterfly(uint64_t& x, uint64_t& y, uint64_t w, uint64_t wq, uint64_t q,
                                              uint64_t q2)
{
    const uint64_t u = x, v = y;
    x = csub_lazy(u + v, q2);
    y = shoup_lazy(u + q2 - v, w, wq, q);
}

// Final inverse stage (axhel/ntt/ntt-native.cpp:126-141): upper branch times
// N^-1, lower branch times scaled_root = N^-1 * w_last.
__device__ __forceinline__ void inv_final_butterfly(uint64_t& x, uint64_t& y, uint64_t ninv, uint64_t ninv_q,
                                                    uint64_t sr, uint64_t sr_q, uint64_t q, uint64_t q2)
{
    const uint64_t gx = csub_lazy(x, q2);
    const uint64_t v = y;
    x = shoup_lazy(gx + v, ninv, ninv_q, q);
    y = shoup_lazy(gx + q2 - v, sr, sr_q, q);
}

// ------------------------------------------------- relaxed integer forms
// For transforms whose outputs are reduced to [0, q), so that intermediate
// values may be any representative.  Bound: the integer multiply pipe, where
// a high 32-bit product costs two low ones; the low-by-low term of the quotient
// and its carries are left out.  768 limbs of N = 2^16 to [0, q): 60-bit moduli
// with the reference's butterflies 567 us forward and 599 inverse, 55-bit ones
// relaxed 530 and 537.

// value * w - e * q with e = floor(value * w' / 2^64) - {0, 1, 2}: the terms
// y1 w'1, floor(y1 w'0 / 2^32) and floor(y0 w'1 / 2^32) only, each floor and
// the missing y0 w'0 / 2^64 below 1.  The result is in [0, 4q) for any
// 64-bit value (Shoup's own error is below q, three units more at most).
__device__ __forceinline__ uint64_t shoup_relaxed(uint64_t v, uint64_t w, uint64_t wq, uint64_t q)
{
    uint64_t e;
    asm("{\n\t"
        ".reg .u32 a0, a1, b0, b1, u, c, r0, r1;\n\t"
        "mov.b64 {a0, a1}, %1;\n\t"
        "mov.b64 {b0, b1}, %2;\n\t"
        "mul.hi.u32 u, a1, b0;\n\t"
        "mad.hi.cc.u32 u, a0, b1, u;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "mad.lo.cc.u32 r0, a1, b1, u;\n\t"
        "madc.hi.u32 r1, a1, b1, c;\n\t"
        "mov.b64 %0, {r0, r1};\n\t"
        "}"
        : "=l"(e)
        : "l"(v), "l"(wq));
    return mul_lo_acc(v, w, e, 0 - q);
}

// ---------------------------------------------------------- FP64 forms
// For q < 2^50.  Residues are integers held in doubles; every value stays
// below 2^53 in magnitude and every result is an exact integer.  The product is
// the fused multiply-add one of J. van der Hoeven, G. Lecerf and G. Quintin,
// "Modular SIMD arithmetic in Mathemagix" (ACM Trans. Math. Softw. 43, 2016): high
// and low part, a rounded quotient, the remainder.  A butterfly is eight FP64
// instructions of two clocks each per warp (the FP64 pipe runs at half the FP32
// rate and is otherwise idle here) against 36 clocks of integer multiplies.  768
// limbs of N = 2^16 to [0, q), 45-bit moduli: 345 us each way (60 bits, integer:
// 567 forward, 599 inverse).

constexpr double kFpRound = 6755399441055744.0;  // 1.5 * 2^52: adding it rounds to an integer
constexpr double kFp2p52 = 4503599627370496.0;

__device__ __forceinline__ double as_fp(uint64_t x) { return __longlong_as_double((long long)x); }
__device__ __forceinline__ uint64_t as_u64(double x) { return (uint64_t)__double_as_longlong(x); }

// Nearest integer to a*b for |a*b| < 2^51 (one rounding).
__device__ __forceinline__ double fp_quot(double a, double b) { return __dadd_rn(__fma_rn(a, b, kFpRound), -kFpRound); }

// y * w - rint(y * w / q) * q for |y| <= Y q, Y <= 4, |w| <= q/2, wq = w/q.
// h + l = y w exactly; h - c q is an integer of magnitude below 2^51, so its
// fma is exact, and so is the sum.  |c - y w / q| <= 1/2 + |y w / q| times the
// relative error of wq: the result is within q/2 + Y q/16 for wq rounded once
// (3q/4 at Y = 4) and within q/2 + Y q/8 for wq = w * (1/q rounded).
__device__ __forceinline__ double fp_mul(double y, double w, double wq, double q)
{
    const double h = __dmul_rn(y, w);
    const double c = fp_quot(y, wq);
    const double l = __fma_rn(y, w, -h);
    return __dadd_rn(__fma_rn(-c, q, h), l);
}

// a * b mod q for |a b| <= 2 q^2, |a|, |b| <= 4q: the quotient from h / q, with
// a relative error of 2^-52, so the result is within q/2 + |a b| / 4q (7q/8 for
// |a| <= 3q/4, |b| <= 2q; q at most).
__device__ __forceinline__ double fp_mulmod(double a, double b, double q, double qi)
{
    const double h = __dmul_rn(a, b);
    const double c = fp_quot(h, qi);
    const double l = __fma_rn(a, b, -h);
    return __dadd_rn(__fma_rn(-c, q, h), l);
}

// x - rint(x / q) * q for |x| < 2^53: within q/2 and a rounding of q/2.
__device__ __forceinline__ double fp_reduce(double x, double q, double qi) { return __fma_rn(-fp_quot(x, qi), q, x); }

// x < 2^52 as a double, less `off - 2^52`.
__device__ __forceinline__ double fp_from_u64(uint64_t x, double off)
{
    return __dadd_rn(as_fp(x | 0x4330000000000000ull), -off);
}

// An integer 0 <= x < 2^52 back to 64-bit form.
__device__ __forceinline__ uint64_t fp_to_u64(double x) { return as_u64(__dadd_rn(x, kFp2p52)) & 0x000fffffffffffffull; }

// The canonical residue of x in (-q, q).
__device__ __forceinline__ uint64_t fp_canon(double x, double q)
{
    const double off = __double2hiint(x) < 0 ? __dadd_rn(q, kFp2p52) : kFp2p52;
    return as_u64(__dadd_rn(x, off)) & 0x000fffffffffffffull;
}

}  // namespace axhel_dev
