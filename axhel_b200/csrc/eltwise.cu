// Element-wise modular kernels for sm_100a (EltwiseAdd/Sub/Mul/FMA/ReduceMod).
//
// HBM-bound streaming kernels: a grid sized to a multiple of the SM count
// walks the vector in chunks of four 16-byte loads per operand and thread,
// each warp access 512 contiguous bytes (all pointers 16-byte aligned), or
// in scalar 8-byte accesses otherwise.  The
// arithmetic of each element is the reference native backend's formula
// (axhel/eltwise/eltwise-*-mod.cpp), so every output is bit-identical.
// result may alias any operand: each element is read before it is written by
// the same thread.
#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"
#include "launch.h"
#include "eltwise_ops.cuh"
#include "modarith.cuh"

namespace axhel_impl {
using namespace axhel_dev;

// ---------------------------------------------------------------- kernels

template <class Op, bool HAS_B>
__global__ void __launch_bounds__(256) eltwise_vec_kernel(uint64_t* r, const uint64_t* a, const uint64_t* b,
                                                          uint64_t n, const Op op)
{
    // 16-byte aligned path.  A CTA takes chunks of V * blockDim 16-byte
    // vectors; vector k of a chunk is read by thread t at k * blockDim + t,
    // so every warp access covers 512 contiguous bytes, and all loads of a
    // chunk are issued before its first store (V loads per operand in flight
    // per thread).
    constexpr int V = 4;
    const uint64_t nv = n >> 1;  // 16-byte vectors
    const ulonglong2* a2 = reinterpret_cast<const ulonglong2*>(a);
    const ulonglong2* b2 = reinterpret_cast<const ulonglong2*>(b);
    ulonglong2* r2 = reinterpret_cast<ulonglong2*>(r);
    const uint64_t chunk = (uint64_t)V * blockDim.x;
    for (uint64_t c = (uint64_t)blockIdx.x * chunk + threadIdx.x; c < nv; c += (uint64_t)gridDim.x * chunk) {
        ulonglong2 x[V], y[V];
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const uint64_t i = c + (uint64_t)k * blockDim.x;
            x[k] = i < nv ? a2[i] : make_ulonglong2(0, 0);
            y[k] = (HAS_B && i < nv) ? b2[i] : make_ulonglong2(0, 0);
        }
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const uint64_t i = c + (uint64_t)k * blockDim.x;
            if (i < nv) r2[i] = make_ulonglong2(op(x[k].x, y[k].x), op(x[k].y, y[k].y));
        }
    }
    // the odd last element by thread 0 of block 0
    if (blockIdx.x == 0 && threadIdx.x == 0 && (n & 1)) r[n - 1] = op(a[n - 1], HAS_B ? b[n - 1] : 0);
}

template <class Op, bool HAS_B>
__global__ void __launch_bounds__(256) eltwise_scalar_kernel(uint64_t* r, const uint64_t* a, const uint64_t* b,
                                                             uint64_t n, const Op op)
{
    // 8-byte aligned path: a CTA takes chunks of kPer * blockDim elements;
    // element k of a chunk is handled by thread t at k * blockDim + t (every
    // warp access 256 contiguous bytes), all loaded before the first store.
    // Two elements per thread measured 1-19 % faster than one (reduce the
    // most) and than four or eight.  Each result depends on its own operands
    // only, so in-place calls hold.
    constexpr int kPer = 2;
    const uint64_t chunk = (uint64_t)kPer * blockDim.x;
    for (uint64_t base = (uint64_t)blockIdx.x * chunk; base < n; base += (uint64_t)gridDim.x * chunk) {
        const uint64_t i = base + threadIdx.x;
        if (base + chunk <= n) {
            uint64_t x[kPer], y[kPer];
#pragma unroll
            for (int k = 0; k < kPer; ++k) {
                x[k] = a[i + (uint64_t)k * blockDim.x];
                y[k] = HAS_B ? b[i + (uint64_t)k * blockDim.x] : 0;
            }
#pragma unroll
            for (int k = 0; k < kPer; ++k) r[i + (uint64_t)k * blockDim.x] = op(x[k], y[k]);
        } else {
            for (int k = 0; k < kPer; ++k) {
                const uint64_t j = i + (uint64_t)k * blockDim.x;
                if (j < n) r[j] = op(a[j], HAS_B ? b[j] : 0);
            }
        }
    }
}

__device__ __forceinline__ void ld_words4(uint64_t (&x)[4], const uint64_t* p)
{
    asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                 : "=l"(x[0]), "=l"(x[1]), "=l"(x[2]), "=l"(x[3])
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void st_words4(uint64_t* p, const uint64_t (&x)[4])
{
    asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(p), "l"(x[0]), "l"(x[1]), "l"(x[2]), "l"(x[3])
                 : "memory");
}

// MulMod and FMAMod.  The Barrett product (about 60 clocks of the multiply
// pipe per warp and element) and the loads have to overlap across warps, so
// what counts is warps in flight: one 32-byte vector per operand and thread,
// 40-48 registers, twice the CTAs, against four 16-byte ones at 64-80
// registers in eltwise_vec_kernel.  MulMod<4>, 59-bit modulus, calls one after
// the other: 2^20 elements 8.8 to 7.1 us, 2^22 21.1 to 18.9, 2^24 76.1 to 65.3;
// factor 1 7.1 to 6.5, 17.6 to 14.9, 64.5 to 63.2 (6.37 TB/s); FMAMod<4> 8.7 to
// 7.7, 23.0 to 21.0, 79.7 to 72.1; factor 1 7.3 to 6.6, 18.9 to 16.8, 65.2 to
// 63.9.  Operands that share their offset from a 32-byte boundary start with
// `head` single elements and end with a tail.
template <class Op, bool HAS_B>
__global__ void __launch_bounds__(256) eltwise_product_kernel(uint64_t* r, const uint64_t* a, const uint64_t* b,
                                                              uint64_t n, uint32_t head, const Op op)
{
    const uint64_t nv = (n - head) / 4;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nv;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t x[4], y[4] = {};
        ld_words4(x, a + head + 4 * i);
        if constexpr (HAS_B) ld_words4(y, b + head + 4 * i);
#pragma unroll
        for (int w = 0; w < 4; ++w) x[w] = op(x[w], y[w]);
        st_words4(r + head + 4 * i, x);
    }
    // the fewer than eight elements outside the vectors, by the first CTA
    if (blockIdx.x == 0) {
        const uint64_t t = threadIdx.x, i = t < head ? t : 4 * nv + t;
        if (i < n) r[i] = op(a[i], HAS_B ? b[i] : 0);
    }
}

template <class Op, bool HAS_B>
static cudaError_t run(uint64_t* r, const uint64_t* a, const uint64_t* b, uint64_t n, const Op& op, cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    const int threads = 256;
    const uintptr_t align = reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(a) |
                            (HAS_B ? reinterpret_cast<uintptr_t>(b) : 0);
    if constexpr (Op::kProduct) {
        const uintptr_t at = reinterpret_cast<uintptr_t>(r);
        const uintptr_t differ = (at ^ reinterpret_cast<uintptr_t>(a)) |
                                 (HAS_B ? at ^ reinterpret_cast<uintptr_t>(b) : 0);
        const uint64_t head = (32 - at % 32) % 32 / 8;
        // A head is a second, dependent round of loads in the first CTA: small
        // calls with one take the kernels below (device us: 8-byte aligned
        // operands, 2^16 elements 1.81 there and 2.32 here, 2^18.5 2.85 and 3.09,
        // 2^19 3.52 and 3.56, 2^20 5.53 and 5.16; 16-byte aligned ones 2^8 1.82
        // and 2.14, 2^10 2.27 and 2.35, 2^12 2.84 and 2.34).
        const uint64_t least = head == 0 ? 0 : ((at & 15) ? 1u << 19 : 1u << 11);
        if ((differ & 31) == 0 && (at & 7) == 0 && n >= least) {
            uint64_t blocks = ((n - head) / 4 + threads - 1) / threads;
            const uint64_t cap = (uint64_t)sm_count() * 16;
            if (blocks > cap) blocks = cap;
            if (blocks == 0) blocks = 1;
            count_launch();
            ProfScope prof(s, "eltwise_%s", Op::kName);
            eltwise_product_kernel<Op, HAS_B><<<(unsigned)blocks, threads, 0, s>>>(r, a, b, n, (uint32_t)head, op);
            return cudaGetLastError();
        }
    }
    const bool vec = (align & 15) == 0;
    const uint64_t work = vec ? (n >> 3) : ((n + 1) >> 1);  // elements per thread per chunk: 8 (vector), 2
    uint64_t blocks = (work + threads - 1) / threads;
    const uint64_t cap = (uint64_t)sm_count() * 8;  // 8 resident CTAs of 256 threads per SM
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    count_launch();
    ProfScope prof(s, "eltwise_%s%s", Op::kName, vec ? "" : "_unaligned");
    if (vec)
        eltwise_vec_kernel<Op, HAS_B><<<(unsigned)blocks, threads, 0, s>>>(r, a, b, n, op);
    else
        eltwise_scalar_kernel<Op, HAS_B><<<(unsigned)blocks, threads, 0, s>>>(r, a, b, n, op);
    return cudaGetLastError();
}

// ------------------------------------------------------------- launchers

static inline uint64_t bit_width(uint64_t x) { return x ? 64 - __builtin_clzll(x) : 0; }

void barrett_params(uint64_t q, uint64_t* mu, uint32_t* shift)
{
    const uint64_t k = bit_width(q);
    const unsigned __int128 num = (unsigned __int128)((uint64_t)1 << (k - 2)) << 64;
    *mu = (uint64_t)(num / q);
    *shift = (uint32_t)(k - 2);
}

cudaError_t eltwise_add(uint64_t* r, const uint64_t* a, const uint64_t* b, uint64_t n, uint64_t q, cudaStream_t s)
{
    return run<OpAddVV, true>(r, a, b, n, OpAddVV{q}, s);
}
cudaError_t eltwise_add_scalar(uint64_t* r, const uint64_t* a, uint64_t b, uint64_t n, uint64_t q, cudaStream_t s)
{
    return run<OpAddVS, false>(r, a, nullptr, n, OpAddVS{q, b}, s);
}
cudaError_t eltwise_sub(uint64_t* r, const uint64_t* a, const uint64_t* b, uint64_t n, uint64_t q, cudaStream_t s)
{
    return run<OpSubVV, true>(r, a, b, n, OpSubVV{q}, s);
}
cudaError_t eltwise_sub_scalar(uint64_t* r, const uint64_t* a, uint64_t b, uint64_t n, uint64_t q, cudaStream_t s)
{
    return run<OpSubVS, false>(r, a, nullptr, n, OpSubVS{q, b}, s);
}

cudaError_t eltwise_mul(uint64_t* r, const uint64_t* a, const uint64_t* b, uint64_t n, uint64_t q, uint64_t f,
                        cudaStream_t s)
{
    uint64_t mu;
    uint32_t sh;
    barrett_params(q, &mu, &sh);
    switch (f) {
    case 1: return run<OpMul<1>, true>(r, a, b, n, OpMul<1>{q, mu, sh}, s);
    case 2: return run<OpMul<2>, true>(r, a, b, n, OpMul<2>{q, mu, sh}, s);
    case 4: return run<OpMul<4>, true>(r, a, b, n, OpMul<4>{q, mu, sh}, s);
    default: return cudaSuccess;  // unsupported factor: no-op, eltwise-mul-mod.cpp:83-93
    }
}

static uint64_t host_reduce_input(uint64_t x, uint64_t q, uint64_t f)
{
    if (f == 8 && x >= 4 * q) x -= 4 * q;
    if (f >= 4 && x >= 2 * q) x -= 2 * q;
    if (f >= 2 && x >= q) x -= q;
    return x;
}

template <int F>
static cudaError_t fma_f(uint64_t* r, const uint64_t* a, uint64_t sc, const uint64_t* c, uint64_t n, uint64_t q,
                         uint64_t mu, uint32_t sh, cudaStream_t s)
{
    const uint64_t sr = host_reduce_input(sc, q, F);  // eltwise-fma-mod.cpp:33
    if (c) return run<OpFma<F, true>, true>(r, a, c, n, OpFma<F, true>{q, mu, sr, sh}, s);
    return run<OpFma<F, false>, false>(r, a, nullptr, n, OpFma<F, false>{q, mu, sr, sh}, s);
}

cudaError_t eltwise_fma(uint64_t* r, const uint64_t* a, uint64_t sc, const uint64_t* c, uint64_t n, uint64_t q,
                        uint64_t f, cudaStream_t s)
{
    uint64_t mu;
    uint32_t sh;
    barrett_params(q, &mu, &sh);
    switch (f) {
    case 1: return fma_f<1>(r, a, sc, c, n, q, mu, sh, s);
    case 2: return fma_f<2>(r, a, sc, c, n, q, mu, sh, s);
    case 4: return fma_f<4>(r, a, sc, c, n, q, mu, sh, s);
    case 8: return fma_f<8>(r, a, sc, c, n, q, mu, sh, s);
    default: return cudaSuccess;  // eltwise-fma-mod.cpp:98-111
    }
}

cudaError_t eltwise_reduce(uint64_t* r, const uint64_t* a, uint64_t n, uint64_t q, uint64_t in_f, uint64_t out_f,
                           cudaStream_t s)
{
    uint64_t mu = 0;
    uint32_t sh = 0;
    // Branch order of EltwiseReduceModNative (eltwise-reduce-mod.cpp:35-127).
    if (in_f == 1 || (out_f == 2 && in_f <= 2)) {
        if (r == a) return cudaSuccess;
        return run<OpReduce<0>, false>(r, a, nullptr, n, OpReduce<0>{q, 0, 0}, s);
    }
    if (in_f == 2 && out_f == 1) return run<OpReduce<1>, false>(r, a, nullptr, n, OpReduce<1>{q, 0, 0}, s);
    if (in_f == 4 && out_f == 1) return run<OpReduce<2>, false>(r, a, nullptr, n, OpReduce<2>{q, 0, 0}, s);
    if (in_f == 4 && out_f == 2) return run<OpReduce<3>, false>(r, a, nullptr, n, OpReduce<3>{q, 0, 0}, s);
    if (in_f == q) {
        barrett_params(q, &mu, &sh);
        return run<OpReduce<4>, false>(r, a, nullptr, n, OpReduce<4>{q, mu, sh}, s);
    }
    return cudaSuccess;  // unmatched pair writes nothing
}

// ------------------------------------------------------ fused tensor product

struct ModConst {
    uint64_t q, mu;
    uint32_t shift, fp;  // fp: q < 2^50, the FP64 form
    double fq, fqi;
};
struct TensorArgs {
    uint64_t *r0, *r1, *r2;
    const uint64_t *c0, *c1, *d0, *d1;
    uint64_t n, count;
    uint32_t nmod, factor;
    ModConst m[kMaxInlineMods];
};

// Per element of limb i (modulus m[i % nmod]):
//   r0 = Mul(c0,d0); r1 = Add(Mul(c0,d1), Mul(c1,d0)); r2 = Mul(c1,d1)
// with EltwiseMulMod<F> / EltwiseAddMod semantics (canonical results, so the
// middle term's evaluation order is free); the trailing EltwiseReduceMod(4,1)
// is the identity on these canonical values.
//
// HBM-bound (56 bytes per element) while the products keep up: three Barrett
// products are about 180 clocks of the multiply pipe per warp and element, of
// the 300 or so that its bytes take.  Moduli below 2^50 take about 40 FP64
// instructions of two clocks instead.  64 pairs x 16 limbs (40-55 bits) of
// N = 2^15: factor 1 305 to 285 us (6.6 TB/s), factor 4 360 to 288.  Calls
// without such moduli run a kernel without that form (59 bits, 1024 limbs of
// N = 2^12: factor 1 48.8 us with it, 41.0 without).
template <int F>
__device__ __forceinline__ void tensor_fp(uint64_t c0, uint64_t c1, uint64_t d0, uint64_t d1, uint64_t& r0,
                                          uint64_t& r1, uint64_t& r2, double q, double qi)
{
    // factor 1: within q; else within 2q, and the first factors brought to q/2
    const double off = F == 1 ? kFp2p52 : __fma_rn(2.0, q, kFp2p52);
    double x0 = fp_from_u64(c0, off), x1 = fp_from_u64(c1, off);
    const double y0 = fp_from_u64(d0, off), y1 = fp_from_u64(d1, off);
    if constexpr (F != 1) {
        x0 = fp_reduce(x0, q, qi);
        x1 = fp_reduce(x1, q, qi);
    }
    const double p0 = fp_mulmod(x0, y0, q, qi), p2 = fp_mulmod(x1, y1, q, qi);
    const double p1 = fp_mulmod(fp_reduce(__dadd_rn(x0, x1), q, qi), __dadd_rn(y0, y1), q, qi);
    r0 = fp_canon(p0, q);
    r2 = fp_canon(p2, q);
    r1 = fp_canon(fp_reduce(__dadd_rn(__dadd_rn(p1, -p0), -p2), q, qi), q);
}

template <int F, bool FP>
__global__ void __launch_bounds__(256) tensor_product_kernel(const __grid_constant__ TensorArgs a)
{
    // grid: x = chunks of one limb, y = limb.  Two elements per thread step.
    const uint64_t limb = blockIdx.y;
    const ModConst& mc = a.m[limb % a.nmod];
    const uint64_t q = mc.q;
    const OpMul<1> mul{q, mc.mu, mc.shift};  // on inputs already reduced to [0, q)
    const OpAddVV add{q};
    const OpSubVV sub{q};
    const uint64_t off = limb * a.n;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * 2;
    // Every output is a canonical residue, so the middle term may be formed
    // as (c0 + c1)(d0 + d1) - c0 d0 - c1 d1: three Barrett products per
    // coefficient instead of four, the same bits.
    auto three = [&](uint64_t c0, uint64_t c1, uint64_t d0, uint64_t d1, uint64_t& r0, uint64_t& r1,
                     uint64_t& r2) {
        c0 = reduce_input<F>(c0, q);
        c1 = reduce_input<F>(c1, q);
        d0 = reduce_input<F>(d0, q);
        d1 = reduce_input<F>(d1, q);
        r0 = mul(c0, d0);
        r2 = mul(c1, d1);
        r1 = sub(sub(mul(add(c0, c1), add(d0, d1)), r0), r2);
    };
    for (uint64_t e = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * 2; e < a.n; e += stride) {
        const ulonglong2 x0 = *reinterpret_cast<const ulonglong2*>(a.c0 + off + e);
        const ulonglong2 x1 = *reinterpret_cast<const ulonglong2*>(a.c1 + off + e);
        const ulonglong2 y0 = *reinterpret_cast<const ulonglong2*>(a.d0 + off + e);
        const ulonglong2 y1 = *reinterpret_cast<const ulonglong2*>(a.d1 + off + e);
        uint64_t r[2][3];
        if (FP && mc.fp) {
            tensor_fp<F>(x0.x, x1.x, y0.x, y1.x, r[0][0], r[0][1], r[0][2], mc.fq, mc.fqi);
            tensor_fp<F>(x0.y, x1.y, y0.y, y1.y, r[1][0], r[1][1], r[1][2], mc.fq, mc.fqi);
        } else {
            three(x0.x, x1.x, y0.x, y1.x, r[0][0], r[0][1], r[0][2]);
            three(x0.y, x1.y, y0.y, y1.y, r[1][0], r[1][1], r[1][2]);
        }
        const ulonglong2 o0 = make_ulonglong2(r[0][0], r[1][0]);
        const ulonglong2 o1 = make_ulonglong2(r[0][1], r[1][1]);
        const ulonglong2 o2 = make_ulonglong2(r[0][2], r[1][2]);
        *reinterpret_cast<ulonglong2*>(a.r0 + off + e) = o0;
        *reinterpret_cast<ulonglong2*>(a.r1 + off + e) = o1;
        *reinterpret_cast<ulonglong2*>(a.r2 + off + e) = o2;
    }
}

cudaError_t tensor_product(uint64_t* r0, uint64_t* r1, uint64_t* r2, const uint64_t* c0, const uint64_t* c1,
                           const uint64_t* d0, const uint64_t* d1, uint64_t n, uint64_t count, const uint64_t* moduli,
                           uint64_t nmod, uint64_t factor, cudaStream_t s)
{
    TensorArgs a{};
    a.r0 = r0; a.r1 = r1; a.r2 = r2;
    a.c0 = c0; a.c1 = c1; a.d0 = d0; a.d1 = d1;
    a.n = n; a.count = count;
    a.nmod = (uint32_t)nmod;
    a.factor = (uint32_t)factor;
    for (uint64_t i = 0; i < nmod; ++i) {
        a.m[i].q = moduli[i];
        barrett_params(moduli[i], &a.m[i].mu, &a.m[i].shift);
        a.m[i].fp = moduli[i] < kFpModulusEnd;
        a.m[i].fq = (double)moduli[i];
        a.m[i].fqi = 1.0 / a.m[i].fq;
    }
    bool fp = false;
    for (uint64_t i = 0; i < nmod; ++i) fp |= a.m[i].fp != 0;
    if (n == 0 || count == 0) return cudaSuccess;
    const int threads = 256;
    uint64_t bx = (n / 2 + threads - 1) / threads;
    // CTAs per SM in total, at least one per limb: 64 with FP64 moduli (8: 305
    // us, 64: 293, one chunk per CTA: 326, on the shape above); 16 without, in
    // a power of two of CTAs per limb, so that they share its chunks evenly
    // (59 bits, against 8: 32 limbs of N = 2^15 12.0 to 10.7 us, 64 of 2^17 83.5
    // to 78.8; 3 CTAs for the 8 chunks of 1024 limbs of 2^12 41.0 to 42.7, 2 41.0).
    uint64_t want = ((uint64_t)sm_count() * (fp ? 64 : 16) + count - 1) / count;
    if (want < 1) want = 1;
    if (!fp)
        while (want & (want - 1)) want &= want - 1;
    if (bx > want) bx = want;
    const dim3 grid((unsigned)bx, (unsigned)count);
    count_launch();
    ProfScope prof(s, "tensor_product f=%d", (int)factor);
    switch (factor) {
    case 1: (fp ? tensor_product_kernel<1, true> : tensor_product_kernel<1, false>)<<<grid, threads, 0, s>>>(a); break;
    case 2: (fp ? tensor_product_kernel<2, true> : tensor_product_kernel<2, false>)<<<grid, threads, 0, s>>>(a); break;
    case 4: (fp ? tensor_product_kernel<4, true> : tensor_product_kernel<4, false>)<<<grid, threads, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace axhel_impl
