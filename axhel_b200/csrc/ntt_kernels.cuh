// NTT pass kernels for sm_100a.
//
// A transform of N = 2^logn points is split into passes; a pass runs the
// reference's radix-2 stages [s0, s0 + LG) on "groups" of G = 2^LG elements
// that only interact with each other inside those stages:
//
//   element r of group (blk, col) sits at  p = blk*G*S + r*S + col
//
// with stride S = 2^(logn - s0 - LG) for the forward (Cooley-Tukey, large gaps
// first) and S = 2^s0 for the inverse (Gentleman-Sande, small gaps first).
// A CTA takes TG consecutive groups (a "tile"): TG adjacent columns of one
// block when S > 1, or TG adjacent contiguous blocks when S == 1.
//
// Each thread holds R = 2^LR elements of one group in registers and applies
// LR consecutive stages to them per round.  The first round loads straight
// from global memory and the last round stores straight back; shared memory
// (XOR-swizzled, bank-conflict free) is used only to exchange elements between rounds,
// with one barrier per exchange.  Global accesses are coalesced: in strided
// tiles consecutive lanes take consecutive columns; in contiguous tiles a
// round whose register bits are the low bits reads R consecutive words per
// thread as 32- or 16-byte vectors, and the other rounds read runs of 2^lo words.
//
// The butterflies are the reference's (ForwardButterflyNative /
// InverseButterflyNative, axhel/ntt/ntt-internal.hpp:20-49, and the final
// inverse stage of axhel/ntt/ntt-native.cpp:126-141) on the same element
// pairs with the same twiddles in the same stage order: operation for
// operation where the output is lazy, on other representatives of the same
// residues where it is canonical (the modes below), so outputs are
// bit-identical, lazy ranges included.  Twiddle indices:
//   forward stage t, position p : fwd[2^t + (p >> (logn - t))]      (ntt-native.cpp:39)
//   inverse stage s, position p : inv[1 + N - N/2^s + (p >> (s+1))]  (ntt-native.cpp:84, the
//                                 sequential root_index over the blocks of each stage)
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

#include "fp_layout.cuh"
#include "internal.h"
#include "modarith.cuh"

namespace axhel_impl {

using namespace axhel_dev;

// Threads per CTA allowed for a register depth: 32 elements per thread need
// more than the 128 registers a 512-thread launch bound leaves.
constexpr int max_threads(int LR) { return LR >= 5 ? 256 : 512; }

// Machine registers of the kernels that hold several arithmetics and two
// transforms or two limbs per thread: left alone the compiler spreads them
// over 100-128.  80 lets three CTAs of 256 threads share an SM (80, 96 and
// 128 measured on 768 limbs of N = 2^16: chain pass 657 / 750 / 675 us,
// product pass 684 / 666 / 701 us).
constexpr int kPairRegs = 80;
constexpr int chain_regs(int LR) { return LR >= 5 ? 255 : (LR == 4 ? 128 : 80); }
constexpr int product_regs(int P) { return P == 2 ? 96 : 80; }

template <int LG, int LR>
constexpr int num_rounds()
{
    return (LG + LR - 1) / LR;
}

// Lowest in-group bit held in registers during round RD.  Forward rounds walk
// the bits from the top, inverse rounds from the bottom; a short final round
// re-covers already processed bits so every round holds LR bits.
template <bool INV, int LG, int LR, int RD>
constexpr int round_lo()
{
    if constexpr (INV) {
        return (RD * LR < LG - LR) ? RD * LR : LG - LR;
    } else {
        return (LG - (RD + 1) * LR > 0) ? LG - (RD + 1) * LR : 0;
    }
}

// XOR swizzle of the in-group index for register depth LR: the low 4 bits
// (the 8-byte bank pair among 16) are flipped by index bits LR..LR+3.  In a
// round whose register bits start at lo < 4, the 16 lanes of a half-warp vary
// in index bits [0, lo) and [lo + LR, LR + 4); the shift by LR lands the
// latter on [lo, 4), so every round's access hits 16 distinct bank pairs.
// (A bijection: each flipped bit is flipped by bits above it.)
template <int LR>
__host__ __device__ constexpr uint32_t swz(uint32_t r)
{
    return r ^ ((r >> LR) & 15u);
}

// Shared-memory slot of in-group index r: groups are stored unpadded, G words
// each; `hmask` (per thread, below) XORs the group's varying bits into the
// bank pairs the element bits leave free, so half-warps that span several
// groups stay conflict-free too.
//
// The swizzle is linear, so the slot of r | c (c the register bits, zero in r)
// is slot(r) with its bank bits flipped by a constant, plus a constant: one
// instruction and an immediate offset per access.
template <int LG, int LR>
__device__ __forceinline__ uint32_t slot(uint32_t r, uint32_t hmask)
{
    return (LG < 4 ? r : swz<LR>(r)) ^ hmask;
}
// Byte offset of slot(r | c, hmask) from slot8 = 8 slot(r, hmask).
template <int LG, int LR>
__device__ __forceinline__ uint32_t slot8_at(uint32_t slot8, uint32_t c)
{
    if constexpr (LG < 4) return slot8 + (c << 3);
    return (slot8 ^ ((swz<LR>(c) & 15u) << 3)) + ((swz<LR>(c) & ~15u) << 3);
}

// Group bits of a half-warp's lanes sit above the element bits: strided tiles
// put the group first in the lane index (lgtg bits), contiguous tiles the
// thread-in-group first (LG - LR bits).
template <int LG, int LR>
__device__ __forceinline__ uint32_t group_mask(bool strided, uint32_t lgtg, uint32_t gi)
{
    const uint32_t nk = strided ? (lgtg >= 4 ? 0u : 4u - lgtg) : ((LG - LR) >= 4 ? 4u : (uint32_t)(LG - LR));
    return (gi << nk) & 15u;
}

// The mask with the group's place in the tile: slots count from the tile's
// first word.
template <int LG, int LR>
__device__ __forceinline__ uint32_t group_slot(bool strided, uint32_t lgtg, uint32_t gi)
{
    return (gi << LG) | (LG < 4 ? 0u : group_mask<LG, LR>(strided, lgtg, gi));
}

// Per-CTA tile geometry.
struct Tile {
    uint32_t g0;    // first group of the tile within the limb
    uint32_t base;  // word offset (in the limb) of element (gi = 0, r = 0)
    uint32_t lgS;   // log2 group stride in words
    uint32_t lgtg;  // log2 groups per tile
    bool strided;   // S > 1
};

// Tile `tile_in_limb` of a limb for a pass with group stride 2^lgS and
// 2^lgtg groups per tile.
template <int LG>
__device__ __forceinline__ Tile make_tile(uint32_t lgS, uint32_t lgtg, uint64_t tile_in_limb, bool strided)
{
    Tile t;
    t.g0 = (uint32_t)tile_in_limb << lgtg;
    t.lgS = lgS;
    t.lgtg = lgtg;
    t.strided = strided;
    if (t.strided) {
        const uint32_t blk = t.g0 >> lgS, col = t.g0 & ((1u << lgS) - 1);
        t.base = (blk << (LG + lgS)) + col;
    } else {
        t.base = t.g0 << LG;
    }
    return t;
}

template <int LG>
__device__ __forceinline__ Tile make_tile(uint32_t lgS, uint32_t lgtg, uint64_t tile_in_limb)
{
    return make_tile<LG>(lgS, lgtg, tile_in_limb, lgS != 0);
}

// Which tiles a kernel is compiled for: strided columns, contiguous rows, or
// either.  One kind alone is half the code: fewer registers, and a launch of
// a few limbs, which runs through its code once, fetches less of it.
enum TileShape : int { kAnyTiles = 0, kColumnTiles = 1, kRowTiles = 2 };

template <int LG>
__device__ __forceinline__ uint32_t tile_blk(const Tile& t, uint32_t gi)
{
    return t.strided ? (t.g0 >> t.lgS) : (t.g0 + gi);
}

// Thread -> (group in tile, thread in group).  Column-fastest when strided so
// a warp touches consecutive columns; thread-in-group-fastest otherwise.
template <int LG, int LR>
__device__ __forceinline__ void thread_role(const Tile& t, uint32_t& gi, uint32_t& k)
{
    constexpr uint32_t KT = 1u << (LG - LR);
    const uint32_t tid = threadIdx.x;
    if (t.strided) {
        gi = tid & ((1u << t.lgtg) - 1);
        k = tid >> t.lgtg;
    } else {
        gi = tid / KT;
        k = tid % KT;
    }
}

// Highest thread-in-group bit (k) whose in-group bit changes between rounds
// RD-1 and RD (-1 if none).  Element r sits in thread k(r) = r's bits below
// the register window, then those above it shifted down by LR; bits move
// between k and the registers, or between k positions, only up to here.
template <bool INV, int LG, int LR, int RD>
constexpr int exchange_max_pos()
{
    constexpr int lp = round_lo<INV, LG, LR, RD - 1>(), ln = round_lo<INV, LG, LR, RD>();
    int m = -1;
    for (int b = 0; b < LG; ++b) {
        const bool rp = b >= lp && b < lp + LR, rn = b >= ln && b < ln + LR;
        const int pp = rp ? -1 : (b < lp ? b : b - LR), pn = rn ? -1 : (b < ln ? b : b - LR);
        if (pp != pn) m = (pp > m ? pp : m) > pn ? (pp > m ? pp : m) : pn;
    }
    return m;
}

// limb mod n, the limb's modulus context.  Limb indexes below 2^32 (every
// real batch) take the 32-bit division, a fraction of the 64-bit one's
// instructions.
__device__ __forceinline__ uint32_t limb_mod(uint64_t limb, uint32_t n)
{
    return (limb >> 32) == 0 ? (uint32_t)limb % n : (uint32_t)(limb % n);
}

// Lane shift of k in the thread index: 0 for contiguous tiles (thread =
// group * threads-per-group + k), log2 groups per tile for strided ones
// (thread = group + k * groups); 32 for CTAs under one warp, which always
// synchronize the whole CTA.
__device__ __forceinline__ uint32_t lane_shift(bool strided, uint32_t lgtg)
{
    return blockDim.x >= 32 ? (strided ? lgtg : 0u) : 32u;
}

// In-group index of register 0 for register bits [lo, lo + LR).
template <int LR>
__device__ __forceinline__ uint32_t round_base(uint32_t k, int lo)
{
    return ((k >> lo) << (lo + LR)) | (k & ((1u << lo) - 1));
}

// ------------------------------------------------------- global <-> registers

// Loads with CG = true bypass L1 (ld.global.cg): used when the data was
// written by other CTAs of the same launch (the persistent batch kernel).
template <bool CG>
__device__ __forceinline__ uint64_t ld64(const uint64_t* p)
{
    if constexpr (CG) return __ldcg(reinterpret_cast<const unsigned long long*>(p));
    return *p;
}
template <bool CG>
__device__ __forceinline__ ulonglong2 ld128(const ulonglong2* p)
{
    if constexpr (CG) return __ldcg(p);
    return *p;
}

// Widest vector access the alignment of a limb's addresses allows: 32, 16 or
// 8 bytes.  Threads that hold 8 or 16 consecutive words are 64 or 128 bytes
// apart, and each request costs the L1 a wavefront per line it touches: 32-byte
// accesses halve them.
enum VecAlign : int { kVec8 = 0, kVec16 = 1, kVec32 = 2 };
__device__ __forceinline__ int vec_align(uintptr_t addrs)
{
    return (addrs & 31) == 0 ? kVec32 : ((addrs & 15) == 0 ? kVec16 : kVec8);
}

// Word `off / 8` of a limb: 32-bit byte offsets (a limb is at most 2^20 bytes)
// on the limb's address, so an access costs one 32-bit addition.
__device__ __forceinline__ const uint64_t* at_bytes(const uint64_t* limb, uint32_t off)
{
    return reinterpret_cast<const uint64_t*>(reinterpret_cast<const char*>(limb) + off);
}
__device__ __forceinline__ uint64_t* at_bytes(uint64_t* limb, uint32_t off)
{
    return reinterpret_cast<uint64_t*>(reinterpret_cast<char*>(limb) + off);
}

template <int LG, int LR, int LO, bool CG = false>
__device__ __forceinline__ void load_global(uint64_t (&v)[1 << LR], const uint64_t* __restrict__ limb_src,
                                            const Tile& t, uint32_t gi, uint32_t rb, int vec_ok)
{
    constexpr int R = 1 << LR;
    if (t.strided) {
        // (uniform offsets on the thread's address)
        const uint64_t* p = limb_src + (t.base + gi + (rb << t.lgS));
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = ld64<CG>(p + ((uint64_t)i << (LO + t.lgS)));
    } else if (LO == 0 && LR >= 3 && !CG && vec_ok == kVec32) {
        const uint32_t off = (t.base + (gi << LG) + rb) << 3;
#pragma unroll
        for (int i = 0; i < R; i += 4)
            asm volatile("ld.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                         : "=l"(v[i]), "=l"(v[i + 1]), "=l"(v[i + 2]), "=l"(v[i + 3])
                         : "l"(at_bytes(limb_src, off) + i)
                         : "memory");
    } else if (LO == 0 && vec_ok) {
        const uint32_t off = (t.base + (gi << LG) + rb) << 3;
#pragma unroll
        for (int i = 0; i < R / 2; ++i) {
            const ulonglong2 w = ld128<CG>(reinterpret_cast<const ulonglong2*>(at_bytes(limb_src, off)) + i);
            v[2 * i] = w.x;
            v[2 * i + 1] = w.y;
        }
    } else {
        const uint32_t off = (t.base + (gi << LG) + rb) << 3;
#pragma unroll
        for (int i = 0; i < R; ++i) v[i] = ld64<CG>(at_bytes(limb_src, off) + (i << LO));
    }
}

template <int LG, int LR, int LO>
__device__ __forceinline__ void store_global(const uint64_t (&v)[1 << LR], uint64_t* __restrict__ limb_dst,
                                             const Tile& t, uint32_t gi, uint32_t rb, int vec_ok)
{
    constexpr int R = 1 << LR;
    if (t.strided) {
        uint64_t* p = limb_dst + (t.base + gi + (rb << t.lgS));
#pragma unroll
        for (int i = 0; i < R; ++i) p[(uint64_t)i << (LO + t.lgS)] = v[i];
    } else if (LO == 0 && LR >= 3 && vec_ok == kVec32) {
        const uint32_t off = (t.base + (gi << LG) + rb) << 3;
#pragma unroll
        for (int i = 0; i < R; i += 4)
            asm volatile("st.global.v4.b64 [%0], {%1, %2, %3, %4};" ::"l"(at_bytes(limb_dst, off) + i), "l"(v[i]),
                         "l"(v[i + 1]), "l"(v[i + 2]), "l"(v[i + 3])
                         : "memory");
    } else if (LO == 0 && vec_ok) {
        const uint32_t off = (t.base + (gi << LG) + rb) << 3;
#pragma unroll
        for (int i = 0; i < R / 2; ++i)
            reinterpret_cast<ulonglong2*>(at_bytes(limb_dst, off))[i] = make_ulonglong2(v[2 * i], v[2 * i + 1]);
    } else {
        const uint32_t off = (t.base + (gi << LG) + rb) << 3;
#pragma unroll
        for (int i = 0; i < R; ++i) at_bytes(limb_dst, off)[i << LO] = v[i];
    }
}

// ------------------------------------------------------------------ stages

// Arithmetic of a transform's stages.  Registers and shared memory hold 64-bit
// words in every mode; the FP64 modes keep doubles in them.
//   kExact   the reference's butterflies, value for value (any q < 2^62)
//   kRelaxed integer residues below 32q (q < 2^59): shoup_relaxed
//   kFp      FP64 integers within 4q (q < 2^50): fp_mul
//   kFpLazy  the reference's forward butterflies on FP64 integers (q < 2^50)
// The relaxed modes serve transforms whose output is reduced to [0, q) at the
// end, where only the residues are visible; kExact and kFpLazy hold the
// reference's lazy values at every stage.
enum Arith : int { kExact = 0, kRelaxed = 1, kFp = 2, kFpLazy = 3 };

// A limb's constants for the stages.  Twiddles are read by 32-bit byte
// offsets on a table's address.
struct ModArith {
    const char* tw;   // {w, w'}, or w alone as a double
    const char* itw;  // kFpLazy: {w, w'} too
    const ModCtx* cx;
    uint32_t n;
    uint64_t q, q2;
    double fq, fqi;   // q, 1/q
    uint32_t lazy_hi; // kFpLazy: high word of the largest remainder that needs the exact quotient
    bool row;         // contiguous pass (group stride 1) with the FP64 tables' tail order
};

// The tables lie at fixed places behind the context header.
template <int MODE, bool INV>
__device__ __forceinline__ ModArith mod_arith(const ModCtx* cx, uint32_t n, bool row)
{
    constexpr bool FP = MODE == kFp || MODE == kFpLazy;
    ModArith a{};
    a.cx = cx;
    a.n = n;
    a.row = row && n >= kFpTailMinN;
    a.q = cx->q;
    a.q2 = cx->q2;
    const char* fwd = reinterpret_cast<const char*>(cx) + kCtxHeaderBytes;
    a.tw = fwd + (FP ? (INV ? 40u : 32u) : (INV ? 16u : 0u)) * n;
    if constexpr (FP) {
        a.itw = fwd;
        a.fq = cx->fq;
        a.fqi = cx->fqi;
        a.lazy_hi = cx->lazy_hi;
    }
    return a;
}

__device__ __forceinline__ ulonglong2 twiddle(const char* table, uint32_t idx)
{
    return __ldg(reinterpret_cast<const ulonglong2*>(table + (idx << 4)));
}

// The exact lazy product of kFpLazy for the operand y: MultiplyUIntModLazy
// on its integer value.
__device__ __forceinline__ double fp_exact_lazy(double y, const ulonglong2 w, uint64_t q)
{
    return fp_from_u64(shoup_lazy(fp_to_u64(y), w.x, w.y, q), kFp2p52);
}

// Twiddles m0, m0 + 1, .. of one stage whose table section starts at `nat`
// (m0 a multiple of how many the thread reads); b = the stage's in-group bit.
//
// In a contiguous pass the stages of in-group bits 2, 1, 0 take 1, 2 and 4
// twiddles for each 8 consecutive elements, so lanes reading them in natural
// order are 16 to 64 bytes apart and a request touches up to 16 lines: the
// L1's data pipe was 91 % busy on the forward 9-stage pass with it (72 us for
// 192 limbs of N = 2^16).  The FP64 tables therefore hold the 7N/8 entries of
// those stages (from `tail` on) for 32 neighbouring groups of 8 side by side,
// one entry of each after the other: fp_tail_pos.
//
// A stage's twiddles: the table and where entry m0 + j lies.  For the FP64
// modes the second word is w / q from the rounded 1/q (relative error 2^-52):
// one FP64 product for each twiddle, shared by its butterflies, instead of
// twice the bytes through the L1, which is what those modes wait for.
struct StageTw {
    const char* at;  // the entry of j = 0
    bool tail;
    template <int MODE>
    __device__ __forceinline__ ulonglong2 get(int j, int b, double fqi) const
    {
        if constexpr (MODE == kFp || MODE == kFpLazy) {
            const double* e = reinterpret_cast<const double*>(at);
            const double w = __ldg(b <= 2 && tail ? e + fp_tail_slot(b, j & ((1 << (2 - b)) - 1)) * kFpTailGroups +
                                                        (j >> (2 - b))
                                                  : e + j);
            return make_ulonglong2(as_u64(w), as_u64(__dmul_rn(w, fqi)));
        } else {
            return __ldg(reinterpret_cast<const ulonglong2*>(at) + j);
        }
    }
};

// `nat`: the stage's section in natural order, `tail`: the slots' part.
template <int MODE>
__device__ __forceinline__ StageTw stage_tw(const ModArith& a, uint32_t nat, uint32_t m0, int b, uint32_t tail)
{
    if constexpr (MODE == kFp || MODE == kFpLazy) {
        if (b <= 2 && a.row) return StageTw{a.tw + ((tail + fp_tail_pos(m0 >> (2 - b), 0)) << 3), true};
        return StageTw{a.tw + ((nat + m0) << 3), false};
    } else {
        return StageTw{a.tw + ((nat + m0) << 4), false};
    }
}

// Forward round RD on registers: stage bits hi-1 .. hi-nb of the in-group
// index (largest gap first); registers hold bits [lo, lo + LR).
//
// kRelaxed: the upper operand enters a round's first stage reduced below
// 16q and both outputs of a stage grow by less than 4q, so up to four stages
// stay below 32q.  kFp: likewise, from q/2 each of a round's three stages adds
// a product of at most q/2 + Y/8 for a multiplicand within Y; with Y = 2.8q at
// the round's start the values end within 2.8q again.
// kFpLazy: the lazy product t = y w - floor(y w' / 2^64) q equals the
// canonical remainder r, plus q when r 2^64 < y (w 2^64 mod q); as y < 4q
// that needs r < 4 q^2 / 2^64, which a random remainder meets with
// probability 4q / 2^64 (2^-12 at most), so a stage whose smallest remainder
// is that small recomputes those products with the integer formula.  A zero
// remainder needs none: y = 0 gives t = 0, and y = kq, k = 1..3, gives y w' =
// k (w 2^64 - (w 2^64 mod q)), whose quotient is kw - 1, so t = q.  (Zeros become
// such multiples in the first stage, x + t and x + 2q - t.  768 limbs of N = 2^16,
// 45 bits: 499 us whatever the values; with the integer formula for every zero
// remainder 480 for values without any and 884-948 for zeros, every second
// coefficient zero or multiples of q; with a second look at them after the check
// 478 and 590, but 2 % more for the wide moduli that share the kernel.  The
// reference's butterflies: 551.)
template <int MODE, int LG, int LR, int RD, int P>
__device__ __forceinline__ void fwd_stages(uint64_t (&v)[P][1 << LR], uint32_t rbase, uint32_t blk, uint32_t s0,
                                           const ModArith& a)
{
    constexpr int R = 1 << LR;
    constexpr int hi = LG - RD * LR;
    constexpr int nb = hi < LR ? hi : LR;
    constexpr int lo = round_lo<false, LG, LR, RD>();
#pragma unroll
    for (int bb = 0; bb < nb; ++bb) {
        const int b = hi - 1 - bb;  // in-group bit = butterfly span
        const int rb = b - lo;      // register bit
        const uint32_t t = s0 + (LG - 1 - b);
        // the twiddles of this stage are consecutive: rbase's register bits
        // are zero, so (rbase | j << (b+1)) >> (b+1) = (rbase >> (b+1)) + j
        const uint32_t m0 = (blk << (LG - 1 - b)) + (rbase >> (b + 1));
        const StageTw tw = stage_tw<MODE>(a, 1u << t, m0, b, a.n >> 3);
        if constexpr (MODE == kFpLazy) {
            double r[P][R / 2];
            uint32_t least = 0xffffffffu;  // high word of the least remainder but zero, less 1
#pragma unroll
            for (int j = 0; j < (R >> (rb + 1)); ++j) {
                const ulonglong2 w = tw.get<MODE>(j, b, a.fqi);
#pragma unroll
                for (int p = 0; p < P; ++p)
#pragma unroll
                    for (int l = 0; l < (1 << rb); ++l) {
                        const int k = (j << rb) | l, i1 = (j << (rb + 1)) | l | (1 << rb);
                        const double y = as_fp(v[p][i1]);
                        double x = fp_mul(y, as_fp(w.x), as_fp(w.y), a.fq);
                        // negative, or zero with y not (only zero has a zero high word)
                        if (__double2hiint(x) < min(__double2hiint(y), 1)) x = __dadd_rn(x, a.fq);
                        r[p][k] = x;
                        least = __viaddmin_u32((uint32_t)__double2hiint(x), 0xffffffffu, least);
                    }
            }
            if (least < a.lazy_hi) {
#pragma unroll
                for (int p = 0; p < P; ++p)
#pragma unroll
                    for (int k = 0; k < R / 2; ++k) {
                        const int j = k >> rb, i1 = (j << (rb + 1)) | (k & ((1 << rb) - 1)) | (1 << rb);
                        if ((uint32_t)__double2hiint(r[p][k]) - 1 < a.lazy_hi)
                            r[p][k] = fp_exact_lazy(as_fp(v[p][i1]), twiddle(a.itw, (1u << t) + m0 + j), a.q);
                    }
            }
            const double q2 = __dadd_rn(a.fq, a.fq);
#pragma unroll
            for (int p = 0; p < P; ++p)
#pragma unroll
                for (int k = 0; k < R / 2; ++k) {
                    const int i0 = ((k >> rb) << (rb + 1)) | (k & ((1 << rb) - 1));
                    double g = as_fp(v[p][i0]);
                    if (g >= q2) g = __dadd_rn(g, -q2);
                    v[p][i0] = as_u64(__dadd_rn(g, r[p][k]));
                    v[p][i0 | (1 << rb)] = as_u64(__dadd_rn(__dadd_rn(g, q2), -r[p][k]));
                }
        } else {
#pragma unroll
            for (int j = 0; j < (R >> (rb + 1)); ++j) {
                const ulonglong2 w = tw.get<MODE>(j, b, a.fqi);
#pragma unroll
                for (int p = 0; p < P; ++p)
#pragma unroll
                    for (int l = 0; l < (1 << rb); ++l) {
                        const int i0 = (j << (rb + 1)) | l;
                        uint64_t &x = v[p][i0], &y = v[p][i0 | (1 << rb)];
                        if constexpr (MODE == kExact) {
                            fwd_butterfly(x, y, w.x, w.y, a.q, a.q2);
                        } else if constexpr (MODE == kRelaxed) {
                            const uint64_t g = bb == 0 ? csub_lazy(x, a.q2 << 3) : x;
                            const uint64_t u = shoup_relaxed(y, w.x, w.y, a.q);
                            x = g + u;
                            y = g + (a.q2 << 1) - u;
                        } else {
                            const double u = fp_mul(as_fp(y), as_fp(w.x), as_fp(w.y), a.fq);
                            const double g = bb == 0 ? fp_reduce(as_fp(x), a.fq, a.fqi) : as_fp(x);
                            x = as_u64(__dadd_rn(g, u));
                            y = as_u64(__dadd_rn(g, -u));
                        }
                    }
            }
        }
    }
}

// kRelaxed: x < (bound)q brought below 4q by conditional subtracts.
__device__ __forceinline__ uint64_t relax_to_4q(uint64_t x, int bound, uint64_t q2)
{
    if (bound > 16) x = csub_lazy(x, q2 << 3);
    if (bound > 8) x = csub_lazy(x, q2 << 2);
    if (bound > 4) x = csub_lazy(x, q2 << 1);
    return x;
}

// Inverse round RD on registers: stage bits b0 .. b1-1 (smallest gap first).
// With `last` set the pass holds global stage logn-1, the N^-1 final stage.
//
// The relaxed modes track each register's bound at compile time.  kRelaxed
// (units of q): a round starts and ends below 4q, a sum is reduced when it
// passes 16q, products are below 4q.  kFp (units of q/4): a round starts and
// ends within 2q, a sum is reduced when it passes 2q, differences are within
// 4q and products within q (the final stage's, by quotients rounded once,
// within 3q/4).
template <int MODE, int LG, int LR, int RD, int P>
__device__ __forceinline__ void inv_stages(uint64_t (&v)[P][1 << LR], uint32_t rbase, uint32_t blk, uint32_t s0,
                                           const ModArith& a, bool last)
{
    constexpr int R = 1 << LR;
    constexpr int b0 = RD * LR;
    constexpr int b1 = (b0 + LR < LG) ? b0 + LR : LG;
    constexpr int lo = round_lo<true, LG, LR, RD>();
    int bnd[R];
#pragma unroll
    for (int i = 0; i < R; ++i) bnd[i] = MODE == kFp ? 8 : 4;
#pragma unroll
    for (int b = b0; b < b1; ++b) {
        const int rb = b - lo;
        if (b == LG - 1 && last) {
            const ModCtx* cx = a.cx;
            const uint64_t ninv = cx->ninv, ninv_q = cx->ninv_q, sr = cx->sroot, sr_q = cx->sroot_q;
#pragma unroll
            for (int p = 0; p < P; ++p) {
#pragma unroll
                for (int k = 0; k < R / 2; ++k) {
                    const int i0 = ((k >> rb) << (rb + 1)) | (k & ((1 << rb) - 1)), i1 = i0 | (1 << rb);
                    if constexpr (MODE == kExact) {
                        inv_final_butterfly(v[p][i0], v[p][i1], ninv, ninv_q, sr, sr_q, a.q, a.q2);
                    } else if constexpr (MODE == kRelaxed) {
                        const uint64_t x = v[p][i0], y = v[p][i1];
                        v[p][i0] = shoup_relaxed(x + y, ninv, ninv_q, a.q);
                        v[p][i1] = shoup_relaxed(x + a.q * bnd[i1] - y, sr, sr_q, a.q);
                    } else {
                        const double x = as_fp(v[p][i0]), y = as_fp(v[p][i1]);
                        v[p][i0] = as_u64(fp_mul(__dadd_rn(x, y), cx->fninv, cx->fninv_q, a.fq));
                        v[p][i1] = as_u64(fp_mul(__dadd_rn(x, -y), cx->fsroot, cx->fsroot_q, a.fq));
                    }
                }
            }
        } else {
            const uint32_t s = s0 + b;
            const uint32_t m0 = (blk << (LG - b - 1)) + (rbase >> (b + 1));
            const StageTw tw = stage_tw<MODE>(a, 1 + a.n - (a.n >> s), m0, b, 0);
#pragma unroll
            for (int j = 0; j < (R >> (rb + 1)); ++j) {
                const ulonglong2 w = tw.get<MODE>(j, b, a.fqi);
#pragma unroll
                for (int p = 0; p < P; ++p)
#pragma unroll
                    for (int l = 0; l < (1 << rb); ++l) {
                        const int i0 = (j << (rb + 1)) | l, i1 = i0 | (1 << rb);
                        uint64_t &x = v[p][i0], &y = v[p][i1];
                        if constexpr (MODE == kExact) {
                            inv_butterfly(x, y, w.x, w.y, a.q, a.q2);
                        } else if constexpr (MODE == kRelaxed) {
                            const uint64_t u = x, d = x + a.q * bnd[i1] - y;
                            x = u + y;
                            if (bnd[i0] + bnd[i1] > 16) x = csub_lazy(x, a.q2 << 3);
                            y = shoup_relaxed(d, w.x, w.y, a.q);
                        } else {
                            const double u = as_fp(x), d = __dadd_rn(u, -as_fp(y));
                            double g = __dadd_rn(u, as_fp(y));
                            if (bnd[i0] + bnd[i1] > 8) g = fp_reduce(g, a.fq, a.fqi);
                            x = as_u64(g);
                            y = as_u64(fp_mul(d, as_fp(w.x), as_fp(w.y), a.fq));
                        }
                    }
            }
#pragma unroll
            for (int k = 0; k < R / 2; ++k) {
                const int i0 = ((k >> rb) << (rb + 1)) | (k & ((1 << rb) - 1)), i1 = i0 | (1 << rb);
                bnd[i0] += bnd[i1];
                if (MODE == kRelaxed && bnd[i0] > 16) bnd[i0] = 16;
                if (MODE == kFp && bnd[i0] > 8) bnd[i0] = 3;
                bnd[i1] = 4;
            }
        }
    }
    if constexpr (MODE == kRelaxed) {
        // the final stage leaves every value below 4q; otherwise bring the
        // sums back (a pass's last round included: the next pass starts there)
        if (!(b1 == LG && last)) {
#pragma unroll
            for (int p = 0; p < P; ++p)
#pragma unroll
                for (int i = 0; i < R; ++i) v[p][i] = relax_to_4q(v[p][i], bnd[i], a.q2);
        }
    }
}

// Register exchange between rounds RD-1 and RD through shared memory.  Each
// thread writes back the slots it held and reads its next slots; the slot
// sets of one round are disjoint across threads, so one barrier suffices.
template <bool INV, int LG, int LR, int RD, int P>
__device__ __forceinline__ void exchange(uint64_t (&v)[P][1 << LR], uint64_t* smg, uint32_t k, uint32_t hmask,
                                         uint32_t lsh, uint32_t pstride)
{
    constexpr int R = 1 << LR;
    constexpr int lp = round_lo<INV, LG, LR, RD - 1>();
    constexpr int ln = round_lo<INV, LG, LR, RD>();
    constexpr int mp = exchange_max_pos<INV, LG, LR, RD>();
    char* sm = reinterpret_cast<char*>(smg);
    const uint32_t bp = slot<LG, LR>(round_base<LR>(k, lp), hmask) << 3;
    const uint32_t bn = slot<LG, LR>(round_base<LR>(k, ln), hmask) << 3;
#pragma unroll
    for (int i = 0; i < R; ++i) {
        uint64_t* at = reinterpret_cast<uint64_t*>(sm + slot8_at<LG, LR>(bp, (uint32_t)i << lp));
#pragma unroll
        for (int p = 0; p < P; ++p) at[p * pstride] = v[p][i];
    }
    // Every thread writes the slots it read at the previous exchange, so when
    // all changed k bits are lane bits (the inner stages) the elements only
    // move inside a warp and a warp barrier orders them.  (Uniform branch.)
    if (mp + (int)lsh < 5)
        __syncwarp();
    else
        __syncthreads();
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const uint64_t* at = reinterpret_cast<const uint64_t*>(sm + slot8_at<LG, LR>(bn, (uint32_t)i << ln));
#pragma unroll
        for (int p = 0; p < P; ++p) v[p][i] = at[p * pstride];
    }
}

// One limb per thread, as the cluster kernels hold it.
template <bool INV, int LG, int LR, int RD>
__device__ __forceinline__ void exchange(uint64_t (&v)[1 << LR], uint64_t* smg, uint32_t k, uint32_t hmask,
                                         uint32_t lsh)
{
    exchange<INV, LG, LR, RD, 1>(reinterpret_cast<uint64_t(&)[1][1 << LR]>(v), smg, k, hmask, lsh, 0);
}

// Rounds 1 .. NR-1 (round 0 runs on the freshly loaded registers).
template <int MODE, int LG, int LR, int P, int... RD>
__device__ __forceinline__ void fwd_rest(std::integer_sequence<int, RD...>, uint64_t (&v)[P][1 << LR], uint64_t* smg,
                                         uint32_t k, uint32_t hmask, uint32_t lsh, uint32_t pstride, uint32_t blk,
                                         uint32_t s0, const ModArith& a)
{
    ((exchange<false, LG, LR, RD + 1, P>(v, smg, k, hmask, lsh, pstride),
      fwd_stages<MODE, LG, LR, RD + 1, P>(v, round_base<LR>(k, round_lo<false, LG, LR, RD + 1>()), blk, s0, a)),
     ...);
}

template <int MODE, int LG, int LR, int P, int... RD>
__device__ __forceinline__ void inv_rest(std::integer_sequence<int, RD...>, uint64_t (&v)[P][1 << LR], uint64_t* smg,
                                         uint32_t k, uint32_t hmask, uint32_t lsh, uint32_t pstride, uint32_t blk,
                                         uint32_t s0, const ModArith& a, bool last)
{
    ((exchange<true, LG, LR, RD + 1, P>(v, smg, k, hmask, lsh, pstride),
      inv_stages<MODE, LG, LR, RD + 1, P>(v, round_base<LR>(k, round_lo<true, LG, LR, RD + 1>()), blk, s0, a, last)),
     ...);
}

// The rounds of a pass on P limbs of one modulus per thread (words pstride
// apart in shared memory); `row`: contiguous groups.
template <bool INV, int LG, int LR, int MODE, int P>
__device__ __forceinline__ void run_rounds(uint64_t (&v)[P][1 << LR], uint64_t* smg, uint32_t k, uint32_t hmask,
                                           uint32_t lsh, uint32_t pstride, uint32_t blk, uint32_t s0, uint32_t n,
                                           const ModCtx* cx, bool row, bool last)
{
    constexpr int NR = num_rounds<LG, LR>();
    const ModArith a = mod_arith<MODE, INV>(cx, n, row);
    if constexpr (INV) {
        inv_stages<MODE, LG, LR, 0, P>(v, round_base<LR>(k, round_lo<true, LG, LR, 0>()), blk, s0, a, last);
        inv_rest<MODE, LG, LR, P>(std::make_integer_sequence<int, NR - 1>{}, v, smg, k, hmask, lsh, pstride, blk, s0,
                                  a, last);
    } else {
        fwd_stages<MODE, LG, LR, 0, P>(v, round_base<LR>(k, round_lo<false, LG, LR, 0>()), blk, s0, a);
        fwd_rest<MODE, LG, LR, P>(std::make_integer_sequence<int, NR - 1>{}, v, smg, k, hmask, lsh, pstride, blk, s0,
                                  a);
    }
}

// The reference's rounds on one limb, as the cluster kernels hold it.
template <bool INV, int LG, int LR>
__device__ __forceinline__ void run_rounds(uint64_t (&v)[1 << LR], uint64_t* smg, uint32_t k, uint32_t hmask,
                                           uint32_t lsh, uint32_t blk, uint32_t s0, uint32_t n, const ModCtx* cx,
                                           bool last)
{
    run_rounds<INV, LG, LR, kExact, 1>(reinterpret_cast<uint64_t(&)[1][1 << LR]>(v), smg, k, hmask, lsh, 0, blk, s0,
                                       n, cx, false, last);
}

// Group sizes and register depth compiled with the relaxed modes: 8 registers
// per thread (16 would take 110-128 machine registers for the modes together).
constexpr bool relaxed_compiled(int lg, int lr) { return lr == 3 && lg >= 4 && (1 << (lg - lr)) <= max_threads(lr); }

// ------------------------------------------------------------------ kernels

// The registers as read from memory in the form the stages of MODE work on.
// The passes of a kFp transform hand each other doubles; its first pass
// reads integers below 4q, centred so that they start within 2q.
template <int MODE, int LR>
__device__ __forceinline__ void to_stages(uint64_t (&v)[1 << LR], bool first, const ModCtx* cx)
{
    if constexpr (MODE == kFp) {
        if (!first) return;
        const double off = __fma_rn(2.0, cx->fq, kFp2p52);
#pragma unroll
        for (int i = 0; i < (1 << LR); ++i) v[i] = as_u64(fp_from_u64(v[i], off));
    } else if constexpr (MODE == kFpLazy) {
#pragma unroll
        for (int i = 0; i < (1 << LR); ++i) v[i] = as_u64(fp_from_u64(v[i], kFp2p52));
    }
}

// The registers after a forward's last stage as the integers of its output.
template <int MODE, int LR>
__device__ __forceinline__ void fwd_output(uint64_t (&v)[1 << LR], bool norm, const ModCtx* cx)
{
    const uint64_t q = cx->q, q2 = cx->q2;
#pragma unroll
    for (int i = 0; i < (1 << LR); ++i) {
        if constexpr (MODE == kFp) {
            v[i] = fp_canon(fp_reduce(as_fp(v[i]), cx->fq, cx->fqi), cx->fq);
        } else if constexpr (MODE == kRelaxed) {
            v[i] = csub_lazy(csub_lazy(relax_to_4q(v[i], 32, q2), q2), q);
        } else {
            if constexpr (MODE == kFpLazy) v[i] = fp_to_u64(as_fp(v[i]));
            if (norm) v[i] = csub_lazy(csub_lazy(v[i], q2), q);
        }
    }
}

// The registers after the inverse's final stage as the integers of its output.
template <int MODE, int LR>
__device__ __forceinline__ void inv_output(uint64_t (&v)[1 << LR], bool norm, const ModCtx* cx)
{
    const uint64_t q = cx->q, q2 = cx->q2;
#pragma unroll
    for (int i = 0; i < (1 << LR); ++i) {
        if constexpr (MODE == kFp) v[i] = fp_canon(as_fp(v[i]), cx->fq);
        else if constexpr (MODE == kRelaxed) v[i] = csub_lazy(csub_lazy(v[i], q2), q);
        else if (norm) v[i] = csub_lazy(v[i], q);
    }
}

// Dyadic product of the registers (round with register bits at LO) with the
// multiplicand at the same positions: EltwiseMulModNative<4>
// (eltwise-mul-mod.cpp:40-60), both operands in [0, 4q), result in [0, q);
// the relaxed modes give a representative of it (kFp within 7q/8).
template <int MODE, int LG, int LR, int LO, bool CG>
__device__ __forceinline__ void mul_operand(uint64_t (&v)[1 << LR], const uint64_t* __restrict__ limb_m,
                                            const Tile& t, uint32_t gi, uint32_t k, const ModCtx* cx, int vec_ok,
                                            int bound)
{
    uint64_t m[1 << LR];
    load_global<LG, LR, LO, CG>(m, limb_m, t, gi, round_base<LR>(k, LO),
                                min(vec_ok, vec_align(reinterpret_cast<uintptr_t>(limb_m))));
    if constexpr (MODE == kFp) {
        const double q = cx->fq, qi = cx->fqi, off = __fma_rn(2.0, q, kFp2p52);
#pragma unroll
        for (int i = 0; i < (1 << LR); ++i)
            v[i] = as_u64(fp_mulmod(fp_reduce(as_fp(v[i]), q, qi), fp_from_u64(m[i], off), q, qi));
    } else {
        const uint64_t q = cx->q, mu = cx->mu;
        const uint32_t shift = cx->shift;
#pragma unroll
        for (int i = 0; i < (1 << LR); ++i) {
            const uint64_t x = MODE == kRelaxed ? relax_to_4q(v[i], bound, q << 1) : v[i];
            v[i] = barrett_mul(reduce_input<4>(x, q), reduce_input<4>(m[i], q), q, mu, shift);
        }
    }
}

// One tile of a pass: stages [s0, s0 + LG) of limb `limb`, or of P limbs of
// one modulus, `lstep` limbs apart.  `sm` holds P times 2^lgtg groups of 2^LG
// words; all threads of the CTA take part.  With MUL, flags kPreMul /
// kPostMul multiply by `operand` (MulMod<4>) after the load / before the
// store.
//
// P = 2: a twiddle read costs the L1's data pipe as much as four coalesced
// residues, and with one limb per thread twiddles were two thirds of its
// wavefronts (profiled at N = 2^16: 78-86 % of the pipe's cycles); two limbs
// of a modulus share every twiddle, its address and the barriers.
template <int MODE, bool INV, int LG, int LR, bool CG, bool MUL, int P, int SHAPE>
__device__ __forceinline__ void pass_tile_as(const uint64_t* src, uint64_t* dst, const ModCtx* cx, uint32_t logn,
                                             uint32_t s0, uint32_t lgtg, uint64_t limb, uint64_t lstep,
                                             uint64_t tile_in_limb, uint32_t flags, uint64_t* sm,
                                             const uint64_t* operand)
{
    constexpr int R = 1 << LR;
    constexpr int NR = num_rounds<LG, LR>();
    constexpr int LO_FIRST = round_lo<INV, LG, LR, 0>();
    constexpr int LO_LAST = round_lo<INV, LG, LR, NR - 1>();
    const uint32_t lgS = SHAPE == kRowTiles ? 0u : (INV ? s0 : (logn - s0 - LG));
    const Tile t = make_tile<LG>(lgS, lgtg, tile_in_limb, SHAPE == kColumnTiles || (SHAPE == kAnyTiles && lgS != 0));
    const uint32_t n = 1u << logn;
    const uint64_t* lsrc = src + (limb << logn);
    uint64_t* ldst = dst + (limb << logn);
    const uint64_t pstep = lstep << logn;
    const int vec_ok = vec_align(reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst));
    const bool last = (flags & kLastPass) != 0;

    uint32_t gi, k;
    thread_role<LG, LR>(t, gi, k);
    const uint32_t blk = tile_blk<LG>(t, gi);

    uint64_t v[P][R];
#pragma unroll
    for (int p = 0; p < P; ++p)
        load_global<LG, LR, LO_FIRST, CG>(v[p], lsrc + p * pstep, t, gi, round_base<LR>(k, LO_FIRST), vec_ok);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        to_stages<MODE, LR>(v[p], s0 == 0, cx);
        if constexpr (MODE == kExact) {
            if (flags & kPreCsub2q) {
#pragma unroll
                for (int i = 0; i < R; ++i) v[p][i] = csub_lazy(v[p][i], cx->q2);
            }
        }
        if constexpr (MUL && INV)
            if (flags & kPreMul)
                mul_operand<MODE, LG, LR, LO_FIRST, CG>(v[p], operand + (limb << logn) + p * pstep, t, gi, k, cx,
                                                        vec_ok, 4);
    }
    run_rounds<INV, LG, LR, MODE, P>(v, sm, k, group_slot<LG, LR>(t.strided, lgtg, gi),
                                     lane_shift(t.strided, lgtg), 1u << (LG + lgtg), blk, s0, n, cx, !t.strided, last);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        bool stored = false;
        if constexpr (MUL && !INV) {
            if (flags & kPostMul) {
                mul_operand<MODE, LG, LR, LO_LAST, CG>(v[p], operand + (limb << logn) + p * pstep, t, gi, k, cx,
                                                       vec_ok, 32);
                if constexpr (MODE == kFp) inv_output<MODE, LR>(v[p], true, cx);
                stored = true;
            }
        }
        // between passes kFp hands on doubles and kRelaxed values below 32q
        // (forward) / 4q (inverse); the others the reference's lazy integers
        if (!stored && (last || MODE == kFpLazy || MODE == kExact)) {
            const bool norm = (flags & kPostNorm) != 0;
            if constexpr (INV) inv_output<MODE, LR>(v[p], norm, cx);
            else fwd_output<MODE, LR>(v[p], norm, cx);
        }
        store_global<LG, LR, LO_LAST>(v[p], ldst + p * pstep, t, gi, round_base<LR>(k, LO_LAST), vec_ok);
    }
}

// The P limbs of a tile one after the other: in the integer arithmetics the
// multiply pipe is the bound, not the twiddles, and two limbs' butterflies
// unrolled side by side overflow the instruction cache (a fifth of the stalls
// in the 9-stage passes).  The chain and product passes of 768 limbs at
// N = 2^16 measured 657 against 675 us and 666 against 788 us so, the lazy
// inverse's 9-stage pass 300 against 316 (only the forward's was 3 % faster
// side by side).
template <int P, class Run>
__device__ __forceinline__ void each_limb(uint64_t limb, uint64_t lstep, const Run& run)
{
    if constexpr (P == 1) {
        run(limb);
    } else {
#pragma unroll 1
        for (int p = 0; p < P; ++p) {
            if (p) {
                if (lstep == 0) break;  // a limb without a partner
                __syncthreads();        // the tile's shared memory is free again
            }
            run(limb + p * lstep);
        }
    }
}

// The same in the arithmetic the limb's modulus and the launch allow: with
// MODES, kRelaxOut transforms of moduli below 2^50 run in FP64 and those
// below 2^59 on relaxed integers, other forward transforms of moduli below
// 2^50 as lazy FP64.  RELAX says which of the two sets a kernel holds, so
// that the sets' registers do not count against each other.  (Every pass of
// a call has the same kRelaxOut flag and every kernel that may be launched
// with it the same modes, so the passes agree on what lies between them.)
template <bool INV, int LG, int LR, bool CG, bool MUL = false, bool MODES = false, bool RELAX = false, int P = 1,
          int SHAPE = kAnyTiles>
__device__ __forceinline__ void pass_tile(const uint64_t* src, uint64_t* dst, const ModCtx* cx, uint32_t logn,
                                          uint32_t s0, uint32_t lgtg, uint64_t limb, uint64_t tile_in_limb,
                                          uint32_t flags, uint64_t* sm, const uint64_t* operand = nullptr,
                                          uint64_t lstep = 0)
{
    if constexpr (MODES && relaxed_compiled(LG, LR)) {
        const uint32_t kind = cx->arith;
        if constexpr (RELAX) {
            if (kind == kFp) {
                pass_tile_as<kFp, INV, LG, LR, CG, MUL, P, SHAPE>(src, dst, cx, logn, s0, lgtg, limb, lstep, tile_in_limb,
                                                           flags, sm, operand);
                return;
            }
            if (kind == kRelaxed) {
                each_limb<P>(limb, lstep, [&](uint64_t l) {
                    pass_tile_as<kRelaxed, INV, LG, LR, CG, MUL, 1, SHAPE>(src, dst, cx, logn, s0, lgtg, l, lstep,
                                                                       tile_in_limb, flags, sm, operand);
                });
                return;
            }
        } else if constexpr (!INV && !MUL) {  // (a product's output is normalized)
            if (kind == kFp && (flags & kLazyFp)) {
                pass_tile_as<kFpLazy, INV, LG, LR, CG, MUL, P, SHAPE>(src, dst, cx, logn, s0, lgtg, limb, lstep,
                                                               tile_in_limb, flags, sm, operand);
                return;
            }
        }
    }
    each_limb<P>(limb, lstep, [&](uint64_t l) {
        pass_tile_as<kExact, INV, LG, LR, CG, MUL, 1, SHAPE>(src, dst, cx, logn, s0, lgtg, l, lstep, tile_in_limb, flags,
                                                         sm, operand);
    });
}

// CTA -> tile: blockIdx.y is the modulus, blockIdx.x the group of nctx limbs
// (with P = 2 the pair of groups) and the tile in the limb.  (No division, and
// the modulus context is uniform over the CTA for the compiler too.)  `lstep`:
// the distance to the second limb of a pair, 0 for a limb without a partner,
// which is then its own (both copies hold the same values and write them to
// the same place).
template <int P>
__device__ __forceinline__ bool cta_tile(const PassArgs& a, uint32_t lg_tiles, uint64_t& limb, uint32_t& tile_in_limb,
                                         uint64_t& lstep)
{
    tile_in_limb = blockIdx.x & ((1u << lg_tiles) - 1);
    limb = (uint64_t)(blockIdx.x >> lg_tiles) * P * a.nctx + blockIdx.y;
    lstep = P == 1 || limb + a.nctx >= a.count ? 0 : a.nctx;
    return limb < a.count;
}

template <bool INV, int LG, int LR, bool RELAX, int SHAPE>
__global__ void __launch_bounds__(max_threads(LR), LR == 3 ? 2 : 1) ntt_pass_kernel(const __grid_constant__ PassArgs a)
{
    extern __shared__ uint64_t sm[];
    const uint32_t lgtg = __ffs(a.tg) - 1;
    uint64_t limb, lstep;
    uint32_t til;
    if (!cta_tile<1>(a, a.logn - LG - lgtg, limb, til, lstep)) return;
    pass_tile<INV, LG, LR, false, false, true, RELAX, 1, SHAPE>(
        a.src, a.dst, a.ctx[blockIdx.y], a.logn, a.s0, lgtg, limb, til, a.flags, sm, nullptr, lstep);
}

// Sixteen registers of the limb per thread: held to the machine registers it
// takes by itself, where four or three CTAs of 256 threads share an SM.
template <bool INV, int LG, int SHAPE>
__global__ void __maxnreg__(INV ? 80 : 72) ntt_pass16_kernel(const __grid_constant__ PassArgs a)
{
    extern __shared__ uint64_t sm[];
    const uint32_t lgtg = __ffs(a.tg) - 1;
    uint64_t limb, lstep;
    uint32_t til;
    if (!cta_tile<1>(a, a.logn - LG - lgtg, limb, til, lstep)) return;
    pass_tile<INV, LG, 4, false, false, true, false, 1, SHAPE>(
        a.src, a.dst, a.ctx[blockIdx.y], a.logn, a.s0, lgtg, limb, til, a.flags, sm, nullptr, lstep);
}

template <bool INV, int LG, int LR, bool RELAX, int SHAPE>
__global__ void __maxnreg__(kPairRegs) ntt_pass_pair_kernel(const __grid_constant__ PassArgs a)
{
    extern __shared__ uint64_t sm[];
    const uint32_t lgtg = __ffs(a.tg) - 1;
    uint64_t limb, lstep;
    uint32_t til;
    if (!cta_tile<2>(a, a.logn - LG - lgtg, limb, til, lstep)) return;
    pass_tile<INV, LG, LR, false, false, true, RELAX, 2, SHAPE>(
        a.src, a.dst, a.ctx[blockIdx.y], a.logn, a.s0, lgtg, limb, til, a.flags, sm, nullptr, lstep);
}

// The same pass with the dyadic product of kPreMul / kPostMul: a kernel of
// its own, so that the product's registers do not count against the plain
// passes.
template <bool INV, int LG, int LR, bool RELAX, int SHAPE>
__global__ void __launch_bounds__(max_threads(LR), LR == 3 ? 2 : 1) ntt_pass_mul_kernel(const __grid_constant__ PassArgs a)
{
    extern __shared__ uint64_t sm[];
    const uint32_t lgtg = __ffs(a.tg) - 1;
    uint64_t limb, lstep;
    uint32_t til;
    if (!cta_tile<1>(a, a.logn - LG - lgtg, limb, til, lstep)) return;
    pass_tile<INV, LG, LR, false, true, true, RELAX, 1, SHAPE>(
        a.src, a.dst, a.ctx[blockIdx.y], a.logn, a.s0, lgtg, limb, til, a.flags, sm, a.operand, lstep);
}

template <bool INV, int LG, int SHAPE>
__global__ void __maxnreg__(128) ntt_pass_mul16_kernel(const __grid_constant__ PassArgs a)
{
    extern __shared__ uint64_t sm[];
    const uint32_t lgtg = __ffs(a.tg) - 1;
    uint64_t limb, lstep;
    uint32_t til;
    if (!cta_tile<1>(a, a.logn - LG - lgtg, limb, til, lstep)) return;
    pass_tile<INV, LG, 4, false, true, true, false, 1, SHAPE>(
        a.src, a.dst, a.ctx[blockIdx.y], a.logn, a.s0, lgtg, limb, til, a.flags, sm, a.operand, lstep);
}

template <bool INV, int LG, int LR, bool RELAX, int SHAPE>
__global__ void __maxnreg__(kPairRegs) ntt_pass_mul_pair_kernel(const __grid_constant__ PassArgs a)
{
    extern __shared__ uint64_t sm[];
    const uint32_t lgtg = __ffs(a.tg) - 1;
    uint64_t limb, lstep;
    uint32_t til;
    if (!cta_tile<2>(a, a.logn - LG - lgtg, limb, til, lstep)) return;
    pass_tile<INV, LG, LR, false, true, true, RELAX, 2, SHAPE>(
        a.src, a.dst, a.ctx[blockIdx.y], a.logn, a.s0, lgtg, limb, til, a.flags, sm, a.operand, lstep);
}

// Fused column pass of an INTT -> op -> NTT chain: the inverse's last pass
// (stages logn-LG .. logn-1, incl. the N^-1 final stage) and the forward's
// first pass (stages 0 .. LG-1) act on the same groups p = r*S + col, and the
// inverse's last round holds the same register bits as the forward's first
// round, so the element-wise op runs in registers between them.  IM / FM: the
// arithmetic of the inverse and of the forward.
template <int IM, int FM, int LG, int LR, bool CG, int P>
__device__ __forceinline__ void chain_tile_as(const uint64_t* src, uint64_t* dst, const uint64_t* operand,
                                              const ModCtx* cx, uint32_t op, uint64_t scalar, uint32_t logn,
                                              uint32_t lgtg, uint64_t limb, uint64_t lstep, uint64_t tile_in_limb,
                                              uint32_t flags, uint64_t* sm)
{
    constexpr int R = 1 << LR;
    constexpr int NR = num_rounds<LG, LR>();
    constexpr int LO_FIRST = round_lo<true, LG, LR, 0>();
    constexpr int LO_MID = round_lo<true, LG, LR, NR - 1>();
    constexpr int LO_LAST = round_lo<false, LG, LR, NR - 1>();
    static_assert(LO_MID == round_lo<false, LG, LR, 0>(), "inverse last round and forward first round differ");
    static_assert(IM != kFp || FM == kFp || FM == kFpLazy, "an FP64 inverse hands doubles to the forward");
    const Tile t = make_tile<LG>(logn - LG, lgtg, tile_in_limb);
    const uint64_t q = cx->q;
    const uint32_t n = 1u << logn;
    const uint64_t* lsrc = src + (limb << logn);
    uint64_t* ldst = dst + (limb << logn);
    const uint64_t pstep = lstep << logn;
    const int vec_ok = vec_align(reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst) |
                                 reinterpret_cast<uintptr_t>(operand));
    const bool one_pass = logn == LG;

    uint32_t gi, k;
    thread_role<LG, LR>(t, gi, k);
    const uint32_t blk = tile_blk<LG>(t, gi);
    const uint32_t hmask = group_slot<LG, LR>(t.strided, lgtg, gi);
    const uint32_t lsh = lane_shift(t.strided, lgtg);
    const uint32_t ps = 1u << (LG + lgtg);

    uint64_t v[P][R];
#pragma unroll
    for (int p = 0; p < P; ++p)
        load_global<LG, LR, LO_FIRST, CG>(v[p], lsrc + p * pstep, t, gi, round_base<LR>(k, LO_FIRST), vec_ok);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        to_stages<IM, LR>(v[p], one_pass, cx);
        if constexpr (IM == kExact) {
            if (flags & kPreCsub2q) {
#pragma unroll
                for (int i = 0; i < R; ++i) v[p][i] = csub_lazy(v[p][i], cx->q2);
            }
        }
    }
    run_rounds<true, LG, LR, IM, P>(v, sm, k, hmask, lsh, ps, blk, logn - LG, n, cx, one_pass, true);

    // Element-wise op on the inverse output (lazy [0, 2q)) with factor-2
    // inputs: EltwiseMulModNative<2> / EltwiseFMAModNative<2> formulas.
    const uint32_t rb = round_base<LR>(k, LO_MID);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const uint64_t* lop = operand + (limb << logn) + p * pstep;
        if constexpr (IM == kFp) {
            const double fq = cx->fq, fqi = cx->fqi, off = __fma_rn(2.0, fq, kFp2p52);
            uint64_t m[R];
            if (operand) load_global<LG, LR, LO_MID, false>(m, lop, t, gi, rb, vec_ok);
            if (op == kChainMul) {
#pragma unroll
                for (int i = 0; i < R; ++i)
                    v[p][i] = as_u64(fp_mulmod(as_fp(v[p][i]), fp_from_u64(m[i], off), fq, fqi));
            } else if (op == kChainFma) {
                const double sc = (double)reduce_input<2>(scalar, q);
#pragma unroll
                for (int i = 0; i < R; ++i) v[p][i] = as_u64(fp_mulmod(as_fp(v[p][i]), sc, fq, fqi));
                if (operand) {
#pragma unroll
                    for (int i = 0; i < R; ++i)
                        v[p][i] = as_u64(__dadd_rn(as_fp(v[p][i]), fp_from_u64(m[i], off)));
                }
            }
            if constexpr (FM == kFpLazy) {
                // the op's result in [0, q), as the reference hands it to the forward
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    double x = fp_reduce(as_fp(v[p][i]), fq, fqi);
                    if (__double2hiint(x) < 0) x = __dadd_rn(x, fq);
                    v[p][i] = as_u64(x);
                }
            }
        } else {
            const uint64_t mu = cx->mu;
            const uint32_t shift = cx->shift;
            if constexpr (IM == kRelaxed) {
#pragma unroll
                for (int i = 0; i < R; ++i) v[p][i] = csub_lazy(v[p][i], cx->q2);
            }
            if (op == kChainMul) {
                uint64_t m[R];
                load_global<LG, LR, LO_MID, false>(m, lop, t, gi, rb, vec_ok);
#pragma unroll
                for (int i = 0; i < R; ++i)
                    v[p][i] = barrett_mul(reduce_input<2>(v[p][i], q), reduce_input<2>(m[i], q), q, mu, shift);
            } else if (op == kChainFma) {
                const uint64_t sc = reduce_input<2>(scalar, q);
#pragma unroll
                for (int i = 0; i < R; ++i) v[p][i] = barrett_mul(reduce_input<2>(v[p][i], q), sc, q, mu, shift);
                if (operand) {
                    uint64_t m[R];
                    load_global<LG, LR, LO_MID, false>(m, lop, t, gi, rb, vec_ok);
#pragma unroll
                    for (int i = 0; i < R; ++i) v[p][i] = csub(v[p][i] + reduce_input<2>(m[i], q), q);
                }
            }
        }
    }

    // The forward's first pass: stages 0 .. LG-1 of block 0.
    const ModArith a = mod_arith<FM, false>(cx, n, one_pass);
    fwd_stages<FM, LG, LR, 0, P>(v, rb, 0, 0, a);
    fwd_rest<FM, LG, LR, P>(std::make_integer_sequence<int, NR - 1>{}, v, sm, k, hmask, lsh, ps, 0, 0, a);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        if (one_pass || FM == kFpLazy || FM == kExact) fwd_output<FM, LR>(v[p], (flags & kPostNorm) != 0, cx);
        store_global<LG, LR, LO_LAST>(v[p], ldst + p * pstep, t, gi, round_base<LR>(k, LO_LAST), vec_ok);
    }
}

// The chain tile in the arithmetic the modulus allows: the inverse feeds a
// MulMod / FMAMod, which takes any representative; RELAX says whether the
// forward's output is normalized too.
template <int LG, int LR, bool CG, bool MODES = false, bool RELAX = false, int P = 1>
__device__ __forceinline__ void chain_tile(const uint64_t* src, uint64_t* dst, const uint64_t* operand,
                                           const ModCtx* cx, uint32_t op, uint64_t scalar, uint32_t logn,
                                           uint32_t lgtg, uint64_t limb, uint64_t tile_in_limb, uint32_t flags,
                                           uint64_t* sm, uint64_t lstep = 0)
{
    if constexpr (MODES && relaxed_compiled(LG, LR)) {
        if (flags & kRelaxIn) {
            const uint32_t kind = cx->arith;
            if (kind == kFp) {
                chain_tile_as<kFp, RELAX ? kFp : kFpLazy, LG, LR, CG, P>(
                    src, dst, operand, cx, op, scalar, logn, lgtg, limb, lstep, tile_in_limb, flags, sm);
                return;
            }
            if (kind == kRelaxed) {
                each_limb<P>(limb, lstep, [&](uint64_t l) {
                    chain_tile_as<kRelaxed, RELAX ? kRelaxed : kExact, LG, LR, CG, 1>(
                        src, dst, operand, cx, op, scalar, logn, lgtg, l, lstep, tile_in_limb, flags, sm);
                });
                return;
            }
        }
    }
    each_limb<P>(limb, lstep, [&](uint64_t l) {
        chain_tile_as<kExact, kExact, LG, LR, CG, 1>(src, dst, operand, cx, op, scalar, logn, lgtg, l, lstep,
                                                        tile_in_limb, flags, sm);
    });
}

// Fused row pass of an NTT -> MulMod -> INTT product (the polynomial product
// in evaluation form, SEAL's multiply_plain): the forward's last pass (stages
// logn-LG .. logn-1) and the inverse's first pass (stages 0 .. LG-1) act on
// the same contiguous groups of 2^LG words, and the forward's last round
// holds the same register bits as the inverse's first round (the low LR
// bits), so the dyadic product runs in registers between them.  The product
// is EltwiseMulModNative<4> (axhel/eltwise/eltwise-mul-mod.cpp:18-63) of the
// forward's lazy output and the multiplicand, both in [0, 4q).  With LG ==
// logn (one pass each way) the tile also holds the inverse's N^-1 stage.
template <int FM, int IM, int LG, int LR, int P>
__device__ __forceinline__ void product_tile_as(const uint64_t* src, uint64_t* dst, const uint64_t* operand,
                                                const ModCtx* cx, uint32_t logn, uint32_t lgtg, uint64_t limb,
                                                uint64_t lstep, uint64_t tile_in_limb, uint32_t flags, uint64_t* sm)
{
    constexpr int R = 1 << LR;
    constexpr int NR = num_rounds<LG, LR>();
    constexpr int LO_FIRST = round_lo<false, LG, LR, 0>();
    constexpr int LO_MID = round_lo<false, LG, LR, NR - 1>();
    constexpr int LO_LAST = round_lo<true, LG, LR, NR - 1>();
    static_assert(LO_MID == round_lo<true, LG, LR, 0>(), "forward last round and inverse first round differ");
    const Tile t = make_tile<LG>(0, lgtg, tile_in_limb);
    const uint32_t n = 1u << logn;
    const uint64_t at = limb << logn, pstep = lstep << logn;
    const int vec_ok = vec_align(reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst) |
                                 reinterpret_cast<uintptr_t>(operand));
    const bool last = (flags & kLastPass) != 0;
    uint32_t gi, k;
    thread_role<LG, LR>(t, gi, k);
    const uint32_t blk = tile_blk<LG>(t, gi);
    const uint32_t hmask = group_slot<LG, LR>(t.strided, lgtg, gi);
    const uint32_t lsh = lane_shift(t.strided, lgtg);
    const uint32_t ps = 1u << (LG + lgtg);

    uint64_t v[P][R];
#pragma unroll
    for (int p = 0; p < P; ++p)
        load_global<LG, LR, LO_FIRST, false>(v[p], src + at + p * pstep, t, gi, round_base<LR>(k, LO_FIRST), vec_ok);
#pragma unroll
    for (int p = 0; p < P; ++p) to_stages<FM, LR>(v[p], logn == LG, cx);
    run_rounds<false, LG, LR, FM, P>(v, sm, k, hmask, lsh, ps, blk, logn - LG, n, cx, true, false);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        mul_operand<FM, LG, LR, LO_MID, false>(v[p], operand + at + p * pstep, t, gi, k, cx, vec_ok, 32);
        if constexpr (FM == kFp && IM != kFp) inv_output<FM, LR>(v[p], true, cx);
    }
    run_rounds<true, LG, LR, IM, P>(v, sm, k, hmask, lsh, ps, blk, 0, n, cx, true, last);
#pragma unroll
    for (int p = 0; p < P; ++p) {
        if (last || IM == kExact) inv_output<IM, LR>(v[p], (flags & kPostNorm) != 0, cx);
        store_global<LG, LR, LO_LAST>(v[p], dst + at + p * pstep, t, gi, round_base<LR>(k, LO_LAST), vec_ok);
    }
}

// The product tile in the arithmetic the modulus allows: the forward feeds
// the MulMod, which takes any representative; RELAX says whether the
// inverse's output is normalized too.
template <int LG, int LR, bool MODES, bool RELAX, int P>
__device__ __forceinline__ void product_tile(const uint64_t* src, uint64_t* dst, const uint64_t* operand,
                                             const ModCtx* cx, uint32_t logn, uint32_t lgtg, uint64_t limb,
                                             uint64_t lstep, uint64_t tile_in_limb, uint32_t flags, uint64_t* sm)
{
    if constexpr (MODES && relaxed_compiled(LG, LR)) {
        if (flags & kRelaxIn) {
            const uint32_t kind = cx->arith;
            if (kind == kFp) {
                product_tile_as<kFp, RELAX ? kFp : kExact, LG, LR, P>(src, dst, operand, cx, logn, lgtg, limb, lstep,
                                                                      tile_in_limb, flags, sm);
                return;
            }
            if (kind == kRelaxed) {
                each_limb<P>(limb, lstep, [&](uint64_t l) {
                    product_tile_as<kRelaxed, RELAX ? kRelaxed : kExact, LG, LR, 1>(
                        src, dst, operand, cx, logn, lgtg, l, lstep, tile_in_limb, flags, sm);
                });
                return;
            }
        }
    }
    each_limb<P>(limb, lstep, [&](uint64_t l) {
        product_tile_as<kExact, kExact, LG, LR, 1>(src, dst, operand, cx, logn, lgtg, l, lstep, tile_in_limb,
                                                      flags, sm);
    });
}

// Kernel of the fused product pass: one CTA per tile of product_tile above;
// MODES false: the reference's butterflies only.
template <int LG, int LR, bool MODES, bool RELAX, int P>
__global__ void __maxnreg__(product_regs(P)) ntt_product_kernel(const __grid_constant__ ChainArgs c)
{
    extern __shared__ uint64_t sm[];
    const PassArgs& a = c.pass;
    const uint32_t lgtg = __ffs(a.tg) - 1;
    uint64_t limb, lstep;
    uint32_t til;
    if (!cta_tile<P>(a, a.logn - LG - lgtg, limb, til, lstep)) return;
    product_tile<LG, LR, MODES, RELAX, P>(a.src, a.dst, c.operand, a.ctx[blockIdx.y], a.logn, lgtg, limb, lstep, til,
                                          a.flags, sm);
}

// Kernel of the fused chain pass: one CTA per tile of chain_tile above; the
// modulus context and the FMA scalar follow the limb.
template <int LG, int LR, bool MODES, bool RELAX, int P>
__global__ void __maxnreg__(chain_regs(LR)) ntt_chain_kernel(const __grid_constant__ ChainArgs c)
{
    extern __shared__ uint64_t sm[];
    const PassArgs& a = c.pass;
    const uint32_t lgtg = __ffs(a.tg) - 1;
    uint64_t limb, lstep;
    uint32_t til;
    if (!cta_tile<P>(a, a.logn - LG - lgtg, limb, til, lstep)) return;
    chain_tile<LG, LR, false, MODES, RELAX, P>(a.src, a.dst, c.operand, a.ctx[blockIdx.y], c.op, c.scalar[blockIdx.y],
                                               a.logn, lgtg, limb, til, a.flags, sm, lstep);
}

}  // namespace axhel_impl
