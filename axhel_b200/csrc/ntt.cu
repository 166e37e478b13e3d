// Launchers of the NTT pass, chain and product kernels (ntt_kernels.cuh).
#include <cuda_runtime.h>

#include <mutex>

#include "device_once.h"
#include "launch.h"
#include "ntt_table.cuh"

namespace axhel_impl {

namespace {

// Kinds of kernels, for the dynamic shared memory attribute.
enum FnKind : int { kFnFwd, kFnInv, kFnChain, kFnProduct, kFnFwdMul, kFnInvMul, kFnKinds };
constexpr int kSmemPlain = 2;  // third "pair" column
// Two limbs per thread halve the CTAs: only where they still fill the GPU.
constexpr uint64_t kPairThreadsPerSm = 1024;

DeviceOnce g_smem_set[kFnKinds][2][3][2][kMaxLG + 1][kMaxLR + 1];

std::mutex g_attr_mu;

size_t smem_bytes(const PassCfg& c) { return (size_t)c.tg * (size_t(1) << c.lg) * sizeof(uint64_t); }

template <class Fn>
cudaError_t ensure_smem(Fn fn, FnKind kind, bool relax, int column, bool row, const PassCfg& c)
{
    const size_t bytes = smem_bytes(c) << (column == 1);
    if (bytes <= 48 * 1024) return cudaSuccess;
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    // Set to the maximum once per kernel; cheaper than tracking each size.
    return g_smem_set[kind][relax][column][row][c.lg][c.lr](dev, g_attr_mu, [&] {
        return cudaFuncSetAttribute(reinterpret_cast<const void*>(fn), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    227 * 1024);
    });
}

// Whether a launch's limbs run two per thread, pairs of the batch's groups of
// nctx limbs (one per modulus).  A limb without a partner costs an FP64 pass as
// much as a pair (41 limbs of 40 45-bit moduli, N = 2^16: lazy product 102 us
// as pairs, 59.4 single), so batches with more than a seventh of them stay single.
// The integer product passes run a pair's limbs in turn and do not have that
// cost (40 limbs of 24 55-bit moduli 3-4 % faster as pairs).
bool pairs(FnKind kind, bool relax, const PassCfg& c, const PassArgs& a)
{
    if (kind == kFnFwd && !relax) return false;  // the lazy forms: 333 against 320 us for 768 limbs of 2^16
    if (!relaxed_compiled(c.lg, c.lr) || (smem_bytes(c) << 1) > 227 * 1024) return false;
    if (((a.count << a.logn) >> (c.lr + 1)) < (uint64_t)sm_count() * kPairThreadsPerSm) return false;
    const uint64_t groups = (a.count + a.nctx - 1) / a.nctx, paired = 2 * a.nctx * ((groups + 1) / 2);
    if (kind == kFnProduct && !(a.flags & kFpLimbs)) return groups >= 7 || groups % 2 == 0;
    return 7 * paired <= 8 * a.count;
}

PassArgs& pass_of(PassArgs& a) { return a; }
PassArgs& pass_of(ChainArgs& a) { return a.pass; }
void copy_scalar(PassArgs&, uint64_t, uint64_t) {}
void copy_scalar(ChainArgs& a, uint64_t to, uint64_t from) { a.scalar[to] = a.scalar[from]; }

// Launches a pass over its limbs; `pass` is the PassArgs inside the kernel's
// argument struct `args`.
template <class Args>
cudaError_t launch_tiles(const FnTable<void (*)(const Args)>& t, FnKind kind, bool relax, const PassCfg& c,
                         const Args& args, const PassArgs& pass, bool row, cudaStream_t s)
{
    const bool plain = (kind == kFnChain || kind == kFnProduct) && !(pass.flags & kRelaxIn);
    const bool pair = !plain && pairs(kind, relax, c, pass);
    auto fn = plain ? t.plain[c.lg][c.lr] : t.at[relax][pair][row][c.lg][c.lr];
    if (!fn) return cudaErrorInvalidValue;
    if (pass.count == 0) return cudaSuccess;
    const cudaError_t e = ensure_smem(fn, kind, relax, plain ? kSmemPlain : pair, row, c);
    if (e != cudaSuccess) return e;
    const uint64_t per_limb = (1ull << (pass.logn - c.lg)) / c.tg;
    if (pass.count * per_limb > 0x7fffffffull) return cudaErrorInvalidValue;
    const unsigned threads = (unsigned)c.tg << (c.lg - c.lr);
    count_launch();
    // A last group that holds only some of the moduli: the CTAs of its missing
    // limbs would lie between the others and leave SMs idle, so few limbs are
    // launched as one group, each with its own context (N = 2^16, 55 bits, us:
    // 9 limbs of 8 moduli forward 13.7 to 10.7, product 30.6 to 22.1; 32 of 24
    // 28.9 to 25.9, 67.9 to 64.1).  (More limbs with the groups in blockIdx.z,
    // which puts the missing ones last: 2-7 % faster, 300 of 24 of 2^13 28.2 to
    // 26.4, but the index costs canonical forwards of full groups 1 %.)
    const uint64_t moduli = pass.count < pass.nctx ? pass.count : pass.nctx;
    if (pass.count % moduli != 0 && !pair && pass.count <= (uint64_t)kMaxInlineMods) {
        Args one = args;
        PassArgs& p = pass_of(one);
        p.nctx = (uint32_t)pass.count;
        for (uint64_t i = moduli; i < pass.count; ++i) {
            p.ctx[i] = p.ctx[i - moduli];
            copy_scalar(one, i, i - moduli);
        }
        fn<<<dim3((unsigned)per_limb, p.nctx), threads, smem_bytes(c), s>>>(one);
        return cudaGetLastError();
    }
    const uint64_t groups = (pass.count + moduli - 1) / moduli, gx = ((groups + pair) >> pair) * per_limb;
    fn<<<dim3((unsigned)gx, (unsigned)moduli), threads, smem_bytes(c) << pair, s>>>(args);
    return cudaGetLastError();
}

bool geometry_ok(const PassCfg& c, uint32_t logn, uint32_t lgS)
{
    if (c.lg < 1 || c.lg > kMaxLG || c.lr < 1 || c.lr > kMaxLR || c.lr > c.lg) return false;
    if (c.tg < 1 || (c.tg & (c.tg - 1))) return false;
    if ((uint32_t)c.lg > logn) return false;
    const uint64_t groups = 1ull << (logn - c.lg);
    if ((uint64_t)c.tg > groups) return false;
    if (lgS > 0 && (uint64_t)c.tg > (1ull << lgS)) return false;
    const uint64_t threads = (uint64_t)c.tg << (c.lg - c.lr);
    if (threads > (uint64_t)max_threads(c.lr) || threads < 1) return false;
    if (smem_bytes(c) > 227 * 1024) return false;
    return true;
}

}  // namespace

bool pass_supported(const PassCfg& c)
{
    if (c.lg < 1 || c.lg > kMaxLG || c.lr < 1 || c.lr > kMaxLR) return false;
    return fwd_table().at[0][0][1][c.lg][c.lr] != nullptr;
}

bool pass_relaxable(const PassCfg& c) { return relaxed_compiled(c.lg, c.lr); }

bool plan_relax(bool inverse, uint32_t logn, NttPlan& p)
{
    NttPlan r = p;
    if (plan_overridden(inverse, logn)) {
        // set by the caller: as it is, or with the reference's butterflies
        for (int i = 0; i < p.npass; ++i)
            if (!pass_relaxable(p.pass[i])) return false;
        return true;
    }
    for (int i = 0; i < p.npass; ++i) {
        PassCfg& c = r.pass[i];
        // A pass tuned with 16 registers per thread takes twice the threads
        // here; back to 128 where the tile keeps 8 columns (64-byte rows).
        // The 7-stage passes of 768 limbs of N = 2^16, 16 against 8 columns:
        // 242 to 224 us forward, 285 to 264 inverse (4 columns at 8 stages
        // or 8 at 6: 3-10 % slower).
        if (c.lr == 4 && (c.tg << (c.lg - 3)) > 128 && c.tg > 8) c.tg >>= 1;
        c.lr = 3;
        if (!pass_relaxable(c) || ((uint64_t)c.tg << (c.lg - c.lr)) > (uint64_t)max_threads(c.lr)) return false;
    }
    p = r;
    return true;
}

cudaError_t launch_ntt_pass(bool inverse, const PassCfg& c, const PassArgs& a, cudaStream_t s)
{
    if (!pass_supported(c)) return cudaErrorInvalidValue;
    const uint32_t lgS = inverse ? a.s0 : (a.logn - a.s0 - c.lg);
    if (!geometry_ok(c, a.logn, lgS) || (uint32_t)c.tg != a.tg) return cudaErrorInvalidValue;
    const bool mul = (a.flags & (kPreMul | kPostMul)) != 0;
    const FnTable<PassFn>& t = mul ? (inverse ? inv_mul_table() : fwd_mul_table())
                                   : (inverse ? inv_table() : fwd_table());
    const FnKind kind = mul ? (inverse ? kFnInvMul : kFnFwdMul) : (inverse ? kFnInv : kFnFwd);
    ProfScope prof(s, "ntt_%s%s_pass lg=%d lr=%d tg=%d", inverse ? "inv" : "fwd", mul ? "_mul" : "", c.lg, c.lr,
                   c.tg);
    return launch_tiles(t, kind, (a.flags & kRelaxOut) != 0, c, a, a, lgS == 0, s);
}

cudaError_t launch_product_pass(const PassCfg& c, const ChainArgs& a, cudaStream_t s)
{
    if (!pass_supported(c) || c.lr > 3) return cudaErrorInvalidValue;
    if (!geometry_ok(c, a.pass.logn, 0) || (uint32_t)c.tg != a.pass.tg) return cudaErrorInvalidValue;
    ProfScope prof(s, "ntt_product_pass lg=%d lr=%d tg=%d", c.lg, c.lr, c.tg);
    return launch_tiles(product_table(), kFnProduct, (a.pass.flags & kRelaxOut) != 0, c, a, a.pass, true, s);
}

cudaError_t launch_chain_pass(const PassCfg& c, const ChainArgs& a, cudaStream_t s)
{
    if (!pass_supported(c)) return cudaErrorInvalidValue;
    if (!geometry_ok(c, a.pass.logn, a.pass.logn - c.lg) || (uint32_t)c.tg != a.pass.tg)
        return cudaErrorInvalidValue;
    ProfScope prof(s, "ntt_chain_pass lg=%d lr=%d tg=%d", c.lg, c.lr, c.tg);
    return launch_tiles(chain_table(), kFnChain, (a.pass.flags & kRelaxOut) != 0, c, a, a.pass, true, s);
}

}  // namespace axhel_impl
