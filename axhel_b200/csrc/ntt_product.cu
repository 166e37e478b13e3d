// The fused NTT -> MulMod -> INTT pass kernels (ntt_kernels.cuh).
#include "ntt_table.cuh"

namespace axhel_impl {

namespace {
template <int LG, int LR, bool RELAX, int P, int SHAPE>
struct Get {
    static constexpr bool compiled = LR <= 3, has_plain = true, exact_pairs = true;
    static constexpr Columns columns = kSameColumns;
    static ChainFn fn() { return ntt_product_kernel<LG, LR, P != 0, RELAX, P == 2 ? 2 : 1>; }
};
}  // namespace

const FnTable<ChainFn>& product_table()
{
    static const FnTable<ChainFn> t = make_table<Get, ChainFn>(AllGroups{});
    return t;
}

}  // namespace axhel_impl
