// The forward pass kernels (ntt_kernels.cuh); lazy forwards run one limb per
// thread (pairs() in ntt.cu).
#include "ntt_table.cuh"

namespace axhel_impl {

namespace {
template <int LG, int LR, bool RELAX, int P, int SHAPE>
struct Get {
    static constexpr bool compiled = true, has_plain = false, exact_pairs = false;
    static constexpr Columns columns = kOwnColumns;
    static PassFn fn()
    {
        if constexpr (P == 2) return ntt_pass_pair_kernel<false, LG, LR, RELAX, SHAPE>;
        else if constexpr (LR == 4) return ntt_pass16_kernel<false, LG, SHAPE>;
        else return ntt_pass_kernel<false, LG, LR, RELAX, SHAPE>;
    }
};
}  // namespace

const FnTable<PassFn>& fwd_table()
{
    static const FnTable<PassFn> t = make_table<Get, PassFn>(AllGroups{});
    return t;
}

}  // namespace axhel_impl
