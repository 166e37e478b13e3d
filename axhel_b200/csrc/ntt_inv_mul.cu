// The inverse pass kernels with the dyadic product (ntt_kernels.cuh): the first pass of a
// transform, on contiguous rows.
#include "ntt_table.cuh"

namespace axhel_impl {

namespace {
template <int LG, int LR, bool RELAX, int P, int SHAPE>
struct Get {
    static constexpr bool compiled = true, has_plain = false, exact_pairs = true;
    static constexpr Columns columns = kNoColumns;
    static PassFn fn()
    {
        if constexpr (P == 2) return ntt_pass_mul_pair_kernel<true, LG, LR, RELAX, SHAPE>;
        else if constexpr (LR == 4) return ntt_pass_mul16_kernel<true, LG, SHAPE>;
        else return ntt_pass_mul_kernel<true, LG, LR, RELAX, SHAPE>;
    }
};
}  // namespace

const FnTable<PassFn>& inv_mul_table()
{
    static const FnTable<PassFn> t = make_table<Get, PassFn>(AllGroups{});
    return t;
}

}  // namespace axhel_impl
