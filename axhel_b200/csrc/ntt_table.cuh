// Tables of the compiled pass, chain and product kernels by group size and
// register depth, one source file per kind (they compile side by side).
#pragma once

#include <utility>

#include "ntt_kernels.cuh"

namespace axhel_impl {

using PassFn = void (*)(const PassArgs);
using ChainFn = void (*)(const ChainArgs);

constexpr int kMaxLG = 13;
constexpr int kMaxLR = 5;

// [1][..]: the kernels launched with kRelaxOut, [..][1]: two limbs per thread;
// both where relaxed_compiled.
template <class Fn>
struct FnTable {
    // Last but two: 0 strided columns, 1 contiguous rows (pass kernels).
    Fn at[2][2][2][kMaxLG + 1][kMaxLR + 1] = {};
    // Chain and product kernels with the reference's butterflies only, for
    // launches of a few limbs: those run through their code once, and a
    // kernel that holds the other arithmetics too takes 13-20 % longer to
    // fetch it (a chain of one limb of N = 2^16 17.3 against 15.2 us).
    Fn plain[kMaxLG + 1][kMaxLR + 1] = {};
};

const FnTable<PassFn>& fwd_table();
const FnTable<PassFn>& inv_table();
const FnTable<PassFn>& fwd_mul_table();  // with the dyadic product (kPreMul / kPostMul)
const FnTable<PassFn>& inv_mul_table();
const FnTable<ChainFn>& chain_table();
const FnTable<ChainFn>& product_table();

// What the launchers reach of a kind's kernels (its Get::): `compiled` register
// depths, `has_plain` kernels, `exact_pairs` -- two limbs per thread without
// kRelaxOut -- and kernels for strided columns: of their own, the same as for
// contiguous rows, or none (no such pass).
enum Columns : int { kNoColumns, kSameColumns, kOwnColumns };

template <template <int, int, bool, int, int> class Get, class Fn, int LG, int LR, int SHAPE>
void add_shape(FnTable<Fn>& t)
{
    constexpr int row = SHAPE == kRowTiles;
    t.at[0][0][row][LG][LR] = Get<LG, LR, false, 1, SHAPE>::fn();
    if constexpr (relaxed_compiled(LG, LR)) {
        t.at[1][0][row][LG][LR] = Get<LG, LR, true, 1, SHAPE>::fn();
        if constexpr (Get<LG, LR, false, 1, SHAPE>::exact_pairs)
            t.at[0][1][row][LG][LR] = Get<LG, LR, false, 2, SHAPE>::fn();
        t.at[1][1][row][LG][LR] = Get<LG, LR, true, 2, SHAPE>::fn();
    }
}

// Fills a table with Get<LG, LR, RELAX, P, SHAPE>::fn(); P limbs per thread, 0: plain.  Register-stage counts
// compiled for each group size: LR = LG for tiny groups, otherwise 3, 4 and 5
// where a group's threads fit a CTA.
template <template <int, int, bool, int, int> class Get, class Fn, int LG, int LR>
void add_one(FnTable<Fn>& t)
{
    using G = Get<LG, LR, false, 1, kRowTiles>;
    if constexpr (LR <= LG && (1 << (LG - LR)) <= max_threads(LR) && G::compiled) {
        add_shape<Get, Fn, LG, LR, kRowTiles>(t);
        if constexpr (G::columns == kOwnColumns) add_shape<Get, Fn, LG, LR, kColumnTiles>(t);
        if constexpr (G::columns == kSameColumns) {
            for (auto& relax : t.at)
                for (auto& pair : relax) pair[0][LG][LR] = pair[1][LG][LR];
        }
        t.plain[LG][LR] = t.at[0][0][1][LG][LR];
        if constexpr (relaxed_compiled(LG, LR) && G::has_plain)
            t.plain[LG][LR] = Get<LG, LR, false, 0, kRowTiles>::fn();
    }
}

template <template <int, int, bool, int, int> class Get, class Fn, int... I>
FnTable<Fn> make_table(std::integer_sequence<int, I...>)
{
    FnTable<Fn> t;
    ((I + 1 <= 3 ? add_one<Get, Fn, I + 1, (I + 1 <= 3 ? I + 1 : 3)>(t) : add_one<Get, Fn, I + 1, 3>(t)), ...);
    ((I + 1 > 3 ? add_one<Get, Fn, I + 1, 4>(t) : void()), ...);
    ((I + 1 > 3 ? add_one<Get, Fn, I + 1, 5>(t) : void()), ...);
    return t;
}

using AllGroups = std::make_integer_sequence<int, kMaxLG>;

}  // namespace axhel_impl
