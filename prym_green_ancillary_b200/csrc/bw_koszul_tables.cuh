// Subset neighbours on the device, for the incidence tables of both forms.
#pragma once

#include "bw_common.cuh"

namespace bw {

// Binomial coefficients C(n, k), n, k <= 31 (below 2^32).
struct BinomTable {
    uint32_t c[32][32];
};

inline BinomTable binom_table() {
    BinomTable t;
    for (int n = 0; n < 32; ++n)
        for (int k = 0; k < 32; ++k) t.c[n][k] = static_cast<uint32_t>(k <= n ? binom(n, k) : 0);
    return t;
}

// The size-subset of 0..r-1 of lexicographic rank blk, as a bit mask.
__device__ __forceinline__ uint32_t subset_of(uint32_t blk, int r, int size, const BinomTable& B) {
    uint32_t set = 0, rem = B.c[r][size] - 1 - blk;
    for (int pos = 0, v = 0; pos < size; ++pos, ++v) {
        while (B.c[r - 1 - v][size - pos] > rem) ++v;
        rem -= B.c[r - 1 - v][size - pos];
        set |= 1u << v;
    }
    return set;
}

// Its inverse.
__device__ __forceinline__ uint32_t rank_of(uint32_t set, int r, int size, const BinomTable& B) {
    uint32_t rank = B.c[r][size] - 1;
    for (int v = 0, left = size; left > 0; ++v)
        if (set >> v & 1) rank -= B.c[r - 1 - v][left--];
    return rank;
}

// Calls f(i, rank, negative) for every neighbour of block blk, i ascending:
//   forward : blk = T, a (k-1)-subset; neighbour S = T u {i} for every i not in T
//   backward: blk = S, a k-subset; neighbour T = S \ {i} for every i in S
// with rank(S) = C(r,k) - 1 - sum_pos C(r-1-S_pos, k-pos) (lexicographic) and
// the sign (-1)^pos of i's position in S.  The subset is unranked once;
// `before` and `after` hold the neighbour's rank terms of the elements below
// and above i, so a block costs O(r).
template <class F>
__device__ __forceinline__ void for_each_neighbour(uint32_t blk, int r, int k, bool forward, const BinomTable& B,
                                                   F&& f) {
    const int size = forward ? k - 1 : k, other = forward ? k : k - 1;   // of blk, of its neighbours
    const uint32_t set = subset_of(blk, r, size, B);
    // an element at position j counts C(r-1-v, other - j) below i; above i its
    // position in the neighbour is j + 1 (forward) or j - 1 (backward)
    const int shift = forward ? 1 : -1;
    auto term = [&](int v, int below) { return below >= 0 ? B.c[r - 1 - v][below] : 0u; };
    uint32_t before = 0, after = 0;
    for (int v = 0, j = 0; v < r; ++v)
        if (set >> v & 1) after += term(v, other - j++ - shift);
    for (int i = 0, pos = 0; i < r; ++i) {
        const bool in = (set >> i & 1) != 0;
        const bool negative = (pos & 1) != 0;
        if (in) after -= term(i, other - pos - shift);
        if (in != forward)
            f(i, B.c[r][other] - 1 - before - after - (forward ? term(i, k - pos) : 0u), negative);
        if (in) before += term(i, other - pos++);
    }
}

inline unsigned blocks_of(uint64_t items, unsigned threads) {
    return static_cast<unsigned>((items + threads - 1) / threads);
}

}  // namespace bw
