// What the INT8-limb kernels share: limb planes, warp roles, the pipeline's
// slot ring, limb arithmetic and the epilogue's byte transpose.
#pragma once

#include "bw_common.cuh"
#include "tc_sm100.cuh"

namespace bw {

namespace {

constexpr uint32_t kAbsent = 0xFFFFFFFFu;

// Warp roles of the cp.async gather kernel with PW producer warps: PW = 8
// (eight epilogue warps, 17 in all) or PW = 16 (four epilogue warps, 21 in
// all; more copy streams for the same register budget of 96 a thread).
template <int PW>
struct GatherWarps {
    static_assert(PW == 8 || PW == 16, "8 or 16 producer warps");
    static constexpr int producers = PW;
    static constexpr int mma = PW;                        // allocates TMEM, issues the MMAs
    static constexpr int epilogue0 = PW + 1;
    static constexpr int epilogue = PW == 16 ? 4 : 8;     // per TMEM lane quadrant: epilogue / 4
    static constexpr int threads = (PW + 1 + epilogue) * 32;
};
constexpr int kMaxSmem = 227 * 1024;

// Plane index inside a four-plane block array.
enum : int { PL_LO = 0, PL_HI = 1, PL_NLO = 2, PL_NHI = 3 };

// Position in a ring of pipeline slots: slot index and the parity of its
// current phase, advanced without dividing (a 64-bit division per stage would
// sit on the producers' and the MMA thread's critical paths).
struct SlotRing {
    int slot = 0, n = 1;
    uint32_t phase = 0;
    __device__ explicit SlotRing(int count) : n(count) {}
    __device__ void next() {
        if (++slot == n) {
            slot = 0;
            phase ^= 1u;
        }
    }
};

// ll + 255 (lh + hl) + 255^2 hh mod p (balanced); c1 = 255, c2 = 255^2 mod p, balanced.
__device__ __forceinline__ int32_t combine(int32_t ll, int32_t lhhl, int32_t hh, const Mod& mod, int32_t c1,
                                           int32_t c2) {
    const int32_t a = reduce_partial(ll, mod);
    const int32_t b = reduce_partial(lhhl, mod);
    const int32_t c = reduce_partial(hh, mod);
    return reduce_balanced(a + c1 * b + c2 * c, mod);
}

__host__ __device__ __forceinline__ void split_limbs(int32_t v, int32_t& lo, int32_t& hi) {
    // v in [-16383, 16383]: q = floor((v + 127) / 255), lo = v - 255 q in [-127, 127]
    hi = static_cast<int32_t>(static_cast<uint32_t>(v + 127 + 255 * 128) / 255u) - 128;
    lo = v - 255 * hi;
}
__host__ __device__ __forceinline__ void split_limbs(int32_t v, int8_t& lo, int8_t& hi) {
    int32_t l, h;
    split_limbs(v, l, h);
    lo = static_cast<int8_t>(l);
    hi = static_cast<int8_t>(h);
}

// The low bytes of four values in one word.
__device__ __forceinline__ uint32_t pack_bytes(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// 16 x 16 byte transpose inside each half-warp.  On entry lane L (L = lane & 15)
// holds row L as four words (byte b of word q = element 4q + b); on exit it
// holds column L the same way.  Two butterfly stages exchange words (lane bits
// 2 and 3 against word-index bits), two exchange bytes (lane bits 0 and 1
// against byte-index bits, recombined with byte permutes).
__device__ __forceinline__ void transpose16(uint32_t (&w)[4], int lane) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const bool upper = (lane >> (k + 2)) & 1;
        const int step = 1 << k;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (q & step) continue;   // the pair (q, q + step)
            const uint32_t send = upper ? w[q] : w[q + step];
            const uint32_t recv = __shfl_xor_sync(0xffffffffu, send, 4 << k);
            if (upper) w[q] = recv;
            else w[q + step] = recv;
        }
    }
    const bool b0 = lane & 1, b1 = (lane >> 1) & 1;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        uint32_t r = __shfl_xor_sync(0xffffffffu, w[q], 1);
        w[q] = __byte_perm(w[q], r, b0 ? 0x3715 : 0x6240);
        r = __shfl_xor_sync(0xffffffffu, w[q], 2);
        w[q] = __byte_perm(w[q], r, b1 ? 0x3276 : 0x5410);
    }
}

}  // namespace

}  // namespace bw
