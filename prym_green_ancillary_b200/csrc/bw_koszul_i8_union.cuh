// Gather-GEMM of the INT8-limb form over the generators that a tile has.
//
// The dense kernels of bw_koszul_i8.cu run K over all r generators, although
// a block has only k of them (d^T) or r - k + 1 (d), and issue two MMAs a
// K-step into two accumulators (input lo limbs, input hi limbs).  Here:
//
//   * Both input limbs lie in K.  With x = lo + 255 hi,
//       x * m = lo * m + hi * m',   m' = 255 m mod p (balanced),
//     so a generator spans 2 * inner K' rows (its lo rows against the limbs of
//     M_i, its hi rows against the limbs of 255 M_i), and one accumulator of
//     N = 2 * ho columns (lo and hi limbs of the maps; ho = outer rounded up
//     to 8) holds  out = acc_lo + 255 acc_hi:  the epilogue reads two partial
//     sums an output instead of four.  |acc| <= 2 * 1024 * 127^2 < 2^26.
//   * K runs over the union of the tile's generators only.  A tile is BT =
//     128 / NB blocks of an order that keeps blocks with nearly the same subset
//     together (see star_quad(); r = 19, k = 9: 13.6 of 19 generators a tile for
//     d and 12.0 for d^T).  A tile's generators come in ascending order; a table
//     holds, per tile and position in the union, the BT neighbours' run offsets.
//   * A generator's K' rows are padded to a multiple of 16, the width of a
//     core matrix of the K-major B operand.  The maps stay resident in shared
//     memory as [generator][16-row chunk][N][16 bytes]; a K-step of 32 rows
//     takes two chunks, and where a generator has an odd number of chunks the
//     step between it and the next generator takes one chunk of each: the
//     descriptor's leading-dimension offset is the distance between the two
//     (positive: generators ascend; a zero chunk after the last generator
//     stands in when the count is odd).  The A rows lie back to back in the
//     stage in the same order, so nothing is copied or multiplied for an
//     absent generator, and padding is at most 15 rows a generator.
//     (An earlier form padded every generator to 32 rows, which cost more
//     than the absent generators did.)
//
// The stages of all tiles of a CTA form one list, built once at set-up
// (union_tables_kernel): per stage the run offsets of its (generator, block)
// pairs and the descriptor words of its K-steps.  That keeps the roles' loops
// short, which is what bounds them: an MMA of 128 x 64 x 32 takes 48 cycles
// (its operands at 128 bytes a cycle from shared memory), but computing
// descriptors in the issuing thread cost 135-150 cycles an MMA, and a stage's
// hand-over between roles costs 200-400 cycles whatever the stage holds.  So
//   * the MMA warps issue from the table, and there are two of them where
//     every tile has two stages: a stage's hand-over (wait, proxy fence, commit)
//     keeps its warp about as long as its MMAs take, and the tensor pipe's queue
//     is too short to bridge it (see their loop);
//   * the producer warps form groups that take the stages in turn, each warp
//     with more copies a stage and fewer hand-overs;
//   * every wait is made by all lanes of a warp (one lane and a shuffle took
//     twice as long).
// A lane's unit -> (table word, source row, destination) map is the same in
// every stage and stays in registers, so a pass is a shuffle of the run
// offset, a compare, an add and the two limbs' cp.async.
//
// Measured on one B200 (1965 MHz), us, dense kernels -> one MMA warp -> two:
// r = 19, k = 9, dims 20 -> 28, 16 columns: d 179 -> 130 -> 92, d^T 228 -> 156 ->
// 127; r = 21, k = 10, dims 32 -> 40, 32 columns: d 1726 -> 1190 -> 1050, d^T
// 2429 -> 1411 -> 1260.  (With lexicographic tiles; the star order takes another 1
// to 5 %.)  With the other roles' work switched off the copies
// alone take 60 / 76 us at the first size and 614 / 745 at the second, the MMAs
// 74 / 78 and 555 / 591, the epilogue 73 / 95 and 728 / 859, and the hand-overs
// without any of them 59 / 60 and 348 / 377: no role is far above the others.
#pragma once

#include "bw_common.cuh"
#include "bw_koszul_i8_dev.cuh"
#include "bw_koszul_tables.cuh"
#include "tc_sm100.cuh"

#include <type_traits>

namespace bw {

namespace {

// Warp roles.  8 producer and 8 epilogue warps: every other split measured was
// slower or within 2 % (d, d^T at (19,9,20,28,16) / (21,10,32,40,32), ms: 8+8
// 0.092, 0.127 / 1.05, 1.26; 12+8 0.097, 0.129 / 1.04, 1.23; 8+12 0.098, 0.134 /
// 1.06, 1.27; 8+16 in two teams 0.097, 0.133 / 1.09, 1.30; 4+12 0.124, 0.189 /
// 1.45, 1.81).
namespace union_warps {
constexpr int producers = 8;
constexpr int mma = 8;                        // two; the first also allocates TMEM
constexpr int epilogue0 = 10;
constexpr int epilogue = 8;
constexpr int threads = (epilogue0 + epilogue) * 32;
}  // namespace union_warps

constexpr int kUnionPasses = 10;   // 32-unit passes a producer warp makes over a stage, at most
constexpr int kUnionSteps = 16;    // K-steps of a stage, at most
constexpr uint32_t kNoBlock = 0xFFFFFFFFu;
constexpr uint32_t kSkip = 0xFFFFFFFEu;      // table word of a generator slot past the tile's union
constexpr uint32_t kStepValid = 1u << 14;    // step word: this K-step exists (a descriptor's free bits)
constexpr uint32_t kStepLast = 1u << 15;     // step word 0: the issuing warp's last stage of its tile

struct I8Union {
    const int8_t* in[2];           // input +planes lo and hi: [blk][h][inner][16]; the -planes follow them
    int8_t* out[4];                // output planes lo, hi, -lo, -hi
    uint32_t* canon;               // CANON: the output as canonical residues, [n_blk * outer][width]
    int width;                     // columns of the caller's block (the rest of NB are zero padding)
    const uint32_t* start;         // [grid + 1]: first stage of every CTA's list
    const uint32_t* order;         // [tile][BT]: the tile's blocks, kNoBlock past the last one
    const uint32_t* words;         // [stage][gs * BT]: the neighbour run's 16-byte offset from the +plane,
                                   // kAbsent (rows of zeros) or kSkip (no rows)
    const uint32_t* steps;         // [stage][row]: low descriptor word of every K-step's maps, relative to them
    const int8_t* maps;            // B operand in its shared-memory layout, the zero chunk last
    const int32_t* diag;           // nullptr, or [n_blk * outer] balanced (scales the output)
    int* err;
    long long n_tiles;
    int r, inner, outer, ho;       // N = 2 * ho, ho = outer rounded up to 8
    int cpg;                       // 16-row chunks of a generator's 2 * inner K' rows
    int gs;                        // generators a stage (even when cpg is odd)
    int row;                       // words of a stage in `steps`: its K-steps rounded up to 4
    int issuers;                   // MMA warps: 2 where every tile has two stages or more, else 1
    int groups;                    // producer groups: group g fills the stages g, g + groups, ...
    int slots;
    uint32_t b_bytes, slot_bytes;
    int wide;                      // the epilogue reduces hi on its own (see plan_union)
    Mod mod;
    uint32_t wait_limit;           // tries of every pipeline wait (tc::kWaitLimit outside the failure tests)
    int late_wait;                 // nothing here depends on the kernel before: wait for it at the end only
                                   // (the input is then read at L2 alone, see pdl_wait())
    int hold_first_stage;          // failure tests only: CTA 0's MMA warp never sees its first stage
};

// Near-balanced representative of x, plus half: result - half = x (mod p) lies
// within (1/2 + |x| / 2^32) p + 1 of 0.  One Barrett step with the rounding
// folded in and no correction: the limb planes need any representative that
// two limbs hold (at most 255 * 127 + 127 in magnitude), not the balanced one.
__device__ __forceinline__ int32_t near_shifted(int32_t x, const Mod& mod) {
    const int32_t y = x + mod.half;
    return y - mulhi_s32(y, mod.barrett) * mod.p;
}

// One output from its two accumulators, shifted by half as above: lo + 255 hi,
// times the diagonal entry when scaling.  WIDE: the sums may pass 2^31 before
// the first reduction, so hi is reduced on its own.
template <bool WIDE>
__device__ __forceinline__ int32_t union_value(int32_t lo, int32_t hi, const Mod& mod, bool scale, int32_t dg) {
    const int32_t v = near_shifted(lo + 255 * (WIDE ? reduce_partial(hi, mod) : hi), mod);
    return scale ? near_shifted((v - mod.half) * dg, mod) : v;
}

// The limbs of four values v - half as packed bytes: with x = v - half + 127 +
// 255 * 128 (16 bits) and q = floor(x / 255), hi = q - 128 and lo = v - half -
// 255 hi, whose low byte is that of v - half + hi.
__device__ __forceinline__ void pack_limbs(const int32_t (&v)[4], const Mod& mod, uint32_t& lo, uint32_t& hi) {
    uint32_t l[4], h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t x = static_cast<uint32_t>(v[i] + (127 + 255 * 128 - mod.half));
        h[i] = __umulhi(x, 16843010u);   // ceil(2^32 / 255): exact for 16-bit x
        l[i] = x + h[i] + 1u;            // v - half + h + 128 (mod 256), as -(127 + 255 * 128) = 1 (mod 256)
    }
    lo = pack_bytes(l[0], l[1], l[2], l[3]) ^ 0x80808080u;
    hi = pack_bytes(h[0], h[1], h[2], h[3]) ^ 0x80808080u;
}

// CANON: the output goes to P.canon as canonical residues, else to the planes.
// (As a branch inside the plane form it cost a step 10 % at r = 19.)
template <int NB, bool CANON>
__global__ void __launch_bounds__(union_warps::threads, 1) i8_union_gemm_kernel(I8Union P) {
    namespace W = union_warps;
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int BT = 128 / NB;        // output blocks a tile
    constexpr int HG = NB / 16;         // 16-byte column groups a block row
    const int N = 2 * P.ho;
    const int kg = P.cpg * 16;          // K' rows of a generator
    const int KS = P.gs * kg;           // K' rows of a stage
    uint8_t* sB = smem;
    uint8_t* sA = smem + P.b_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(sA + static_cast<size_t>(P.slots) * P.slot_bytes);
    uint64_t* empty = full + P.slots;      // empty[s] lies slots * 8 bytes after full[s]
    uint64_t* accfull = empty + P.slots;
    uint64_t* accempty = accfull + 2;
    uint64_t* drained = accempty + 2;
    uint64_t* maps_in = drained + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(maps_in + 1);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);   // CTA give-up flag

    // the warp index through a shuffle, so that role and pass branches are uniform
    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x / 32), 0), lane = threadIdx.x % 32;
    const long long n_tiles = P.n_tiles;
    if (threadIdx.x == 0) {
        for (int s = 0; s < P.slots; ++s) {
            tc::mbar_init(&full[s], W::producers / P.groups * 32);   // per thread: its copies have landed
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&accfull[b], P.issuers);
            tc::mbar_init(&accempty[b], W::epilogue * 32);
        }
        tc::mbar_init(drained, P.issuers);
        tc::mbar_init(maps_in, 1);
        tc::fence_mbar_init();
        *abort = 0;
    }
    uint32_t tmem_cols = 32;
    // two buffers of an accumulator a warp
    while (tmem_cols < static_cast<uint32_t>(2 * N * P.issuers)) tmem_cols *= 2;
    if (warp == W::mma) {
        tc::tmem_alloc(tmem_slot, tmem_cols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    // Only now may the next kernel begin: one that shares the SM could otherwise
    // take TMEM that this CTA still waits for, and then wait for this kernel.
    pdl_trigger();
    const uint32_t tmem = *tmem_slot;
    const uint32_t stage0 = __ldg(P.start + blockIdx.x);
    const int n_stages = static_cast<int>(__ldg(P.start + blockIdx.x + 1) - stage0);

    const uint32_t full0 = tc::smem_u32(full), empty0 = tc::smem_u32(empty);
    const uint32_t accfull0 = tc::smem_u32(accfull), accempty0 = tc::smem_u32(accempty);

    if (warp < W::producers) {
        // ------------------------------------------------------------ producers
        // Unit x of a stage: generator q of the stage, block t of the tile and
        // row w of its run (h and u), x = (q * BT + t) * HG * inner + w; warp v
        // of a group takes the passes v, v + WPG, ... of 32 units.  Lane q * BT
        // + t holds that run's table word (loaded one stage ahead).
        const int wpg = W::producers / P.groups;         // warps a group
        const int group = warp / wpg, v = warp - group * wpg;
        const int run = HG * P.inner, words = P.gs * BT;
        const int units = words * run;
        uint32_t unit[kUnionPasses];    // w | word lane << 7 | destination (16-byte units in the slot) << 12
#pragma unroll
        for (int j = 0; j < kUnionPasses; ++j) {
            const int x = (v + j * wpg) * 32 + lane;
            const int qt = x / run, w = x - qt * run;
            const int q = qt / BT, t = qt - q * BT;
            const int h = w / P.inner, u = w - h * P.inner;
            unit[j] = static_cast<uint32_t>(w) | (static_cast<uint32_t>(qt & 31) << 7) |
                      (static_cast<uint32_t>((t * HG + h) * KS + q * kg + u) << 12);
        }
        const uint32_t hi_rows = static_cast<uint32_t>(P.inner) * 16u;   // a generator's hi rows follow its lo rows
        const uint32_t sA_u32 = tc::smem_u32(sA);
        // the group's stages: table pointer, slot, its barriers and its shared memory, all advanced by adding
        const bool has_word = lane < words;
        const uint32_t* tab = P.words + static_cast<size_t>(stage0 + group) * words + lane;
        const int tab_step = P.groups * words;
        int slot = group;      // groups <= slots
        uint32_t parity = 1;   // of the slot's release that a fill waits for
        uint32_t bar = empty0 + static_cast<uint32_t>(group) * 8u;
        uint32_t slotA = sA_u32 + static_cast<uint32_t>(group) * P.slot_bytes;
        const uint32_t bar_step = static_cast<uint32_t>(P.groups) * 8u, slots_bar = static_cast<uint32_t>(P.slots) * 8u;
        const uint32_t slotA_step = static_cast<uint32_t>(P.groups) * P.slot_bytes;
        const uint32_t ring_bytes = static_cast<uint32_t>(P.slots) * P.slot_bytes;
        // two stages' words in flight: the list streams from DRAM
        uint32_t word0 = has_word && group < n_stages ? __ldg(tab) : kSkip;
        uint32_t word1 = has_word && group + P.groups < n_stages ? __ldg(tab + tab_step) : kSkip;
        tab += 2 * tab_step;
        if (!P.late_wait) pdl_wait();   // the input planes; the maps and lists are constant
        for (int left = n_stages - group; left > 0; left -= P.groups) {
            const uint32_t word = word0;
            word0 = word1;
            if (has_word && left > 2 * P.groups) word1 = __ldg(tab);
            tab += tab_step;
            if (!tc::warp_wait(bar, parity, abort, P.err, tc::ERR_WAIT_EMPTY, P.wait_limit)) break;
#pragma unroll
            for (int j = 0; j < kUnionPasses; ++j) {
                const int x0 = (v + j * wpg) * 32;
                if (x0 >= units) break;
                const uint32_t o16 = __shfl_sync(0xffffffffu, word, (unit[j] >> 7) & 31u);
                if (x0 + lane < units && o16 != kSkip) {
                    // an absent neighbour's rows are zero-filled by the copy itself (source size 0)
                    const bool present = o16 != kAbsent;
                    const uint32_t src16 = (present ? o16 : 0u) + (unit[j] & 127u);
                    const uint32_t nbytes = present ? 16u : 0u;
                    const uint32_t dst = slotA + (unit[j] >> 12) * 16u;
                    // .cg: late_wait allows no read of the input through L1
                    tc::cp_async16_zfill(dst, P.in[0] + static_cast<size_t>(src16) * 16u, nbytes);
                    tc::cp_async16_zfill(dst + hi_rows, P.in[1] + static_cast<size_t>(src16) * 16u, nbytes);
                }
            }
            tc::cp_async_arrive_noinc(bar - slots_bar);   // full[slot]: when this thread's copies have landed
            slot += P.groups;
            bar += bar_step;
            slotA += slotA_step;
            if (slot >= P.slots) {
                slot -= P.slots;
                bar -= slots_bar;
                slotA -= ring_bytes;
                parity ^= 1u;
            }
        }
        tc::cp_async_wait_all();   // no copy may still be landing when the CTA exits
    } else if (warp < W::epilogue0) {
        // ------------------------------------------------------------ MMA issuers
        // A whole warp waits and walks its stages, lane k holding K-step k's
        // descriptor word (loaded four stages ahead), and one elected lane
        // issues: an MMA costs a shuffle and no descriptor arithmetic.  The
        // tensor pipe's queue is short, so while a warp waits for a stage, takes
        // the proxy fence and commits (about 400 cycles) nothing runs behind the
        // MMAs that it has issued (6 of 48 cycles a stage at the first size
        // above): two warps take the stages in turn, each with an accumulator of
        // its own.
        const int issuer = warp - W::mma;
        if (issuer < P.issuers) {
            // the maps, in pieces of at most 32 KB; nothing leaves this block before they have landed
            if (issuer == 0 && lane == 0) {
                tc::mbar_arrive_expect_tx(maps_in, P.b_bytes);
                for (uint32_t off = 0; off < P.b_bytes; off += 32768u)
                    tc::bulk_g2s(sB + off, P.maps + off, min(32768u, P.b_bytes - off), maps_in);
            }
            __syncwarp();
            const uint32_t idesc = tc::idesc_i8(128, N, true, false);
            const uint32_t a_hi = tc::desc_hi(static_cast<uint32_t>(KS) * 16u), b_hi = tc::desc_hi(128u);
            const uint32_t a_slot0 = tc::desc_lo(tc::smem_u32(sA), 128u), b0 = tc::desc_lo(tc::smem_u32(sB), 0u);
            const uint32_t slot_units = P.slot_bytes >> 4, step_units = static_cast<uint32_t>(P.issuers) * slot_units;
            const bool has_word = lane < P.row;
            const int tab_step = P.issuers * P.row;
            const uint32_t* tab = P.steps + static_cast<size_t>(stage0 + issuer) * P.row + lane;
            uint32_t ahead[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
                ahead[q] = has_word && issuer + q * P.issuers < n_stages ? __ldg(tab + q * tab_step) : 0u;
            tab += 4 * tab_step;
            const uint32_t acc0 = tmem + static_cast<uint32_t>(issuer * N);
            const uint32_t buf_cols = static_cast<uint32_t>(P.issuers * N);
            uint32_t acc = 0, buf = 0, acc_parity = 1;   // acc = 0: the next stage is the warp's first of a tile
            int slot = issuer % P.slots;
            uint32_t bar = full0 + static_cast<uint32_t>(slot) * 8u;
            uint32_t parity = static_cast<uint32_t>(issuer / P.slots) & 1u;
            uint32_t a_lo = a_slot0 + static_cast<uint32_t>(slot) * slot_units;
            const bool ok = tc::warp_wait(tc::smem_u32(maps_in), 0, nullptr, P.err, tc::ERR_WAIT_FINAL);
            // The producers fill nothing before the kernel before this one is done:
            // the limit of the waits below is for this kernel's own work.
            if (!P.late_wait) pdl_wait();
            // failure tests: CTA 0 waits for its first stage on a barrier that
            // nothing completes before the final drain, so the wait runs out
            const bool held = P.hold_first_stage && blockIdx.x == 0 && issuer == 0 && ok &&
                              !tc::warp_wait(tc::smem_u32(drained), 0, abort, P.err, tc::ERR_WAIT_FULL, P.wait_limit);
            for (int left = ok && !held ? n_stages - issuer : 0; left > 0; left -= P.issuers) {
                const uint32_t word = ahead[0];
#pragma unroll
                for (int q = 0; q < 3; ++q) ahead[q] = ahead[q + 1];
                if (has_word && left > 4 * P.issuers) ahead[3] = __ldg(tab);
                tab += tab_step;
                const int n = __popc(__ballot_sync(0xffffffffu, (word & kStepValid) != 0));
                const bool last = __any_sync(0xffffffffu, (word & kStepLast) != 0);
                const uint32_t bw = (word & 0x3FFF3FFFu) + b0;
                if (acc == 0 && !tc::warp_wait(accempty0 + buf * 8u, acc_parity, abort, P.err, tc::ERR_WAIT_ACCUM_FREE,
                                               P.wait_limit))
                    break;
                if (!tc::warp_wait(bar, parity, abort, P.err, tc::ERR_WAIT_FULL, P.wait_limit)) break;
                tc::fence_proxy_async_smem();
                tc::tc_fence_after();
                const uint32_t dcol = acc0 + buf * buf_cols;
#pragma unroll
                for (int k = 0; k < kUnionSteps; ++k) {
                    if (k >= n) break;
                    const uint32_t b = __shfl_sync(0xffffffffu, bw, k);
                    tc::mma_i8_elect(dcol, tc::desc_make(a_lo + static_cast<uint32_t>(k) * (512u >> 4), a_hi),
                                     tc::desc_make(b, b_hi), idesc, acc);
                    acc = 1;
                }
                tc::mma_commit_elect(bar + static_cast<uint32_t>(P.slots) * 8u);   // empty[slot]
                if (last) {
                    tc::mma_commit_elect(accfull0 + buf * 8u);
                    acc = 0;
                    buf ^= 1u;
                    acc_parity ^= buf == 0 ? 1u : 0u;
                }
                slot += P.issuers;
                bar += static_cast<uint32_t>(P.issuers) * 8u;
                a_lo += step_units;
                if (slot >= P.slots) {   // at least two slots
                    slot -= P.slots;
                    bar -= static_cast<uint32_t>(P.slots) * 8u;
                    a_lo -= static_cast<uint32_t>(P.slots) * slot_units;
                    parity ^= 1u;
                }
            }
            // drain: every MMA issued above completes before TMEM is released
            // (this wait ignores the give-up flag; issued MMAs always finish)
            tc::mma_commit_elect(tc::smem_u32(drained));
            tc::warp_wait(tc::smem_u32(drained), 0, nullptr, P.err, tc::ERR_WAIT_FINAL);
        }
    } else {
        // ------------------------------------------------------------ epilogue
        // warp & 3 is the TMEM lane quadrant a warp may read; the warps of a
        // quadrant split the 16-column output chunks between them.
        const int quad = warp & 3;
        constexpr int EPQ = W::epilogue / 4;
        const int part = (warp - W::epilogue0) >> 2;
        const int m = quad * 32 + lane;            // tile row = (block t, column j)
        const int t = m / NB, j = m % NB;
        const uint32_t lane_off = static_cast<uint32_t>(quad * 32) << 16;
        const int chunks = (P.outer + 15) / 16;
        const uint32_t h_off = static_cast<uint32_t>((j >> 4) * P.outer * 16);
        const bool vec = (P.outer & 3) == 0;       // whole int4 of the diagonal (its base is 16-byte aligned)
        // a loop for every case, so that each is short (one loop for all four: 235
        // instead of 232 us a step at r = 19, k = 9, 20 -> 28, 16 columns)
        auto epilogue = [&](auto wide_c, auto scale_c) {
            constexpr bool WIDE = decltype(wide_c)::value, SCALE = decltype(scale_c)::value;
            // diagonal entries of chunk c of block bk
            auto load_diag = [&](int32_t (&dg)[16], uint32_t bk, int c) {
                const bool any = SCALE && bk != kNoBlock;
                const int32_t* src = P.diag + static_cast<long long>(bk) * P.outer + c * 16;
                if (vec) {
#pragma unroll
                    for (int o4 = 0; o4 < 4; ++o4) {
                        const int4 d4 = any && c * 16 + o4 * 4 < P.outer ? __ldg(reinterpret_cast<const int4*>(src) + o4)
                                                                         : make_int4(0, 0, 0, 0);
                        dg[o4 * 4] = d4.x;
                        dg[o4 * 4 + 1] = d4.y;
                        dg[o4 * 4 + 2] = d4.z;
                        dg[o4 * 4 + 3] = d4.w;
                    }
                } else {
#pragma unroll
                    for (int oo = 0; oo < 16; ++oo) dg[oo] = any && c * 16 + oo < P.outer ? __ldg(src + oo) : 0;
                }
            };
            if (!P.late_wait) pdl_wait();   // the output planes may still be read by earlier kernels
            // a tile's first chunk is loaded one tile ahead (the diagonal streams from DRAM)
            int32_t dg_next[16];
            auto block_of = [&](long long tl) { return tl < n_tiles ? __ldg(P.order + tl * BT + t) : kNoBlock; };
            uint32_t blk_next = block_of(blockIdx.x), blk_after = block_of(blockIdx.x + gridDim.x);
            load_diag(dg_next, blk_next, part);
            long long tcount = 0;
            for (long long tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++tcount) {
                const int buf = static_cast<int>(tcount & 1);
                const uint32_t aph = static_cast<uint32_t>((tcount >> 1) & 1);
                const uint32_t blk_now = blk_next;
                const bool valid = blk_now != kNoBlock;
                const long long blk = blk_now;
                blk_next = blk_after;
                blk_after = block_of(tile + 2ll * gridDim.x);
                int32_t dg[16];
#pragma unroll
                for (int oo = 0; oo < 16; ++oo) dg[oo] = dg_next[oo];
                load_diag(dg_next, blk_next, part);
                if (!tc::warp_wait(accfull0 + static_cast<uint32_t>(buf) * 8u, aph, abort, P.err, tc::ERR_WAIT_ACCUM,
                                   P.wait_limit))
                    break;
                tc::tc_fence_after();
                const uint32_t col0 = tmem + lane_off + static_cast<uint32_t>(buf * P.issuers * N);
                const long long base = blk * static_cast<long long>(NB) * P.outer + h_off;
                for (int c = part; c < chunks; c += EPQ) {
                    const int o0 = c * 16;
                    if (c != part) load_diag(dg, blk_now, c);
                    // this lane's 16 outputs (o0..o0+15 of its column j) as limb bytes; only groups of
                    // eight columns that reach below outer are read (the accumulator has ho of each limb)
                    uint32_t lw[4] = {0, 0, 0, 0}, hw[4] = {0, 0, 0, 0};
                    const int live = P.outer - o0;
#pragma unroll
                    for (int h8 = 0; h8 < 2; ++h8) {
                        if (h8 * 8 >= live) break;
                        int32_t lo[8], hi[8];
                        const uint32_t cb = col0 + static_cast<uint32_t>(o0 + h8 * 8);
                        tc::tmem_ld8(cb, lo);
                        tc::tmem_ld8(cb + P.ho, hi);
                        if (P.issuers == 2) {   // the second warp's sums
                            int32_t lo2[8], hi2[8];
                            tc::tmem_ld8(cb + N, lo2);
                            tc::tmem_ld8(cb + N + P.ho, hi2);
                            tc::tmem_ld_wait();
#pragma unroll
                            for (int q = 0; q < 8; ++q) {
                                lo[q] += lo2[q];
                                hi[q] += hi2[q];
                            }
                        } else {
                            tc::tmem_ld_wait();
                        }
#pragma unroll
                        for (int g4 = 0; g4 < 2; ++g4) {
                            if (h8 * 8 + g4 * 4 >= live) break;
                            int32_t v[4];
#pragma unroll
                            for (int oi = 0; oi < 4; ++oi) {
                                const int o = g4 * 4 + oi;
                                v[oi] = union_value<WIDE>(lo[o], hi[o], P.mod, SCALE, dg[h8 * 8 + o]);
                            }
                            if constexpr (CANON) {   // a row's columns are neighbouring lanes: whole sectors
                                const int o = o0 + h8 * 8 + g4 * 4;
                                uint32_t* at = P.canon + (blk * P.outer + o) * P.width + j;
                                if (valid && j < P.width)
#pragma unroll
                                    for (int oi = 0; oi < 4; ++oi)
                                        if (o + oi < P.outer)
                                            at[oi * P.width] =
                                                to_canonical(reduce_balanced_fast(v[oi] - P.mod.half, P.mod), P.mod);
                            } else {
                                pack_limbs(v, P.mod, lw[h8 * 2 + g4], hw[h8 * 2 + g4]);
                            }
                        }
                    }
                    if constexpr (CANON) continue;
                    // transposed, lane L of the half-warp holds output row o0 + L: 16 bytes, one per j
                    transpose16(lw, lane);
                    transpose16(hw, lane);
                    const int o = o0 + (lane & 15);
                    if (valid && o < P.outer) {
                        const long long at = base + o * 16;
                        *reinterpret_cast<uint4*>(P.out[PL_LO] + at) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
                        *reinterpret_cast<uint4*>(P.out[PL_HI] + at) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                        *reinterpret_cast<uint4*>(P.out[PL_NLO] + at) =
                            make_uint4(neg_bytes4(lw[0]), neg_bytes4(lw[1]), neg_bytes4(lw[2]), neg_bytes4(lw[3]));
                        *reinterpret_cast<uint4*>(P.out[PL_NHI] + at) =
                            make_uint4(neg_bytes4(hw[0]), neg_bytes4(hw[1]), neg_bytes4(hw[2]), neg_bytes4(hw[3]));
                    }
                }
                tc::tc_fence_before();
                tc::mbar_arrive(&accempty[buf]);
            }
        };
        using Yes = std::true_type;
        using No = std::false_type;
        if (P.diag != nullptr)
            P.wide ? epilogue(Yes{}, Yes{}) : epilogue(No{}, Yes{});
        else
            P.wide ? epilogue(Yes{}, No{}) : epilogue(No{}, No{});
    }

    tc::tc_fence_before();
    __syncthreads();
    if (warp == W::mma) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, tmem_cols);
    }
    if (P.late_wait) pdl_wait();   // this kernel's completion implies that of all kernels before it
}

// ---- the order of the blocks
//
// The fewer generators the blocks of a tile have between them, the fewer rows
// it gathers and multiplies.  Four blocks that agree but for the place of one
// element have the least: d's T = C u {x} lack only C's generators in common,
// d^T's S = Q \ {x} lie in one set Q of k + 1.  So the elements are cut into
// quads (from the last element down); a block whose set meets some quad in one
// element (d) or three (d^T), the last such quad, goes with the three blocks
// that differ from it there (its star: they have the same last such quad, so
// stars are disjoint).  The blocks without such a quad go four by four as they
// come.  Both kinds follow the lexicographic order of their first block, which
// keeps the gathered rows of neighbouring tiles close.  A tile is one such four
// (32 columns) or two.  Generators of a tile, lexicographic tiles -> these: r = 21,
// k = 10, tiles of four: d 14.4 -> 13.2, d^T 12.7 -> 11.4; r = 19, k = 9, tiles of
// eight: d 14.0 -> 13.6, d^T 12.6 -> 11.9.  (us: d^T at r = 20,
// k = 8, 21 -> 29, 32 columns and a step of r = 23, k = 11, 32 -> 40, 32 columns:
// 552 -> 548 with its conversion, 13100 -> 12750.)

// First element of the set's star quad, or -1.
__device__ __forceinline__ int star_quad(uint32_t set, int r, bool forward) {
    for (int base = r - 4; base >= 0; base -= 4)
        if (__popc(set >> base & 15u) == (forward ? 1 : 3)) return base;
    return -1;
}

constexpr int kOrderThreads = 256;

// 0: no star; 1: first of its star (lexicographically); 2: another of it.
__device__ __forceinline__ int star_role(uint32_t set, int base, bool forward) {
    return base < 0 ? 0 : (set >> base & 15u) == (forward ? 1u : 7u) ? 1 : 2;
}

// counts[CTA] = its stars and its blocks without one.
__global__ void __launch_bounds__(kOrderThreads) order_count_kernel(uint2* counts, long long n_blk, int r, int size,
                                                                    bool forward,
                                                                    const __grid_constant__ BinomTable B) {
    const long long blk = blockIdx.x * static_cast<long long>(kOrderThreads) + threadIdx.x;
    int role = 2;
    if (blk < n_blk) {
        const uint32_t set = subset_of(static_cast<uint32_t>(blk), r, size, B);
        role = star_role(set, star_quad(set, r, forward), forward);
    }
    const unsigned stars = __syncthreads_count(role == 1), rest = __syncthreads_count(role == 0);
    if (threadIdx.x == 0) counts[blockIdx.x] = make_uint2(stars, rest);
}

// Exclusive sums in place; the totals follow the last entry.  One CTA of 1024.
__global__ void __launch_bounds__(1024) order_scan_kernel(uint2* counts, int n) {
    __shared__ uint2 part[1024];
    const int per = (n + 1023) / 1024, lo = min(n, static_cast<int>(threadIdx.x) * per), hi = min(n, lo + per);
    uint2 sum = make_uint2(0, 0);
    for (int i = lo; i < hi; ++i) sum = make_uint2(sum.x + counts[i].x, sum.y + counts[i].y);
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int d = 1; d < 1024; d *= 2) {
        const uint2 v = static_cast<int>(threadIdx.x) >= d ? part[threadIdx.x - d] : make_uint2(0, 0);
        __syncthreads();
        part[threadIdx.x].x += v.x;
        part[threadIdx.x].y += v.y;
        __syncthreads();
    }
    uint2 at = make_uint2(part[threadIdx.x].x - sum.x, part[threadIdx.x].y - sum.y);
    for (int i = lo; i < hi; ++i) {
        const uint2 c = counts[i];
        counts[i] = at;
        at = make_uint2(at.x + c.x, at.y + c.y);
    }
    if (threadIdx.x == 1023) counts[n] = at;
}

// Writes the stars to order and the other blocks, in order, to rest; with l stars
// and q other blocks before it, a star is the four number l + ceil(q / 4), and
// the other blocks q .. q + 3 (4 | q) are the four number l + q / 4, kept in four[q / 4].
__global__ void __launch_bounds__(kOrderThreads) order_place_kernel(const uint2* counts, uint32_t* order, uint32_t* rest,
                                                                    uint32_t* four, long long n_blk, int r, int size,
                                                                    bool forward,
                                                                    const __grid_constant__ BinomTable B) {
    __shared__ uint2 warps[kOrderThreads / 32];
    const long long blk = blockIdx.x * static_cast<long long>(kOrderThreads) + threadIdx.x;
    const unsigned warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    uint32_t set = 0;
    int base = -1, role = 2;
    if (blk < n_blk) {
        set = subset_of(static_cast<uint32_t>(blk), r, size, B);
        base = star_quad(set, r, forward);
        role = star_role(set, base, forward);
    }
    const uint32_t stars = __ballot_sync(0xffffffffu, role == 1), others = __ballot_sync(0xffffffffu, role == 0);
    if (lane == 0) warps[warp] = make_uint2(__popc(stars), __popc(others));
    __syncthreads();
    const uint32_t below = (1u << lane) - 1;
    uint32_t l = counts[blockIdx.x].x + __popc(stars & below), q = counts[blockIdx.x].y + __popc(others & below);
    for (unsigned w = 0; w < warp; ++w) {
        l += warps[w].x;
        q += warps[w].y;
    }
    if (role == 1) {
        uint32_t* out = order + 4ull * (l + (q + 3) / 4);
        const uint32_t rem = set & ~(15u << base);
        for (int j = 0; j < 4; ++j)   // ascending ranks: d's one element rises, d^T's missing one falls
            out[j] = rank_of(rem | (forward ? 1u << j : 15u & ~(8u >> j)) << base, r, size, B);
    } else if (role == 0) {
        rest[q] = static_cast<uint32_t>(blk);
        if (q % 4 == 0) four[q / 4] = l + q / 4;
    }
}

// Lexicographic order.
__global__ void __launch_bounds__(kOrderThreads) order_plain_kernel(uint32_t* order, uint32_t n_blk, uint32_t n_order) {
    const uint32_t i = blockIdx.x * kOrderThreads + threadIdx.x;
    if (i < n_order) order[i] = i < n_blk ? i : kNoBlock;
}

__global__ void __launch_bounds__(kOrderThreads) order_rest_kernel(const uint2* total, const uint32_t* rest,
                                                                   const uint32_t* four, uint32_t* order) {
    const uint32_t q = blockIdx.x * kOrderThreads + threadIdx.x;
    if (q < total->y) order[4ull * four[q / 4] + q % 4] = rest[q];
}

// The union kernel's stage list (see I8Union): tile t's stages start at
// tile_stage[t]; mask[t] is its union, inc the dense [n_blk][r] table
// (neighbour rank | negative << 31, or kAbsent).
__global__ void union_tables_kernel(const uint32_t* __restrict__ inc, const uint32_t* __restrict__ order,
                                    const uint32_t* __restrict__ mask, const uint32_t* __restrict__ tile_stage,
                                    uint32_t* __restrict__ words, uint32_t* __restrict__ steps, long long n_tiles, int r,
                                    int bt, int gs, int cpg, int n_cols, int row, int issuers, uint32_t run16,
                                    uint32_t neg16) {
    const long long tile = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (tile >= n_tiles) return;
    const uint32_t all = mask[tile];
    const int cnt = __popc(all), stages = (cnt + gs - 1) / gs;
    uint32_t* w = words + static_cast<size_t>(tile_stage[tile]) * gs * bt;
    uint32_t left = all;
    for (int q = 0; q < stages * gs; ++q) {
        const int i = left ? __ffs(left) - 1 : -1;
        left &= left - 1;
        for (int t = 0; t < bt; ++t) {
            uint32_t v = kSkip;
            if (i >= 0) {
                const uint32_t blk = order[tile * bt + t];
                const uint32_t e = blk != kNoBlock ? inc[static_cast<size_t>(blk) * r + i] : kAbsent;
                v = e == kAbsent ? kAbsent : (e >> 31 ? neg16 : 0u) + (e & 0x7FFFFFFFu) * run16;
            }
            w[q * bt + t] = v;
        }
    }
    // a K-step takes the chunks 2k and 2k + 1 of the stage's generators, back
    // to back; a chunk past the last generator is the zero chunk
    left = all;
    for (int s = 0; s < stages; ++s) {
        uint32_t* out = steps + (static_cast<size_t>(tile_stage[tile]) + s) * row;
        const int chunks = min(gs, cnt - s * gs) * cpg;
        uint32_t at[2] = {0, 0};
        int c = 0;
        for (int q = 0; q < gs && left; ++q, left &= left - 1)
            for (int j = 0; j < cpg; ++j, ++c) {
                at[c & 1] = static_cast<uint32_t>((__ffs(left) - 1) * cpg + j) * n_cols;
                if ((c & 1) || c == chunks - 1) {
                    if (!(c & 1)) at[1] = static_cast<uint32_t>(r * cpg) * n_cols;
                    out[c >> 1] = at[0] | ((at[1] - at[0]) << 16) | kStepValid |
                                  (c <= 1 && s + issuers >= stages ? kStepLast : 0u);
                }
            }
        for (int k = (chunks + 1) / 2; k < row; ++k) out[k] = 0;
    }
}

}  // namespace

}  // namespace bw
