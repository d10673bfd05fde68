// INT8-limb tensor-core form of the synthetic Koszul operator (tcgen05 kind::i8).
//
// Every residue x is stored in HBM as two signed 8-bit limbs in base 255:
// x = 255*hi + lo, both in [-127, 127].  Inputs and maps are split from the
// balanced residue (|x| <= (p-1)/2 <= 16383 = 255 * 64 + 63: hi in [-64, 64]);
// the union kernel stores any representative that two limbs hold (|x| <= 255 *
// 127 + 127), so what reads a stored block relies on 127 for either limb.  The
// symmetric range makes negation exact in int8, which is how the Koszul signs
// are applied while operands are staged.
//
// d and d^T are one gather-GEMM.  bw_koszul_i8_union.cuh has the kernel that runs
// it wherever its resident maps leave room for stages; this file has the dense
// kernels for the other sizes (described here), the conversions, the projection
// and the host side of both.  For a tile of 128/n output blocks (n = block width)
// the output is
//   out[blk][o][j] = sum_{i < r} sum_{u < inner} A[(blk, j)][(i, u)] * Bm[o][(i, u)]
// with A[(blk, j)][(i, u)] = sign * in[nbr(blk, i)][u][j] (zero when the
// generator i is not incident to blk) and Bm = the r maps side by side.  The
// tile is an M = 128 GEMM: A = the gathered input blocks (MN-major in shared
// memory: 16 limbs of one input row form one 16-byte core-matrix row),
// B = the maps' lo and hi limbs stacked along N (K-major, resident in shared
// memory for the whole kernel), K = r * inner in steps of 32.  Two MMAs per
// K-step (A = input lo limbs, A = input hi limbs) give four int32 partial
// products per output, recombined exactly mod p in the epilogue:
//   x*m = lo*lo + 255*(lo*hi + hi*lo) + 255^2*hi*hi.
// int32 accumulation is exact: |K * 127 * 127| < 2^24 for K <= 1024.
//
// Limb planes in HBM: four planes per block array (lo, hi, -lo, -hi), each
// laid out [blk][h][u][16 bytes] (h = j / 16), so that every (block, h) is one
// contiguous run of inner * 16 bytes.  The producers fill a stage with 16-byte
// cp.async copies (one per K' row, limb and column group) from the +plane or
// the -plane by the Koszul sign; the rows of an absent generator (about half
// of all rows) are zero-filled by the same copy with source size 0, which
// reads nothing (a common zero source in global memory would funnel that half
// of the traffic through one L2 slice).
// The epilogue writes all four planes of its output.
//
// Warp roles (persistent, one CTA per SM; PW = 8 or 16 producer warps, chosen
// per direction by the set-up autotuner):
//   warps 0..PW-1  producers: each owns one of the tile's output blocks (or,
//               with fewer blocks per tile than producer warps, a share of one
//               block's rows) and keeps their incidence rows in registers (one
//               generator per lane); every thread arrives on the stage barrier
//               through cp.async.mbarrier.arrive.noinc when its copies have
//               landed;
//   warp PW     allocates TMEM and issues tcgen05.mma / tcgen05.commit (after a
//               proxy fence: the stage was written through the generic proxy);
//   the rest    epilogue (eight warps with PW = 8, four with PW = 16), one or two
//               warps per TMEM lane quadrant: tcgen05.ld the four partials,
//               recombine, reduce mod p, scale by D (d^T only), split into
//               limbs, transpose 16 x 16 bytes per half-warp and store one
//               16-byte plane row per lane.
// Stages are tracked with mbarriers; accumulators are double-buffered in TMEM.
// Every wait is bounded and polls only a shared-memory give-up flag: on a
// timeout the kernel records an error code, all roles wind down, in-flight
// copies and MMAs are drained and TMEM is freed.
#include "bw_koszul.cuh"
#include "bw_koszul_i8_dev.cuh"
#include "bw_koszul_tables.cuh"
#include "bw_koszul_i8_union.cuh"
#include "tc_sm100.cuh"

#include <cuda.h>   // CUtensorMap and cuTensorMapEncodeTiled's types (the function is reached through the runtime)

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

namespace bw {

namespace {

constexpr int kEpilogueWarps = 8;                 // hybrid kernel; per TMEM lane quadrant: kEpilogueWarps / 4
constexpr int kMaxRowTable = 2048;    // bytes of the K'-row -> generator table

struct I8Dir {
    const int8_t* in[4];      // input planes lo, hi, -lo, -hi: [blk][h][inner][16]
    long long in_neg_off;     // bytes from an input +plane to its -plane (they share one allocation)
    int8_t* out[4];           // output planes, same layout with `outer`
    const uint32_t* inc;      // [n_blk][r]: neighbour rank | negative << 31, or kAbsent
    const int8_t* b_tiles;    // B operand, already in its shared-memory layout
    const int32_t* diag;      // nullptr, or [n_blk * outer] balanced (scales the output)
    int* err;
    long long n_blk;
    int r, inner, outer, half;   // N = 2 * half, half = outer rounded up to 16
    int gi;                      // generators per stage
    int stages_per_tile;         // ceil(r / gi)
    int ks_full;                 // K-steps of a full stage (gi * inner rows padded to a multiple of 32)
    int ks_last;                 // K-steps of the last stage
    int slots;                   // pipeline depth
    uint32_t b_bytes, slot_bytes, limb_bytes;
    Mod mod;
    int32_t c1, c2;              // 255 and 255^2 mod p, balanced
    uint32_t wait_limit;         // tries of every pipeline wait (tc::kWaitLimit outside the failure tests)
    int hold_first_stage;        // failure tests only: CTA 0's MMA thread never sees its first stage
    // hybrid producer (i8_gather_hybrid_kernel)
    const int4* rows4;           // [n_blk][groups]: plane rows of the four generators of a group (h = 0)
    int groups;                  // ceil(r / 4)
    int gs;                      // groups per stage
    int inner_pad;               // K' rows of a generator: inner rounded up to even (128-byte aligned groups)
    int32_t row_oob;             // a plane row past the input tensor (2 * input blocks * HG): zero-filled
    int t_tma;                   // hybrid producer: output blocks of a tile gathered by TMA (the rest by cp.async)
    uint32_t tx_full, tx_last;   // bytes a full / the last stage of a tile receives
};

// The gather-GEMM epilogue's value of one output, balanced: ll + 255 (lh + hl)
// + 255^2 hh, times the diagonal entry dg when scaling (d^T).  The sum before
// the last reduction stays below 1.11e9 in magnitude: |ll| <= 1024 * 127^2
// (at most 1024 K rows), 255 * |lh + hl reduced| < 255 * 2p and
// |c2 * hh reduced| < 16383 * 2p; the scaled product is below 2p * (p - 1) / 2.
// Both are within reduce_balanced_fast's range.
__device__ __forceinline__ int32_t epilogue_value(int32_t ll, int32_t lhhl, int32_t hh, const Mod& mod, int32_t c2,
                                                  bool scale, int32_t dg) {
    const int32_t t = ll + 255 * reduce_partial(lhhl, mod) + c2 * reduce_partial(hh, mod);
    return reduce_balanced_fast(scale ? reduce_partial(t, mod) * dg : t, mod);
}

template <int NB, int PW>
__global__ void __launch_bounds__(GatherWarps<PW>::threads, 1) i8_gather_gemm_kernel(I8Dir P) {
    using W = GatherWarps<PW>;
    constexpr int kProducerWarps = W::producers, kMmaWarp = W::mma, kEpilogueWarp0 = W::epilogue0;
    constexpr int kGatherEpilogueWarps = W::epilogue;
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int BT = 128 / NB;        // output blocks per tile
    constexpr int HG = NB / 16;         // 16-byte column groups per block row
    const int N = 2 * P.half;
    uint8_t* sB = smem;
    uint8_t* sA = smem + P.b_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(sA + static_cast<size_t>(P.slots) * P.slot_bytes);
    uint64_t* empty = full + P.slots;
    uint64_t* accfull = empty + P.slots;
    uint64_t* accempty = accfull + 2;
    uint64_t* drained = accempty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);   // CTA give-up flag
    uint8_t* il_of_row = reinterpret_cast<uint8_t*>(tmem_slot + 4);   // K' row of a slot -> generator slot

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const long long n_tiles = (P.n_blk + BT - 1) / BT;

    // B operand: global -> shared (generic stores, made visible to the tensor core below)
    for (uint32_t off = threadIdx.x * 16; off < P.b_bytes; off += blockDim.x * 16)
        *reinterpret_cast<int4*>(sB + off) = __ldg(reinterpret_cast<const int4*>(P.b_tiles + off));
    tc::fence_proxy_async_smem();
    if (threadIdx.x == 0) {
        for (int s = 0; s < P.slots; ++s) {
            tc::mbar_init(&full[s], kProducerWarps * 32);   // per thread: its copies have landed
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&accfull[b], 1);
            tc::mbar_init(&accempty[b], kGatherEpilogueWarps * 32);
        }
        tc::mbar_init(drained, 1);
        tc::fence_mbar_init();
        *abort = 0;
    }
    const uint32_t tmem_cols = (4 * N <= 256) ? 256u : 512u;
    if (warp == kMmaWarp) {
        tc::tmem_alloc(tmem_slot, tmem_cols);
        tc::tmem_relinquish();
    }
    const int KS = P.ks_full * 32;                       // K' rows of a slot group (gi * inner, padded)
    for (int w = threadIdx.x; w < KS; w += blockDim.x) il_of_row[w] = static_cast<uint8_t>(w / P.inner);
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp < kProducerWarps) {
        // ------------------------------------------------------------ producers
        // Warp w stages the output blocks t = w % GROUPS, + GROUPS, ... of each tile.  Lane
        // i holds, for those blocks, where generator i's neighbour run starts: its offset
        // from the limb's +plane in 16-byte units, the -plane's offset added for a negative
        // sign, or kAbsent (read by shuffle; the next tile's entries are loaded one tile
        // ahead).  The warp's lanes walk the K' rows of every (limb, block, column group):
        // a 16-byte cp.async from the +plane or -plane of the neighbour block,
        // or a zero-filling one (source size 0) for an absent generator.  Each
        // thread arrives on the stage barrier once, through
        // cp.async.mbarrier.arrive.noinc, when its copies have landed.
        // More producer warps than blocks: RPW warps share a block, interleaving its rows.
        constexpr int RPW = kProducerWarps > BT ? kProducerWarps / BT : 1;
        constexpr int GROUPS = kProducerWarps / RPW;                     // distinct block positions
        constexpr int TPW = (BT + GROUPS - 1) / GROUPS;                  // blocks per producer warp
        const int group = warp % GROUPS, sub = warp / GROUPS;
        const uint32_t neg16 = static_cast<uint32_t>(P.in_neg_off >> 4);
        const uint32_t run16 = static_cast<uint32_t>(HG * P.inner);   // 16-byte rows of one neighbour block
        auto load_inc = [&](long long tile, uint32_t (&dst)[TPW]) {
#pragma unroll
            for (int k = 0; k < TPW; ++k) {
                const int t = group + k * GROUPS;
                const long long blk = tile * BT + t;
                const uint32_t e = (tile < n_tiles && t < BT && blk < P.n_blk && lane < P.r)
                                       ? __ldg(P.inc + blk * P.r + lane) : kAbsent;
                dst[k] = e == kAbsent ? kAbsent : ((e >> 31) ? neg16 : 0u) + (e & 0x7FFFFFFFu) * run16;
            }
        };
        const uint32_t sA_u32 = tc::smem_u32(sA);
        SlotRing ring(P.slots);
        bool ok = true;
        uint32_t incr[TPW], incn[TPW];
        load_inc(blockIdx.x, incn);
        for (long long tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
#pragma unroll
            for (int k = 0; k < TPW; ++k) incr[k] = incn[k];
            load_inc(tile + gridDim.x, incn);
            for (int s = 0; s < P.stages_per_tile; ++s, ring.next()) {
                const int slot = ring.slot;
                const uint32_t ph = ring.phase;
                int got = 1;
                if (lane == 0)
                    got = tc::mbar_wait(&empty[slot], ph ^ 1u, abort, P.err, tc::ERR_WAIT_EMPTY, P.wait_limit) ? 1 : 0;
                got = __shfl_sync(0xffffffffu, got, 0);
                if (!got) {
                    ok = false;
                    break;
                }
                // failure tests: the first stage of CTA 0 is never filled, so its consumer's wait runs out
                const int g_s = min(P.gi, P.r - s * P.gi);
                const int rows = g_s * P.inner;             // K' rows filled in this stage
                const uint32_t slotA = sA_u32 + static_cast<uint32_t>(slot) * P.slot_bytes;
#pragma unroll
                for (int k = 0; k < TPW; ++k) {
                    const int t = group + k * GROUPS;
                    if (t >= BT) break;
                    for (int w0 = sub * 32; w0 < rows; w0 += RPW * 32) {
                        const int w = w0 + lane;
                        const int il = il_of_row[min(w, rows - 1)];
                        const uint32_t o16 = __shfl_sync(0xffffffffu, incr[k], s * P.gi + il);
                        if (w >= rows) continue;
                        const int b = w - il * P.inner;
                        const uint32_t dst0 = slotA + static_cast<uint32_t>(t * HG * KS + w) * 16u;
                        // one code path for every lane: an absent generator's rows are zero-filled by
                        // the copy itself (source size 0: nothing is read), so the warp does not diverge
                        const bool present = o16 != kAbsent;
                        const uint32_t src16 = (present ? o16 : 0u) + static_cast<uint32_t>(b);
                        const uint32_t nbytes = present ? 16u : 0u;
#pragma unroll
                        for (int limb = 0; limb < 2; ++limb)
#pragma unroll
                            for (int h = 0; h < HG; ++h)
                                tc::cp_async16_zfill(dst0 + static_cast<uint32_t>(limb) * P.limb_bytes +
                                                         static_cast<uint32_t>(h * KS * 16),
                                                     P.in[limb] + static_cast<size_t>(src16 + h * P.inner) * 16u,
                                                     nbytes);
                    }
                }
                tc::cp_async_arrive_noinc(&full[slot]);   // when this thread's copies have landed
            }
        }
        tc::cp_async_wait_all();   // no copy may still be landing when the CTA exits
    } else if (warp == kMmaWarp) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            const uint32_t idesc = tc::idesc_i8(128, N, true, false);
            const uint32_t sA0 = tc::smem_u32(sA), sB0 = tc::smem_u32(sB);
            const uint32_t a_hi = tc::desc_hi(static_cast<uint32_t>(KS) * 16u), b_hi = tc::desc_hi(256u);
            const uint32_t b_kstep = static_cast<uint32_t>(N) * 32u;   // bytes of B per K-step
            const uint32_t a_limb = P.limb_bytes >> 4;                 // hi limb of A, in descriptor units
            long long tcount = 0;
            SlotRing ring(P.slots);
            bool ok = true;
            bool held = P.hold_first_stage && blockIdx.x == 0;
            for (long long tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++tcount) {
                const int buf = static_cast<int>(tcount & 1);
                const uint32_t aph = static_cast<uint32_t>((tcount >> 1) & 1);
                if (!tc::mbar_wait(&accempty[buf], aph ^ 1u, abort, P.err, tc::ERR_WAIT_ACCUM_FREE, P.wait_limit)) break;
                tc::tc_fence_after();
                const uint32_t dbase = tmem + static_cast<uint32_t>(buf * 2 * N);
                for (int s = 0; s < P.stages_per_tile; ++s, ring.next()) {
                    const int slot = ring.slot;
                    const uint32_t ph = ring.phase;
                    // failure tests: CTA 0 waits for its first stage on a barrier that
                    // nothing completes before the final drain, so the wait runs out
                    uint64_t* wait_bar = (held && s == 0) ? drained : &full[slot];
                    const uint32_t wait_ph = (held && s == 0) ? 0u : ph;
                    held = false;
                    if (!tc::mbar_wait(wait_bar, wait_ph, abort, P.err, tc::ERR_WAIT_FULL, P.wait_limit)) {
                        ok = false;
                        break;
                    }
                    tc::fence_proxy_async_smem();
                    tc::tc_fence_after();
                    const int ks_n = (s == P.stages_per_tile - 1) ? P.ks_last : P.ks_full;
                    // descriptors advance by adding to their low words: A by one K-step (32 rows of
                    // 16 bytes), B by one K-step of the maps (N x 32 bytes); the two limbs of the
                    // input go to the tile's two accumulators
                    const uint32_t a_lo = tc::desc_lo(sA0 + static_cast<uint32_t>(slot) * P.slot_bytes, 128u);
                    const uint32_t b_lo = tc::desc_lo(sB0 + static_cast<uint32_t>(s * P.ks_full) * b_kstep, 128u);
#pragma unroll 2
                    for (int ks = 0; ks < ks_n; ++ks) {
                        const uint64_t bd = tc::desc_make(b_lo + static_cast<uint32_t>(ks) * (b_kstep >> 4), b_hi);
                        const uint32_t acc = (s > 0 || ks > 0) ? 1u : 0u;
                        const uint32_t a_k = a_lo + static_cast<uint32_t>(ks) * (512u >> 4);
                        tc::mma_i8(dbase, tc::desc_make(a_k, a_hi), bd, idesc, acc);
                        tc::mma_i8(dbase + static_cast<uint32_t>(N), tc::desc_make(a_k + a_limb, a_hi), bd, idesc, acc);
                    }
                    tc::mma_commit(&empty[slot]);
                }
                if (!ok) break;
                tc::mma_commit(&accfull[buf]);
            }
            // drain: every MMA issued above completes before TMEM is released
            // (this wait ignores the give-up flag; issued MMAs always finish)
            tc::mma_commit(drained);
            tc::mbar_wait(drained, 0, nullptr, P.err, tc::ERR_WAIT_FINAL);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue
        // Warps PW+1 on: warp & 3 is the TMEM lane quadrant a warp may read; the
        // warps of a quadrant (two with PW = 8, one with PW = 16) split the
        // 16-column output chunks between them.
        const int q = warp & 3;
        constexpr int EPQ = kGatherEpilogueWarps / 4;          // epilogue warps per quadrant
        const int half_id = (warp - kEpilogueWarp0) >> 2;      // this warp's part of the chunks
        const int m = q * 32 + lane;               // tile row = (block t, column j)
        const int t = m / NB, j = m % NB;
        const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
        const int chunks = P.half / 16;
        const uint32_t h_off = static_cast<uint32_t>((j >> 4) * P.outer * 16);   // this half-warp's column group
        long long tcount = 0;
        for (long long tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++tcount) {
            const int buf = static_cast<int>(tcount & 1);
            const uint32_t aph = static_cast<uint32_t>((tcount >> 1) & 1);
            const long long blk = tile * BT + t;
            const bool valid = blk < P.n_blk;
            // prefetch the diagonal entries of this warp's first chunk before waiting for the accumulator
            int32_t dg[16];
            auto load_diag = [&](int c) {
#pragma unroll
                for (int oo = 0; oo < 16; ++oo) {
                    const int o = c * 16 + oo;
                    dg[oo] = (P.diag && valid && o < P.outer) ? __ldg(P.diag + blk * P.outer + o) : 0;
                }
            };
            load_diag(half_id);
            if (!tc::mbar_wait(&accfull[buf], aph, abort, P.err, tc::ERR_WAIT_ACCUM, P.wait_limit)) break;
            tc::tc_fence_after();
            const uint32_t col0 = tmem + lane_off + static_cast<uint32_t>(buf * 2 * N);
            const long long base = blk * static_cast<long long>(NB) * P.outer;
            int8_t* o_lo = P.out[PL_LO] + base;
            int8_t* o_hi = P.out[PL_HI] + base;
            int8_t* o_nlo = P.out[PL_NLO] + base;
            int8_t* o_nhi = P.out[PL_NHI] + base;
            for (int c = half_id; c < chunks; c += EPQ) {
                const int o0 = c * 16;
                if (c != half_id) load_diag(c);
                // this lane's 16 outputs (o0..o0+15 of its column j) as limb bytes; columns o >= outer
                // hold zeros (zero rows of the maps, zero diagonal entries) and are not stored
                uint32_t lw[4] = {0, 0, 0, 0}, hw[4] = {0, 0, 0, 0};
                // Eight columns at a time (the four partials of eight outputs live together), and only
                // the groups of four columns that reach below outer need arithmetic (the rest stay zero).
                const int live = P.outer - o0;
                const bool scale = P.diag != nullptr;
#pragma unroll
                for (int h8 = 0; h8 < 2; ++h8) {
                    if (h8 * 8 >= live) break;
                    int32_t ll[8], lh[8], hl[8], hh[8];
                    const uint32_t cb = col0 + static_cast<uint32_t>(o0 + h8 * 8);
                    tc::tmem_ld8(cb, ll);
                    tc::tmem_ld8(cb + P.half, lh);
                    tc::tmem_ld8(cb + N, hl);
                    tc::tmem_ld8(cb + N + P.half, hh);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        if (h8 * 8 + q * 4 >= live) break;
#pragma unroll
                        for (int oi = 0; oi < 4; ++oi) {
                            const int oo = q * 4 + oi;
                            const int32_t v = epilogue_value(ll[oo], lh[oo] + hl[oo], hh[oo], P.mod, P.c2, scale,
                                                             dg[h8 * 8 + oo]);
                            int8_t lo, hi;
                            split_limbs(v, lo, hi);
                            lw[h8 * 2 + q] |= static_cast<uint32_t>(static_cast<uint8_t>(lo)) << (8 * oi);
                            hw[h8 * 2 + q] |= static_cast<uint32_t>(static_cast<uint8_t>(hi)) << (8 * oi);
                        }
                    }
                }
                // transposed, lane L of the half-warp holds output row o0 + L: 16 bytes, one per j
                transpose16(lw, lane);
                transpose16(hw, lane);
                const int o = o0 + (lane & 15);
                if (valid && o < P.outer) {
                    const uint32_t off = h_off + static_cast<uint32_t>(o) * 16u;
                    *reinterpret_cast<uint4*>(o_lo + off) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
                    *reinterpret_cast<uint4*>(o_hi + off) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                    *reinterpret_cast<uint4*>(o_nlo + off) =
                        make_uint4(neg_bytes4(lw[0]), neg_bytes4(lw[1]), neg_bytes4(lw[2]), neg_bytes4(lw[3]));
                    *reinterpret_cast<uint4*>(o_nhi + off) =
                        make_uint4(neg_bytes4(hw[0]), neg_bytes4(hw[1]), neg_bytes4(hw[2]), neg_bytes4(hw[3]));
                }
            }
            tc::tc_fence_before();
            tc::mbar_arrive(&accempty[buf]);
        }
    }

    tc::tc_fence_before();
    __syncthreads();
    if (warp == kMmaWarp) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, tmem_cols);
    }
}

// ---- gather-GEMM with a hybrid producer: TMA gathers beside cp.async warps
//
// Same tile, MMA issue and epilogue as i8_gather_gemm_kernel; a stage holds
// gs groups of four generators, each generator inner_pad (inner rounded up to
// even) K' rows, so that every group starts 128-byte aligned.  The tile's
// output blocks t < t_tma are filled by the tensor-memory accelerator, the
// others by eight cp.async warps, both into the same stage and completing on
// the same barrier (257 arrivals: one per cp.async thread when its copies have
// landed, one from the TMA warp with the stage's TMA byte count), so the two
// copy engines work side by side.
//
// TMA part: the +plane and the -plane of a limb are one 2-D tensor (rows =
// (block, h) runs of inner * 16 bytes, the -plane's rows after the +plane's),
// so one tile::gather4 copies the runs of four neighbour blocks, each from the
// plane its Koszul sign selects: row = neg * n_blk_in * HG + nbr * HG + h,
// precomputed on the host per group of four generators (rows4).  An absent
// generator (or a padding generator past r) has a row beyond the tensor: the
// copy fills its rows with zeros and reads nothing.  The odd padding row of a
// generator is beyond the tensor's row width (zero-filled) and meets zero rows
// of the maps.
//
// cp.async part: as in i8_gather_gemm_kernel (16-byte copies from the +plane
// or -plane, zero-filling ones for absent generators), with the rows of a
// block shared by 8 / (BT - t_tma) warps.
//
// Warp roles: warps 0-7 cp.async producers, warp 8 TMA producer, warp 9 MMA
// issuer (allocates TMEM), warps 10-17 epilogue.  On a give-up every producer
// still waits (bounded) for the copies it issued before the CTA exits.
constexpr int kCpWarps = 8;
constexpr int kTmaWarp = kCpWarps;
constexpr int kHyMmaWarp = kCpWarps + 1;
constexpr int kHyEpi0 = kCpWarps + 2;
constexpr int kHyThreads = (kCpWarps + 2 + kEpilogueWarps) * 32;

template <int NB>
__global__ void __launch_bounds__(kHyThreads, 1)
    i8_gather_hybrid_kernel(const __grid_constant__ CUtensorMap map_lo, const __grid_constant__ CUtensorMap map_hi,
                            I8Dir P) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int BT = 128 / NB;        // output blocks per tile
    constexpr int HG = NB / 16;         // 16-byte column groups per block row
    constexpr int kMaxSlots = 8;
    const int N = 2 * P.half;
    uint8_t* sB = smem;
    uint8_t* sA = smem + P.b_bytes;
    uint64_t* full = reinterpret_cast<uint64_t*>(sA + static_cast<size_t>(P.slots) * P.slot_bytes);
    uint64_t* empty = full + P.slots;
    uint64_t* accfull = empty + P.slots;
    uint64_t* accempty = accfull + 2;
    uint64_t* drained = accempty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);   // CTA give-up flag
    uint8_t* il_of_row = reinterpret_cast<uint8_t*>(tmem_slot + 4);        // K' row -> generator in stage (255: pad)

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const long long n_tiles = (P.n_blk + BT - 1) / BT;
    const int KS = P.ks_full * 32;                    // K' rows of a slot's column (full stage, padded)
    // every TMA destination is 128-byte aligned relative to the base
    if ((tc::smem_u32(smem) & 127u) != 0 || P.slots > kMaxSlots || P.t_tma < 0 || P.t_tma > BT ||
        KS > kMaxRowTable) {
        if (threadIdx.x == 0) atomicCAS(P.err, tc::ERR_NONE, tc::ERR_LAYOUT);
        return;
    }

    for (uint32_t off = threadIdx.x * 16; off < P.b_bytes; off += blockDim.x * 16)
        *reinterpret_cast<int4*>(sB + off) = __ldg(reinterpret_cast<const int4*>(P.b_tiles + off));
    tc::fence_proxy_async_smem();
    for (int w = threadIdx.x; w < KS; w += blockDim.x) {
        const int il = w / P.inner_pad, u = w - il * P.inner_pad;
        il_of_row[w] = static_cast<uint8_t>(u < P.inner ? il : 255);
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < P.slots; ++s) {
            tc::mbar_init(&full[s], kCpWarps * 32 + 1);   // cp.async threads + the TMA warp's expect_tx arrive
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&accfull[b], 1);
            tc::mbar_init(&accempty[b], kEpilogueWarps * 32);
        }
        tc::mbar_init(drained, 1);
        tc::fence_mbar_init();
        *abort = 0;
    }
    const uint32_t tmem_cols = (4 * N <= 256) ? 256u : 512u;
    if (warp == kHyMmaWarp) {
        tc::tmem_alloc(tmem_slot, tmem_cols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp < kCpWarps) {
        // ------------------------------------------------------------ cp.async producers
        // Blocks t_tma..BT-1 of every tile; a block's stage rows are shared by
        // wpb = 8 / n_cp warps (interleaved by 32 rows); lane i holds the
        // incidence entry of generator i for its warp's block (the next tile's
        // entry is loaded one tile ahead).  Every producer thread arrives once
        // per stage, after waiting for the slot to be free.
        const int n_cp = BT - P.t_tma;
        const int wpb = n_cp > 0 ? kCpWarps / n_cp : 1;
        const bool active = n_cp > 0 && warp < n_cp * wpb;
        const int t = active ? P.t_tma + warp / wpb : 0, sub = active ? warp % wpb : 0;
        // lane i: where generator i's neighbour run starts (16-byte units from the limb's +plane,
        // the -plane's offset added for a negative sign), or kAbsent
        const uint32_t neg16 = static_cast<uint32_t>(P.in_neg_off >> 4);
        const uint32_t run16 = static_cast<uint32_t>(HG * P.inner);
        auto load_inc = [&](long long tile) -> uint32_t {
            const long long blk = tile * BT + t;
            const uint32_t e = (active && tile < n_tiles && blk < P.n_blk && lane < P.r)
                                   ? __ldg(P.inc + blk * P.r + lane) : kAbsent;
            return e == kAbsent ? kAbsent : ((e >> 31) ? neg16 : 0u) + (e & 0x7FFFFFFFu) * run16;
        };
        const uint32_t sA_u32 = tc::smem_u32(sA);
        SlotRing ring(P.slots);
        bool ok = true;
        uint32_t incn = load_inc(blockIdx.x);
        for (long long tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            const uint32_t incr = incn;
            incn = load_inc(tile + gridDim.x);
            for (int s = 0; s < P.stages_per_tile; ++s, ring.next()) {
                const int slot = ring.slot;
                const uint32_t ph = ring.phase;
                int got = 1;
                if (lane == 0)
                    got = tc::mbar_wait(&empty[slot], ph ^ 1u, abort, P.err, tc::ERR_WAIT_EMPTY, P.wait_limit) ? 1 : 0;
                got = __shfl_sync(0xffffffffu, got, 0);
                if (!got) {
                    ok = false;
                    break;
                }
                if (active) {
                    const bool last = s == P.stages_per_tile - 1;
                    const int rows = (last ? P.groups - s * P.gs : P.gs) * 4 * P.inner_pad;
                    const uint32_t col0 = sA_u32 + static_cast<uint32_t>(slot) * P.slot_bytes +
                                          static_cast<uint32_t>(t * HG * KS) * 16u;
                    for (int w0 = sub * 32; w0 < rows; w0 += wpb * 32) {
                        const int w = w0 + lane;
                        const int il = il_of_row[min(w, rows - 1)];
                        const int gen = s * P.gi + (il == 255 ? 0 : il);
                        const uint32_t o16 = __shfl_sync(0xffffffffu, incr, min(gen, 31));
                        // padding rows and generators past r: their B rows are zero, nothing to copy
                        if (w >= rows || il == 255 || gen >= P.r) continue;
                        const int u = w - il * P.inner_pad;
                        const bool present = o16 != kAbsent;
                        const uint32_t src16 = (present ? o16 : 0u) + static_cast<uint32_t>(u);
                        const uint32_t nbytes = present ? 16u : 0u;
                        const uint32_t dst0 = col0 + static_cast<uint32_t>(w) * 16u;
#pragma unroll
                        for (int limb = 0; limb < 2; ++limb)
#pragma unroll
                            for (int h = 0; h < HG; ++h)
                                tc::cp_async16_zfill(dst0 + static_cast<uint32_t>(limb) * P.limb_bytes +
                                                         static_cast<uint32_t>(h * KS * 16),
                                                     P.in[limb] + static_cast<size_t>(src16 + h * P.inner) * 16u,
                                                     nbytes);
                    }
                }
                tc::cp_async_arrive_noinc(&full[slot]);   // when this thread's copies have landed
            }
        }
        tc::cp_async_wait_all();   // no copy may still be landing when the CTA exits
    } else if (warp == kTmaWarp) {
        // ------------------------------------------------------------ TMA producer
        // Blocks 0..t_tma-1: stage s holds groups s * gs .. of every (block,
        // limb, h): 2 * t_tma * HG * g_n gathers; lane j issues j, j + 32, ...
        // Lane 0 posts the stage's TMA byte count first (an arrive with zero
        // bytes when t_tma = 0).
        tc::prefetch_tmap(&map_lo);
        tc::prefetch_tmap(&map_hi);
        const int32_t oob = P.row_oob;   // beyond the input tensor: zero rows, nothing read
        const uint32_t gbytes = static_cast<uint32_t>(P.inner_pad) * 64;   // one group: 4 generators x inner_pad rows
        SlotRing ring(P.slots);
        uint32_t issued_phase[kMaxSlots];
        bool issued[kMaxSlots];
#pragma unroll
        for (int q = 0; q < kMaxSlots; ++q) issued[q] = false, issued_phase[q] = 0;
        bool ok = true;
        for (long long tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
            for (int s = 0; s < P.stages_per_tile; ++s, ring.next()) {
                const int slot = ring.slot;
                const uint32_t ph = ring.phase;
                int got = 1;
                if (lane == 0)
                    got = tc::mbar_wait(&empty[slot], ph ^ 1u, abort, P.err, tc::ERR_WAIT_EMPTY, P.wait_limit) ? 1 : 0;
                got = __shfl_sync(0xffffffffu, got, 0);
                if (!got) {
                    ok = false;
                    break;
                }
                const bool last = s == P.stages_per_tile - 1;
                const int g_n = last ? P.groups - s * P.gs : P.gs;   // groups in this stage
                const int n_g = 2 * P.t_tma * HG * g_n;
                if (lane == 0) tc::mbar_arrive_expect_tx(&full[slot], static_cast<uint32_t>(n_g) * gbytes);
                __syncwarp();
                uint8_t* slotA = sA + static_cast<size_t>(slot) * P.slot_bytes;
                for (int j = lane; j < n_g; j += 32) {
                    const int gl = j % g_n;                 // group within the stage
                    const int rest = j / g_n;
                    const int limb = rest & 1;
                    const int col = rest >> 1;              // t * HG + h, t < t_tma
                    const int tt = col / HG, h = col - (col / HG) * HG;
                    const long long blk = tile * BT + tt;
                    int4 rr = make_int4(oob, oob, oob, oob);
                    if (blk < P.n_blk) rr = __ldg(P.rows4 + blk * P.groups + s * P.gs + gl);
                    uint8_t* dst = slotA + static_cast<size_t>(limb) * P.limb_bytes +
                                   static_cast<size_t>(col) * KS * 16 + static_cast<size_t>(gl) * gbytes;
                    tc::tma_gather4(dst, limb ? static_cast<const void*>(&map_hi) : static_cast<const void*>(&map_lo),
                                    0, rr.x + h, rr.y + h, rr.z + h, rr.w + h, &full[slot]);
                }
                if (n_g > 0) {
                    issued[slot] = true;
                    issued_phase[slot] = ph;
                }
            }
        }
        // no copy may still be landing when the CTA exits: wait (bounded) for
        // the last stage with gathers in every slot (a consumed stage has completed)
        if (lane == 0) {
#pragma unroll
            for (int q = 0; q < kMaxSlots; ++q)
                if (q < P.slots && issued[q]) tc::mbar_wait(&full[q], issued_phase[q], nullptr, P.err, tc::ERR_WAIT_FINAL);
        }
        __syncwarp();
    } else if (warp == kHyMmaWarp) {
        // ------------------------------------------------------------ MMA issuer
        if (lane == 0) {
            const uint32_t idesc = tc::idesc_i8(128, N, true, false);
            const uint32_t sA0 = tc::smem_u32(sA), sB0 = tc::smem_u32(sB);
            const uint32_t a_hi = tc::desc_hi(static_cast<uint32_t>(KS) * 16u), b_hi = tc::desc_hi(256u);
            const uint32_t b_kstep = static_cast<uint32_t>(N) * 32u;   // bytes of B per K-step
            const uint32_t a_limb = P.limb_bytes >> 4;                 // hi limb of A, in descriptor units
            long long tcount = 0;
            SlotRing ring(P.slots);
            bool ok = true;
            bool held = P.hold_first_stage && blockIdx.x == 0;
            for (long long tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x, ++tcount) {
                const int buf = static_cast<int>(tcount & 1);
                const uint32_t aph = static_cast<uint32_t>((tcount >> 1) & 1);
                if (!tc::mbar_wait(&accempty[buf], aph ^ 1u, abort, P.err, tc::ERR_WAIT_ACCUM_FREE, P.wait_limit)) break;
                tc::tc_fence_after();
                const uint32_t dbase = tmem + static_cast<uint32_t>(buf * 2 * N);
                for (int s = 0; s < P.stages_per_tile; ++s, ring.next()) {
                    const int slot = ring.slot;
                    const uint32_t ph = ring.phase;
                    // failure tests: CTA 0 waits for its first stage on a barrier that
                    // nothing completes before the final drain, so the wait runs out
                    uint64_t* wait_bar = (held && s == 0) ? drained : &full[slot];
                    const uint32_t wait_ph = (held && s == 0) ? 0u : ph;
                    held = false;
                    if (!tc::mbar_wait(wait_bar, wait_ph, abort, P.err, tc::ERR_WAIT_FULL, P.wait_limit)) {
                        ok = false;
                        break;
                    }
                    // the cp.async part was written through the generic proxy
                    tc::fence_proxy_async_smem();
                    tc::tc_fence_after();
                    const int ks_n = (s == P.stages_per_tile - 1) ? P.ks_last : P.ks_full;
                    // descriptors advance by adding to their low words: A by one K-step (32 rows of
                    // 16 bytes), B by one K-step of the maps (N x 32 bytes); the two limbs of the
                    // input go to the tile's two accumulators
                    const uint32_t a_lo = tc::desc_lo(sA0 + static_cast<uint32_t>(slot) * P.slot_bytes, 128u);
                    const uint32_t b_lo = tc::desc_lo(sB0 + static_cast<uint32_t>(s * P.ks_full) * b_kstep, 128u);
#pragma unroll 2
                    for (int ks = 0; ks < ks_n; ++ks) {
                        const uint64_t bd = tc::desc_make(b_lo + static_cast<uint32_t>(ks) * (b_kstep >> 4), b_hi);
                        const uint32_t acc = (s > 0 || ks > 0) ? 1u : 0u;
                        const uint32_t a_k = a_lo + static_cast<uint32_t>(ks) * (512u >> 4);
                        tc::mma_i8(dbase, tc::desc_make(a_k, a_hi), bd, idesc, acc);
                        tc::mma_i8(dbase + static_cast<uint32_t>(N), tc::desc_make(a_k + a_limb, a_hi), bd, idesc, acc);
                    }
                    tc::mma_commit(&empty[slot]);
                }
                if (!ok) break;
                tc::mma_commit(&accfull[buf]);
            }
            // drain: every MMA issued above completes before TMEM is released
            tc::mma_commit(drained);
            tc::mbar_wait(drained, 0, nullptr, P.err, tc::ERR_WAIT_FINAL);
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue
        // Warps 10..17: warp & 3 is the TMEM lane quadrant it may read; the two
        // warps of a quadrant split the 16-column output chunks between them.
        const int q = warp & 3;
        constexpr int EPQ = kEpilogueWarps / 4;
        const int half_id = (warp - kHyEpi0) >> 2;
        const int m = q * 32 + lane;               // tile row = (block t, column j)
        const int t = m / NB, j = m % NB;
        const uint32_t lane_off = static_cast<uint32_t>(q * 32) << 16;
        const int chunks = P.half / 16;
        const uint32_t h_off = static_cast<uint32_t>((j >> 4) * P.outer * 16);
        long long tcount = 0;
        for (long long tile = blockIdx.x; tile < n_tiles; tile += gridDim.x, ++tcount) {
            const int buf = static_cast<int>(tcount & 1);
            const uint32_t aph = static_cast<uint32_t>((tcount >> 1) & 1);
            const long long blk = tile * BT + t;
            const bool valid = blk < P.n_blk;
            int32_t dg[16];
            auto load_diag = [&](int c) {
#pragma unroll
                for (int oo = 0; oo < 16; ++oo) {
                    const int o = c * 16 + oo;
                    dg[oo] = (P.diag && valid && o < P.outer) ? __ldg(P.diag + blk * P.outer + o) : 0;
                }
            };
            load_diag(half_id);
            if (!tc::mbar_wait(&accfull[buf], aph, abort, P.err, tc::ERR_WAIT_ACCUM, P.wait_limit)) break;
            tc::tc_fence_after();
            const uint32_t col0 = tmem + lane_off + static_cast<uint32_t>(buf * 2 * N);
            const long long base = blk * static_cast<long long>(NB) * P.outer;
            int8_t* o_lo = P.out[PL_LO] + base;
            int8_t* o_hi = P.out[PL_HI] + base;
            int8_t* o_nlo = P.out[PL_NLO] + base;
            int8_t* o_nhi = P.out[PL_NHI] + base;
            for (int c = half_id; c < chunks; c += EPQ) {
                const int o0 = c * 16;
                if (c != half_id) load_diag(c);
                uint32_t lw[4] = {0, 0, 0, 0}, hw[4] = {0, 0, 0, 0};
                // Eight columns at a time (the four partials of eight outputs live together), and only
                // the groups of four columns that reach below outer need arithmetic (the rest stay zero).
                const int live = P.outer - o0;
                const bool scale = P.diag != nullptr;
#pragma unroll
                for (int h8 = 0; h8 < 2; ++h8) {
                    if (h8 * 8 >= live) break;
                    int32_t ll[8], lh[8], hl[8], hh[8];
                    const uint32_t cb = col0 + static_cast<uint32_t>(o0 + h8 * 8);
                    tc::tmem_ld8(cb, ll);
                    tc::tmem_ld8(cb + P.half, lh);
                    tc::tmem_ld8(cb + N, hl);
                    tc::tmem_ld8(cb + N + P.half, hh);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        if (h8 * 8 + q * 4 >= live) break;
#pragma unroll
                        for (int oi = 0; oi < 4; ++oi) {
                            const int oo = q * 4 + oi;
                            const int32_t v = epilogue_value(ll[oo], lh[oo] + hl[oo], hh[oo], P.mod, P.c2, scale,
                                                             dg[h8 * 8 + oo]);
                            int8_t lo, hi;
                            split_limbs(v, lo, hi);
                            lw[h8 * 2 + q] |= static_cast<uint32_t>(static_cast<uint8_t>(lo)) << (8 * oi);
                            hw[h8 * 2 + q] |= static_cast<uint32_t>(static_cast<uint8_t>(hi)) << (8 * oi);
                        }
                    }
                }
                transpose16(lw, lane);
                transpose16(hw, lane);
                const int o = o0 + (lane & 15);
                if (valid && o < P.outer) {
                    const uint32_t off = h_off + static_cast<uint32_t>(o) * 16u;
                    *reinterpret_cast<uint4*>(o_lo + off) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
                    *reinterpret_cast<uint4*>(o_hi + off) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                    *reinterpret_cast<uint4*>(o_nlo + off) =
                        make_uint4(neg_bytes4(lw[0]), neg_bytes4(lw[1]), neg_bytes4(lw[2]), neg_bytes4(lw[3]));
                    *reinterpret_cast<uint4*>(o_nhi + off) =
                        make_uint4(neg_bytes4(hw[0]), neg_bytes4(hw[1]), neg_bytes4(hw[2]), neg_bytes4(hw[3]));
                }
            }
            tc::tc_fence_before();
            tc::mbar_arrive(&accempty[buf]);
        }
    }

    tc::tc_fence_before();
    __syncthreads();
    if (warp == kHyMmaWarp) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, tmem_cols);
    }
}

// ---- limb conversions and the projection on limb planes
//
// Memory-bound: a thread takes four columns of a row (16 bytes of residues, 4
// bytes of each plane), so a warp's loads and stores are whole lines; one
// byte a thread with 64-bit divisions ran at a sixth of the copy bandwidth
// (genus-20-like Y, 1.85 M x 16, with the call around d: 514 us against 254).

// Offset of the four columns 4 q .. 4 q + 3 of a row in a plane of NB columns.
template <int NB>
__device__ __forceinline__ size_t quad_offset(uint32_t row, uint32_t q, uint32_t dim) {
    if constexpr (NB == 16) {
        return static_cast<size_t>(row) * 16 + q * 4;   // one column group: a block's rows are its plane rows
    } else {
        const uint32_t blk = row / dim, u = row - blk * dim;
        return (static_cast<size_t>(blk) * (NB / 16) + (q >> 2)) * dim * 16 + u * 16 + (q & 3) * 4;
    }
}

// Four residues as packed limb bytes (any 32-bit values; reduced mod p).
__device__ __forceinline__ void limbs4(const uint4& x, const Mod& mod, uint32_t& lo, uint32_t& hi) {
    const uint32_t v[4] = {x.x, x.y, x.z, x.w};
    int32_t l[4], h[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        split_limbs(to_balanced(reduce_u32(v[j], mod), mod), l[j], h[j]);
    }
    lo = pack_bytes(l[0], l[1], l[2], l[3]);
    hi = pack_bytes(h[0], h[1], h[2], h[3]);
}

// canonical row-major (rows x w_in) -> four planes of NB columns (columns
// w_in..NB-1 are zero); rows below 2^32
template <int NB>
__global__ void __launch_bounds__(256) to_limbs_kernel(const uint32_t* __restrict__ in, int8_t* __restrict__ lo,
                                                       int8_t* __restrict__ hi, int8_t* __restrict__ nlo,
                                                       int8_t* __restrict__ nhi, long long quads, uint32_t dim,
                                                       uint32_t w_in, bool aligned, Mod mod) {
    constexpr uint32_t Q = NB / 4;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < quads; i += stride) {
        const uint32_t row = static_cast<uint32_t>(i / Q), q = static_cast<uint32_t>(i) % Q;
        uint32_t a = 0, b = 0;
        if (q * 4 < w_in) limbs4(load_quad(in + static_cast<size_t>(row) * w_in + q * 4, aligned), mod, a, b);
        const size_t off = quad_offset<NB>(row, q, dim);
        *reinterpret_cast<uint32_t*>(lo + off) = a;
        *reinterpret_cast<uint32_t*>(hi + off) = b;
        *reinterpret_cast<uint32_t*>(nlo + off) = neg_bytes4(a);
        *reinterpret_cast<uint32_t*>(nhi + off) = neg_bytes4(b);
    }
}

// four planes of NB columns -> canonical row-major with the first w_out columns
template <int NB>
__global__ void __launch_bounds__(256) from_limbs_kernel(const int8_t* __restrict__ lo, const int8_t* __restrict__ hi,
                                                         uint32_t* __restrict__ out, long long quads, uint32_t dim,
                                                         uint32_t w_shift, bool aligned, Mod mod) {
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < quads; i += stride) {
        const uint32_t row = static_cast<uint32_t>(i >> w_shift), q = static_cast<uint32_t>(i) & ((1u << w_shift) - 1);
        const size_t off = quad_offset<NB>(row, q, dim);
        const uint32_t a = __ldg(reinterpret_cast<const uint32_t*>(lo + off));
        const uint32_t b = __ldg(reinterpret_cast<const uint32_t*>(hi + off));
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int32_t x = 255 * static_cast<int8_t>(b >> (8 * j)) + static_cast<int8_t>(a >> (8 * j));
            v[j] = to_canonical(reduce_balanced_fast(x, mod), mod);
        }
        store_quad(out + i * 4, make_uint4(v[0], v[1], v[2], v[3]), aligned);
    }
}

// ---- projection a = X^T W on the tensor cores
//
// K = the source rows.  A = X in limbs: M rows = the lo limbs of the m
// projection columns in groups of 16, then their hi limbs (MN-major; laid out
// once per session as one contiguous tile per stage).  B = the lo and hi
// planes of W side by side (N = 2 NB, MN-major: one 16-byte plane row is one
// core-matrix row, so a block's rows copy straight from HBM).  A stage is SB
// whole source blocks, SB * dim rows padded to KP (a multiple of 32); the
// padding rows of the X tile are zero, so whatever the stage buffer holds
// there adds nothing.  The M = 128 descriptor also reads past the X tile: the
// TMEM rows at and above 32 * MG are never read back.
//   D[lo x][j]      = sum lo(X) lo(W),   D[lo x][NB + j] = sum lo(X) hi(W),
//   D[hi x][j]      = sum hi(X) lo(W),   D[hi x][NB + j] = sum hi(X) hi(W)
// int32 accumulation is exact for at most 2^31 / 127^2 > 131072 rows, so the
// accumulator is drained (double-buffered) every `drain` stages.
//
// Warps: 0 producer (the stage's X tile and W runs), 1 MMA issuer (allocates
// TMEM), 2-5 epilogue (tcgen05.ld + reduction mod p).  The W runs of 16-column
// blocks are back to back in a plane and take one bulk copy a limb.  Those of
// 32-column blocks alternate between the two column groups: a box of a 3-D
// tensor map (run, group, block) collects a group's runs of the whole stage.
// (One bulk copy a run, 32 a stage, held the copies at half the rate: 427 us at
// r = 21, k = 10, dim 32, 32 columns, 409 with warp-uniform MMA issue, 221 with
// the boxes.)  The
// CTA's combined sums are added into an m x n int32 accumulator; the last CTA
// to finish writes them to the session's buffer, clears them and advances the
// index.
constexpr int kProjThreads = 6 * 32;
constexpr int kProjStageTarget = 32 * 1024;   // bytes of X tile + W runs per stage

struct I8Proj {
    const int8_t* xt;           // [stage][2 MG][KP][16]
    const int8_t* w[2];         // W lo, hi planes: [blk][h][u][16]
    int32_t* partials;          // [m][NB] accumulator, zero between launches
    unsigned int* counter;
    SeqState* state;
    int* err;
    long long n_blk;
    int dim, m, mg, sb, kp, n_stages, slots, drain;
    int n_out;                  // columns of W that are the caller's (the rest are zero padding)
    uint32_t a_bytes, slot_bytes, pad_bytes;
    Mod mod;
    int32_t c1, c2;
    uint32_t wait_limit;        // tries of every pipeline wait (tc::kWaitLimit outside the failure tests)
};

template <int NB>
__global__ void __launch_bounds__(kProjThreads, 1)
    i8_project_tc_kernel(const __grid_constant__ CUtensorMap w_lo, const __grid_constant__ CUtensorMap w_hi, I8Proj P) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr int HG = NB / 16;
    constexpr int N = 2 * NB;
    int32_t* red = reinterpret_cast<int32_t*>(smem + static_cast<size_t>(P.slots) * P.slot_bytes + P.pad_bytes);
    uint64_t* full = reinterpret_cast<uint64_t*>(red + 32 * P.mg * N);
    uint64_t* empty = full + P.slots;
    uint64_t* accfull = empty + P.slots;
    uint64_t* accempty = accfull + 2;
    uint64_t* drained = accempty + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(drained + 1);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    __shared__ bool am_last;

    const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x / 32), 0), lane = threadIdx.x % 32;
    const long long n_my = blockIdx.x < P.n_stages ? (P.n_stages - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    const long long n_chunks = (n_my + P.drain - 1) / P.drain;
    const uint32_t tmem_cols = 2 * N;   // two accumulators (64 or 128 columns)
    if (threadIdx.x == 0) {
        for (int s = 0; s < P.slots; ++s) {
            tc::mbar_init(&full[s], 1);
            tc::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&accfull[b], 1);
            tc::mbar_init(&accempty[b], 4 * 32);
        }
        tc::mbar_init(drained, 1);
        tc::fence_mbar_init();
        *abort = 0;
    }
    if (warp == 1) {
        tc::tmem_alloc(tmem_slot, tmem_cols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t run_bytes = static_cast<uint32_t>(P.dim) * 16;   // one (block, h) run of a plane
    // In this order: when the next kernel begins, W is complete (see
    // i8_step_once: the next step's d does not wait for this kernel).
    pdl_wait();
    pdl_trigger();

    if (warp == 0) {
        // ------------------------------------------------------------ producer
        SlotRing ring(P.slots);
        for (long long i = 0; i < n_my; ++i, ring.next()) {
            const int slot = ring.slot;
            const uint32_t ph = ring.phase;
            const long long st = blockIdx.x + i * gridDim.x;
            const long long blk0 = st * P.sb;
            // a box is copied whole (past the last block: zeros)
            const int nbh = HG == 1 ? static_cast<int>(min(static_cast<long long>(P.sb), P.n_blk - blk0)) : P.sb;
            int got = 1;
            if (lane == 0) {
                got = tc::mbar_wait(&empty[slot], ph ^ 1u, abort, P.err, tc::ERR_WAIT_EMPTY, P.wait_limit) ? 1 : 0;
                if (got)
                    tc::mbar_arrive_expect_tx(&full[slot], P.a_bytes + 2u * HG * nbh * run_bytes);
            }
            got = __shfl_sync(0xffffffffu, got, 0);
            if (!got) break;
            uint8_t* sA = smem + static_cast<size_t>(slot) * P.slot_bytes;
            uint8_t* sB = sA + P.a_bytes;
            const uint32_t group_bytes = static_cast<uint32_t>(P.kp) * 16;
            if (lane == 0) tc::bulk_g2s(sA, P.xt + st * P.a_bytes, P.a_bytes, &full[slot]);
            if (HG == 1) {
                // consecutive blocks are consecutive rows of a 16-column plane
                if (lane < 2)
                    tc::bulk_g2s(sB + lane * group_bytes, P.w[lane] + blk0 * run_bytes, nbh * run_bytes, &full[slot]);
            } else {
                if (lane < 2 * HG)
                    tc::tma_load3(sB + lane * group_bytes, lane < HG ? &w_lo : &w_hi, 0, lane % HG,
                                  static_cast<int32_t>(blk0), &full[slot]);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer
        // A whole warp waits and walks the stages and one elected lane issues, so
        // that descriptors are warp-uniform (issued by lane 0 in a branch of its
        // own, each MMA took 140 cycles instead of its 40 to 48).
        const uint32_t idesc = tc::idesc_i8(128, N, true, true);
        const uint32_t gb = static_cast<uint32_t>(P.kp) * 16, d_hi = tc::desc_hi(gb);
        const uint32_t a_first = tc::desc_lo(tc::smem_u32(smem), 128u), slot_units = P.slot_bytes >> 4;
        const uint32_t b_off = P.a_bytes >> 4;
        const uint32_t full0 = tc::smem_u32(full), empty0 = tc::smem_u32(empty);
        const uint32_t accfull0 = tc::smem_u32(accfull), accempty0 = tc::smem_u32(accempty);
        const int ksteps = P.kp / 32;
        int slot = 0, left = 0;          // stages left of the accumulator's share
        uint32_t parity = 0, buf = 0, acc_parity = 1, acc = 0;
        for (int todo = static_cast<int>(n_my); todo > 0; --todo) {
            if (left == 0) {
                if (!tc::warp_wait(accempty0 + buf * 8u, acc_parity, abort, P.err, tc::ERR_WAIT_ACCUM_FREE, P.wait_limit))
                    break;
                left = min(todo, P.drain);
                acc = 0;
            }
            if (!tc::warp_wait(full0 + static_cast<uint32_t>(slot) * 8u, parity, abort, P.err, tc::ERR_WAIT_FULL,
                               P.wait_limit))
                break;
            tc::tc_fence_after();
            const uint32_t a_lo = a_first + static_cast<uint32_t>(slot) * slot_units;
            const uint32_t dcol = tmem + buf * N;
#pragma unroll 4
            for (int ks = 0; ks < ksteps; ++ks) {
                const uint32_t a = a_lo + static_cast<uint32_t>(ks) * 32u;
                tc::mma_i8_elect(dcol, tc::desc_make(a, d_hi), tc::desc_make(a + b_off, d_hi), idesc, acc);
                acc = 1;
            }
            tc::mma_commit_elect(empty0 + static_cast<uint32_t>(slot) * 8u);
            if (--left == 0) {
                tc::mma_commit_elect(accfull0 + buf * 8u);
                buf ^= 1u;
                acc_parity ^= buf == 0 ? 1u : 0u;
            }
            if (++slot == P.slots) {
                slot = 0;
                parity ^= 1u;
            }
        }
        // drain: every MMA issued above completes before TMEM is released
        tc::mma_commit_elect(tc::smem_u32(drained));
        tc::warp_wait(tc::smem_u32(drained), 0, nullptr, P.err, tc::ERR_WAIT_FINAL);
    } else {
        // ------------------------------------------------------------ epilogue
        const int q = warp & 3;                  // TMEM lane quadrant of this warp
        const int row = q * 32 + lane;           // D row
        const bool active = q < P.mg;            // rows below 32 * MG carry the X limbs
        int32_t acc[N];
#pragma unroll
        for (int c = 0; c < N; ++c) acc[c] = 0;
        for (long long c = 0; c < n_chunks; ++c) {
            const int buf = static_cast<int>(c & 1);
            const uint32_t aph = static_cast<uint32_t>((c >> 1) & 1);
            if (!tc::mbar_wait(&accfull[buf], aph, abort, P.err, tc::ERR_WAIT_ACCUM, P.wait_limit)) break;
            tc::tc_fence_after();
            if (active) {
                const uint32_t col0 = tmem + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(buf * N);
#pragma unroll
                for (int c0 = 0; c0 < N; c0 += 16) {
                    int32_t v[16];
                    tc::tmem_ld16(col0 + c0, v);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int cc = 0; cc < 16; ++cc) acc[c0 + cc] = reduce_balanced(acc[c0 + cc] + reduce_partial(v[cc], P.mod), P.mod);
                }
            }
            tc::tc_fence_before();
            tc::mbar_arrive(&accempty[buf]);
        }
        if (active)
#pragma unroll
            for (int c = 0; c < N; ++c) red[row * N + c] = acc[c];
    }

    tc::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc::tc_fence_after();
        tc::tmem_dealloc(tmem, tmem_cols);
    }
    // x * w = lo*lo + 255 (lo*hi + hi*lo) + 255^2 hi*hi, per (x, j); the
    // CTA's balanced sums meet in one int32 accumulator by atomics (148 CTAs x
    // (p-1)/2 stay far below 2^31: exact and order-independent), which the
    // last CTA reads and clears
    const int entries = P.m * NB;
    const int hi_row = 16 * P.mg;
    for (int e = threadIdx.x; e < entries; e += blockDim.x) {
        const int x = e / NB, j = e - (e / NB) * NB;
        const int32_t ll = red[x * N + j], lh = red[x * N + NB + j];
        const int32_t hl = red[(hi_row + x) * N + j], hh = red[(hi_row + x) * N + NB + j];
        atomicAdd(P.partials + e, combine(ll, lh + hl, hh, P.mod, P.c1, P.c2));
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) am_last = (atomicAdd(P.counter, 1u) == gridDim.x - 1);
    __syncthreads();
    if (!am_last) return;
    __threadfence();
    const unsigned long long pos = P.state->index;
    uint32_t* seq = P.state->seq;
    for (int e = threadIdx.x; e < entries; e += blockDim.x) {
        const int x = e / NB, j = e - (e / NB) * NB;
        const int32_t sum = atomicExch(P.partials + e, 0);
        if (j >= P.n_out) continue;
        seq[pos * (static_cast<unsigned long long>(P.m) * P.n_out) + x * P.n_out + j] =
            to_canonical(reduce_balanced(sum, P.mod), P.mod);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        P.state->index = pos + 1;
        *P.counter = 0;
        __threadfence();
    }
}

// X (canonical, rows x m) -> the projection's A tiles [stage][2 MG][KP][16]:
// group g < MG holds the lo limbs of columns 16 g .. 16 g + 15, group MG + g
// their hi limbs; rows past the stage's SB * dim, past the last row or columns
// past m are zero.  A thread takes four columns of one row, both limbs.
__global__ void __launch_bounds__(256) x_tiles_kernel(const uint32_t* __restrict__ X, int8_t* __restrict__ xt,
                                                      long long rows, int m, int mg, int dim, int sb, int kp,
                                                      long long quads, bool aligned, Mod mod) {
    const uint32_t per_stage = static_cast<uint32_t>(mg) * kp * 4;   // quads
    for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < quads;
         i += static_cast<long long>(gridDim.x) * blockDim.x) {
        const long long st = i / per_stage;
        const uint32_t rem = static_cast<uint32_t>(i - st * per_stage);
        const uint32_t q = rem % 4, gk = rem / 4, g = gk / kp, kr = gk - g * kp;
        const long long row = st * sb * dim + kr;
        const int x0 = static_cast<int>(g) * 16 + static_cast<int>(q) * 4;
        uint32_t a = 0, b = 0;
        if (kr < static_cast<uint32_t>(sb * dim) && row < rows && x0 < m)
            limbs4(load_quad(X + row * m + x0, aligned), mod, a, b);
        int8_t* at = xt + ((st * 2 * mg + g) * kp + kr) * 16 + q * 4;
        *reinterpret_cast<uint32_t*>(at) = a;
        *reinterpret_cast<uint32_t*>(at + static_cast<size_t>(mg) * kp * 16) = b;
    }
}

template <class F>
void dispatch_i8_nb(int nb, F&& f) {
    switch (nb) {
        case 16: f(std::integral_constant<int, 16>{}); break;
        case 32: f(std::integral_constant<int, 32>{}); break;
        default: throw Error("INT8 form supports block widths 16 and 32", 1);
    }
}

}  // namespace

// Host-side state of the INT8 form.
struct KoszulCtx::I8State {
    struct Dir {
        I8Dir p{};
        int8_t* b_tiles = nullptr;
        uint32_t* inc = nullptr;
        int4* rows4 = nullptr;     // TMA gather rows per group of four generators
        bool gather4 = false;      // hybrid producer (TMA gathers beside cp.async warps), else cp.async only
        int pw = 8;                // cp.async producer warps (8 or 16)
        size_t smem = 0;
        unsigned grid = 0;
        // union kernel (bw_koszul_i8_union.cuh); the dense producers' tables above are then not built
        bool use_union = false;
        I8Union u{};
        int8_t* maps = nullptr;
        std::vector<uint32_t> mask;      // [tile] union of its blocks' generators
        uint32_t* d_mask = nullptr;
        uint32_t* order = nullptr;       // [tile][BT] blocks (see I8Union)
        uint32_t *start = nullptr, *words = nullptr, *steps = nullptr;   // stage list of list_gs generators a stage
        int list_gs = 0, list_issuers = 0;
    } fwd, bwd;
    // Y_a, Y_b, Z: lo, hi, -lo, -hi; each -plane directly follows its +plane in
    // memory, so that one tensor map covers both signs of a limb
    int8_t* planes[3][4] = {};
    CUtensorMap runs[2][2] = {};       // Y_a, Y_b: [limb], the projection's boxes of 32-column blocks
    CUtensorMap maps[3][2];        // [block array][limb]: rows = (sign, block, h) runs
    std::string plan_text;         // the chosen stage plans and the autotuner's timings
    I8Proj proj{};             // projection plan (X tiles, stage shape, grid)
    int8_t* xt = nullptr;
    size_t proj_smem = 0;
    unsigned proj_grid = 0;
    int* err = nullptr;        // the kernels' error word (device address)
    volatile int* h_err = nullptr;   // the same word: mapped host memory, written only when a kernel gives up
    unsigned long long err_context = 0;   // the CUDA context that the word's page belongs to
};

namespace {

// Autotuner cache: the chosen producer and stage size per operator shape and
// device, shared by every context of the process.
struct TuneKey {
    int r, k, inner, outer, nbi, dir, sms, allowed;
    bool operator<(const TuneKey& o) const {
        return std::tie(r, k, inner, outer, nbi, dir, sms, allowed) <
               std::tie(o.r, o.k, o.inner, o.outer, o.nbi, o.dir, o.sms, o.allowed);
    }
};
struct TuneChoice {
    int kind = 0;           // 0 dense cp.async, 1 dense hybrid, 2 union
    int pw = 8;             // cp.async producer warps
    int gps = 0;            // generators per stage (dense and union kernels)
    int t_tma = 0;          // hybrid: blocks of a tile gathered by TMA; union: producer groups
    int issuers = 1;        // union: MMA warps
    double ms = 0;
};
std::mutex g_tune_mutex;
std::map<TuneKey, TuneChoice> g_tune_cache;

bool tune_lookup(const TuneKey& k, TuneChoice& out) {
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    const auto it = g_tune_cache.find(k);
    if (it == g_tune_cache.end()) return false;
    out = it->second;
    return true;
}

void tune_store(const TuneKey& k, const TuneChoice& c) {
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    g_tune_cache[k] = c;
}

// Error words: engine contexts alive at the same time share mapped allocations
// of 64 words each (allocating one took a small context a fifth of its set-up);
// one goes back with its last word.  A page belongs to the CUDA context that it
// was allocated in and serves only that one: cudaDeviceReset, which an engine
// context may outlive, takes the memory of the device's pages with it.
struct ErrorPage {
    unsigned long long context;   // id of the CUDA context (never used again in the process)
    int* words;
    uint64_t used;
};
std::mutex g_error_mutex;
std::vector<ErrorPage> g_error_pages;

// Id of the calling thread's current CUDA context, 0 without one.
unsigned long long current_context_id() {
    using GetIdFn = CUresult (*)(CUcontext, unsigned long long*);
    static const GetIdFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<GetIdFn>(f);
    }();
    unsigned long long id = 0;
    if (fn == nullptr || fn(nullptr, &id) != CUDA_SUCCESS) return 0;
    return id;
}

// A word of the current CUDA context's pages; `context` receives its id.
volatile int* error_word_acquire(unsigned long long& context) {
    context = current_context_id();
    BW_REQUIRE(context != 0, "INT8 form: no current CUDA context");
    std::lock_guard<std::mutex> lock(g_error_mutex);
    auto at = std::find_if(g_error_pages.begin(), g_error_pages.end(),
                           [&](const ErrorPage& g) { return g.context == context && ~g.used != 0; });
    if (at == g_error_pages.end()) {
        void* p = nullptr;
        g_error_pages.reserve(g_error_pages.size() + 1);
        BW_CUDA(cudaHostAlloc(&p, 64 * sizeof(int), cudaHostAllocMapped));
        g_error_pages.push_back({context, static_cast<int*>(p), 0});
        at = g_error_pages.end() - 1;
    }
    const int bit = __builtin_ctzll(~at->used);
    at->used |= 1ull << bit;
    return at->words + bit;
}

void error_word_release(volatile int* word, unsigned long long context) {
    std::lock_guard<std::mutex> lock(g_error_mutex);
    for (auto at = g_error_pages.begin(); at != g_error_pages.end(); ++at) {
        if (at->context != context || word < at->words || word >= at->words + 64) continue;
        at->used &= ~(1ull << (word - at->words));
        if (at->used == 0) {
            if (current_context_id() == context) cudaFreeHost(at->words);   // else it went with its CUDA context
            g_error_pages.erase(at);
        }
        return;
    }
}

// Plans one direction: stage size, pipeline depth, B operand (host layout).
//
// A generator spans `inner_pad` K' rows (inner, rounded up to even for the TMA
// gather producer so that every group of four generators starts 128-byte
// aligned).  A stage holds `gps` generators (gather producer: gs groups of
// four), padded to whole K-steps of 32 rows; B is zero in every padding row
// and for every generator past r, so the A rows there may hold anything.
// Returns false when the maps and stages do not fit in shared memory.
bool plan_direction(KoszulCtx& c, KoszulCtx::I8State::Dir& D, int inner, int outer, bool transpose_maps,
                    bool gather4, int gps_forced = 0) {
    I8Dir& P = D.p;
    P.r = c.r;
    P.inner = inner;
    P.outer = outer;
    P.half = (outer + 15) / 16 * 16;
    const int N = 2 * P.half;
    BW_REQUIRE(N <= 256, "INT8 form: output dimension above 128 is not supported");
    const size_t extra = (2 * 8 + 2 * 2 + 1) * 8 + 16 + kMaxRowTable;
    const int inner_pad = gather4 ? inner + (inner & 1) : inner;
    auto b_bytes_of = [&](int gps) {
        const int stages = (c.r + gps - 1) / gps;
        const int ks_full = (gps * inner_pad + 31) / 32;
        const int last = c.r - (stages - 1) * gps;
        const int last_rows = gather4 ? (last + 3) / 4 * 4 * inner_pad : last * inner_pad;
        return static_cast<size_t>((stages - 1) * ks_full + (last_rows + 31) / 32) * N * 32;
    };
    int gps = 0;
    if (gps_forced > 0) {
        // a stage size chosen by the autotuner (checked below against shared memory)
        if (gather4 && gps_forced % 4 != 0) return false;
        gps = std::min(gps_forced, gather4 ? (c.r + 3) / 4 * 4 : c.r);
        if (gather4) {
            P.groups = (c.r + 3) / 4;
            P.gs = gps / 4;
        } else if (gps * inner > kMaxRowTable) {
            return false;
        }
    } else if (gather4) {
        // groups of four generators per stage: the best-filled choice that
        // leaves at least three pipeline slots, the fewer stages on ties
        P.groups = (c.r + 3) / 4;
        double best = -1;
        for (int gs = 1; gs <= P.groups; ++gs) {
            const int rows = gs * 4 * inner_pad, padded = (rows + 31) / 32 * 32;
            const size_t slot = static_cast<size_t>(2) * 8 * padded * 16;
            const size_t bb = b_bytes_of(4 * gs);
            if (bb + 3 * slot + extra > static_cast<size_t>(kMaxSmem)) break;
            const double fill = static_cast<double>(rows) / padded;
            if (fill > best + 1e-9) {
                best = fill;
                gps = 4 * gs;
            }
        }
        if (gps == 0) return false;
        P.gs = gps / 4;
    } else {
        // the best-filled stage of at most 56 KB of A per slot, the largest such on ties
        double best_fill = -1;
        for (int g = 1; g <= c.r; ++g) {
            const int rows = g * inner, padded = (rows + 31) / 32 * 32;
            if (g > 1 && static_cast<size_t>(2) * 8 * padded * 16 > 56 * 1024) break;
            const double fill = static_cast<double>(rows) / padded;
            if (fill > best_fill - 1e-9) {
                best_fill = std::max(best_fill, fill);
                gps = g;
            }
        }
        BW_REQUIRE(gps * inner <= kMaxRowTable, "INT8 form: stage too deep for the row table");
    }
    P.inner_pad = inner_pad;
    P.gi = gps;
    P.stages_per_tile = (c.r + gps - 1) / gps;
    P.ks_full = (gps * inner_pad + 31) / 32;
    const int last_g = c.r - (P.stages_per_tile - 1) * gps;
    const int last_rows = gather4 ? (last_g + 3) / 4 * 4 * inner_pad : last_g * inner_pad;
    P.ks_last = (last_rows + 31) / 32;
    const int total_ks = (P.stages_per_tile - 1) * P.ks_full + P.ks_last;
    P.b_bytes = static_cast<uint32_t>(total_ks) * N * 32;
    P.limb_bytes = static_cast<uint32_t>(8 * P.ks_full * 32 * 16);
    P.slot_bytes = 2 * P.limb_bytes;
    P.tx_full = static_cast<uint32_t>(16 * gps * inner_pad * 16);              // 2 limbs x 8 columns x rows x 16 B
    P.tx_last = static_cast<uint32_t>(16 * ((last_g + 3) / 4 * 4) * inner_pad * 16);
    int slots = 8;
    while (slots > 1 && P.b_bytes + static_cast<size_t>(slots) * P.slot_bytes + extra > static_cast<size_t>(kMaxSmem))
        --slots;
    if (P.b_bytes + static_cast<size_t>(slots) * P.slot_bytes + extra > static_cast<size_t>(kMaxSmem)) return false;
    if (gather4 && P.ks_full * 32 > kMaxRowTable) return false;
    P.slots = slots;
    D.smem = P.b_bytes + static_cast<size_t>(slots) * P.slot_bytes + extra;
    D.gather4 = gather4;
    P.mod = c.mod;
    P.c1 = to_balanced(255u % c.p, c.mod);
    P.c2 = to_balanced(static_cast<uint32_t>((255ull * 255ull) % c.p), c.mod);

    // B: row n < half -> lo limb, n >= half -> hi limb of map coefficient (o = n mod half),
    // column K' = stage row base + (generator in stage) * inner_pad + u; K-major,
    // 8x16-byte core matrices, LBO 128, SBO 256.
    std::vector<int8_t> B(P.b_bytes, 0);
    const int kp_total = total_ks * 32;
    for (int kp = 0; kp < kp_total; ++kp) {
        const int s = std::min(kp / (P.ks_full * 32), P.stages_per_tile - 1);
        const int local = kp - s * P.ks_full * 32;
        const int gen_local = local / inner_pad, u = local % inner_pad;
        const int i = s * gps + gen_local;
        if (u >= inner || gen_local >= (s == P.stages_per_tile - 1 ? last_g : gps) || i >= c.r) continue;   // padding
        for (int n = 0; n < N; ++n) {
            const int o = n % P.half;
            if (o >= outer) continue;
            // forward: coefficient M_i[o = c][u = b]; transpose: M_i[u = c][o = b]
            const uint32_t raw = transpose_maps
                                     ? c.maps_canonical[(static_cast<size_t>(i) * c.co + u) * c.ci + o]
                                     : c.maps_canonical[(static_cast<size_t>(i) * c.co + o) * c.ci + u];
            int8_t lo, hi;
            split_limbs(to_balanced(raw % c.p, c.mod), lo, hi);
            const int ks = kp / 32, kk = kp % 32;
            const size_t off = static_cast<size_t>(ks) * N * 32 + (n / 8) * 256 + (kk / 16) * 128 + (n % 8) * 16 + (kk % 16);
            B[off] = n < P.half ? lo : hi;
        }
    }
    D.b_tiles = c.alloc<int8_t>(P.b_bytes);
    BW_CUDA(cudaMemcpyAsync(D.b_tiles, B.data(), B.size(), cudaMemcpyHostToDevice, c.own_stream));
    BW_CUDA(cudaStreamSynchronize(c.own_stream));
    P.b_tiles = D.b_tiles;
    return true;
}

// Dense incidence table [blk][r]: neighbour rank | negative << 31, or kAbsent
// (forward: blk = T; backward: blk = S; see for_each_neighbour).
__global__ void incidence_kernel(uint32_t* __restrict__ inc, long long n_blk, int r, int k, bool forward,
                                 const __grid_constant__ BinomTable B) {
    const long long blk = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (blk >= n_blk) return;
    uint32_t* out = inc + blk * r;
    for (int i = 0; i < r; ++i) out[i] = kAbsent;
    for_each_neighbour(static_cast<uint32_t>(blk), r, k, forward, B, [&](int i, uint32_t rank, bool negative) {
        out[i] = rank | (negative ? 0x80000000u : 0u);
    });
}

// Rows of the TMA gathers: for output block blk and group g (generators
// 4g..4g+3), the plane row of each generator's neighbour run at h = 0:
// neg * n_blk_in * HG + nbr * HG, or one past the last row (zero-filled) for an
// absent generator or one past r.
__global__ void gather_rows_kernel(const uint32_t* __restrict__ inc, int4* __restrict__ rows, long long n_blk, int r,
                                   int groups, long long n_blk_in, int hg) {
    const long long q = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (q >= n_blk * groups) return;
    const long long blk = q / groups;
    const int g = static_cast<int>(q - blk * groups);
    int32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int i = 4 * g + j;
        const uint32_t e = i < r ? inc[blk * r + i] : kAbsent;
        v[j] = static_cast<int32_t>(e == kAbsent ? 2 * n_blk_in * hg
                                                 : (e >> 31) * n_blk_in * hg + (e & 0x7FFFFFFFu) * static_cast<long long>(hg));
    }
    rows[q] = make_int4(v[0], v[1], v[2], v[3]);
}

// Per tile of bt blocks, the generators that any of its blocks has.
__global__ void union_mask_kernel(const uint32_t* __restrict__ inc, const uint32_t* __restrict__ order,
                                  uint32_t* __restrict__ mask, long long n_tiles, int r, int bt) {
    const long long tile = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (tile >= n_tiles) return;
    uint32_t m = 0;
    for (int t = 0; t < bt; ++t) {
        const uint32_t blk = order[tile * bt + t];
        for (int i = 0; blk != kNoBlock && i < r; ++i)
            if (inc[static_cast<size_t>(blk) * r + i] != kAbsent) m |= 1u << i;
    }
    mask[tile] = m;
}

// Plans one direction of the union kernel with gs generators a stage, the
// producer warps in so many groups and one or two MMA warps; false when it does
// not fit (shared memory for the resident maps and at least two slots, one
// table word and one step word a lane, kUnionPasses passes, a stage a tile for
// either MMA warp).
bool plan_union(KoszulCtx& c, KoszulCtx::I8State::Dir& D, int inner, int outer, bool transpose_dir, int gs, int groups,
                int issuers) {
    I8Union& U = D.u;
    const int bt = 128 / c.nbi, run = (c.nbi / 16) * inner;
    U.r = c.r;
    U.inner = inner;
    U.outer = outer;
    U.ho = (outer + 7) / 8 * 8;
    U.cpg = (2 * inner + 15) / 16;
    U.gs = gs;
    U.groups = groups;
    U.issuers = issuers;
    U.row = ((gs * U.cpg + 1) / 2 + 3) / 4 * 4;
    // Without a reduction of hi on its own the epilogue's first sum is lo + 255
    // hi over at most n = incident generators x inner pairs of rows, each below
    // 127 * (127 + 127) in lo and 64 * (127 + 127) in hi (the maps' hi limbs are
    // at most 64): 4.18e6 n, which must stay within the range near_shifted()
    // brings back below 255 * 127 + 127, 0.49 * 2^32 at p = 32749: n <= 500.
    U.wide = (transpose_dir ? c.k : c.r - c.k + 1) * inner > 500;
    const bool odd = (U.cpg & 1) != 0;
    if (gs < 1 || (odd && gs % 2 != 0) || gs * bt > 32 || U.row > kUnionSteps) return false;
    if (gs * bt * run > union_warps::producers / groups * 32 * kUnionPasses) return false;
    const size_t b = (static_cast<size_t>(c.r) * U.cpg + (odd ? 1 : 0)) * 2 * U.ho * 16;
    const size_t slot = static_cast<size_t>(gs) * U.cpg * 16 * 128;
    const size_t extra = (2 * 8 + 2 * 2 + 2) * 8 + 16;
    if (b + 2 * slot + extra > static_cast<size_t>(kMaxSmem)) return false;
    U.b_bytes = static_cast<uint32_t>(b);
    U.slot_bytes = static_cast<uint32_t>(slot);
    U.slots = static_cast<int>(std::min<size_t>(8, (kMaxSmem - b - extra) / slot));
    // Two MMA warps take the stages in turn: every tile has to have a stage for
    // either (a block alone has so many generators), and a slot has to belong to
    // one of them for good, or one could run a lap ahead of the other and take a
    // barrier's phase for the next but one.
    const int least = transpose_dir ? c.k : c.r - c.k + 1;
    if (issuers == 2) U.slots &= ~1;
    if (U.slots < std::max(2, groups) || (issuers == 2 && least <= gs)) return false;
    U.mod = c.mod;
    U.maps = D.maps;
    D.smem = b + U.slots * slot + extra;
    return true;
}

// The maps as the union kernel's B operand, in their shared-memory layout.
std::vector<int8_t> union_maps(const KoszulCtx& c, int inner, int outer, bool transpose_maps) {
    const int cpg = (2 * inner + 15) / 16, ho = (outer + 7) / 8 * 8, N = 2 * ho;
    std::vector<int8_t> maps((static_cast<size_t>(c.r) * cpg + (cpg & 1)) * N * 16, 0);
    for (int i = 0; i < c.r; ++i)
        for (int row = 0; row < 2 * inner; ++row) {
            const int limb = row / inner, u = row - limb * inner;
            for (int o = 0; o < outer; ++o) {
                // forward: coefficient M_i[o][u]; transpose: M_i[u][o]; times 255 for the hi rows
                const uint64_t raw = transpose_maps
                                         ? c.maps_canonical[(static_cast<size_t>(i) * c.co + u) * c.ci + o]
                                         : c.maps_canonical[(static_cast<size_t>(i) * c.co + o) * c.ci + u];
                const uint32_t v = static_cast<uint32_t>((limb ? 255u : 1u) * raw % c.p);
                int8_t lo, hi;
                split_limbs(to_balanced(v, c.mod), lo, hi);
                int8_t* at = maps.data() + (static_cast<size_t>(i) * cpg + row / 16) * N * 16 + row % 16;
                at[static_cast<size_t>(o) * 16] = lo;
                at[static_cast<size_t>(ho + o) * 16] = hi;
            }
        }
    return maps;
}

// D.order: the blocks of a direction in the order of star_quad(), n_order >=
// n_blk entries, kNoBlock where the last four of a kind have no block.
void build_order(KoszulCtx& c, KoszulCtx::I8State::Dir& D, uint64_t n_blk, uint64_t n_order, bool forward,
                 const BinomTable& binoms) {
    const int size = forward ? c.k - 1 : c.k;
    const unsigned ctas = blocks_of(n_blk, kOrderThreads);
    D.order = c.alloc<uint32_t>(n_order);
    // With a tile a CTA at most, a kernel is one tile's latency whatever its
    // generators: lexicographic (the order's set-up took 0.1 ms of 0.8).
    if (n_order * c.nbi <= static_cast<uint64_t>(c.sms) * 128) {
        order_plain_kernel<<<blocks_of(n_order, kOrderThreads), kOrderThreads, 0, c.own_stream>>>(
            D.order, static_cast<uint32_t>(n_blk), static_cast<uint32_t>(n_order));
        BW_CHECK_LAUNCH();
        return;
    }
    uint32_t* tmp = c.alloc<uint32_t>(2 * (ctas + 1ull) + n_blk + n_blk / 4 + 1);
    uint2* counts = reinterpret_cast<uint2*>(tmp);
    uint32_t *rest = tmp + 2 * (ctas + 1ull), *four = rest + n_blk;
    const long long n = static_cast<long long>(n_blk);
    BW_CUDA(cudaMemsetAsync(D.order, 0xFF, n_order * 4, c.own_stream));
    order_count_kernel<<<ctas, kOrderThreads, 0, c.own_stream>>>(counts, n, c.r, size, forward, binoms);
    order_scan_kernel<<<1, 1024, 0, c.own_stream>>>(counts, static_cast<int>(ctas));
    order_place_kernel<<<ctas, kOrderThreads, 0, c.own_stream>>>(counts, D.order, rest, four, n, c.r, size, forward,
                                                                 binoms);
    order_rest_kernel<<<ctas, kOrderThreads, 0, c.own_stream>>>(counts + ctas, rest, four, D.order);
    BW_CHECK_LAUNCH();
    c.release(tmp);   // cudaFree waits for the kernels
}

// Builds the stage list for D.u's generators a stage: CTA c's tiles are c,
// c + grid, ..., their stages one after the other.
void build_stage_list(KoszulCtx& c, KoszulCtx::I8State::Dir& D, uint64_t n_in, int inner) {
    I8Union& U = D.u;
    if (D.list_gs != U.gs || D.list_issuers != U.issuers) {
        for (uint32_t** p : {&D.start, &D.words, &D.steps})
            if (*p) {
                c.release(*p);
                *p = nullptr;
            }
        const uint64_t tiles = D.mask.size();
        const int bt = 128 / c.nbi;
        std::vector<uint32_t> start(D.grid + 1, 0u), tile_stage(tiles);
        uint32_t at = 0;
        for (unsigned cta = 0; cta < D.grid; ++cta) {
            start[cta] = at;
            for (uint64_t t = cta; t < tiles; t += D.grid) {
                tile_stage[t] = at;
                at += static_cast<uint32_t>((__builtin_popcount(D.mask[t]) + U.gs - 1) / U.gs);
            }
        }
        start[D.grid] = at;
        D.start = c.alloc<uint32_t>(start.size());
        D.words = c.alloc<uint32_t>(static_cast<uint64_t>(at) * U.gs * bt);
        D.steps = c.alloc<uint32_t>(static_cast<uint64_t>(at) * U.row);
        uint32_t* d_ts = c.alloc<uint32_t>(tiles);
        BW_CUDA(cudaMemcpyAsync(D.start, start.data(), start.size() * 4, cudaMemcpyHostToDevice, c.own_stream));
        BW_CUDA(cudaMemcpyAsync(d_ts, tile_stage.data(), tiles * 4, cudaMemcpyHostToDevice, c.own_stream));
        const uint32_t run16 = static_cast<uint32_t>((c.nbi / 16) * inner);
        union_tables_kernel<<<blocks_of(tiles, 128), 128, 0, c.own_stream>>>(
            D.inc, D.order, D.d_mask, d_ts, D.words, D.steps, static_cast<long long>(tiles), c.r, bt, U.gs, U.cpg,
            2 * U.ho, U.row, U.issuers, run16, static_cast<uint32_t>(n_in * run16));
        BW_CHECK_LAUNCH();
        BW_CUDA(cudaStreamSynchronize(c.own_stream));
        c.release(d_ts);
        D.list_gs = U.gs;
        D.list_issuers = U.issuers;
    }
    U.n_tiles = static_cast<long long>(D.mask.size());
    U.order = D.order;
    U.start = D.start;
    U.words = D.words;
    U.steps = D.steps;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn tensor_map_encoder() {
    static const EncodeTiledFn encode = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<EncodeTiledFn>(f);
    }();
    BW_REQUIRE(encode != nullptr, "INT8 form: cuTensorMapEncodeTiled is not available from the driver");
    return encode;
}

// One limb of a block array as a 2-D tensor for the gathers: rows = the
// (sign, block, h) runs of dim * 16 bytes (the -plane's rows after the
// +plane's), 8-byte elements; box = one run of dim_pad * 16 bytes.
void encode_plane_map(CUtensorMap* map, const int8_t* base, uint64_t n_blk, int dim, int dim_pad, int hg) {
    BW_REQUIRE(reinterpret_cast<uintptr_t>(base) % 16 == 0, "INT8 form: plane not 16-byte aligned");
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(2 * dim), static_cast<cuuint64_t>(2 * n_blk * hg)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(dim) * 16};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(2 * dim_pad), 1};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult rc = tensor_map_encoder()(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 2, const_cast<int8_t*>(base), dims,
                                             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    BW_REQUIRE(rc == CUDA_SUCCESS, "INT8 form: cuTensorMapEncodeTiled failed (code " + std::to_string(rc) + ")");
}

// One limb of a source block array as a 3-D tensor for the projection: (bytes of
// a run, column group, block), 8-byte elements; box = one group's runs of sb
// blocks (sb and 2 * dim are at most 256).
void encode_run_map(CUtensorMap* map, const int8_t* base, uint64_t n_blk, int dim, int hg, int sb) {
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(2 * dim), static_cast<cuuint64_t>(hg), n_blk};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(dim) * 16, static_cast<cuuint64_t>(dim) * 16 * hg};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(2 * dim), 1, static_cast<cuuint32_t>(sb)};
    const cuuint32_t estr[3] = {1, 1, 1};
    const CUresult rc = tensor_map_encoder()(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, const_cast<int8_t*>(base), dims,
                                             strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    BW_REQUIRE(rc == CUDA_SUCCESS, "INT8 form: cuTensorMapEncodeTiled failed (code " + std::to_string(rc) + ")");
}

// Projection stage shape: SB whole source blocks per stage, KP = SB * dim
// rounded up to 32, about kProjStageTarget bytes of X tile and W runs, the
// least padding first.  Allocates the X tiles.
void plan_projection(KoszulCtx& c, KoszulCtx::I8State& S) {
    I8Proj& P = S.proj;
    BW_REQUIRE(c.m >= 1 && c.m <= 64, "INT8 form: projection width must be 1..64");
    P.m = c.m;
    P.n_out = c.nb;
    P.mg = (c.m + 15) / 16;
    P.dim = c.ci;
    P.n_blk = static_cast<long long>(c.n_s);
    const int row_bytes = (2 * P.mg + 2 * (c.nbi / 16)) * 16;
    int best_sb = 1;
    double best_fill = 0;
    const int max_sb = c.nbi == 16 ? 4096 : 256;   // a box has at most 256 blocks
    for (int sb = 1; sb <= max_sb; ++sb) {
        const int kp = (sb * P.dim + 31) / 32 * 32;
        if (sb > 1 && kp * row_bytes > kProjStageTarget) break;
        const double fill = static_cast<double>(sb * P.dim) / kp;
        if (fill >= best_fill) {
            best_fill = fill;
            best_sb = sb;
        }
    }
    P.sb = best_sb;
    P.kp = (best_sb * P.dim + 31) / 32 * 32;
    P.n_stages = static_cast<int>((P.n_blk + P.sb - 1) / P.sb);
    P.drain = std::max(1, 131072 / P.kp);
    const uint32_t group_bytes = static_cast<uint32_t>(P.kp) * 16;
    P.a_bytes = 2 * P.mg * group_bytes;
    P.slot_bytes = P.a_bytes + 2 * (c.nbi / 16) * group_bytes;
    // the M = 128 A descriptor spans 8 groups from the tile start
    const uint32_t reach = 8 * group_bytes;
    P.pad_bytes = reach > P.slot_bytes ? reach - P.slot_bytes : 0;
    const size_t extra = static_cast<size_t>(32) * P.mg * 2 * c.nbi * 4 + (2 * 8 + 2 * 2 + 1) * 8 + 16;
    const size_t limit = static_cast<size_t>(kMaxSmem) - 1024;   // headroom for the kernel's static flag
    int slots = 4;
    while (slots > 2 && static_cast<size_t>(slots) * P.slot_bytes + P.pad_bytes + extra > limit) --slots;
    BW_REQUIRE(static_cast<size_t>(slots) * P.slot_bytes + P.pad_bytes + extra <= limit,
               "INT8 form: projection stage does not fit in shared memory");
    P.slots = slots;
    S.proj_smem = static_cast<size_t>(slots) * P.slot_bytes + P.pad_bytes + extra;
    P.mod = c.mod;
    P.c1 = to_balanced(255u % c.p, c.mod);
    P.c2 = to_balanced(static_cast<uint32_t>((255ull * 255ull) % c.p), c.mod);
    P.err = S.err;
    S.proj_grid = static_cast<unsigned>(std::max(1, std::min(P.n_stages, c.sms)));
    BW_REQUIRE(S.proj_grid <= std::max<unsigned>(c.proj_grid, static_cast<unsigned>(c.sms)),
               "INT8 form: projection grid above the partials buffer");
    S.xt = c.alloc<int8_t>(static_cast<uint64_t>(P.n_stages) * P.a_bytes);
    P.xt = S.xt;
}

template <int NB>
void launch_i8(KoszulCtx& c, KoszulCtx::I8State::Dir& D, const CUtensorMap* maps, bool after_projection,
               cudaStream_t st) {
    if (D.use_union) {
        D.u.late_wait = after_projection ? 1 : 0;
        BW_REQUIRE(D.u.start != nullptr && D.u.words != nullptr && D.u.steps != nullptr && D.u.maps != nullptr,
                   "internal: INT8 stage list missing for the union kernel");
        launch_dependent(D.u.canon ? i8_union_gemm_kernel<NB, true> : i8_union_gemm_kernel<NB, false>, D.grid,
                         union_warps::threads, D.smem, st, D.u);
        BW_CHECK_LAUNCH();
        ++c.launches;
        return;
    }
    BW_REQUIRE(D.p.inc != nullptr && (!D.gather4 || D.p.rows4 != nullptr) && D.p.b_tiles != nullptr,
               "internal: INT8 gather tables missing for the chosen producer");
    if (D.gather4)
        i8_gather_hybrid_kernel<NB><<<D.grid, kHyThreads, D.smem, st>>>(maps[0], maps[1], D.p);
    else if (D.pw == 16)
        i8_gather_gemm_kernel<NB, 16><<<D.grid, GatherWarps<16>::threads, D.smem, st>>>(D.p);
    else
        i8_gather_gemm_kernel<NB, 8><<<D.grid, GatherWarps<8>::threads, D.smem, st>>>(D.p);
    BW_CHECK_LAUNCH();
    ++c.launches;
}

}  // namespace

void KoszulCtx::i8_destroy() {
    if (i8 != nullptr && i8->h_err != nullptr) error_word_release(i8->h_err, i8->err_context);
    delete i8;
    i8 = nullptr;
}

void KoszulCtx::i8_setup() {
    BW_REQUIRE(nbi == 16 || nbi == 32, "INT8 form: internal block width must be 16 or 32");
    // two double-buffered accumulators of 2 N <= 256 columns each fill the 512 TMEM columns
    BW_REQUIRE(ci <= 64 && co <= 64, "INT8 form: dim_in and dim_out must be at most 64");
    BW_REQUIRE(static_cast<long long>(r) * std::max(ci, co) <= 1024, "INT8 form: r * dim above 1024 (int32 bound)");
    BW_REQUIRE(r <= 32, "INT8 form: at most 32 generators (one per lane)");
    int major = 0;
    BW_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
    BW_REQUIRE(major == 10, "INT8 form needs an sm_100 GPU (tcgen05)");
    i8 = new I8State();
    I8State& S = *i8;
    // each limb's -plane directly after its +plane (one tensor map covers both signs)
    for (int b = 0; b < 3; ++b) {
        const uint64_t plane = (b < 2 ? n_src : n_tgt) * nbi;
        // the gather producers address a +plane and its -plane in 16-byte units below 2^32 - 1
        BW_REQUIRE(2 * plane / 16 < 0xFFFFFFFFull, "INT8 form: limb planes above the 16-byte offset range");
        for (int limb = 0; limb < 2; ++limb) {
            int8_t* pair = alloc<int8_t>(2 * plane);
            S.planes[b][limb] = pair;
            S.planes[b][limb + 2] = pair + plane;
        }
    }
    S.h_err = error_word_acquire(S.err_context);
    *S.h_err = 0;
    BW_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&S.err), const_cast<int*>(S.h_err), 0));
    plan_projection(*this, S);
    const int hg = nbi / 16;
    // The producers that may be used.  BW_I8_PRODUCER=union, =cpasync or
    // =hybrid restricts the choice to one, two of them with a comma between d's
    // and d^T's to one each.
    struct {
        bool uni = true, g4 = true, cp = true;
    } allow[2];
    bool tune = true;
    if (const char* e = std::getenv("BW_I8_PRODUCER")) {
        const std::string text = e;
        const size_t comma = text.find(',');
        for (int dir = 0; dir < 2; ++dir) {
            const std::string want =
                comma == std::string::npos ? text : dir == 0 ? text.substr(0, comma) : text.substr(comma + 1);
            allow[dir] = {want != "cpasync" && want != "hybrid", want != "cpasync" && want != "union",
                          want != "hybrid" && want != "union"};
        }
    }
    if (const char* e = std::getenv("BW_I8_TUNE")) tune = std::string(e) != "0";
    // BW_I8_PRODUCER_WARPS=8 or =16 restricts the cp.async producers' warp count
    std::vector<int> pws{8, 16};
    if (const char* e = std::getenv("BW_I8_PRODUCER_WARPS")) {
        const int v = std::atoi(e);
        if (v == 8 || v == 16) pws = {v};
    }
    // Plans of a direction (see Cand): the union kernel's, and the dense
    // producers' only where the union kernel's resident maps leave room for
    // fewer than eight generators in flight (maps of 2 r inner rows: r * inner
    // * outer above about 32,000).  With more room the union kernel won at every
    // shape timed (us, dense against union: r=19 k=9 20->28 n=16 179/92 d and
    // 228/127 d^T; r=21 k=10 32->40 n=32 1726/1050 and 2429/1260), also where it
    // pads most, at dims 1 to 16 (a step, dense / union: r=20 k=10 1->1 n=32
    // 683/398, 4->5 921/448; r=16 k=8 1->1 n=16 34.6/27.4; r=31 k=5 1->1 n=16
    // 158/149; r=31 k=28 1->1 n=16 40.4/35.7; 150 shapes, 1.06 to 2.0 times).  Its
    // kernels alone are there within 15 % of the dense ones or faster.
    struct Cand {
        int kind;                        // 0 dense cp.async, 1 dense hybrid, 2 union
        int gps, t_tma, pw, issuers;     // as in TuneChoice
    };
    std::vector<Cand> cands[2];
    TuneKey keys[2];
    const BinomTable binoms = binom_table();
    for (int dir = 0; dir < 2; ++dir) {
        I8State::Dir& D = dir == 0 ? S.fwd : S.bwd;
        const uint64_t n_out = dir == 0 ? n_t : n_s, n_in = dir == 0 ? n_s : n_t;
        const int inner = dir == 0 ? ci : co, outer = dir == 0 ? co : ci, bt = 128 / nbi;
        int in_flight = 0;      // generators, of the roomiest union plan
        // four generators a stage or near it (fewer leave room for more slots but
        // pay a hand-over between the roles for less work), in 2 or 4 groups; two
        // MMA warps where they fit (us at the two sizes of bw_koszul_i8_union.cuh,
        // one warp / two: d 130/92 and 1190/1050, d^T 156/127 and 1410/1260)
        for (int g : {4, 3, 6, 8, 2}) {
            for (int groups : {2, 4})
                for (int issuers : {2, 1})
                    if (allow[dir].uni && plan_union(*this, D, inner, outer, dir == 1, g, groups, issuers)) {
                        cands[dir].push_back({2, g, groups, 8, issuers});
                        in_flight = std::max(in_flight, D.u.slots * g);
                    }
        }
        const bool dense = (allow[dir].g4 || allow[dir].cp) && in_flight < 8;
        BW_REQUIRE(!cands[dir].empty() || dense, "INT8 form: no union plan fits in shared memory");
        if (dense) {
            if (allow[dir].cp)
                // the fill heuristic's stage, and fewer or more generators a stage
                // (smaller stages leave room for more pipeline slots)
                for (int pw : pws) {
                    cands[dir].push_back({0, 0, 0, pw, 1});
                    for (int g : {4, 6, 8, 12})
                        if (g < r) cands[dir].push_back({0, g, 0, pw, 1});
                }
            if (allow[dir].g4)
                for (int gs = 1; gs <= std::min(3, (r + 3) / 4); ++gs)
                    for (int qt = 1; qt <= 3; ++qt) cands[dir].push_back({1, 4 * gs, qt * bt / 4, 8, 1});
        }
        keys[dir] = TuneKey{r, k, inner, outer, nbi, dir, sms,
                            (allow[dir].g4 ? 1 : 0) | (allow[dir].cp ? 2 : 0) | (pws.size() == 1 ? pws[0] * 4 : 0) |
                                (allow[dir].uni ? 128 : 0)};
        TuneChoice known{};
        // a shape tuned earlier in this process: its choice alone
        if (tune && tune_lookup(keys[dir], known))
            cands[dir] = {{known.kind, known.gps, known.t_tma, known.pw, known.issuers}};
        // the tables that the candidates read
        bool any_union = false, any_rows = false;
        for (const Cand& c : cands[dir]) {
            any_union = any_union || c.kind == 2;
            any_rows = any_rows || c.kind == 1;
        }
        D.inc = alloc<uint32_t>(n_out * r);
        incidence_kernel<<<blocks_of(n_out, 128), 128, 0, own_stream>>>(D.inc, static_cast<long long>(n_out), r, k,
                                                                         dir == 0, binoms);
        if (any_rows) {
            const int groups = (r + 3) / 4;
            BW_REQUIRE(2 * n_in * hg + hg < (1ull << 31), "INT8 form: plane rows above the TMA coordinate range");
            D.rows4 = alloc<int4>(n_out * groups);
            gather_rows_kernel<<<blocks_of(n_out * groups, 256), 256, 0, own_stream>>>(
                D.inc, D.rows4, static_cast<long long>(n_out), r, groups, static_cast<long long>(n_in), hg);
        }
        if (any_union) {
            const uint64_t tiles = (n_out + bt - 1) / bt;
            D.d_mask = alloc<uint32_t>(tiles);
            build_order(*this, D, n_out, tiles * bt, dir == 0, binoms);
            union_mask_kernel<<<blocks_of(tiles, 128), 128, 0, own_stream>>>(D.inc, D.order, D.d_mask,
                                                                             static_cast<long long>(tiles), r, bt);
            D.mask.resize(tiles);
            BW_CUDA(cudaMemcpyAsync(D.mask.data(), D.d_mask, tiles * 4, cudaMemcpyDeviceToHost, own_stream));
            const std::vector<int8_t> maps = union_maps(*this, inner, outer, dir == 1);
            D.maps = alloc<int8_t>(maps.size());
            BW_CUDA(cudaMemcpyAsync(D.maps, maps.data(), maps.size(), cudaMemcpyHostToDevice, own_stream));
            BW_CUDA(cudaStreamSynchronize(own_stream));
        }
        BW_CHECK_LAUNCH();
    }
    for (int b = 0; b < 3; ++b) {
        const uint64_t n_blk = b < 2 ? n_s : n_t;
        const int dim = b < 2 ? ci : co;
        for (int limb = 0; limb < 2; ++limb)
            encode_plane_map(&S.maps[b][limb], S.planes[b][limb], n_blk, dim, dim + (dim & 1), hg);
        for (int limb = 0; limb < 2 && b < 2 && hg > 1; ++limb)
            encode_run_map(&S.runs[b][limb], S.planes[b][limb], n_blk, dim, hg, S.proj.sb);
    }
    // Failure tests only (the environment of the creating process): a short
    // limit on every pipeline wait, and a first stage that CTA 0 of the d/d^T
    // kernel never fills, so that its consumer's wait runs out and the kernel
    // gives up, frees its TMEM and returns; the host then reports status 2.
    // (The hold starts after the set-up's own timing launches.)
    uint32_t wait_limit = tc::kWaitLimit;
    if (const char* e = std::getenv("BW_TEST_WAIT_LIMIT")) {
        const unsigned long v = std::strtoul(e, nullptr, 10);
        if (v >= 1 && v < tc::kWaitLimit) wait_limit = static_cast<uint32_t>(v);
    }
    int hold = 0;
    if (const char* e = std::getenv("BW_TEST_HOLD_FIRST_STAGE")) hold = (*e && std::string(e) != "0") ? 1 : 0;
    S.proj.wait_limit = wait_limit;
    int cap_g = 0, cap_4 = 0, cap_u = 0;
    dispatch_i8_nb(nbi, [&](auto NBc) {
        cap_g = std::min(allow_dynamic_smem(i8_gather_gemm_kernel<decltype(NBc)::value, 8>, device),
                         allow_dynamic_smem(i8_gather_gemm_kernel<decltype(NBc)::value, 16>, device));
        cap_u = std::min(allow_dynamic_smem(i8_union_gemm_kernel<decltype(NBc)::value, false>, device),
                         allow_dynamic_smem(i8_union_gemm_kernel<decltype(NBc)::value, true>, device));
        cap_4 = allow_dynamic_smem(i8_gather_hybrid_kernel<decltype(NBc)::value>, device);
        const int cap_p = allow_dynamic_smem(i8_project_tc_kernel<decltype(NBc)::value>, device);
        BW_REQUIRE(static_cast<int>(S.proj_smem) <= cap_p, "INT8 form: shared-memory plan above the device limit");
    });
    const int bt = 128 / nbi;
    S.fwd.p.n_blk = static_cast<long long>(n_t);
    S.bwd.p.n_blk = static_cast<long long>(n_s);
    S.fwd.p.row_oob = static_cast<int32_t>(2 * n_s * hg);   // the forward gathers Y (source blocks)
    S.bwd.p.row_oob = static_cast<int32_t>(2 * n_t * hg);   // d^T gathers Z (target blocks)
    S.fwd.grid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>((n_t + bt - 1) / bt, sms)));
    S.bwd.grid = static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>((n_s + bt - 1) / bt, sms)));

    // Stage plans.  Each direction's plan is chosen by timing every candidate
    // that fits in shared memory on this device, at set-up, on the context's
    // own buffers (the kernels' work does not depend on the values); the choice
    // is cached per shape for the life of the process.  BW_I8_TUNE=0 takes the
    // first candidate that fits instead.
    std::string text;
    for (int dir = 0; dir < 2; ++dir) {
        I8State::Dir& D = dir == 0 ? S.fwd : S.bwd;
        const int inner = dir == 0 ? ci : co, outer = dir == 0 ? co : ci;
        const int in_buf = dir == 0 ? I8_YA : I8_Z, out_buf = dir == 0 ? I8_Z : I8_YB;
        auto plan = [&](const Cand& c) {
            D.use_union = c.kind == 2;
            if (D.use_union) {
                if (!plan_union(*this, D, inner, outer, dir == 1, c.gps, c.t_tma, c.issuers) ||
                    static_cast<int>(D.smem) > cap_u)
                    return false;
                build_stage_list(*this, D, dir == 0 ? n_s : n_t, inner);
                D.u.err = S.err;
                D.u.wait_limit = wait_limit;
                D.u.hold_first_stage = 0;
                return true;
            }
            const bool g4 = c.kind == 1;
            if (D.b_tiles) release(D.b_tiles);
            D.b_tiles = nullptr;
            if (!plan_direction(*this, D, inner, outer, dir == 1, g4, c.gps)) return false;
            if (static_cast<int>(D.smem) > (g4 ? cap_4 : cap_g)) return false;
            D.pw = g4 ? 8 : c.pw;
            D.p.t_tma = g4 ? c.t_tma : 0;
            D.p.err = S.err;
            D.p.wait_limit = wait_limit;
            D.p.hold_first_stage = 0;
            D.p.inc = D.inc;
            D.p.rows4 = D.rows4;
            return true;
        };
        std::string tried;
        Cand choice = cands[dir][0];
        if (!tune) {
            for (const Cand& cand : cands[dir])
                if (plan(cand)) {
                    choice = cand;
                    break;
                }
        } else if (cands[dir].size() > 1) {
            double best = 1e30;
            for (const Cand& cand : cands[dir]) {
                if (!plan(cand)) continue;
                const double ms = i8_time_direction(dir == 0, in_buf, out_buf);
                char buf[96];
                const char* sep = tried.empty() ? "" : ", ";
                if (cand.kind == 2)
                    std::snprintf(buf, sizeof buf, "%su%d/%d/%d %.4f", sep, cand.gps, cand.t_tma,
                                  cand.issuers, ms);
                else if (cand.kind == 1)
                    std::snprintf(buf, sizeof buf, "%shybrid stage=%d tma=%d/%d: %.4f ms", sep, D.p.gi, cand.t_tma, bt,
                                  ms);
                else
                    std::snprintf(buf, sizeof buf, "%scp.async stage=%d warps=%d: %.4f ms", sep, D.p.gi, cand.pw, ms);
                tried += buf;
                if (ms < best) {
                    best = ms;
                    choice = {cand.kind, cand.kind == 2 ? cand.gps : D.p.gi, cand.t_tma, cand.pw, cand.issuers};
                }
            }
            BW_REQUIRE(best < 1e30, "INT8 form: no stage plan fits in shared memory");
            tune_store(keys[dir], TuneChoice{choice.kind, choice.pw, choice.gps, choice.t_tma, choice.issuers, best});
        }
        BW_REQUIRE(plan(choice), "INT8 form: maps too large for shared memory");
        D.gather4 = !D.use_union && D.gather4;
        char buf[256];
        if (D.use_union)
            std::snprintf(buf, sizeof buf, "%s: union stage=%d generators, %d producer groups, %d MMA warps, %d slots, "
                          "%zu B shared", dir == 0 ? "d" : "d^T", D.u.gs, D.u.groups, D.u.issuers, D.u.slots, D.smem);
        else if (D.gather4)
            std::snprintf(buf, sizeof buf, "%s: hybrid (TMA gathers for %d of %d blocks) stage=%d generators, %d slots, "
                          "%zu B shared", dir == 0 ? "d" : "d^T", D.p.t_tma, bt, D.p.gi, D.p.slots, D.smem);
        else
            std::snprintf(buf, sizeof buf, "%s: cp.async stage=%d generators, %d producer warps, %d slots, %zu B shared",
                          dir == 0 ? "d" : "d^T", D.p.gi, D.pw, D.p.slots, D.smem);
        text += (text.empty() ? "" : "; ") + std::string(buf);
        if (!tried.empty()) text += " (tuned: " + tried + ")";
    }
    // the tables of the producers that were not chosen are freed: the union
    // kernel reads its stage list only, the hybrid producer both dense tables
    for (I8State::Dir* D : {&S.fwd, &S.bwd}) {
        auto drop = [&](auto*& p) {
            if (p) release(p);
            p = nullptr;
        };
        if (D->use_union) {
            drop(D->inc);
        } else {
            drop(D->start);
            drop(D->words);
            drop(D->steps);
            drop(D->maps);
            drop(D->order);
        }
        if (!D->gather4) drop(D->rows4);
        drop(D->d_mask);
        D->mask = std::vector<uint32_t>();
        D->u.hold_first_stage = hold;
        D->p.inc = D->inc;
        D->p.rows4 = D->rows4;
        D->p.hold_first_stage = hold;
    }
    char pbuf[160];
    std::snprintf(pbuf, sizeof pbuf, "; projection: %d blocks a stage (%d rows), %d slots", S.proj.sb, S.proj.kp,
                  S.proj.slots);
    S.plan_text = text + pbuf;
    BW_CUDA(cudaStreamSynchronize(own_stream));
}

const std::string& KoszulCtx::i8_plan_text() const { return i8->plan_text; }

// Device time of one direction's gather-GEMM on the context's buffers: one
// warm-up launch, then the mean of three (CUDA events on the own stream).
double KoszulCtx::i8_time_direction(bool forward_dir, int in_buf, int out_buf) {
    cudaEvent_t e0, e1;
    BW_CUDA(cudaEventCreate(&e0));
    BW_CUDA(cudaEventCreate(&e1));
    i8_run(forward_dir, in_buf, out_buf, !forward_dir, own_stream);
    BW_CUDA(cudaEventRecord(e0, own_stream));
    for (int i = 0; i < 3; ++i) i8_run(forward_dir, in_buf, out_buf, !forward_dir, own_stream);
    BW_CUDA(cudaEventRecord(e1, own_stream));
    BW_CUDA(cudaEventSynchronize(e1));
    float ms = 0;
    BW_CUDA(cudaEventElapsedTime(&ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    i8_check_error();
    return ms / 3.0;
}

uint64_t KoszulCtx::i8_kernels_per_step() const { return 3; }

void KoszulCtx::i8_run(bool forward_dir, int in_buf, int out_buf, bool scale, cudaStream_t st, bool after_projection,
                       uint32_t* canon) {
    I8State::Dir& D = forward_dir ? i8->fwd : i8->bwd;
    if (D.use_union) {
        D.u.in[0] = i8->planes[in_buf][PL_LO];
        D.u.in[1] = i8->planes[in_buf][PL_HI];
        for (int pl = 0; pl < 4; ++pl) D.u.out[pl] = i8->planes[out_buf][pl];
        D.u.diag = (!forward_dir && scale) ? d_diag : nullptr;
        D.u.canon = canon;
        D.u.width = nb;
    }
    for (int pl = 0; pl < 4; ++pl) {
        D.p.in[pl] = i8->planes[in_buf][pl];
        D.p.out[pl] = i8->planes[out_buf][pl];
    }
    D.p.in_neg_off = i8->planes[in_buf][PL_NLO] - i8->planes[in_buf][PL_LO];
    D.p.diag = (!forward_dir && scale) ? d_diag : nullptr;
    dispatch_i8_nb(nbi, [&](auto NBc) { launch_i8<decltype(NBc)::value>(*this, D, i8->maps[in_buf], after_projection, st); });
}

// d or d^T with its result as canonical residues in the caller's buffer.  The
// union kernel's epilogue writes them (limb planes and a conversion kernel after
// it: forward at r = 19, k = 9, 20 -> 28, 16 columns 197 us, now 169).
void KoszulCtx::i8_run_to(bool forward_dir, int in_buf, int out_buf, bool scale, uint32_t* out, cudaStream_t st) {
    const bool direct = (forward_dir ? i8->fwd : i8->bwd).use_union;
    i8_run(forward_dir, in_buf, out_buf, scale, st, false, direct ? out : nullptr);
    if (!direct) i8_from_limbs(out_buf, out, st);
}

void KoszulCtx::i8_check_error() {
    const int err = *i8->h_err;   // the caller has synchronised with the kernels
    if (err != 0) {
        *i8->h_err = 0;
        static const char* const names[] = {"", "ERR_WAIT_FULL: consumer waited for a loaded stage",
                                            "ERR_WAIT_EMPTY: producer waited for a free stage",
                                            "ERR_WAIT_ACCUM: epilogue waited for an accumulator",
                                            "ERR_WAIT_ACCUM_FREE: MMA waited for a free accumulator",
                                            "ERR_WAIT_FINAL: final drain of in-flight MMAs",
                                            "ERR_LAYOUT: shared-memory layout check failed"};
        const std::string what = (err >= 1 && err <= 6) ? names[err] : "code " + std::to_string(err);
        throw Error("INT8 tensor-core kernel gave up waiting (" + what + ")", 2);
    }
}

int KoszulCtx::i8_dim(int buf) const { return buf == I8_Z ? co : ci; }
uint64_t KoszulCtx::i8_rows(int buf) const { return buf == I8_Z ? n_tgt : n_src; }

void KoszulCtx::i8_to_limbs(const uint32_t* in, int buf, cudaStream_t st) {
    const uint64_t quads = i8_rows(buf) * nbi / 4;
    int8_t** pl = i8->planes[buf];
    dispatch_i8_nb(nbi, [&](auto NBc) {
        to_limbs_kernel<decltype(NBc)::value><<<quad_grid(quads, sms), 256, 0, st>>>(
            in, pl[0], pl[1], pl[2], pl[3], static_cast<long long>(quads), static_cast<uint32_t>(i8_dim(buf)),
            static_cast<uint32_t>(nb), quad_aligned(in), mod);
    });
    BW_CHECK_LAUNCH();
    ++launches;
}

void KoszulCtx::i8_from_limbs(int buf, uint32_t* out, cudaStream_t st) {
    const uint64_t quads = i8_rows(buf) * nb / 4;
    const uint32_t w_shift = nb == 4 ? 0 : nb == 8 ? 1 : nb == 16 ? 2 : 3;
    int8_t** pl = i8->planes[buf];
    dispatch_i8_nb(nbi, [&](auto NBc) {
        from_limbs_kernel<decltype(NBc)::value><<<quad_grid(quads, sms), 256, 0, st>>>(
            pl[0], pl[1], out, static_cast<long long>(quads), static_cast<uint32_t>(i8_dim(buf)), w_shift,
            quad_aligned(out), mod);
    });
    BW_CHECK_LAUNCH();
    ++launches;
}

void KoszulCtx::i8_load_x(const uint32_t* x, cudaStream_t st) {
    const I8Proj& P = i8->proj;
    const long long quads = static_cast<long long>(P.n_stages) * P.mg * P.kp * 4;
    x_tiles_kernel<<<quad_grid(quads, sms), 256, 0, st>>>(x, i8->xt, static_cast<long long>(n_src), m, P.mg, ci, P.sb,
                                                          P.kp, quads, quad_aligned(x), mod);
    BW_CHECK_LAUNCH();
    ++launches;
}

void KoszulCtx::i8_project(int buf, cudaStream_t st) {
    I8Proj P = i8->proj;
    P.w[0] = i8->planes[buf][0];
    P.w[1] = i8->planes[buf][1];
    P.partials = d_partials;
    P.counter = d_counter;
    P.state = d_seq_state;
    dispatch_i8_nb(nbi, [&](auto NBc) {
        launch_dependent(i8_project_tc_kernel<decltype(NBc)::value>, i8->proj_grid, kProjThreads, i8->proj_smem, st,
                         i8->runs[buf][0], i8->runs[buf][1], P);
    });
    BW_CHECK_LAUNCH();
    ++launches;
}

// One INT8 step on the limb state: cur -> other, append a_i.
//
// d reads what the step before it wrote in d^T and writes Z, which that d^T
// has read: it has nothing to do with the projection between them.  Where the
// kernel launched before it on `st` is this state's projection, d therefore
// runs without waiting for that kernel (it begins once every CTA of the
// projection has seen d^T complete, and waits for it before it ends, so that a
// completed kernel still implies all earlier ones).  A step takes, us, waiting
// at the start / at the end: r = 10, k = 4, 16 -> 24, 8 columns 14.9 / 12.0;
// r = 19, k = 9, 20 -> 28, 16 columns 236 / 235; r = 21, k = 10, 32 -> 40, 32
// columns 3050 / 2930; r = 23, k = 11, 32 -> 40, 32 columns 13350 / 12900.
void KoszulCtx::i8_step_once(cudaStream_t st, bool after_step) {
    const int src = cur_is_a ? I8_YA : I8_YB, dst = cur_is_a ? I8_YB : I8_YA;
    i8_run(true, src, I8_Z, false, st, after_step);
    i8_run(false, I8_Z, dst, true, st);
    i8_project(dst, st);
    cur_is_a = !cur_is_a;
}

}  // namespace bw
