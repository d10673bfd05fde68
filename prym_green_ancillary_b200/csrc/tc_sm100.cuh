// Thin inline-PTX layer over the sm_100a tensor-core path used by the INT8-limb
// kernels: mbarriers, bulk global->shared copies, TMEM allocation, tcgen05.mma
// (kind::i8), tcgen05.commit and tcgen05.ld.  Shared-memory matrix descriptors
// and the instruction descriptor follow the PTX ISA layouts for tcgen05 (no
// swizzle; K-major and MN-major canonical layouts).
#pragma once

#include <cstdint>

namespace bw {
namespace tc {

// Bounded waits: a wait that runs out records an error code and returns false
// so that the kernel can wind down instead of hanging the GPU.
constexpr uint32_t kWaitLimit = 1u << 25;

enum WaitError : int {
    ERR_NONE = 0,
    ERR_WAIT_FULL = 1,      // consumer waited for a loaded stage
    ERR_WAIT_EMPTY = 2,     // producer waited for a free stage
    ERR_WAIT_ACCUM = 3,     // epilogue waited for an accumulator
    ERR_WAIT_ACCUM_FREE = 4,// MMA waited for the epilogue to free an accumulator
    ERR_WAIT_FINAL = 5,     // final drain of in-flight MMAs
    ERR_LAYOUT = 6,         // shared-memory layout check failed before any copy was issued
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Wait for the phase with the given parity to complete, at most `limit`
// tries.  `abort` (shared memory, or null) is the CTA's give-up flag: the wait
// returns false once another role of the CTA has given up, and a wait that
// runs out sets it and records `code` in the global error word.  Polling only
// the shared flag keeps every spin on-chip.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort, int* err, int code,
                                          uint32_t limit = kWaitLimit) {
    for (uint32_t i = 0; i < limit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (abort != nullptr && *abort != 0) return false;
    }
    if (abort != nullptr) *abort = 1;
    atomicCAS(err, ERR_NONE, code);
    return false;
}

// The same wait made by a whole converged warp (bar, a shared-memory address,
// and parity uniform): the outcome comes from warp votes, so every branch on
// it is uniform.  With one lane waiting (or lanes branching on their own
// outcome) a wait on a phase that is already complete costs about 230-330
// cycles of divergence handling; voted, about 70.
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int* abort, int* err, int code,
                                          uint32_t limit = kWaitLimit) {
    for (uint32_t i = 0; i < limit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (__all_sync(0xffffffffu, ok != 0)) return true;
        if (abort != nullptr && __any_sync(0xffffffffu, *abort != 0)) return false;
    }
    if (abort != nullptr) *abort = 1;
    atomicCAS(err, ERR_NONE, code);
    return false;
}

// Bulk copy of `bytes` (multiple of 16, both addresses 16-byte aligned) from
// global to this CTA's shared memory, completing on `bar` (tx bytes).
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// TMA load of a box of a 3-D tensor map (this GPU's memory, no multicast) to
// shared memory (128-byte aligned), completing on `bar` with the bytes of the
// whole box; what lies outside the tensor is filled with zeros.
__device__ __forceinline__ void tma_load3(void* dst, const void* tmap, int32_t x, int32_t y, int32_t z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// TMA gather of four rows of a 2-D tensor map (sm_100 tile::gather4): rows
// y0..y3 (any order; a row outside the tensor is filled with zeros and read
// from nowhere), columns from x for the map's box width, written back to back
// at dst (128-byte aligned shared memory of this CTA), completing on `bar`
// (tx bytes = 4 x box bytes).  No multicast: the map covers this GPU's memory.
__device__ __forceinline__ void tma_gather4(void* dst, const void* tmap, int32_t x, int32_t y0, int32_t y1,
                                            int32_t y2, int32_t y3, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y0), "r"(y1), "r"(y2), "r"(y3), "r"(smem_u32(bar))
        : "memory");
}

// Prefetch a tensor map (kernel parameter) into the descriptor cache.
__device__ __forceinline__ void prefetch_tmap(const void* tmap) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(tmap)) : "memory");
}

// 16-byte asynchronous copy global -> shared through L2 (cp.async.cg) that reads
// src_size (0 or 16) bytes and zero-fills the rest:
// src_size 0 writes 16 zero bytes without reading global memory.
__device__ __forceinline__ void cp_async16_zfill(void* dst, const void* src, uint32_t src_size) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_size)
                 : "memory");
}

// The same with the destination given as a shared-memory address.
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst_smem, const void* src, uint32_t src_size) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst_smem), "l"(src), "r"(src_size) : "memory");
}

// Arrive on `bar` once every cp.async issued so far by this thread has landed
// (the arrival is one of the barrier's expected arrivals).
__device__ __forceinline__ void cp_async_arrive_noinc(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void cp_async_arrive_noinc(uint32_t bar) {   // bar: a shared-memory address
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// Wait until every cp.async issued by this thread has completed.
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ---- TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// ---- descriptors
// Shared-memory matrix descriptor, no swizzle: start address, leading-dimension
// byte offset (LBO) and stride-dimension byte offset (SBO), version 1.  Two
// 32-bit words, so that a loop can advance the start address by adding to the
// low word (the address field holds addr >> 4 in 14 bits; shared-memory
// addresses stay below 2^18, so the sum never carries out).
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr, uint32_t lbo) {
    return ((saddr >> 4) & 0x3FFFu) | (((lbo >> 4) & 0x3FFFu) << 16);
}
__device__ __forceinline__ uint32_t desc_hi(uint32_t sbo) { return ((sbo >> 4) & 0x3FFFu) | (1u << 14); }
__device__ __forceinline__ uint64_t desc_make(uint32_t lo, uint32_t hi) {
    return (static_cast<uint64_t>(hi) << 32) | lo;
}

// Instruction descriptor of tcgen05.mma kind::i8: D = s32, A = B = s8, dense.
__host__ __device__ constexpr uint32_t idesc_i8(int M, int N, bool a_mn_major, bool b_mn_major) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) |
           (static_cast<uint32_t>(N >> 3) << 17) | (static_cast<uint32_t>(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem]^T, issued by one thread.
__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// The same issued by one elected lane of a converged warp.  The operands have
// to be values the compiler can prove warp-uniform (kernel parameters, warp
// votes and shuffles): from such values an MMA issues at the tensor pipe's
// rate, from others it costs about 100 cycles more.
__device__ __forceinline__ void mma_i8_elect(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Arrive on `bar` once all tcgen05 operations issued so far by this thread complete.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// The same by one elected lane of a converged warp (the lane that
// mma_i8_elect() elects), the barrier as a shared-memory address.
__device__ __forceinline__ void mma_commit_elect(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "elect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar)
        : "memory");
}

// 32 lanes x 16 consecutive 32-bit columns (lane = warp quadrant base + lane id).
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, int32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
// 32 lanes x 8 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, int32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

}  // namespace tc
}  // namespace bw
