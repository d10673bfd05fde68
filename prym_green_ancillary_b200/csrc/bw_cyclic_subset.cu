// Subset-major paper-mode operator: the four Koszul gathers of the eliminated
// operator with one thread per subset, on 16-bit vectors in padded blocks.
//
// Every character block of the shipped instances has at most two rows (A0
// blocks two, A1 blocks one or two, kernel-weight blocks at most one), and
// the rows of one subset's block read the same neighbour blocks with
// different coefficients.  So:
//   * the internal vectors (scaled source x, y, u, u2, t_adj) hold balanced
//     residues as int16 and give every subset's block two row slots: a block
//     is one aligned 16-byte load, found from the subset's rank alone;
//   * one thread takes a subset, loads each incidence word (neighbour rank,
//     generator, sign) and each neighbour block once, and accumulates both
//     rows of its own block;
//   * the signed coefficients of mu for (sign, generator, own character) are
//     four int32 in shared memory: one 16-byte load per incidence, indexed by
//     the code the incidence word carries (sign * n + generator).
// An incidence thus costs one coalesced word, one 16-byte load, one 16-byte
// shared load and sixteen multiply-adds.
//
// Two of the reference's kernel pairs are fused, with their intermediates in
// registers:
//   * D_m forward (cuda/cyclic_cuda_helpers.h:145-204) with the elimination
//     y = B z - R t (cyclic_elim_z_to_y_kernel, cyclic_elim_subtract_Rt_kernel,
//     :718-791): t never reaches memory;
//   * D_(m-1) transpose (:206-266) with t_adj = R^t h, z_adj = B^t h and the
//     z part of the adjoint assembly (cyclic_elim_RT_h_kernel,
//     cyclic_elim_BT_h_kernel, cyclic_elim_assemble_adjoint_kernel, :793-895):
//     h never reaches memory.
// The folded target preconditioner runs in ELL form with int16 values; it
// reads u kept in an order with row-mixing partners adjacent (so a row's
// sixteen columns lie within nine consecutive rows) and writes u2 in the
// padded subset layout.  The operator's inputs and outputs (the block B,
// S B) stay compact int32; results are the same canonical residues as the
// generic row kernels of bw_cyclic.cu, which remain for instances outside
// this format.
#include "bw_cyclic.cuh"
#include "bw_cyclic_dev.cuh"

#include <algorithm>

namespace bw {

namespace {

constexpr int kThreads = 256;
constexpr uint32_t kLow26 = (1u << 26) - 1;
constexpr int kResidentThreads = 512, kMomentThreads = 128, kResidentChunks = 4;   // sub_rounds_kernel: threads a CTA, chunks a gather, at most

using cyc::Acc4;
using cyc::ld4;
using cyc::neg4;
using cyc::scale4;
using cyc::st4;

// ----- 16-bit rows: 4 columns in 8 bytes, a block of two rows in 16
__device__ __forceinline__ uint32_t pack2(int32_t a, int32_t b) {
    return (static_cast<uint32_t>(a) & 0xFFFFu) | (static_cast<uint32_t>(b) << 16);
}
__device__ __forceinline__ int32_t lo16(uint32_t w) { return static_cast<int16_t>(w & 0xFFFFu); }
__device__ __forceinline__ int32_t hi16(uint32_t w) { return static_cast<int32_t>(w) >> 16; }
__device__ __forceinline__ uint2 pack_row(const int4& v) { return make_uint2(pack2(v.x, v.y), pack2(v.z, v.w)); }
__device__ __forceinline__ int4 unpack_row(uint32_t a, uint32_t b) { return make_int4(lo16(a), hi16(a), lo16(b), hi16(b)); }
__device__ __forceinline__ void st_block(uint4* v, uint32_t s, const int4& r0, const int4& r1) {
    const uint2 a = pack_row(r0), b = pack_row(r1);
    v[s] = make_uint4(a.x, a.y, b.x, b.y);
}

// Views of the shared-memory tables.
struct Tables {
    const int4* coef;
    const int32_t *R, *B, *a0off, *a0idx, *a1off, *a1idx, *koff, *kidx, *ych;
};

__device__ __forceinline__ Tables views(const SubsetDev& D, const int32_t* sm) {
    Tables t;
    t.coef = reinterpret_cast<const int4*>(sm);
    t.R = sm + D.o_R;
    t.B = sm + D.o_B;
    t.a0off = sm + D.o_a0off;
    t.a0idx = sm + D.o_a0idx;
    t.a1off = sm + D.o_a1off;
    t.a1idx = sm + D.o_a1idx;
    t.koff = sm + D.o_koff;
    t.kidx = sm + D.o_kidx;
    t.ych = sm + D.o_ych;
    return t;
}

// Staging reads only the constant tables, so it overlaps the end of the kernel
// before (programmatic dependent launch); the wait follows it.
__device__ __forceinline__ Tables stage(const SubsetDev& D, const int32_t* __restrict__ blob, int32_t* sm) {
    pdl_trigger();
    for (int w = threadIdx.x; w < D.blob_words; w += blockDim.x) sm[w] = __ldg(blob + w);
    __syncthreads();
    pdl_wait();
    return views(D, sm);
}

// Streamed table words: evict-first when the sector's tables exceed the L2
// (they would only push the gathered vector out), cached otherwise (small
// sectors keep tables and vectors in L2 from one application to the next).
template <bool STREAM, class T>
__device__ __forceinline__ T ld_table(const T* p) {
    if constexpr (STREAM)
        return __ldcs(p);
    else
        return __ldg(p);
}

// acc_k += c_k0 * row0 + c_k1 * row1 for the neighbour block b (two int16
// rows) and c = (c_00, c_01, c_10, c_11).
template <bool SMALL>
__device__ __forceinline__ void mac_block(const int4& c, const uint4& b, Acc4<SMALL>& acc0, Acc4<SMALL>& acc1) {
    const int4 r0 = unpack_row(b.x, b.y), r1 = unpack_row(b.z, b.w);
    acc0.mac(c.x, r0);
    acc0.mac(c.y, r1);
    acc1.mac(c.z, r0);
    acc1.mac(c.w, r1);
}

// Both rows of subset s against its `width` neighbour blocks.  The coefficient
// table is [code = sign * n + generator][own character]; a neighbour block with
// one row has zero coefficients for its second slot (which holds zeros).
// Incidence words are read once per application (ld_table).  `nin` is the
// number of blocks of `in`, which carries one more, all-zero block at nin.
template <bool SMALL, bool STREAM>
__device__ __forceinline__ void gather_block(const uint32_t* __restrict__ inc, uint32_t nsub, uint32_t s,
                                             uint32_t width, const int4* coef, int r, int ch,
                                             const uint4* __restrict__ in, uint32_t nin, Acc4<SMALL>& acc0,
                                             Acc4<SMALL>& acc1) {
    // Chunks of four incidences: a chunk's blocks are loaded together, and
    // the next chunk's words while those blocks are in flight.  Only the
    // words of a last, partial chunk are loaded under a mask; its empty slots
    // hold the zero block (code 0), so the products run unmasked.
    constexpr int U = 4;
    const uint32_t* p = inc + s;
    const size_t step = nsub;
    const uint32_t full = width / U, rem = width % U, chunks = full + (rem ? 1u : 0u);
    auto words = [&](uint32_t k, uint32_t (&w)[U]) {
        const uint32_t* q = p + static_cast<size_t>(k) * U * step;
        if (k < full) {
#pragma unroll
            for (int u = 0; u < U; ++u) w[u] = ld_table<STREAM>(q + u * step);
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) w[u] = static_cast<uint32_t>(u) < rem ? ld_table<STREAM>(q + u * step) : nin;
        }
    };
    uint32_t e[U];
    if (chunks == 0) return;
    words(0, e);
    for (uint32_t k = 0; k < chunks; ++k) {
        uint4 b[U];
#pragma unroll
        for (int u = 0; u < U; ++u) b[u] = __ldg(in + (e[u] & kLow26));
        uint32_t next[U];
        if (k + 1 < chunks) words(k + 1, next);
#pragma unroll
        for (int u = 0; u < U; ++u) mac_block<SMALL>(coef[static_cast<int>(e[u] >> 26) * r + ch], b[u], acc0, acc1);
        if (k + 1 < chunks) {
#pragma unroll
            for (int u = 0; u < U; ++u) e[u] = next[u];
        }
    }
}

#define BW_ITEMS(var, count)                                                                         \
    for (long long var = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; var < (count); \
         var += static_cast<long long>(gridDim.x) * blockDim.x)

// Scaled source: items [0, n0) are m-subsets, whose x block (compact rows
// x_off, x_off + 1 of the operator column op_col, times dc) goes to the padded
// xs; items n0 + j are the compact z rows and the extra dense columns (int32).
__global__ void __launch_bounds__(kThreads) sub_source_kernel(SubsetDev D, const int32_t* __restrict__ in,
                                                              const int32_t* __restrict__ dc, uint4* __restrict__ xs,
                                                              int32_t* __restrict__ zs) {
    extern __shared__ __align__(16) int32_t sm[];
    const Tables T = stage(D, D.blob_f, sm);
    const long long n0 = D.n0, total = n0 + static_cast<long long>(D.z_cols) + D.n_extra;
    BW_ITEMS(item, total) {
        if (item < n0) {
            const uint32_t dx = __ldg(D.m0 + item);
            const int xch = static_cast<int>(dx >> 26);
            const int nx = T.a0off[xch + 1] - T.a0off[xch];
            int4 r[2] = {make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0)};
            for (int q = 0; q < nx; ++q) {
                const long long c = cyc::op_col(D.drop0, D.drop1, static_cast<long long>(dx & kLow26) + q);
                if (c < 0) continue;   // dropped base column (replacement): zero
                const int4 v = ld4(in, c);
                r[q] = dc ? scale4(v, __ldg(dc + c), D.mod) : v;
            }
            st_block(xs, static_cast<uint32_t>(item), r[0], r[1]);
        } else {
            const long long zq = item - n0;
            const long long src = zq < static_cast<long long>(D.z_cols)
                                      ? cyc::op_col(D.drop0, D.drop1, static_cast<long long>(D.x_cols) + zq)
                                      : static_cast<long long>(D.kept_cols) + (zq - static_cast<long long>(D.z_cols));
            int4 v = make_int4(0, 0, 0, 0);
            if (src >= 0) {
                v = ld4(in, src);
                if (dc) v = scale4(v, __ldg(dc + src), D.mod);
            }
            st4(zs, zq, v);
        }
    }
}

// (m-1)-subset S: its t rows t(S, beta) = (D_m xs)(S, beta), then its y block
//   y(S, a) = sum_kappa B[a,kappa] zs(S, kappa) - sum_beta R[a,beta] t(S, beta).
template <bool SMALL, bool STREAM>
__global__ void __launch_bounds__(kThreads) sub_dm_forward_elim_kernel(SubsetDev D, const uint4* __restrict__ xs,
                                                                       const int32_t* __restrict__ zs,
                                                                       uint4* __restrict__ y) {
    extern __shared__ __align__(16) int32_t sm[];
    const Tables T = stage(D, D.blob_f, sm);
    BW_ITEMS(item, D.n1) {
        const uint32_t s = static_cast<uint32_t>(item);
        const uint32_t d = __ldg(D.m1 + s);
        const int tch = static_cast<int>(d >> 26), ych = T.ych[tch];
        const int ya = T.a0off[ych], ny = T.a0off[ych + 1] - ya;
        int4 out[2] = {make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0)};
        if (ny > 0) {
            const int tb = T.a1off[tch], nt = T.a1off[tch + 1] - tb;
            int4 t0 = make_int4(0, 0, 0, 0), t1 = t0;
            if (nt > 0) {
                Acc4<SMALL> acc0, acc1;
                gather_block<SMALL, STREAM>(D.inc_dmf, D.n1, s, D.w_dmf, T.coef, D.r, tch, xs, D.n0, acc0, acc1);
                t0 = acc0.reduce(D.mod);
                t1 = acc1.reduce(D.mod);
            }
            const int beta0 = nt > 0 ? T.a1idx[tb] : 0, beta1 = nt > 1 ? T.a1idx[tb + 1] : beta0;
            const int kb = T.koff[ych], nz = T.koff[ych + 1] - kb;
            int4 z0 = make_int4(0, 0, 0, 0), z1 = z0;
            if (nz > 0) {
                const long long zr = d & kLow26;
                z0 = ld4(zs, zr);
                if (nz > 1) z1 = ld4(zs, zr + 1);
            }
            for (int q = 0; q < ny; ++q) {
                const int a = T.a0idx[ya + q];
                Acc4<SMALL> acc;
                if (nz > 0) acc.mac(T.B[a * D.kdim + T.kidx[kb]], z0);
                if (nz > 1) acc.mac(T.B[a * D.kdim + T.kidx[kb + 1]], z1);
                if (nt > 0) acc.mac(-T.R[a * D.n + beta0], t0);
                if (nt > 1) acc.mac(-T.R[a * D.n + beta1], t1);
                out[q] = acc.reduce(D.mod);
            }
        }
        st_block(y, s, out[0], out[1]);
    }
}

// (m-2)-subset S2: its u rows u(S2, beta) = (D_(m-1) y)(S2, beta), plus
// dense_sign * dense zs_extra for the deformation variants (|terms| stay below
// 2^31: a balanced residue plus two products of balanced residues), each
// written to its position u_pos in the row-mixing locality order.
template <bool SMALL, bool STREAM>
__global__ void __launch_bounds__(kThreads) sub_d2_forward_kernel(SubsetDev D, const uint4* __restrict__ y,
                                                                  const int32_t* __restrict__ zs,
                                                                  uint2* __restrict__ u) {
    extern __shared__ __align__(16) int32_t sm[];
    const Tables T = stage(D, D.blob_f, sm);
    BW_ITEMS(item, D.n2) {
        const uint32_t s = static_cast<uint32_t>(item);
        const uint32_t d = __ldg(D.m2 + s);
        const int uch = static_cast<int>(d >> 26);
        const int nu = T.a1off[uch + 1] - T.a1off[uch];
        const long long urow = d & kLow26;
        int4 out[2] = {make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0)};
        if (nu > 0) {
            Acc4<SMALL> acc0, acc1;
            gather_block<SMALL, STREAM>(D.inc_d2f, D.n2, s, D.w_d2f, T.coef, D.r, uch, y, D.n1, acc0, acc1);
            out[0] = acc0.reduce(D.mod);
            if (nu > 1) out[1] = acc1.reduce(D.mod);
            if (D.n_extra) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q >= nu) break;
                    int4 v = out[q];
                    for (int j = 0; j < D.n_extra; ++j) {
                        const int32_t c = D.dense_sign * __ldg(D.dense + (urow + q) * D.n_extra + j);
                        const int4 e = ld4(zs, static_cast<long long>(D.z_cols) + j);
                        v.x += c * e.x;
                        v.y += c * e.y;
                        v.z += c * e.z;
                        v.w += c * e.w;
                    }
                    out[q] = make_int4(reduce_balanced(v.x, D.mod), reduce_balanced(v.y, D.mod),
                                       reduce_balanced(v.z, D.mod), reduce_balanced(v.w, D.mod));
                }
            }
        }
        // rows to their positions in the row-mixing locality order
#pragma unroll
        for (int q = 0; q < 2; ++q)
            if (q < nu) u[__ldg(D.u_pos + urow + q)] = pack_row(out[q]);
    }
}

// u2 = P u for the folded target preconditioner P = T^t Dr T in ELL form
// ([slot][row] over the padded u2 slots, `ell` slots a row, coalesced across
// threads; columns are positions of u in the locality order; empty slots hold
// value 0).  SIX: a row of two rounds' pairings M1, M2 has the columns i, M1 i,
// M2 i, M1 M2 i, M2 M1 i and M1 M2 M1 i, so `ell` is six and a row's words and
// then its six rows of u are loaded together.  Otherwise four slots at a time:
// their rows are gathered together, and the next four slots' words are loaded
// meanwhile.  Bound by the latency of those loads: registers for all of them
// (four CTAs an SM) are worth more than occupancy (an application at genus 26
// 177.7 -> 165.4 us; with eight slots and eight CTAs 171.8).
template <bool SMALL, bool STREAM, bool SIX>
__global__ void __launch_bounds__(kThreads, 4) sub_ell_kernel(SubsetDev D, const uint2* __restrict__ u,
                                                           uint2* __restrict__ u2) {
    constexpr int U = SIX ? 6 : 4;
    pdl_trigger();
    pdl_wait();
    const long long rows = 2 * static_cast<long long>(D.n2);
    BW_ITEMS(row, rows) {
        Acc4<SMALL> acc;
        const uint32_t* c = D.e_col + row;
        const int16_t* v = D.e_val + row;
        uint32_t cc[U];
        int32_t vv[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            cc[q] = ld_table<STREAM>(c + q * rows);
            vv[q] = ld_table<STREAM>(v + q * rows);
        }
        for (uint32_t k = 0; k < (SIX ? 1u : D.ell); k += U) {
            uint2 x[U];
#pragma unroll
            for (int q = 0; q < U; ++q) x[q] = __ldg(u + cc[q]);
            uint32_t nc[U];
            int32_t nv[U];
            const bool more = !SIX && k + U < D.ell;
            if (more) {
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    nc[q] = ld_table<STREAM>(c + (k + U + q) * rows);
                    nv[q] = ld_table<STREAM>(v + (k + U + q) * rows);
                }
            }
#pragma unroll
            for (int q = 0; q < U; ++q) acc.mac(vv[q], unpack_row(x[q].x, x[q].y));
            if (more) {
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    cc[q] = nc[q];
                    vv[q] = nv[q];
                }
            }
        }
        u2[row] = pack_row(acc.reduce(D.mod));
    }
}

// (m-1)-subset S: its h rows h(S, a) = (D_(m-1)^t u2)(S, a), then
//   t_adj(S, beta) = sum_a R[a,beta] h(S, a)               (padded t block)
//   out_z(S, kappa) = dc * sum_a B[a,kappa] h(S, a)        (compact, through op_col)
// and, with next_zs, the next application's source row dc * out_z (zero for
// a dropped column), so that apply_square needs no source kernel.
template <bool SMALL, bool STREAM>
__global__ void __launch_bounds__(kThreads) sub_d2_transpose_adjoint_kernel(SubsetDev D,
                                                                            const uint4* __restrict__ u2,
                                                                            const int32_t* __restrict__ dc,
                                                                            uint4* __restrict__ t_adj,
                                                                            int32_t* __restrict__ out,
                                                                            int32_t* __restrict__ next_zs) {
    extern __shared__ __align__(16) int32_t sm[];
    const Tables T = stage(D, D.blob_t, sm);
    BW_ITEMS(item, D.n1) {
        const uint32_t s = static_cast<uint32_t>(item);
        const uint32_t d = __ldg(D.m1 + s);
        const int tch = static_cast<int>(d >> 26), ych = T.ych[tch];
        const int ya = T.a0off[ych], ny = T.a0off[ych + 1] - ya;
        const int a0 = ny > 0 ? T.a0idx[ya] : 0, a1 = ny > 1 ? T.a0idx[ya + 1] : a0;
        int4 h0 = make_int4(0, 0, 0, 0), h1 = h0;
        if (ny > 0) {
            Acc4<SMALL> acc0, acc1;
            gather_block<SMALL, STREAM>(D.inc_d2t, D.n1, s, D.w_d2t, T.coef, D.r, ych, u2, D.n2, acc0, acc1);
            h0 = acc0.reduce(D.mod);
            h1 = acc1.reduce(D.mod);
        }
        const int tb = T.a1off[tch], nt = T.a1off[tch + 1] - tb;
        int4 tv[2] = {make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0)};
        for (int q = 0; q < nt; ++q) {
            const int beta = T.a1idx[tb + q];
            Acc4<SMALL> acc;
            if (ny > 0) acc.mac(T.R[a0 * D.n + beta], h0);
            if (ny > 1) acc.mac(T.R[a1 * D.n + beta], h1);
            tv[q] = acc.reduce(D.mod);
        }
        st_block(t_adj, s, tv[0], tv[1]);
        const int kb = T.koff[ych], nz = T.koff[ych + 1] - kb;
        const long long zq0 = d & kLow26, zfirst = static_cast<long long>(D.x_cols) + zq0;
        for (int q = 0; q < nz; ++q) {
            const long long orow = cyc::op_col(D.drop0, D.drop1, zfirst + q);
            if (orow < 0) {   // dropped base column (replacement)
                if (next_zs) st4(next_zs, zq0 + q, make_int4(0, 0, 0, 0));
                continue;
            }
            const int kap = T.kidx[kb + q];
            Acc4<SMALL> acc;
            if (ny > 0) acc.mac(T.B[a0 * D.kdim + kap], h0);
            if (ny > 1) acc.mac(T.B[a1 * D.kdim + kap], h1);
            const int4 v = acc.reduce(D.mod);
            const int4 o = dc ? scale4(v, __ldg(dc + orow), D.mod) : v;
            st4(out, orow, o);
            if (next_zs) st4(next_zs, zq0 + q, scale4(o, __ldg(dc + orow), D.mod));   // next source row
        }
    }
}

// m-subset S': its x rows out_x(S', a) = -dc * (D_m^t t_adj)(S', a), compact
// through op_col, and, with next_xs, the next application's padded source
// block dc * out_x (as the source kernel would build it from out).
template <bool SMALL, bool STREAM>
__global__ void __launch_bounds__(kThreads) sub_dm_transpose_kernel(SubsetDev D, const uint4* __restrict__ t_adj,
                                                                    const int32_t* __restrict__ dc,
                                                                    int32_t* __restrict__ out,
                                                                    uint4* __restrict__ next_xs) {
    extern __shared__ __align__(16) int32_t sm[];
    const Tables T = stage(D, D.blob_t, sm);
    BW_ITEMS(item, D.n0) {
        const uint32_t s = static_cast<uint32_t>(item);
        const uint32_t d = __ldg(D.m0 + s);
        const int xch = static_cast<int>(d >> 26);
        const int nx = T.a0off[xch + 1] - T.a0off[xch];
        if (nx == 0) continue;
        Acc4<SMALL> acc0, acc1;
        gather_block<SMALL, STREAM>(D.inc_dmt, D.n0, s, D.w_dmt, T.coef, D.r, xch, t_adj, D.n1, acc0, acc1);
        const long long xrow = d & kLow26;
        int4 nxt[2] = {make_int4(0, 0, 0, 0), make_int4(0, 0, 0, 0)};
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            if (q >= nx) break;
            const long long orow = cyc::op_col(D.drop0, D.drop1, xrow + q);
            if (orow < 0) continue;   // dropped base column (replacement): its source slot stays zero
            const int4 v = neg4(q == 0 ? acc0.reduce(D.mod) : acc1.reduce(D.mod));
            const int4 o = dc ? scale4(v, __ldg(dc + orow), D.mod) : v;
            st4(out, orow, o);
            if (next_xs) nxt[q] = scale4(o, __ldg(dc + orow), D.mod);
        }
        if (next_xs) st_block(next_xs, s, nxt[0], nxt[1]);   // next application's source block
    }
}

// Extra source rows of the deformation transpose from the padded u2:
//   out[kept_cols + j][c] = dense_sign * dc[kept_cols + j] * sum_row dense[row][j] u2[row][c]
// Each CTA sums a stripe of padded rows; the CTA sums meet in an 8-entry
// accumulator (cyc::grid_sum) and the last CTA writes the n_extra rows (and,
// with next_zs, their next source rows).
__global__ void __launch_bounds__(kThreads) sub_dense_t_kernel(SubsetDev D, const uint2* __restrict__ u2,
                                                               const int32_t* __restrict__ dc,
                                                               int32_t* __restrict__ out,
                                                               int32_t* __restrict__ partials,
                                                               unsigned int* __restrict__ counter,
                                                               int32_t* __restrict__ next_zs) {
    extern __shared__ __align__(16) int32_t sm[];
    const Tables T = stage(D, D.blob_f, sm);
    int32_t acc[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] = 0;
    int cnt = 0;
    BW_ITEMS(row, 2 * static_cast<long long>(D.n2)) {
        const uint32_t d = __ldg(D.m2 + (row >> 1));
        const int uch = static_cast<int>(d >> 26);
        const int q = static_cast<int>(row & 1);
        if (q >= T.a1off[uch + 1] - T.a1off[uch]) continue;   // padding slot
        const long long crow = static_cast<long long>(d & kLow26) + q;
        const uint2 w = __ldg(u2 + row);
        const int4 v = unpack_row(w.x, w.y);
        for (int j = 0; j < D.n_extra; ++j) {
            const int32_t c = __ldg(D.dense + crow * D.n_extra + j);
            acc[4 * j] += c * v.x;
            acc[4 * j + 1] += c * v.y;
            acc[4 * j + 2] += c * v.z;
            acc[4 * j + 3] += c * v.w;
        }
        if (++cnt == 8) {   // 8 products of balanced residues stay below 2^31
            cnt = 0;
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[e] = reduce_partial(acc[e], D.mod);
        }
    }
    __shared__ int32_t red[kThreads / 32][8];
    __shared__ bool am_last;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        int32_t v = reduce_balanced(acc[e], D.mod);
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if (lane == 0) red[warp][e] = reduce_balanced(v, D.mod);
    }
    __syncthreads();
    int32_t mine = 0, total = 0;
    if (threadIdx.x < 8) {
        for (int w = 0; w < kThreads / 32; ++w) mine += red[w][threadIdx.x];
        mine = reduce_balanced(mine, D.mod);
    }
    if (!cyc::grid_sum(partials, counter, 8, mine, total, &am_last)) return;
    if (threadIdx.x < 4 * D.n_extra) {
        const int j = threadIdx.x / 4, c = threadIdx.x % 4;
        const long long orow = static_cast<long long>(D.kept_cols) + j;
        int32_t v = D.dense_sign * reduce_balanced(total, D.mod);
        if (dc) v = reduce_balanced(v * __ldg(dc + orow), D.mod);
        out[orow * 4 + c] = v;
        if (next_zs)   // next application's source row of extra column j
            next_zs[(static_cast<long long>(D.z_cols) + j) * 4 + c] = reduce_balanced(v * __ldg(dc + orow), D.mod);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        *counter = 0;
        __threadfence();
    }
}

// ----- whole rounds in one launch
//
// An application is five kernels, and on a small sector each costs about 4 us
// whatever it does: the launch, the wait for the kernel before, and a chain of
// dependent loads (a subset's word, its incidence words, its blocks chunk
// after chunk).  Where every subset has a thread of its own and the tables fit
// in shared memory, one cooperative launch runs many rounds instead: a
// thread's incidence words and preconditioner entries stay in shared memory
// and its coefficients in registers, so a phase is one round of gathers, all
// in flight together, between two grid-wide barriers; the Gram moments of an
// application are added up beside the next one's first phase.
//
// Microseconds an application, kernel by kernel -> so: genus 12 15.4 -> 7.8, 16
// 20.3 -> 10.7, 20 24.1 -> 13.4, 22 34.5 -> 19.2, of which the five barriers
// take 3.6 (one CTA pair) to 6.7.  (With the tables read from L2 it was 17.5,
// 18.2, 22.7 and 29.1: the chain, not the launches, is what a phase costs.)
struct RoundsArgs {
    uint4 *xs, *y, *t_adj, *u2;
    uint2* u;
    int32_t *zs, *b, *d;          // scaled source's compact rows; the two compact blocks
    const int32_t* dc;
    long long rows;               // of the compact blocks
    int32_t* sums;                // 20 accumulators, zero between launches
    uint32_t* seq;
    unsigned long long* seq_index;
    unsigned int* arrivals;       // of all CTAs at all barriers (zero at launch)
    int* err;                     // written only on a give-up
    unsigned int wait_limit;
    int hold;                     // failure test: CTA 0 never arrives
    int rounds;
};

// All CTAs of a cooperative launch meet (the `count`-th time); `threads` of
// every CTA take part at hardware barrier `id`, the subset threads here and the
// others in grid_barrier_join.  Thread 0 releases its CTA's writes and acquires
// the others'; data written in this launch is read at L2 (__ldcg).  One counter
// that one thread a CTA polls: 1.0 to 1.2 us (148 flags polled side by side by
// every CTA: 3.5 us).  The wait is bounded: a CTA that runs out of tries
// reports it and returns, and so do then the others.
__device__ __forceinline__ void cta_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ bool grid_barrier(const RoundsArgs& A, unsigned int count, int id, int threads,
                                             volatile unsigned int* gave_up) {
    cta_sync(id, threads);
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(A.arrivals) : "memory");
        const unsigned int target = count * gridDim.x;
        unsigned int tries = 0, v;
        do {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(A.arrivals) : "memory");
        } while (v < target && ++tries < A.wait_limit);
        if (v < target) {
            *gave_up = count;
            *reinterpret_cast<volatile int*>(A.err) = 1;
        }
    }
    cta_sync(id, threads);
    return *gave_up == 0;
}

// The part in the `count`-th of threads that only wait for the CTA's polling
// thread.  That thread may have run into a later barrier, and given it up,
// before they read the word: they take that for what it is then and go on to
// the next barrier they join, where the CTA's other threads meet them.  (Were
// some to leave at once and others not, those would wait there for good.)
__device__ __forceinline__ bool grid_barrier_join(unsigned int count, volatile unsigned int* gave_up, int all) {
    cta_sync(0, all);
    cta_sync(0, all);
    const unsigned int at = *gave_up;
    return at == 0 || at > count;
}

// Adds the packed upper triangles of B^t D and O^t O (O: the newer of the two)
// over all rows to A.sums, by the kMomentThreads threads that call it in every
// CTA (t: the thread's number among them).
__device__ __forceinline__ void add_moments(const RoundsArgs& A, bool b_is_newer, const Mod& mod, int t) {
    int32_t acc[20];
#pragma unroll
    for (int e = 0; e < 20; ++e) acc[e] = 0;
    int cnt = 0;
    for (long long row = static_cast<long long>(blockIdx.x) * kMomentThreads + t; row < A.rows;
         row += static_cast<long long>(gridDim.x) * kMomentThreads) {
        const int4 b = __ldcg(reinterpret_cast<const int4*>(A.b) + row);
        const int4 d = __ldcg(reinterpret_cast<const int4*>(A.d) + row), o = b_is_newer ? b : d;
        const int bv[4] = {b.x, b.y, b.z, b.w}, dv[4] = {d.x, d.y, d.z, d.w}, ov[4] = {o.x, o.y, o.z, o.w};
#pragma unroll
        for (int r0 = 0; r0 < 4; ++r0)
#pragma unroll
            for (int c0 = r0; c0 < 4; ++c0) {
                acc[cyc::tri_index(r0, c0)] += bv[r0] * dv[c0];
                acc[10 + cyc::tri_index(r0, c0)] += ov[r0] * ov[c0];
            }
        if (++cnt == 8) {
            cnt = 0;
#pragma unroll
            for (int e = 0; e < 20; ++e) acc[e] = reduce_partial(acc[e], mod);
        }
    }
    const int lane = t % 32;
    int32_t mine = 0;
#pragma unroll
    for (int e = 0; e < 20; ++e) {
        const int32_t v = __reduce_add_sync(0xffffffffu, reduce_balanced(acc[e], mod));
        if (lane == e) mine = v;
    }
    // at most 148 * 4 warps of 32 balanced values: far below 2^31
    if (lane < 20) atomicAdd(A.sums + lane, mine);
}

// Gathers of one subset whose words lie in shared memory ([position][thread],
// padded to chunks of four with words of the zero block): eight blocks are in
// flight before their products.
template <bool SMALL>
__device__ __forceinline__ void gather_resident(const uint32_t* words, int stride, int chunks, const int4* coef, int r,
                                                int ch, const uint4* in, Acc4<SMALL>& acc0, Acc4<SMALL>& acc1) {
#pragma unroll
    for (int c0 = 0; c0 < kResidentChunks; c0 += 2) {
        if (c0 >= chunks) break;
        const bool two = c0 + 1 < chunks;
        uint32_t w[8];
        uint4 b[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (u < 4 || two) {
                w[u] = words[(4 * c0 + u) * stride];
                b[u] = __ldcg(in + (w[u] & kLow26));
            }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (u < 4 || two) mac_block<SMALL>(coef[static_cast<int>(w[u] >> 26) * r + ch], b[u], acc0, acc1);
    }
}

// Shared memory: the two coefficient blobs, then per subset thread (stride T)
// the padded words of the four gathers and the columns and values of its two
// preconditioner rows.  Subset thread t of the grid owns the t-th m-, (m-1)-
// and (m-2)-subset; each CTA's last kMomentThreads threads add up the moments
// of the application before, beside the first three phases (in the subset
// threads that took 3.5 us an application).
template <bool SMALL>
__global__ void __launch_bounds__(kResidentThreads, 1) sub_rounds_kernel(SubsetDev D, RoundsArgs A) {
    extern __shared__ __align__(16) int32_t sm[];
    __shared__ unsigned int gave_up;   // number of the barrier that the CTA gave up at, or 0
    const int all = blockDim.x, T = all - kMomentThreads, tid = threadIdx.x;
    const int blob4 = (D.blob_words + 3) / 4 * 4;
    for (int w = tid; w < D.blob_words; w += all) {
        sm[w] = __ldg(D.blob_f + w);
        sm[blob4 + w] = __ldg(D.blob_t + w);
    }
    if (tid == 0) gave_up = 0;
    if (A.hold && blockIdx.x == 0) return;
    if (tid >= T) {
        // ------------------------------------------------ moments
        // joins the third barrier (the older block is overwritten after it)
        // and the fifth (the newer one is complete)
        __syncthreads();
        for (int app = 0; app < 2 * A.rounds; ++app) {
            if (app > 0) add_moments(A, (app & 1) == 0, D.mod, tid - T);
            if (!grid_barrier_join(5u * app + 3, &gave_up, all) || !grid_barrier_join(5u * app + 5, &gave_up, all)) return;
        }
        add_moments(A, true, D.mod, tid - T);
        grid_barrier_join(10u * A.rounds + 1, &gave_up, all);
        return;
    }
    const uint32_t id = blockIdx.x * static_cast<uint32_t>(T) + tid;
    const bool has0 = id < D.n0, has1 = id < D.n1, has2 = id < D.n2;
    const int c_dmf = (D.w_dmf + 3) / 4, c_d2f = (D.w_d2f + 3) / 4, c_d2t = (D.w_d2t + 3) / 4, c_dmt = (D.w_dmt + 3) / 4;
    uint32_t* const w_dmf = reinterpret_cast<uint32_t*>(sm) + 2 * blob4 + tid;
    uint32_t* const w_d2f = w_dmf + 4 * c_dmf * T;
    uint32_t* const w_d2t = w_d2f + 4 * c_d2f * T;
    uint32_t* const w_dmt = w_d2t + 4 * c_d2t * T;
    uint32_t* const e_col = w_dmt + 4 * c_dmt * T;     // [12][T]: six slots of either row
    int32_t* const e_val = reinterpret_cast<int32_t*>(e_col + 12 * T);
    auto keep_words = [&](uint32_t* dst, const uint32_t* inc, bool has, uint32_t n, uint32_t width, uint32_t nin) {
        for (uint32_t k = 0; k < (width + 3) / 4 * 4; ++k)
            dst[k * T] = has && k < width ? __ldg(inc + static_cast<size_t>(k) * n + id) : nin;
    };
    keep_words(w_dmf, D.inc_dmf, has1, D.n1, D.w_dmf, D.n0);
    keep_words(w_d2f, D.inc_d2f, has2, D.n2, D.w_d2f, D.n1);
    keep_words(w_d2t, D.inc_d2t, has1, D.n1, D.w_d2t, D.n2);
    keep_words(w_dmt, D.inc_dmt, has0, D.n0, D.w_dmt, D.n1);
    for (int q = 0; q < 12; ++q) {
        const long long at = (q % 6) * (2 * static_cast<long long>(D.n2)) + 2 * static_cast<long long>(id) + q / 6;
        e_col[q * T] = has2 ? __ldg(D.e_col + at) : 0u;
        e_val[q * T] = has2 ? __ldg(D.e_val + at) : 0;
    }
    __syncthreads();
    const Tables F = views(D, sm), B = views(D, sm + blob4);

    // (m-1)-subset: y = B z - R t forward, t_adj = R^t h and z = B^t h back, with
    // zero coefficients where the block has fewer rows
    int tch = 0, ych = 0, ny = 0, nt = 0, nz = 0;
    long long zrow = 0;
    int32_t cB[2][2] = {}, cR[2][2] = {}, dcz[2] = {};   // [y row][z or t row]
    if (has1) {
        const uint32_t d = __ldg(D.m1 + id);
        tch = static_cast<int>(d >> 26);
        ych = F.ych[tch];
        zrow = d & kLow26;
        ny = F.a0off[ych + 1] - F.a0off[ych];
        nt = F.a1off[tch + 1] - F.a1off[tch];
        nz = F.koff[ych + 1] - F.koff[ych];
        for (int q = 0; q < ny; ++q) {
            const int a = F.a0idx[F.a0off[ych] + q];
            for (int j = 0; j < nz; ++j) cB[q][j] = F.B[a * D.kdim + F.kidx[F.koff[ych] + j]];
            for (int j = 0; j < nt; ++j) cR[q][j] = F.R[a * D.n + F.a1idx[F.a1off[tch] + j]];
        }
        for (int j = 0; j < nz; ++j) dcz[j] = __ldg(A.dc + D.x_cols + zrow + j);
    }
    // (m-2)-subset: the positions of its u rows
    int uch = 0, nu = 0;
    uint32_t upos[2] = {};
    if (has2) {
        const uint32_t d = __ldg(D.m2 + id);
        uch = static_cast<int>(d >> 26);
        nu = F.a1off[uch + 1] - F.a1off[uch];
        for (int q = 0; q < nu; ++q) upos[q] = __ldg(D.u_pos + (d & kLow26) + q);
    }
    // m-subset: its compact rows and their column preconditioner
    int xch = 0, nx = 0;
    long long xrow = 0;
    int32_t dcx[2] = {};
    if (has0) {
        const uint32_t d = __ldg(D.m0 + id);
        xch = static_cast<int>(d >> 26);
        nx = F.a0off[xch + 1] - F.a0off[xch];
        xrow = d & kLow26;
        for (int q = 0; q < nx; ++q) dcx[q] = __ldg(A.dc + xrow + q);
    }

    const unsigned long long pos = *A.seq_index;
    unsigned int met = 0;
    // the sums of application `app`, complete after a barrier, to the sequence
    auto write_moments = [&](int app) {
        if (blockIdx.x == 0 && tid < 20) {
            const int32_t total = atomicExch(A.sums + tid, 0);
            A.seq[(pos + 2ull * app) * 10 + tid] = to_canonical(reduce_balanced(total, D.mod), D.mod);
        }
    };
    const int4 zero = make_int4(0, 0, 0, 0);
    // subset threads alone, or with the moments' threads
    // (a give-up there lets the moments' threads out of the barrier they wait at)
    auto subset_barrier = [&] {
        if (grid_barrier(A, ++met, 1, T, &gave_up)) return true;
        grid_barrier_join(met, &gave_up, all);
        return false;
    };
    auto full_barrier = [&] { return grid_barrier(A, ++met, 0, all, &gave_up); };
    for (int app = 0; app < 2 * A.rounds; ++app) {
        int32_t* out = (app & 1) ? A.b : A.d;
        if (has1) {
            int4 z[2] = {zero, zero};
#pragma unroll
            for (int j = 0; j < 2; ++j)
                if (j < nz) z[j] = __ldcg(reinterpret_cast<const int4*>(A.zs) + zrow + j);
            Acc4<SMALL> t0, t1;
            gather_resident<SMALL>(w_dmf, T, c_dmf, F.coef, D.r, tch, A.xs, t0, t1);
            const int4 t[2] = {t0.reduce(D.mod), t1.reduce(D.mod)};
            int4 y[2];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                Acc4<SMALL> acc;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    acc.mac(cB[q][j], z[j]);
                    acc.mac(-cR[q][j], t[j]);
                }
                y[q] = acc.reduce(D.mod);
            }
            st_block(A.y, id, y[0], y[1]);
        }
        if (!subset_barrier()) return;
        if (has2) {
            Acc4<SMALL> u0, u1;
            gather_resident<SMALL>(w_d2f, T, c_d2f, F.coef, D.r, uch, A.y, u0, u1);
            if (nu > 0) A.u[upos[0]] = pack_row(u0.reduce(D.mod));
            if (nu > 1) A.u[upos[1]] = pack_row(u1.reduce(D.mod));
        }
        if (!subset_barrier()) return;
        if (has2) {
            uint2 x[12];
#pragma unroll
            for (int q = 0; q < 12; ++q) x[q] = __ldcg(A.u + e_col[q * T]);
            Acc4<SMALL> p[2];
#pragma unroll
            for (int q = 0; q < 12; ++q) p[q / 6].mac(e_val[q * T], unpack_row(x[q].x, x[q].y));
            st_block(A.u2, id, p[0].reduce(D.mod), p[1].reduce(D.mod));
        }
        if (!full_barrier()) return;
        if (app > 0) write_moments(app - 1);   // complete since the third barrier
        if (has1) {
            Acc4<SMALL> h0, h1;
            gather_resident<SMALL>(w_d2t, T, c_d2t, B.coef, D.r, ych, A.u2, h0, h1);
            const int4 h[2] = {ny > 0 ? h0.reduce(D.mod) : zero, ny > 1 ? h1.reduce(D.mod) : zero};
            int4 t[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                Acc4<SMALL> acc, az;
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    acc.mac(cR[q][j], h[q]);
                    az.mac(cB[q][j], h[q]);
                }
                t[j] = acc.reduce(D.mod);
                if (j < nz) {
                    const int4 o = scale4(az.reduce(D.mod), dcz[j], D.mod);
                    st4(out, static_cast<long long>(D.x_cols) + zrow + j, o);
                    st4(A.zs, zrow + j, scale4(o, dcz[j], D.mod));   // next source row
                }
            }
            st_block(A.t_adj, id, t[0], t[1]);
        }
        if (!subset_barrier()) return;
        if (has0 && nx > 0) {
            Acc4<SMALL> x0, x1;
            gather_resident<SMALL>(w_dmt, T, c_dmt, B.coef, D.r, xch, A.t_adj, x0, x1);
            int4 next[2] = {zero, zero};
#pragma unroll
            for (int q = 0; q < 2; ++q)
                if (q < nx) {
                    const int4 o = scale4(neg4(q == 0 ? x0.reduce(D.mod) : x1.reduce(D.mod)), dcx[q], D.mod);
                    st4(out, xrow + q, o);
                    next[q] = scale4(o, dcx[q], D.mod);
                }
            st_block(A.xs, id, next[0], next[1]);   // next application's source block
        }
        if (!full_barrier()) return;
    }
    if (!full_barrier()) return;   // the last application's moments
    write_moments(2 * A.rounds - 1);
    if (blockIdx.x == 0 && tid == 0) *A.seq_index = pos + 4ull * A.rounds;
}

// Compact int32 rows <-> padded int16 blocks of the (m-2)-subsets: u2 in the
// non-hot entry points (backward / target_precondition on compact vectors).
__global__ void __launch_bounds__(kThreads) sub_u_pack_kernel(SubsetDev D, const int32_t* __restrict__ u32,
                                                              uint4* __restrict__ u16) {
    extern __shared__ __align__(16) int32_t sm[];
    const Tables T = stage(D, D.blob_f, sm);
    BW_ITEMS(item, D.n2) {
        const uint32_t d = __ldg(D.m2 + item);
        const int uch = static_cast<int>(d >> 26);
        const int nu = T.a1off[uch + 1] - T.a1off[uch];
        const long long first = d & kLow26;
        const int4 zero = make_int4(0, 0, 0, 0);
        st_block(u16, static_cast<uint32_t>(item), nu > 0 ? ld4(u32, first) : zero,
                 nu > 1 ? ld4(u32, first + 1) : zero);
    }
}
__global__ void __launch_bounds__(kThreads) sub_u_unpack_kernel(SubsetDev D, const uint4* __restrict__ u16,
                                                                int32_t* __restrict__ u32) {
    extern __shared__ __align__(16) int32_t sm[];
    const Tables T = stage(D, D.blob_f, sm);
    BW_ITEMS(item, D.n2) {
        const uint32_t d = __ldg(D.m2 + item);
        const int uch = static_cast<int>(d >> 26);
        const int nu = T.a1off[uch + 1] - T.a1off[uch];
        const long long first = d & kLow26;
        const uint4 b = __ldg(u16 + item);
        if (nu > 0) st4(u32, first, unpack_row(b.x, b.y));
        if (nu > 1) st4(u32, first + 1, unpack_row(b.z, b.w));
    }
}

// Compact int32 u rows <-> u in the row-mixing locality order (int16 rows).
__global__ void __launch_bounds__(kThreads) sub_u_to_walk_kernel(SubsetDev D, const int32_t* __restrict__ u32,
                                                                 uint2* __restrict__ u, long long rows) {
    BW_ITEMS(q, rows) u[__ldg(D.u_pos + q)] = pack_row(ld4(u32, q));
}
__global__ void __launch_bounds__(kThreads) sub_u_from_walk_kernel(SubsetDev D, const uint2* __restrict__ u,
                                                                   int32_t* __restrict__ u32, long long rows) {
    BW_ITEMS(q, rows) {
        const uint2 w = __ldg(u + __ldg(D.u_pos + q));
        st4(u32, q, unpack_row(w.x, w.y));
    }
}

int32_t balanced_of(uint32_t v, const Mod& m) { return to_balanced(v % static_cast<uint32_t>(m.p), m); }

}  // namespace

// Builds the subset tables, the padded preconditioner and the two
// shared-memory blobs, and allocates the padded int16 vectors; leaves
// subset_path false (and says why in subset_reason) when the sector does not
// fit the format or BW_CYCLIC_GENERIC asks for the generic row kernels.
void CyclicCtx::setup_subset_path() {
    subset_path = false;
    if (const char* env = std::getenv("BW_CYCLIC_GENERIC")) {
        if (*env && std::string(env) != "0") {
            subset_reason = "BW_CYCLIC_GENERIC is set";
            return;
        }
    }
    cyclic::SubsetTables tab;
    // u is kept in an order with row-mixing partners adjacent, so the folded
    // preconditioner's sixteen columns of a row fall within a few sectors
    const std::vector<uint32_t> u_pos = cyclic::rowmix_locality_order(plan);
    subset_reason = cyclic::build_subset_tables(inst, es, precond, u_pos, tab);
    if (!subset_reason.empty()) return;

    const cyclic::CharMap a0 = cyclic::build_char_map(inst.weight_a0, inst.r);
    const cyclic::CharMap a1 = cyclic::build_char_map(inst.weight_a1, inst.r);
    const cyclic::CharMap km = cyclic::build_char_map(inst.kernel_weights, inst.r);
    const int n = static_cast<int>(inst.n), g = static_cast<int>(inst.genus), r = static_cast<int>(inst.r);
    const int kdim = static_cast<int>(inst.kernel_dim());
    SubsetDev& D = S;
    D.mod = mod;
    D.n = n;
    D.g = g;
    D.kdim = kdim;
    D.r = r;
    int w = 8 * n * r;   // coefficients: [2 n codes][r] x int4
    D.o_R = w;
    w += g * n;
    D.o_B = w;
    w += g * kdim;
    D.o_a0off = w;
    w += r + 1;
    D.o_a0idx = w;
    w += g;
    D.o_a1off = w;
    w += r + 1;
    D.o_a1idx = w;
    w += n;
    D.o_koff = w;
    w += r + 1;
    D.o_kidx = w;
    w += kdim;
    D.o_ych = w;
    w += r;
    D.blob_words = w;
    if (static_cast<size_t>(w) * 4 > 48 * 1024) {
        subset_reason = "shared-memory tables above 48 KB";
        return;
    }
    std::vector<int32_t> common(w, 0);
    for (int a = 0; a < g; ++a) {
        for (int b = 0; b < n; ++b) common[D.o_R + a * n + b] = balanced_of(inst.right_inverse[a * n + b], mod);
        for (int k = 0; k < kdim; ++k) common[D.o_B + a * kdim + k] = balanced_of(inst.kernel_basis[a * kdim + k], mod);
    }
    for (int c = 0; c <= r; ++c) {
        common[D.o_a0off + c] = static_cast<int32_t>(a0.offsets[c]);
        common[D.o_a1off + c] = static_cast<int32_t>(a1.offsets[c]);
        common[D.o_koff + c] = static_cast<int32_t>(km.offsets[c]);
    }
    for (int e = 0; e < g; ++e) common[D.o_a0idx + e] = a0.indices[e];
    for (int e = 0; e < n; ++e) common[D.o_a1idx + e] = a1.indices[e];
    for (int e = 0; e < kdim; ++e) common[D.o_kidx + e] = km.indices[e];
    for (int c = 0; c < r; ++c)
        common[D.o_ych + c] = static_cast<int32_t>((c + r - static_cast<int>(inst.w_weight % inst.r)) % r);
    // Coefficients of code (sign, generator i) and own character ch: own rows
    // k = 0, 1 (the first two keys of ch's block), neighbour slots l = 0, 1,
    // at int32 number 2 k + l of the entry.
    auto put = [&](std::vector<int32_t>& blob, int i, int ch, int k, int l, uint32_t mu) {
        const int32_t b = balanced_of(mu, mod);
        for (int neg = 0; neg < 2; ++neg) blob[4 * ((neg * n + i) * r + ch) + 2 * k + l] = neg ? -b : b;
    };
    std::vector<int32_t> blob_f = common, blob_t = common;
    for (int i = 0; i < n; ++i)
        for (int ch = 0; ch < r; ++ch) {
            // forward: own rows beta in the A1 block of ch; neighbour rows a in
            // the A0 block of A1(beta) - V(i) (the same block for both betas)
            for (uint32_t kb = a1.offsets[ch]; kb < a1.offsets[ch + 1]; ++kb) {
                const int beta = a1.indices[kb];
                const uint32_t q = (inst.weight_a1[beta] + inst.r - inst.weight_v[i] % inst.r) % inst.r;
                for (uint32_t lb = a0.offsets[q]; lb < a0.offsets[q + 1]; ++lb)
                    put(blob_f, i, ch, static_cast<int>(kb - a1.offsets[ch]), static_cast<int>(lb - a0.offsets[q]),
                        inst.mu_at(i, beta, a0.indices[lb]));
            }
            // transpose: own rows a in the A0 block of ch; neighbour rows beta
            // in the A1 block of A0(a) + V(i)
            for (uint32_t kb = a0.offsets[ch]; kb < a0.offsets[ch + 1]; ++kb) {
                const int a = a0.indices[kb];
                const uint32_t q = (inst.weight_a0[a] + inst.weight_v[i]) % inst.r;
                for (uint32_t lb = a1.offsets[q]; lb < a1.offsets[q + 1]; ++lb)
                    put(blob_t, i, ch, static_cast<int>(kb - a0.offsets[ch]), static_cast<int>(lb - a1.offsets[q]),
                        inst.mu_at(i, a1.indices[lb], a));
            }
        }

    D.n1 = static_cast<uint32_t>(tab.m1.size());
    D.n2 = static_cast<uint32_t>(tab.m2.size());
    D.n0 = static_cast<uint32_t>(tab.m0.size());
    D.w_dmf = static_cast<uint32_t>(es.dm.row_width);
    D.w_d2f = static_cast<uint32_t>(es.d2.row_width);
    D.w_d2t = static_cast<uint32_t>(es.d2.column_width);
    D.w_dmt = static_cast<uint32_t>(es.dm.column_width);
    D.m1 = upload(tab.m1);
    D.m2 = upload(tab.m2);
    D.m0 = upload(tab.m0);
    D.inc_dmf = upload(tab.inc_dmf);
    D.inc_d2f = upload(tab.inc_d2f);
    D.inc_d2t = upload(tab.inc_d2t);
    D.inc_dmt = upload(tab.inc_dmt);
    D.u_pos = upload(u_pos);
    D.e_col = upload(tab.e_col);
    D.e_val = upload(tab.e_val);
    D.ell = static_cast<uint32_t>(tab.ell);
    D.blob_f = upload(blob_f);
    D.blob_t = upload(blob_t);
    D.x_cols = es.x_cols;
    D.z_cols = es.z_cols;
    D.kept_cols = E.kept_cols;
    D.drop0 = E.drop0;
    D.drop1 = E.drop1;
    D.n_extra = E.n_extra;
    D.dense_sign = E.dense_sign;
    D.dense = E.dense;
    // Tables read once per application: evict-first when they exceed half the L2.
    size_t table_bytes = 4 * (tab.inc_dmf.size() + tab.inc_d2f.size() + tab.inc_d2t.size() + tab.inc_dmt.size());
    table_bytes += 4 * tab.e_col.size() + 2 * tab.e_val.size();
    int l2 = 0;
    BW_CUDA(cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, device));
    stream_tables = table_bytes > static_cast<size_t>(l2) / 2;
    if (const char* env = std::getenv("BW_CYCLIC_PDL")) pdl = std::string(env) != "0";
    // BW_CYCLIC_STREAM_TABLES=1 / =0 forces the evict-first (or the cached)
    // table reads at any size, so that small sectors run either instantiation.
    if (const char* env = std::getenv("BW_CYCLIC_STREAM_TABLES")) {
        if (*env) stream_tables = std::string(env) != "0";
    }
    // Gathered vectors carry one more block, all zero, for the empty slots of
    // a partial chunk of incidences (their words point at it).
    d_xs16 = alloc<uint4>(D.n0 + 1);
    d_zs = alloc<int32_t>((es.z_cols + dense.columns) * num_v);
    d_y16 = alloc<uint4>(D.n1 + 1);
    d_t16 = alloc<uint4>(D.n1 + 1);
    d_u16 = alloc<uint4>((es.target_rows + 1) / 2 + 1);   // u rows (int16) in the locality order
    d_u2_16 = alloc<uint4>(D.n2 + 1);
    BW_CUDA(cudaMemsetAsync(d_xs16, 0, (D.n0 + 1) * sizeof(uint4), stream));
    BW_CUDA(cudaMemsetAsync(d_y16, 0, (D.n1 + 1) * sizeof(uint4), stream));
    BW_CUDA(cudaMemsetAsync(d_t16, 0, (D.n1 + 1) * sizeof(uint4), stream));
    BW_CUDA(cudaMemsetAsync(d_u2_16, 0, (D.n2 + 1) * sizeof(uint4), stream));
    subset_path = true;
}

// Whether generate() runs whole rounds in one cooperative launch
// (sub_rounds_kernel): the eliminated operator with two row-mixing rounds,
// every subset with a thread of its own in one CTA an SM, and the tables in
// shared memory (the published genera up to 22).  BW_CYCLIC_PERSISTENT=0 turns
// it off.  Settled by the first generate(): loading the kernel in open() made
// that 3 ms longer.
void CyclicCtx::setup_rounds() {
    if (const char* env = std::getenv("BW_CYCLIC_PERSISTENT"))
        if (std::string(env) == "0") return;
    if (S.n_extra != 0 || S.drop0 >= 0 || S.ell != 6) return;
    auto chunks = [](uint32_t w) { return (w + 3) / 4; };
    if (std::max({chunks(S.w_dmf), chunks(S.w_d2f), chunks(S.w_d2t), chunks(S.w_dmt)}) > kResidentChunks) return;
    const uint32_t items = std::max({S.n0, S.n1, S.n2});
    const uint32_t per_sm = (items + sms - 1) / sms, threads = std::max(64u, (per_sm + 31) / 32 * 32);
    if (threads + kMomentThreads > kResidentThreads) return;
    const uint32_t words = 4 * (chunks(S.w_dmf) + chunks(S.w_d2f) + chunks(S.w_d2t) + chunks(S.w_dmt)) + 24;
    rounds_smem = (static_cast<size_t>(2 * ((S.blob_words + 3) / 4 * 4)) + static_cast<size_t>(words) * threads) * 4;
    auto kern = small ? sub_rounds_kernel<true> : sub_rounds_kernel<false>;
    if (rounds_smem > static_cast<size_t>(allow_dynamic_smem(kern, device))) return;
    int coop = 0, occ = 0;
    BW_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device));
    BW_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, static_cast<int>(threads) + kMomentThreads,
                                                          rounds_smem));
    if (!coop || occ < 1) return;
    rounds_threads = static_cast<int>(threads) + kMomentThreads;
    rounds_grid = (items + threads - 1) / threads;
    d_barrier = alloc<uint32_t>(1);
    d_err = alloc<int>(1);
    BW_CUDA(cudaMemsetAsync(d_err, 0, sizeof(int), stream));
    if (const char* e = std::getenv("BW_TEST_WAIT_LIMIT")) {
        const unsigned long v = std::strtoul(e, nullptr, 10);
        if (v >= 1 && v < rounds_wait_limit) rounds_wait_limit = static_cast<uint32_t>(v);
    }
    if (const char* e = std::getenv("BW_TEST_HOLD_FIRST_STAGE")) rounds_hold = (*e && std::string(e) != "0") ? 1 : 0;
    persistent = true;
}

void CyclicCtx::subset_rounds(size_t rounds) {
    RoundsArgs A{d_xs16, d_y16, d_t16, d_u2_16, reinterpret_cast<uint2*>(d_u16), d_zs, d_b, d_d, d_dc,
                 static_cast<long long>(op_cols), d_partials, d_seq, d_seq_index, d_barrier, d_err, rounds_wait_limit,
                 rounds_hold, 0};
    auto kern = small ? sub_rounds_kernel<true> : sub_rounds_kernel<false>;
    for (size_t done = 0; done < rounds; done += A.rounds) {
        // bounded launches: 10 barriers a round keep the arrival count far below 2^32
        A.rounds = static_cast<int>(std::min<size_t>(rounds - done, 1024));
        BW_CUDA(cudaMemsetAsync(d_barrier, 0, sizeof(uint32_t), stream));
        void* args[] = {&S, &A};
        BW_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(rounds_grid),
                                            dim3(rounds_threads), args, rounds_smem, stream));
        ++launches;
    }
    xs_for = d_b;
}

// Kernel template dispatch: SMALL (int32 sums exact) x STREAM (tables above L2).
#define BW_SUBSET_DISPATCH(launch)      \
    do {                                \
        if (small && stream_tables) {   \
            launch(true, true);         \
        } else if (small) {             \
            launch(true, false);        \
        } else if (stream_tables) {     \
            launch(false, true);        \
        } else {                        \
            launch(false, false);       \
        }                               \
    } while (0)

void CyclicCtx::subset_source16(const int32_t* in, const int32_t* dc) {
    const size_t smem = static_cast<size_t>(S.blob_words) * 4;
    const size_t items = static_cast<size_t>(S.n0) + es.z_cols + dense.columns;
    sub_source_kernel<<<grid_for(items), kThreads, smem, stream>>>(S, in, dc, d_xs16, d_zs);
    BW_CHECK_LAUNCH();
    ++launches;
    xs_for = dc == d_dc ? in : nullptr;
}

void CyclicCtx::subset_forward16() {
    const size_t smem = static_cast<size_t>(S.blob_words) * 4;
#define BW_LAUNCH(A, B)                                                                                    \
    launch_pdl(sub_dm_forward_elim_kernel<A, B>, grid_for(S.n1), smem, S, static_cast<const uint4*>(d_xs16), \
               static_cast<const int32_t*>(d_zs), d_y16);                                                  \
    launch_pdl(sub_d2_forward_kernel<A, B>, grid_for(S.n2), smem, S, static_cast<const uint4*>(d_y16),     \
               static_cast<const int32_t*>(d_zs), reinterpret_cast<uint2*>(d_u16))
    BW_SUBSET_DISPATCH(BW_LAUNCH);
#undef BW_LAUNCH
    BW_CHECK_LAUNCH();
    launches += 2;
}

void CyclicCtx::subset_precondition16() {
    const uint2* u = reinterpret_cast<const uint2*>(d_u16);
    uint2* u2 = reinterpret_cast<uint2*>(d_u2_16);
    const unsigned grid = grid_for(2 * static_cast<size_t>(S.n2));
#define BW_LAUNCH(A, B)                                            \
    if (S.ell == 6)                                                \
        launch_pdl(sub_ell_kernel<A, B, true>, grid, 0, S, u, u2); \
    else                                                           \
        launch_pdl(sub_ell_kernel<A, B, false>, grid, 0, S, u, u2)
    BW_SUBSET_DISPATCH(BW_LAUNCH);
#undef BW_LAUNCH
    BW_CHECK_LAUNCH();
    ++launches;
}

void CyclicCtx::subset_backward16(const int32_t* dc, int32_t* out, bool next_source) {
    const size_t smem = static_cast<size_t>(S.blob_words) * 4;
    // next_source (apply_square, dc = the column preconditioner): the kernels
    // also write the next application's source from `out`
    uint4* nxs = next_source ? d_xs16 : nullptr;
    int32_t* nzs = next_source ? d_zs : nullptr;
#define BW_LAUNCH(A, B)                                                                                       \
    launch_pdl(sub_d2_transpose_adjoint_kernel<A, B>, grid_for(S.n1), smem, S,                               \
               static_cast<const uint4*>(d_u2_16), dc, d_t16, out, nzs);                                      \
    launch_pdl(sub_dm_transpose_kernel<A, B>, grid_for(S.n0), smem, S, static_cast<const uint4*>(d_t16), dc, \
               out, nxs)
    BW_SUBSET_DISPATCH(BW_LAUNCH);
#undef BW_LAUNCH
    BW_CHECK_LAUNCH();
    launches += 2;
    if (S.n_extra) {
        launch_pdl(sub_dense_t_kernel, dense_grid, smem, S, reinterpret_cast<const uint2*>(d_u2_16), dc, out,
                   d_dpart, d_dcounter, nzs);
        BW_CHECK_LAUNCH();
        ++launches;
    }
    if (next_source)
        xs_for = out;
    else if (xs_for == out)
        xs_for = nullptr;
}

void CyclicCtx::subset_u_to_walk(const int32_t* u32) {
    const long long rows = static_cast<long long>(es.target_rows);
    sub_u_to_walk_kernel<<<grid_for(es.target_rows), kThreads, 0, stream>>>(S, u32, reinterpret_cast<uint2*>(d_u16),
                                                                            rows);
    BW_CHECK_LAUNCH();
    ++launches;
}

void CyclicCtx::subset_u_from_walk(int32_t* u32) {
    const long long rows = static_cast<long long>(es.target_rows);
    sub_u_from_walk_kernel<<<grid_for(es.target_rows), kThreads, 0, stream>>>(
        S, reinterpret_cast<const uint2*>(d_u16), u32, rows);
    BW_CHECK_LAUNCH();
    ++launches;
}

void CyclicCtx::subset_pack_u(const int32_t* u32, uint4* u16) {
    sub_u_pack_kernel<<<grid_for(S.n2), kThreads, static_cast<size_t>(S.blob_words) * 4, stream>>>(S, u32, u16);
    BW_CHECK_LAUNCH();
    ++launches;
}

void CyclicCtx::subset_unpack_u(const uint4* u16, int32_t* u32) {
    sub_u_unpack_kernel<<<grid_for(S.n2), kThreads, static_cast<size_t>(S.blob_words) * 4, stream>>>(S, u16, u32);
    BW_CHECK_LAUNCH();
    ++launches;
}

}  // namespace bw
