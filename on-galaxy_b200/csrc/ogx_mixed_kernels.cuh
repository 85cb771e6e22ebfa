// ogx_mixed_kernels.cuh -- kernels of the mixed-precision form.
//
// M2L on the 5th-generation tensor cores (tcgen05, kind::f16, TMEM accumulators).
// The reference applies fmm::M2L pair by pair (src3d/FmmExpansions3D.hpp:273-299,
// called per V-list entry in src3d/AdaptiveFMM3D.hpp:78-81).  Here:
//   * a CTA owns 128 targets that share their octant t inside their parents
//     (any level: the scaled operator is level independent);
//   * the V list of every such target is the children s of its parent's
//     colleague slots D with offset o = 2(D-1) + s - t, max|o| >= 2 (189
//     combinations for a given t); for one combination every target has at
//     most one source, so the sources of the 128 targets form the rows of a
//     dense operand A (128 x K, zero rows where absent) and the translation is
//     D[128 x N] = A . T_o^T with one operator matrix T_o for the whole tile;
//   * split precision: multipoles and operators are split into FP16 hi + lo
//     parts (11 + 11 significant bits) and D accumulates A_hi B_hi + A_hi B_lo +
//     A_lo B_hi in FP32 (the dropped lo x lo term is ~2^-22 relative).  FP16
//     has the significand of TF32 at half the bytes, and the tensor cores' operand
//     reads (shared memory) bound this kernel; its narrow exponent range is met by
//     scaling every multipole row and every operator by a power of two that puts
//     its largest entry in [0.5, 1), undone exactly per row and combination when
//     the result is drained;
//   * a small tree has fewer tiles than SMs (8,192 bodies: 8, each a serial walk of ~150
//     combinations, 183 us): its tiles are cut into ranges of colleague slots (ogx_m2l64.cuh),
//     one CTA each, whose sums are added in range order;
//   * accumulation: FP32 accumulation over all ~6000 MMA steps of a tile loses
//     ~1e-5 of the (strongly cancelling) far field, so every combination gets a
//     fresh FP32 accumulator (a ring of buffers in TMEM) that the epilogue warps
//     drain while the MMA warp proceeds with the next combination.  The drain
//     unscales each combination's result, sums the (at most eight) combinations
//     of one colleague slot D in FP32 registers, and folds each slot's sum into
//     an FP64 accumulator (registers for p <= 8, TMEM otherwise);
//   * operands: K is cut into chunks of 64 fp16 (one 128-byte line per row) in
//     the K-major 128-byte-swizzle layout; A rows are gathered with cp.async,
//     each T_o chunk is a pre-laid-out image copied by the TMA bulk engine
//     (cp.async.bulk, no multicast); up to 4 stages pipeline through mbarriers.
//     A producer thread hands its rows of a stage over with an asynchronous
//     mbarrier arrival that fires when its copies have landed, so it never waits
//     for its own copies and every stage of the ring can be in flight;
//   * warp specialisation: four warps gather the A rows (the colleague table
//     of the tile is staged in shared memory and the next combination's source
//     index is fetched one combination ahead), one lane issues the MMAs, and
//     eight drain warps fold each combination into FP64 and write the result.
// Output degree 0 (L_0^0, only needed for potentials) is excluded from N.
// An MMA of N <= ~160 columns costs about the same time, so for p <= 8 the
// operator's hi and lo images form one N = 2 N operand: A_hi x [B_hi | B_lo] and
// A_lo x B_hi are two MMAs per K step (three otherwise).  TMEM holds two FP32
// buffers (2 x 2N or 2 x N columns) + 2 x N FP64-halves columns, which fits
// N <= 128 (p <= 10).  For p = 11 and 12 the output columns are cut into NSPLIT
// slices (2 x 72 and 3 x 56 dofs), each handled by its own CTA (grid y) in the
// paired form with one 64- or 80-column operand; the A rows are gathered once per
// slice.
#pragma once

#include <cuda_fp16.h>

#include "ogx_m2l64.cuh"
#include "ogx_sm100.cuh"

namespace ogx {
namespace mixed {

// column slices of the M2L output: 1 while the unsplit operand fits TMEM (4 NPAD
// <= 512), else the fewest slices whose width allows the paired form (6 NPAD <= 512)
constexpr int tc_round16(int v) { return (v + 15) / 16 * 16; }
constexpr int tc_nsplit(int nfull) {
    if (4 * tc_round16(nfull) <= 512) return 1;
    int s = 2;
    while (6 * tc_round16((nfull + s - 1) / s) > 512) ++s;
    return s;
}

template <int P>
struct TcCfg {
    static constexpr int K = (P + 1) * (P + 1);
    static constexpr int KPAD = (K + 15) / 16 * 16;
    static constexpr int NKS = KPAD / 16;     // K-steps of the MMA (16 fp16 each)
    static constexpr int CH = 4;              // K-steps per pipeline chunk (64 fp16 = one 128-byte line)
    static constexpr int NCH = (NKS + CH - 1) / CH;
    static constexpr int NFULL = K - 1;       // output dofs 1..K-1
    static constexpr int NSPLIT = tc_nsplit(NFULL);
    static constexpr int N = (NFULL + NSPLIT - 1) / NSPLIT;   // dofs of one slice: 1 + z N .. z N + N
    static constexpr int NPAD = (N + 15) / 16 * 16;
    static constexpr int M = 128;
    static constexpr int SBO = 1024;          // bytes between 8-row groups (one swizzle atom)
    static constexpr int A_BYTES = (M / 8) * SBO;
    static constexpr int B_BYTES = (NPAD / 8) * SBO;
    static constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * B_BYTES;
    static constexpr int STAGES = (220 * 1024 / STAGE_BYTES) >= 4 ? 4 : (220 * 1024 / STAGE_BYTES);
    static constexpr int SMEM = STAGES * STAGE_BYTES + 1024;
    // Paired form (p <= 8): B_hi and B_lo are adjacent rows of one N = 2 NPAD operand,
    // so A_hi x [B_hi | B_lo] is one MMA and A_lo x B_hi a second one (two MMAs per
    // K-step instead of three; an MMA costs about the same time up to N ~ 160).
    // A combination buffer then holds [hh + lh | hl], summed when drained.
    static constexpr bool PAIR = 6 * NPAD <= 512;
    static constexpr int DBUF = PAIR ? 2 * NPAD : NPAD;  // TMEM columns of one FP32 buffer
    // REGACC (p <= 8): one group of four drain warps per 16-column slice of the
    // output, each lane keeping its 16 FP64 sums in registers (a combination costs a
    // drain warp one TMEM load round trip); TMEM then holds only FP32 buffers, NBUF
    // of them in a ring, so the MMA runs NBUF - 1 combinations ahead of the drain.
    // Otherwise two column slices, FP64 sums in TMEM at column ACC64, two buffers.
    static constexpr bool REGACC = PAIR;
    static constexpr int NGRP = REGACC ? NPAD / 16 : 2;  // column slices
    static constexpr int MAXG = (NPAD / 16 + NGRP - 1) / NGRP;
    static constexpr int DRAIN_WARPS = 4 * NGRP;
    static constexpr int THREADS = 128 + 32 + 32 * DRAIN_WARPS;   // producers, MMA warp, drain warps
    static constexpr int NBUF = REGACC ? 512 / DBUF : 2;
    static constexpr int ACC64 = 2 * DBUF;    // first column of the FP64 accumulator (TMEM form)
    static constexpr int TMEM_COLS = 512;
    static constexpr bool SUPPORTED = 4 * NPAD <= 512 && STAGES >= 2;
    static_assert(CH * 16 * 2 == 128, "a chunk row must fill exactly one 128-byte swizzle line");
};

// Byte offset of fp16 element (row, kk), kk < 64, inside one operand of a stage,
// in the K-major 128-byte-swizzle layout: each row's 64 fp16 of the chunk fill
// one 128-byte line, 8 rows form a 1024-byte atom, and 16-byte piece j of row r
// sits at piece position j ^ (r mod 8) so the tensor core reads the 8 rows of an
// atom from different banks.  Operand bases are 1024-byte aligned.
__host__ __device__ __forceinline__ int tile_off(int row, int kk) {
    return (row >> 3) * 1024 + (row & 7) * 128 + ((((kk >> 3) ^ row) & 7) << 4) + (kk & 7) * 2;
}

// Warp roles: warps 0-3 gather the A rows (thread r owns target row r), warp 4
// issues the MMAs (one lane), warps 5..5+TcCfg::DRAIN_WARPS-1 fold every
// combination's FP32 result into the FP64 accumulator and write the tile's result.
// A warp may only touch the TMEM lane quarter (warp index mod 4), so the drain warps
// come in groups of four, each group owning a slice of the output columns.
constexpr int TC_PRODUCERS = 128;

__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Add the FP32 combination result in D buffer `a` (16-column groups g0..g1-1) to
// the FP64 accumulator of this warp's 32 lanes; `first` initialises it instead.
// PAIR: the buffer holds two partial products NPAD columns apart.  `unscale`
// (a power of two) undoes the row's source scale and the operator's scale.
template <int NPAD, int DBUF, int ACC64, bool PAIR>
__device__ __forceinline__ void drain_combo(uint32_t tmem_lane, int a, bool first, int g0, int g1, float unscale) {
#pragma unroll 1
    for (int c16 = g0; c16 < g1; ++c16) {
        uint32_t v[16], w[16], lo[16], hi[16];
        sm100::tmem_ld16(tmem_lane + a * DBUF + c16 * 16, v);
        if (PAIR) sm100::tmem_ld16(tmem_lane + a * DBUF + NPAD + c16 * 16, w);
        if (!first) {
            sm100::tmem_ld16(tmem_lane + ACC64 + c16 * 32, lo);
            sm100::tmem_ld16(tmem_lane + ACC64 + c16 * 32 + 16, hi);
        }
        sm100::tmem_ld_wait();
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            double s = (double)(__uint_as_float(v[k]) * unscale);
            if (PAIR) s += (double)(__uint_as_float(w[k]) * unscale);
            if (!first) s += __hiloint2double((int)hi[k], (int)lo[k]);
            lo[k] = (uint32_t)__double2loint(s);
            hi[k] = (uint32_t)__double2hiint(s);
        }
        tmem_st16(tmem_lane + ACC64 + c16 * 32, lo);
        tmem_st16(tmem_lane + ACC64 + c16 * 32 + 16, hi);
    }
    tmem_st_wait();
}

template <int P>
__global__ void __launch_bounds__(TcCfg<P>::THREADS, 1)
    k_m2l_tc(TreeView tv, M2L64Args ar, const __half* __restrict__ mhi, const __half* __restrict__ mlo, const float* __restrict__ munscale,
             const uint8_t* __restrict__ btab, const float* __restrict__ ounscale, double* __restrict__ lown, int* err) {
    using C = TcCfg<P>;
    static_assert(C::SUPPORTED, "tensor-core M2L: operand does not fit");
    const int zs = blockIdx.y;                    // output column slice
    constexpr int NG = C::NPAD / 16;
    constexpr int NGRP = C::NGRP;
    constexpr int NBUF = C::NBUF;
    static_assert(NBUF * C::DBUF + (C::REGACC ? 0 : 2 * C::NPAD) <= C::TMEM_COLS, "TMEM budget");
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    __shared__ uint64_t afull[C::STAGES], bfull[C::STAGES], empty[C::STAGES], dfull[C::NBUF], dempty[C::NBUF], fin;
    __shared__ uint32_t s_tmem;
    __shared__ volatile int s_abort;
    __shared__ int s_t, s_ncombo;
    __shared__ int s_box[128];
    __shared__ int s_Q[27][128];      // colleague slot D of each target's parent
    __shared__ int s_par[128];
    __shared__ uint32_t s_mask[7];    // bit D * 8 + s: some target of the tile has that V source
    __shared__ int s_wcnt[7];
    __shared__ int s_combo[189];      // present combinations: D | s << 5 | o << 8
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int base = blockIdx.x * 128;
    const uint32_t* __restrict__ tgt_key = ar.tgt_key;
    const uint32_t* __restrict__ tgt_box = ar.tgt_box;
    if (tv_over(tv)) return;
    // this CTA's ranges of colleague slots: [zlo, zhi) of the S ranges (any grid z is correct)
    static_assert(C::NSPLIT <= 3, "k_target_groups writes the split for up to three slices");
    const int S = ar.gs[GS_TC_SPLIT + C::NSPLIT - 1];
    const int zlo = S * (int)blockIdx.z / (int)gridDim.z, zhi = S * ((int)blockIdx.z + 1) / (int)gridDim.z;
    if (zlo == zhi) return;
    if (tid == 0) {
        s_t = (tgt_key[base] == 0xFFFFFFFFu) ? -1 : (int)tgt_key[base];
        s_abort = 0;
        for (int s = 0; s < C::STAGES; ++s) {
            sm100::mbar_init(&afull[s], TC_PRODUCERS);
            sm100::mbar_init(&bfull[s], 1);
            sm100::mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < C::NBUF; ++a) {
            sm100::mbar_init(&dfull[a], 1);
            sm100::mbar_init(&dempty[a], 32 * C::DRAIN_WARPS);
        }
        sm100::mbar_init(&fin, 1);
        sm100::fence_mbar_init();
    }
    if (tid < 7) s_mask[tid] = 0;
    __syncthreads();
    const int t = s_t;
    if (t < 0) return;
    const int D0 = m2l64_first_slot(zlo, S, t), D1 = m2l64_first_slot(zhi, S, t);
    // the A operands of every stage start at zero (rows without a source are not copied)
    for (int i = tid; i < C::STAGES * 2 * C::A_BYTES / 16; i += blockDim.x) {
        const int sg = i / (2 * C::A_BYTES / 16), off = i - sg * (2 * C::A_BYTES / 16);
        reinterpret_cast<uint4*>(smem + (size_t)sg * C::STAGE_BYTES)[off] = make_uint4(0u, 0u, 0u, 0u);
    }
    sm100::fence_proxy_async();
    const int tx = t & 1, ty = (t >> 1) & 1, tz = (t >> 2) & 1;
    if (warp == 4) sm100::tmem_alloc(&s_tmem, C::TMEM_COLS);
    if (tid < 128) {
        const uint32_t key = tgt_key[base + tid];
        const int myb = (key == (uint32_t)t) ? (int)tgt_box[base + tid] : -1;
        s_box[tid] = myb;
        s_par[tid] = (myb >= 0) ? tv.parent[myb] : -1;
    }
    __syncthreads();
    // Colleague slots and the children they offer, spread over the whole CTA: thread
    // (group g, row r) takes slots D = g, g + NGS, ... of target r, with all its loads
    // in flight together.  A warp holds one g and 32 targets, so one OR over the warp
    // gives the presence bits of its slots.
    {
        constexpr int NGS = C::THREADS / 128;
        constexpr int DPT = (27 + NGS - 1) / NGS;
        constexpr int NW = (DPT * 8 + 31) / 32;
        const int r = tid & 127, g = tid >> 7;
        if (g < NGS) {
            const int par = s_par[r];
            int Qv[DPT];
#pragma unroll
            for (int i = 0; i < DPT; ++i) {
                const int D = g + i * NGS;
                Qv[i] = (D >= D0 && D < D1 && par >= 0) ? __ldg(tv.col + 27 * (size_t)par + D) : -1;
            }
            int4 cr[DPT][2];
#pragma unroll
            for (int i = 0; i < DPT; ++i) {
                const int D = g + i * NGS;
                if (D < 27) s_Q[D][r] = Qv[i];
                if (Qv[i] >= 0) {
                    cr[i][0] = __ldg(reinterpret_cast<const int4*>(tv.child + 8 * (size_t)Qv[i]));
                    cr[i][1] = __ldg(reinterpret_cast<const int4*>(tv.child + 8 * (size_t)Qv[i]) + 1);
                } else {
                    cr[i][0] = cr[i][1] = make_int4(-1, -1, -1, -1);
                }
            }
            uint32_t bw[NW];
#pragma unroll
            for (int w = 0; w < NW; ++w) bw[w] = 0;
#pragma unroll
            for (int i = 0; i < DPT; ++i) {
                const int D = g + i * NGS;
                const int Dx = D % 3 - 1, Dy = (D / 3) % 3 - 1, Dz = D / 9 - 1;
                const int ch[8] = {cr[i][0].x, cr[i][0].y, cr[i][0].z, cr[i][0].w,
                                   cr[i][1].x, cr[i][1].y, cr[i][1].z, cr[i][1].w};
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const int ox = 2 * Dx + (s & 1) - tx, oy = 2 * Dy + ((s >> 1) & 1) - ty, oz = 2 * Dz + ((s >> 2) & 1) - tz;
                    if (D < 27 && max(abs(ox), max(abs(oy), abs(oz))) > 1 && ch[s] >= 0) bw[i >> 2] |= 1u << (8 * (i & 3) + s);
                }
            }
#pragma unroll
            for (int w = 0; w < NW; ++w) bw[w] = __reduce_or_sync(0xffffffffu, bw[w]);
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < DPT; ++i) {
                    const int D = g + i * NGS;
                    const uint32_t byte = (bw[i >> 2] >> (8 * (i & 3))) & 0xFFu;
                    if (D < 27 && byte) atomicOr(&s_mask[D >> 2], byte << (8 * (D & 3)));
                }
            }
        }
    }
    __syncthreads();
    // the present combinations in (D, s) order, placed by a ballot prefix over 7 warps
    {
        bool pres = false;
        int code = 0;
        unsigned bal = 0;
        if (tid < 224) {
            const int c = tid, D = c >> 3, s = c & 7;
            if (c < 216 && ((s_mask[c >> 5] >> (c & 31)) & 1u)) {
                const int Dx = D % 3 - 1, Dy = (D / 3) % 3 - 1, Dz = D / 9 - 1;
                const int ox = 2 * Dx + (s & 1) - tx, oy = 2 * Dy + ((s >> 1) & 1) - ty, oz = 2 * Dz + ((s >> 2) & 1) - tz;
                pres = true;
                code = D | (s << 5) | (((ox + 3) + 7 * (oy + 3) + 49 * (oz + 3)) << 8);
            }
            bal = __ballot_sync(0xffffffffu, pres);
            if (lane == 0) s_wcnt[warp] = __popc(bal);
        }
        __syncthreads();
        if (pres) {
            int pos = __popc(bal & ((1u << lane) - 1u));
            for (int w = 0; w < warp; ++w) pos += s_wcnt[w];
            s_combo[pos] = code;
        }
        if (tid == 0) {
            int n = 0;
            for (int w = 0; w < 7; ++w) n += s_wcnt[w];
            s_ncombo = n;
        }
    }
    sm100::tc_fence_before();
    __syncthreads();
    sm100::tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int nco = s_ncombo;

    if (warp == 4) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            constexpr uint32_t idesc = sm100::idesc_f16(C::M, C::NPAD);
            constexpr uint32_t idesc2 = sm100::idesc_f16(C::M, 2 * C::NPAD);
            // descriptors differ only in their 14-bit start-address field (bytes >> 4):
            // build stage 0's once and add the stage / K-step / operand offsets
            const uint64_t desc0 = sm100::smem_desc_sw128(sm100::smem_u32(smem), C::SBO);
            constexpr uint32_t D_LO = C::A_BYTES >> 4, D_BHI = (2 * C::A_BYTES) >> 4,
                               D_BLO = (2 * C::A_BYTES + C::B_BYTES) >> 4, D_STAGE = C::STAGE_BYTES >> 4;
            int u = 0;
            for (int k = 0; k < nco && !s_abort; ++k) {
                const int a = k % NBUF;
                if (k >= NBUF) {
                    if (!sm100::mbar_wait(&dempty[a], ((k / NBUF) - 1) & 1, &s_abort)) {
                        s_abort = 1;
                        atomicExch(err, 1);
                        break;
                    }
                    sm100::tc_fence_after();
                }
                const uint32_t dcol = tmem + a * C::DBUF;
                uint32_t accum = 0;
                for (int c = 0; c < C::NCH && !s_abort; ++c, ++u) {
                    const int s = u % C::STAGES;
                    const uint32_t ph = (u / C::STAGES) & 1;
                    if (!sm100::mbar_wait(&afull[s], ph, &s_abort) || !sm100::mbar_wait(&bfull[s], ph, &s_abort)) {
                        s_abort = 1;
                        atomicExch(err, 1);
                        break;
                    }
                    // the A rows were written by cp.async (generic proxy); the MMA reads
                    // them through the async proxy
                    sm100::fence_proxy_async();
                    sm100::tc_fence_after();
                    const uint64_t ds = desc0 + (uint64_t)(s * D_STAGE);
                    const int nks = min(C::CH, C::NKS - c * C::CH);
#pragma unroll
                    for (int ks = 0; ks < C::CH; ++ks) {
                        if (ks < nks) {
                            const uint64_t dk = ds + (uint64_t)(ks * 2);    // 32 bytes per K-step inside the line
                            if constexpr (C::PAIR) {
                                sm100::mma_f16(dcol, dk, dk + D_BHI, idesc2, accum);      // A_hi x [B_hi | B_lo]
                                accum = 1;
                                sm100::mma_f16(dcol, dk + D_LO, dk + D_BHI, idesc, 1);    // A_lo x B_hi
                            } else {
                                sm100::mma_f16(dcol, dk, dk + D_BHI, idesc, accum);
                                accum = 1;
                                sm100::mma_f16(dcol, dk, dk + D_BLO, idesc, 1);
                                sm100::mma_f16(dcol, dk + D_LO, dk + D_BHI, idesc, 1);
                            }
                        }
                    }
                    sm100::mma_commit(&empty[s]);
                }
                sm100::mma_commit(&dfull[a]);
            }
            // completion of every MMA this thread issued (normal end and abort alike)
            sm100::mma_commit(&fin);
            if (!sm100::mbar_wait(&fin, 0, nullptr)) atomicExch(err, 1);
        }
        __syncwarp();
    } else if (warp < 4) {
        // ---------------- producers: thread r gathers target row r ----------------
        const int r = tid;
        int u = 0;
        bool bulk_pending[C::STAGES];
        uint32_t bulk_phase[C::STAGES];
        for (int s = 0; s < C::STAGES; ++s) bulk_pending[s] = false, bulk_phase[s] = 0;
        // source box of the next combination, fetched one combination ahead
        int src_next = -1;
        if (nco > 0) {
            const int c0 = s_combo[0];
            const int Q = s_Q[c0 & 31][r];
            src_next = (Q >= 0) ? __ldg(tv.child + 8 * (size_t)Q + ((c0 >> 5) & 7)) : -1;
        }
        // exits are warp-uniform: the row copies below shuffle across the warp
        for (int k = 0; k < nco && !__any_sync(0xffffffffu, s_abort != 0); ++k) {
            const int code = s_combo[k];
            const int src = src_next;
            if (k + 1 < nco) {
                const int c1 = s_combo[k + 1];
                const int Q = s_Q[c1 & 31][r];
                src_next = (Q >= 0) ? __ldg(tv.child + 8 * (size_t)Q + ((c1 >> 5) & 7)) : -1;
            }
            const int o = code >> 8;
            for (int c = 0; c < C::NCH; ++c, ++u) {
                const int s = u % C::STAGES;
                if (u >= C::STAGES) {
                    const bool ok = sm100::mbar_wait(&empty[s], ((u / C::STAGES) - 1) & 1, &s_abort);
                    if (!__all_sync(0xffffffffu, ok)) {
                        s_abort = 1;
                        atomicExch(err, 1);
                        break;
                    }
                    bulk_pending[s] = false;
                }
                uint8_t* st = smem + (size_t)s * C::STAGE_BYTES;
                if (r == 0) {
                    const uint8_t* bsrc = btab + ((size_t)((o * C::NSPLIT + zs) * C::NCH + c) * 2) * C::B_BYTES;
                    sm100::mbar_arrive_expect_tx(&bfull[s], 2 * C::B_BYTES);
                    sm100::bulk_g2s(st + 2 * C::A_BYTES, bsrc, C::B_BYTES, &bfull[s]);
                    sm100::bulk_g2s(st + 2 * C::A_BYTES + C::B_BYTES, bsrc + C::B_BYTES, C::B_BYTES, &bfull[s]);
                    bulk_pending[s] = true;
                    bulk_phase[s] = (u / C::STAGES) & 1;
                }
                // the warp copies its 32 rows cooperatively: one instruction moves
                // 16-byte pieces q0..q0+3 of 8 rows, so each source row is read in
                // whole 64-byte runs and a quarter-warp fills 8 consecutive slots
                const int k0 = c * C::CH * 16;
                const int nq = min(8, (C::KPAD - k0) / 8);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int rl = 8 * (i >> 2) + (lane & 7);         // row within the warp
                    const int part = (i >> 1) & 1;                    // 0: hi, 1: lo
                    const int q = (i & 1) * 4 + (lane >> 3);          // 16-byte piece (8 fp16) of the chunk
                    const int rs = __shfl_sync(0xffffffffu, src, rl);
                    if (q < nq) {
                        // an absent source leaves the row's previous contents (finite
                        // values of an earlier row, or the zeros written at start): the
                        // drain multiplies that row's result by an unscale of 0
                        if (rs >= 0)
                            sm100::cp_async16(st + part * C::A_BYTES + tile_off(32 * warp + rl, 8 * q),
                                              (part ? mlo : mhi) + (size_t)rs * C::KPAD + k0 + 8 * q);
                    }
                }
                // the stage's A barrier counts one arrival per producer thread, made
                // when that thread's copies have landed: the producer moves on at once,
                // so every stage of the ring can have its gathers in flight
                sm100::cp_async_mbar_arrive_noinc(&afull[s]);
            }
        }
        sm100::cp_async_wait_all();
        if (s_abort && r == 0) {
            // let this thread's bulk copies land before the CTA exits
            for (int s = 0; s < C::STAGES; ++s)
                if (bulk_pending[s]) sm100::mbar_wait(&bfull[s], bulk_phase[s], nullptr);
        }
    } else {
        // ---------------- drain warps: FP32 combination -> FP64 accumulator -> L_own ----------------
        const int quarter = warp & 3;                 // the TMEM lane quarter this warp may access
        const int grp = (warp - 5) >> 2;              // column slice of this warp
        const int g0 = grp * NG / NGRP, g1 = (grp + 1) * NG / NGRP;
        const uint32_t tmem_lane = tmem + ((uint32_t)(quarter * 32) << 16);
        const int row = quarter * 32 + lane;
        double racc[C::REGACC ? C::MAXG : 1][16];
        float part[C::REGACC ? C::MAXG : 1][16];
#pragma unroll
        for (int g = 0; g < (C::REGACC ? C::MAXG : 1); ++g)
#pragma unroll
            for (int i = 0; i < 16; ++i) racc[g][i] = 0.0, part[g][i] = 0.f;
        int z = zlo, zend = m2l64_first_slot(zlo + 1, S, t);   // the range of the current combination, its first slot behind
        bool fresh = true;                                     // no combination of this range yet
        // the finished range's sums (zeros where it had no combination) to its row
        auto flush = [&]() {
            // to the box's local (one range), else to the range's row of the partial sums
            // (k_m2l64_sum adds them in range order)
            const int myb = s_box[row];
            double inv = 1.0;
            double* o = nullptr;
            if (myb >= 0 && S == 1) {
                inv = 1.0 / (2.0 * tv.center[4 * (size_t)myb + 3]);
                o = lown + (size_t)myb * C::K;
            } else if (myb >= 0) {
                const int pq = base + row - ar.gs[9 + t];
                o = ar.part + ((size_t)z * tv.cnt->ntgt32 + ar.gs[t] + (int64_t)(pq / 128) * ar.gs[GS_FILL] + pq % 128) * C::K;
            }
            if constexpr (C::REGACC) {
#pragma unroll
                for (int g = 0; g < C::MAXG; ++g) {
                    const int c16 = g0 + g;
                    if (c16 < g1 && myb >= 0) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const int col = c16 * 16 + i, dof = 1 + zs * C::N + col;
                            if (col < C::N && dof < C::K) o[dof] = racc[g][i] * inv;
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 16; ++i) racc[g][i] = 0.0;
                }
            } else {
#pragma unroll 1
                for (int c16 = g0; c16 < g1; ++c16) {
                    uint32_t lo[16], hi[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) lo[k] = hi[k] = 0u;
                    if (!fresh) {
                        sm100::tmem_ld16(tmem_lane + C::ACC64 + c16 * 32, lo);
                        sm100::tmem_ld16(tmem_lane + C::ACC64 + c16 * 32 + 16, hi);
                        sm100::tmem_ld_wait();
                    }
                    if (myb >= 0) {
#pragma unroll
                        for (int k = 0; k < 16; ++k) {
                            const int col = c16 * 16 + k, dof = 1 + zs * C::N + col;
                            if (col < C::N && dof < C::K) o[dof] = __hiloint2double((int)hi[k], (int)lo[k]) * inv;
                        }
                    }
                }
            }
            fresh = true;
            ++z;
            zend = m2l64_first_slot(z + 1, S, t);
        };
        for (int k = 0; k < nco && !s_abort; ++k) {
            const int a = k % NBUF;
            // this row's source for combination k and the scales its operands carry
            const int code = s_combo[k];
            while ((code & 31) >= zend && z + 1 < zhi) flush();
            // combinations come grouped by colleague slot D (the eight children of one
            // colleague, at similar distances): their FP32 results are summed in FP32 and
            // the slot's sum is folded into FP64 once, after its last combination
            const bool fold = (k + 1 == nco) || ((s_combo[k + 1] & 31) != (code & 31));
            const int Q = s_Q[code & 31][row];
            const int srcb = (Q >= 0) ? __ldg(tv.child + 8 * (size_t)Q + ((code >> 5) & 7)) : -1;
            const float unscale = (srcb >= 0) ? __ldg(munscale + srcb) * __ldg(ounscale + (code >> 8)) : 0.f;
            if (!sm100::mbar_wait(&dfull[a], (k / NBUF) & 1, &s_abort)) {
                s_abort = 1;
                atomicExch(err, 1);
                break;
            }
            sm100::tc_fence_after();
            if constexpr (C::REGACC) {
#pragma unroll
                for (int g = 0; g < C::MAXG; ++g) {
                    const int c16 = g0 + g;
                    if (c16 < g1) {
                        // two halves of 8 columns keep the drain's registers within the
                        // launch's budget; the two partial products meet in FP32 (w is
                        // ~2^-11 of v)
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            uint32_t v[8], w[8];
                            sm100::tmem_ld8(tmem_lane + a * C::DBUF + c16 * 16 + 8 * h, v);
                            sm100::tmem_ld8(tmem_lane + a * C::DBUF + C::NPAD + c16 * 16 + 8 * h, w);
                            sm100::tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                                part[g][8 * h + i] = fmaf(__uint_as_float(v[i]) + __uint_as_float(w[i]), unscale, part[g][8 * h + i]);
                        }
                        if (fold) {
#pragma unroll
                            for (int i = 0; i < 16; ++i) {
                                racc[g][i] += (double)part[g][i];
                                part[g][i] = 0.f;
                            }
                        }
                    }
                }
            } else {
                drain_combo<C::NPAD, C::DBUF, C::ACC64, C::PAIR>(tmem_lane, a, fresh, g0, g1, unscale);
            }
            fresh = false;
            sm100::tc_fence_before();
            sm100::mbar_arrive(&dempty[a]);
        }
        // (one range and no combination: the local stays zero)
        if (!s_abort && (nco >= 1 || S > 1))
            while (z < zhi) flush();
    }
    sm100::tc_fence_before();
    __syncthreads();
    if (warp == 4) {
        // the MMA lane waited on `fin` above, so no MMA still writes TMEM here
        sm100::tc_fence_after();
        sm100::tmem_dealloc(tmem, C::TMEM_COLS);
    }
}

// FP64 multipoles -> scaled FP16 hi/lo pairs, rows padded to KPAD with zeros.  Warp
// per box: the row is scaled by a power of two 2^-e so that its largest entry lies
// in [0.5, 1) (FP16 keeps 11 significant bits like TF32 but has a narrow exponent
// range); hi = fp16(x), lo = fp16(x - hi); munscale[b] = 2^e undoes the scaling
// exactly when the M2L result is drained.
template <int P>
__global__ void __launch_bounds__(128) k_split_mpole(const double* __restrict__ M, int nb, __half* __restrict__ hi,
                                                     __half* __restrict__ lo, float* __restrict__ munscale,
                                                     const DevCounts* counts) {
    using C = TcCfg<P>;
    const int lane = threadIdx.x & 31;
    const int b = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (b >= nb || b >= counts->nb32 || counts->overflow) return;
    const double* row = M + (size_t)b * C::K;
    double mx = 0.0;
    for (int k = lane; k < C::K; k += 32) mx = fmax(mx, fabs(row[k]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    int e = 0;
    if (mx > 0.0) frexp(mx, &e);
    const double scale = ldexp(1.0, -e);
    for (int k = lane; k < C::KPAD; k += 32) {
        const double x = (k < C::K) ? row[k] * scale : 0.0;
        const __half h = __double2half(x);
        hi[(size_t)b * C::KPAD + k] = h;
        lo[(size_t)b * C::KPAD + k] = __double2half(x - (double)__half2float(h));
    }
    if (lane == 0) munscale[b] = ldexpf(1.0f, e);
}

// L_0^0 of the M2L (needed only for potentials): FP64 row 0 of every T_o.  Warp per target:
// lane D lists the V children of colleague slot D, then the lanes run over the coefficients
// of one source after another (a thread per target read K doubles of 189 sources on its own,
// 510 us on 262,144 bodies at p = 4).
template <int P>
__global__ void __launch_bounds__(128) k_m2l_dof0(TreeView tv, int ntgt_bound, const uint32_t* __restrict__ box,
                                                  const double* __restrict__ row0 /* 343 x K */, const double* __restrict__ M,
                                                  double* __restrict__ lown) {
    constexpr int K = (P + 1) * (P + 1), NPL = (K + 31) / 32;
    __shared__ int s_src[4][192], s_op[4][192];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int i = blockIdx.x * 4 + w;
    if (i >= ntgt_bound || tv_over(tv) || i >= tv.cnt->ntgt32) return;
    const int b = (int)box[i], par = tv.parent[b];
    const int tx = tv.coord[3 * (size_t)b] & 1, ty = tv.coord[3 * (size_t)b + 1] & 1, tz = tv.coord[3 * (size_t)b + 2] & 1;
    const int Q = lane < 27 ? tv.col[27 * (size_t)par + lane] : -1;
    int4 c0 = make_int4(-1, -1, -1, -1), c1 = c0;
    if (Q >= 0) {
        c0 = __ldg(reinterpret_cast<const int4*>(tv.child + 8 * (size_t)Q));
        c1 = __ldg(reinterpret_cast<const int4*>(tv.child + 8 * (size_t)Q) + 1);
    }
    const int ch[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
    const int Dx = lane % 3 - 1, Dy = (lane / 3) % 3 - 1, Dz = lane / 9 - 1;
    int n = 0;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const int ox = 2 * Dx + (s & 1) - tx, oy = 2 * Dy + ((s >> 1) & 1) - ty, oz = 2 * Dz + ((s >> 2) & 1) - tz;
        const bool v = ch[s] >= 0 && max(abs(ox), max(abs(oy), abs(oz))) > 1;
        const unsigned m = __ballot_sync(0xffffffffu, v);
        if (v) {
            const int q = n + __popc(m & ((1u << lane) - 1u));
            s_src[w][q] = ch[s];
            s_op[w][q] = (ox + 3) + 7 * (oy + 3) + 49 * (oz + 3);
        }
        n += __popc(m);
    }
    __syncwarp();
    double acc = 0.0;
#pragma unroll 4
    for (int q = 0; q < n; ++q) {
        const double* m = M + (size_t)s_src[w][q] * K;
        const double* r = row0 + (size_t)s_op[w][q] * K;
#pragma unroll
        for (int u = 0; u < NPL; ++u)
            if (lane + 32 * u < K) acc = fma(__ldg(r + lane + 32 * u), __ldg(m + lane + 32 * u), acc);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) lown[(size_t)b * K] += acc / (2.0 * tv.center[4 * (size_t)b + 3]);
}

// acc[orig] = G (far + near), pot[orig] = -G (far + near) (AdaptiveFMM3D.hpp:104)
// far = far_l (L2P) + far_m (M2P) when the two parts ran apart (far_m non-null)
template <bool POT>
__global__ void k_combine(int n, const int* __restrict__ perm, double G, const double* __restrict__ far,
                          const double* __restrict__ far_m, const double* __restrict__ near, double* __restrict__ acc,
                          double* __restrict__ pot, const DevCounts* counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || counts->overflow) return;
    const int o = perm[i];
    double2 f0 = reinterpret_cast<const double2*>(far)[2 * (size_t)i];
    double2 f1 = reinterpret_cast<const double2*>(far)[2 * (size_t)i + 1];
    if (far_m) {
        const double2 m0 = reinterpret_cast<const double2*>(far_m)[2 * (size_t)i];
        const double2 m1 = reinterpret_cast<const double2*>(far_m)[2 * (size_t)i + 1];
        f0.x += m0.x; f0.y += m0.y; f1.x += m1.x; f1.y += m1.y;
    }
    const double2 n0 = reinterpret_cast<const double2*>(near)[2 * (size_t)i];
    const double2 n1 = reinterpret_cast<const double2*>(near)[2 * (size_t)i + 1];
    acc[3 * (size_t)o] = G * (f0.x + n0.x);
    acc[3 * (size_t)o + 1] = G * (f0.y + n0.y);
    acc[3 * (size_t)o + 2] = G * (f1.x + n1.x);
    if (POT) pot[o] = -G * (f1.y + n1.y);
}

}  // namespace mixed
}  // namespace ogx
