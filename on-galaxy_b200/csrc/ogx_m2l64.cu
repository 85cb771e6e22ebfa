// ogx_m2l64.cu -- the plain form's M2L on the FP64 matrix instructions.
//
// The reference applies fmm::M2L pair by pair (src3d/FmmExpansions3D.hpp:273-299, called
// per V-list entry in src3d/AdaptiveFMM3D.hpp:78-81).  Here 64 targets that share their
// octant in the parent form a tile; for one (colleague slot D, child s) combination every
// target has at most one source, so the sources' multipoles are the rows of A (64 x K,
// zero rows where absent) and L += A T_o^T with one operator for the tile.
//
// Bound: the FP64 pipe (mma.sync f64 and DFMA measured alike, 18.4e12 FMA/s on the whole
// GPU).  A kernel of plain FMAs needs ten loads per 24 FMAs and ran at a fifth of that, so
// the product goes through mma.sync m16n8k4: a warp holds 16 targets x all K outputs in
// registers and reads one operand double per 16 x 4 FMAs.  Operator chunks (28 rows) and
// source chunks come by cp.async, three stages deep, two CTAs per SM (one DMMA warp per
// scheduler leaves the pipe idle at the chunk barriers).  A warp whose 16 targets have no
// source in a combination skips its products.
#include <algorithm>

#include "ogx_m2l64.cuh"
#include "ogx_sm100.cuh"

namespace ogx {
namespace {

template <int P>
struct M64 {
    static constexpr int K = (P + 1) * (P + 1);
    static constexpr int K4 = (K + 3) / 4 * 4;            // contraction, padded with zeros
    static constexpr int NT = (K + 7) / 8;                // 8-column tiles of the output
    static constexpr int NP = 8 * NT;
    static constexpr int LDN = NP + 4;                    // 4 or 12 mod 16: conflict-free operand reads
    static constexpr int NCH = (K4 + 27) / 28;            // chunks of at most 28 rows
    static constexpr int KC = ((K4 + NCH - 1) / NCH + 3) / 4 * 4;
    static constexpr int LDA = (KC % 16 == 4 || KC % 16 == 12) ? KC : KC + 4;
    static constexpr int WN = NT > 16 ? 2 : 1;            // warps along the output (P >= 11: registers)
    static constexpr int NTW = NT / WN;        // column tiles of one warp
    static constexpr int THREADS = 128 * WN;
    static constexpr int A_D = M2L64_TGT * LDA, B_D = KC * LDN;   // doubles of a stage
    static constexpr int STAGE = (A_D + B_D) * 8;
    static constexpr bool THREE = 3 * STAGE <= 105 * 1024 || 2 * STAGE > 105 * 1024;
    static constexpr int STAGES = THREE ? 3 : 2;
    static constexpr int SMEM = STAGES * STAGE;
    static constexpr int MINB = SMEM <= 105 * 1024 ? 2 : 1;
    static_assert(LDA % 16 == 4 || LDA % 16 == 12, "A rows: conflict-free operand reads");
    static_assert(LDN % 16 == 4 || LDN % 16 == 12, "B rows: conflict-free operand reads");
    static_assert(NT % WN == 0, "column halves");
    static_assert(SMEM <= 218 * 1024, "stages fit the SM");
};

template <int P>
__global__ void __launch_bounds__(M64<P>::THREADS, M64<P>::MINB)
    k_m2l_fp64(TreeView tv, M2L64Args ar, const double* __restrict__ ops, const double* __restrict__ mpole, double* lown) {
    using C = M64<P>;
    constexpr int K = C::K, TH = C::THREADS;
    extern __shared__ __align__(16) double s_dyn[];
    __shared__ int s_Q[27][M2L64_TGT];       // colleague slots of each target's parent
    __shared__ uint32_t s_mask[7];           // bit 8 D + s: some target of the tile has that source
    __shared__ int s_combo[189];             // the item's combinations: D | s << 5 | o << 8
    __shared__ int s_src[2][M2L64_TGT];      // source boxes of one combination, double buffered
    __shared__ uint32_t s_act[8];            // which 16-target groups have a source (ring)
    __shared__ int s_tgt[M2L64_TGT];
    __shared__ int s_n, s_item;
    if (tv_over(tv)) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = warp & 3, wn = warp >> 2;               // row group, column half
    const int S = ar.gs[GS_SPLIT], tiles = ar.gs[GS_TILES];
    const int ntgt = tv.cnt->ntgt32;
    for (;;) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(ar.gs + GS_TICKET, 1);
        if (tid < 7) s_mask[tid] = 0;
        __syncthreads();
        const int item = s_item;
        if (item >= tiles * S) return;
        const int z = item / tiles, base = (item - z * tiles) * M2L64_TGT;
        // the padded target layout never mixes octants inside a tile; an empty tile starts empty
        const int t = (int)ar.tgt_key[base];
        if (t < 0) continue;
        const int D0 = m2l64_first_slot(z, S, t), D1 = m2l64_first_slot(z + 1, S, t);
        if (tid < M2L64_TGT) s_tgt[tid] = ((int)ar.tgt_key[base + tid] == t) ? (int)ar.tgt_box[base + tid] : -1;
        __syncthreads();
        const int tx = t & 1, ty = (t >> 1) & 1, tz = (t >> 2) & 1;
        // colleague slots and the children they offer: thread = (target, slot group)
        for (int i = tid; i < (D1 - D0) * M2L64_TGT; i += TH) {
            const int D = D0 + i / M2L64_TGT, r = i % M2L64_TGT;
            const int b = s_tgt[r];
            const int Q = b >= 0 ? tv.col[27 * (size_t)tv.parent[b] + D] : -1;
            s_Q[D][r] = Q;
            uint32_t bits = 0;
            if (Q >= 0) {
                const int4 c0 = __ldg(reinterpret_cast<const int4*>(tv.child + 8 * (size_t)Q));
                const int4 c1 = __ldg(reinterpret_cast<const int4*>(tv.child + 8 * (size_t)Q) + 1);
                const int ch[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
                const int Dx = D % 3 - 1, Dy = (D / 3) % 3 - 1, Dz = D / 9 - 1;
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const int ox = 2 * Dx + (s & 1) - tx, oy = 2 * Dy + ((s >> 1) & 1) - ty, oz = 2 * Dz + ((s >> 2) & 1) - tz;
                    if (ch[s] >= 0 && max(abs(ox), max(abs(oy), abs(oz))) > 1) bits |= 1u << s;
                }
            }
            bits = __reduce_or_sync(0xffffffffu, bits);   // whole warps share a slot
            if (lane == 0 && bits) atomicOr(&s_mask[D >> 2], bits << (8 * (D & 3)));
        }
        __syncthreads();
        if (warp == 0) {   // the present combinations in (D, s) order
            int n = 0;
            for (int w = 0; w < 7; ++w) {
                const uint32_t m = s_mask[w];
                if (m >> lane & 1) {
                    const int c = 32 * w + lane, D = c >> 3, s = c & 7;
                    const int ox = 2 * (D % 3 - 1) + (s & 1) - tx, oy = 2 * ((D / 3) % 3 - 1) + ((s >> 1) & 1) - ty,
                              oz = 2 * (D / 9 - 1) + ((s >> 2) & 1) - tz;
                    s_combo[n + __popc(m & ((1u << lane) - 1u))] = D | (s << 5) | (((ox + 3) + 7 * (oy + 3) + 49 * (oz + 3)) << 8);
                }
                n += __popc(m);
            }
            if (lane == 0) s_n = n;
        }
        __syncthreads();
        const int nco = s_n, nch = nco * C::NCH;
        double acc[C::NTW][4];
#pragma unroll
        for (int i = 0; i < C::NTW; ++i)
#pragma unroll
            for (int q = 0; q < 4; ++q) acc[i][q] = 0.0;
        // source of row tid (< 64) in combination k
        auto source = [&](int k) {
            if (k >= nco) return -1;
            const int code = s_combo[k], Q = s_Q[code & 31][tid];
            return Q >= 0 ? __ldg(tv.child + 8 * (size_t)Q + ((code >> 5) & 7)) : -1;
        };
        auto put_source = [&](int k, int src) {   // warps 0 and 1
            s_src[k & 1][tid] = src;
            const unsigned b = __ballot_sync(0xffffffffu, src >= 0);
            if (lane == 0) {   // rows 32 w .. 32 w + 31: bits 2 w and 2 w + 1
                const uint32_t two = ((b & 0xFFFFu) ? 1u : 0u) | ((b >> 16) ? 2u : 0u);
                reinterpret_cast<volatile uint8_t*>(s_act)[(k & 7) * 4 + warp] = (uint8_t)two;
            }
        };
        int src_next = -1;                         // source for combination k + 1, one ahead
        if (tid < M2L64_TGT) {
            put_source(0, source(0));
            src_next = source(1);
        }
        __syncthreads();
        // issue the copies of chunk u into its stage
        auto issue = [&](int u) {
            if (u < nch) {
                const int k = u / C::NCH, c = u - k * C::NCH;
                double* sa = s_dyn + (size_t)(u % C::STAGES) * (C::A_D + C::B_D);
                double* sb = sa + C::A_D;
                const int kn = min(C::KC, C::K4 - c * C::KC);
                const double* T = ops + ((size_t)(s_combo[k] >> 8) * C::K4 + c * C::KC) * C::LDN;
                for (int i = tid; i < kn * C::LDN / 2; i += TH) sm100::cp_async16(sb + 2 * i, T + 2 * i);
                const int* src = s_src[k & 1];
#pragma unroll 4
                for (int i = tid; i < M2L64_TGT * C::KC; i += TH) {
                    const int r = i / C::KC, q = i - r * C::KC, kk = c * C::KC + q;
                    const int b = src[r];
                    const bool ok = b >= 0 && kk < K;
                    if (q < kn) sm100::cp_async8_zfill(sa + r * C::LDA + q, ok ? mpole + (size_t)b * K + kk : mpole, ok ? 8u : 0u);
                }
                if (c == 0 && tid < M2L64_TGT) {   // sources of the next combination; the buffer's last reader was chunk u - 1
                    put_source(k + 1, src_next);
                    src_next = source(k + 2);
                }
            }
            sm100::cp_async_commit();
        };
        for (int u = 0; u < C::STAGES - 1; ++u) {
            issue(u);
            __syncthreads();
        }
        for (int u = 0; u < nch; ++u) {
            sm100::cp_async_wait<C::STAGES - 2>();
            __syncthreads();           // chunk u has landed; the stage of chunk u - 1 is free
            issue(u + C::STAGES - 1);
            const int k = u / C::NCH, c = u - k * C::NCH;
            const uint32_t act = reinterpret_cast<const volatile uint8_t*>(s_act)[(k & 7) * 4 + (wr >> 1)];
            if (!(act >> (wr & 1) & 1u)) continue;   // none of this warp's 16 targets has a source
            const double* sa = s_dyn + (size_t)(u % C::STAGES) * (C::A_D + C::B_D);
            const double* sb = sa + C::A_D + (lane & 3) * C::LDN + (lane >> 2) + wn * C::NTW * 8;
            sa += (16 * wr + (lane >> 2)) * C::LDA + (lane & 3);
            const int kn = min(C::KC, C::K4 - c * C::KC);
            auto step = [&](int k4) {
                const double a0 = sa[k4], a1 = sa[k4 + 8 * C::LDA];
#pragma unroll
                for (int i = 0; i < C::NTW; ++i)
                    sm100::dmma(acc[i], a0, a1, sb[k4 * C::LDN + 8 * i]);
            };
            if (kn == C::KC) {
#pragma unroll
                for (int k4 = 0; k4 < C::KC; k4 += 4) step(k4);
            } else {
#pragma unroll 1
                for (int k4 = 0; k4 < kn; k4 += 4) step(k4);
            }
        }
        sm100::cp_async_wait_all();
        // rows lane / 4 and lane / 4 + 8 of the warp's group, columns 2 (lane % 4) + {0, 1} of each tile
#pragma unroll
        for (int hrow = 0; hrow < 2; ++hrow) {
            const int r = 16 * wr + (lane >> 2) + 8 * hrow, b = s_tgt[r];
            if (b < 0) continue;
            const int q = base + r - ar.gs[9 + t], fill = ar.gs[GS_FILL];
            const int64_t j = ar.gs[t] + (int64_t)(q / 128) * fill + q % 128;   // sorted target
            double* o = S == 1 ? lown + (size_t)b * K : ar.part + ((size_t)z * ntgt + j) * K;
            const double sc = S == 1 ? 1.0 / (2.0 * tv.center[4 * b + 3]) : 1.0;
#pragma unroll
            for (int i = 0; i < C::NTW; ++i) {
                const int d = 8 * (wn * C::NTW + i) + 2 * (lane & 3);
                if (d < K) o[d] = acc[i][2 * hrow] * sc;
                if (d + 1 < K) o[d + 1] = acc[i][2 * hrow + 1] * sc;
            }
        }
    }
}

// Lown of every target = its ranges' sums in range order / side (split above 1)
__global__ void __launch_bounds__(256) k_m2l64_sum(TreeView tv, M2L64Args ar, int K, int slices, double* __restrict__ lown) {
    const int S = ar.gs[slices > 0 ? GS_TC_SPLIT + slices - 1 : GS_SPLIT];
    if (tv_over(tv) || S == 1) return;
    const int ntgt = tv.cnt->ntgt32;
    const int64_t total = (int64_t)ntgt * K;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
        const int j = (int)(i / K), d = (int)(i - (int64_t)j * K);
        if (slices > 0 && d == 0) continue;
        double v = 0.0;
#pragma unroll 9
        for (int z = 0; z < S; ++z) v += ar.part[(size_t)z * total + i];
        const int b = (int)ar.sorted_box[j];
        lown[(size_t)b * K + d] = v * (1.0 / (2.0 * tv.center[4 * b + 3]));
    }
}

template <int P>
int launch(Handle& h, const double* M, double* Lown) {
    using C = M64<P>;
    M2L64Args a;
    OGX_TRY(m2l64_args(h, 0, &a));
    OGX_CUDA(smem_optin((const void*)k_m2l_fp64<P>, C::SMEM));
    const int tiles = h.ntgt_pad / M2L64_TGT;
    const int grid = (int)std::min<int64_t>((int64_t)tiles * M2L64_MAXSPLIT, C::MINB * h.num_sms);
    k_m2l_fp64<P><<<grid, C::THREADS, C::SMEM, h.stream>>>(h.tv, a, h.d_m2l, M, Lown); ++h.launches;
    return m2l64_sum_launch(h, a, 0, Lown, h.stream);
}

}  // namespace

int m2l64_pad_rows(int p) { return ((p + 1) * (p + 1) + 3) / 4 * 4; }
int m2l64_pad_cols(int p) { return ((p + 1) * (p + 1) + 7) / 8 * 8 + 4; }

int m2l64_args(Handle& h, int slices, M2L64Args* a) {
    a->tgt_key = h.tgt_tile_key;
    a->tgt_box = h.tgt_tile_box;
    a->sorted_box = h.tgt_box;
    a->gs = h.tgt_groups;
    const size_t rows = slices > 0 ? m2l_tc_partial_rows(h.ntgt, slices) : m2l64_partial_rows(h.ntgt);
    return arena_get(h.ws, S_M2L_PART, rows * num_dofs(h.prm.p), &a->part);
}

int m2l64_sum_launch(Handle& h, const M2L64Args& a, int slices, double* Lown, cudaStream_t st) {
    const int K = num_dofs(h.prm.p);
    const int grid = (int)std::min<int64_t>(((int64_t)h.ntgt * K + 255) / 256, 8 * h.num_sms);
    k_m2l64_sum<<<grid, 256, 0, st>>>(h.tv, a, K, slices, Lown); ++h.launches;
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

int m2l_fp64_launch(Handle& h, const double* M, double* Lown) {
    if (!h.d_m2l || h.m2l_ops_p != h.prm.p) return OGX_ERR_STATE;   // no operators on the device
    switch (h.prm.p) {
        case 1: return launch<1>(h, M, Lown);
        case 2: return launch<2>(h, M, Lown);
        case 3: return launch<3>(h, M, Lown);
        case 4: return launch<4>(h, M, Lown);
        case 5: return launch<5>(h, M, Lown);
        case 6: return launch<6>(h, M, Lown);
        case 7: return launch<7>(h, M, Lown);
        case 8: return launch<8>(h, M, Lown);
        case 9: return launch<9>(h, M, Lown);
        case 10: return launch<10>(h, M, Lown);
        case 11: return launch<11>(h, M, Lown);
        case 12: return launch<12>(h, M, Lown);
        default: return OGX_ERR_INVALID;
    }
}

}  // namespace ogx
