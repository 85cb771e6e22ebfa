// ogx_m2l_rot.cu -- the third form's M2L: every operator factored into rotations.
//
// The reference applies each M2L with the dense O(p^4) formulas (fmm::M2L,
// src3d/FmmExpansions3D.hpp:273-300) and defers an O(p^3) rotation scheme (its
// README.md:75).  Here T_o = Q_o^-1 Z_|o| Q_o (factors from build_rot_pack in
// ogx_tables.cpp), applied tile by tile over the same target tiles and (colleague
// slot, child) combinations as the plain form's k_m2l_fp64.  Kept in a file of its
// own: the fully unrolled blocks of twelve orders take minutes to compile, and the
// build then runs it beside the other units.
#include <algorithm>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

#include "ogx_m2l64.cuh"
#include "ogx_sm100.cuh"

namespace ogx {
namespace {

constexpr int ROT_TGT = M2L64_TGT;   // targets per CTA

// ---- M2L by rotations (the third form) ------------------------------------------------
// T_o = Q_o^-1 Z_|o| Q_o (build_rot_pack): per tile of ROT_TGT targets sharing octant t
// and per present (D, s) combination (offset o) the 64 source multipoles are staged,
// then y = Q_o m (degree blocks) -> z = Z_|o| y (order blocks) -> acc += Q_o^-1 z
// (degree blocks), the last sums kept in registers over all combinations.
// Thread (g, a) = (tid / 64, tid % 64) owns source / target row a and, in each stage, a
// fixed set of blocks: the four groups g take the blocks in snake order of size
// (largest to g = 0, 1, 2, 3, 3, 2, 1, 0, 0, ...), so they carry about equal work.  A
// block runs fully unrolled: its inputs sit in registers and its outputs are
// independent FMA chains, so a thread keeps up to 2p + 1 of them in flight.  The
// factors are read with warp-uniform addresses (every lane of a warp is in the same
// block).  FP64 throughout.
template <int P>
struct RotCfg {
    static constexpr int K = (P + 1) * (P + 1);
    static constexpr int LD = K | 1;
    static constexpr int QSZ = (P + 1) * (2 * P + 1) * (2 * P + 3) / 3;   // sum_n (2n+1)^2
    static constexpr int ZSZ = (P + 1) * (P + 2) * (2 * P + 3) / 6;       // sum_m (P+1-m)^2
    static constexpr int PACK = 2 * QSZ + ZSZ;
    // the device's packs: Q_o, Q_o^-1 and Z, each from a 16-byte boundary
    static constexpr int QS = (QSZ + 1) / 2 * 2, ZS = (ZSZ + 1) / 2 * 2, DPACK = 2 * QS + ZS;
    static constexpr size_t ROWS_BYTES = (size_t)2 * ROT_TGT * LD * sizeof(double);
    // factors staged in shared memory where they fit beside the rows (p <= 11)
    static constexpr bool STAGE = ROWS_BYTES + DPACK * sizeof(double) <= 212 * 1024;
    static constexpr size_t SMEM = ROWS_BYTES + (STAGE ? DPACK * sizeof(double) : 0);
    // rows per thread: each factor entry loaded feeds RB FMAs (2 where the registers allow)
    static constexpr int RB = P <= 10 ? 2 : 1;
    static constexpr int ROWS = ROT_TGT / RB;          // threads of one block group
    static constexpr int THREADS = 4 * ROWS;
    static constexpr int snake(int i) { return ((i / 4) % 2 == 0) ? i % 4 : 3 - i % 4; }
    // degree blocks: block n has 2n+1 rows; the i-th largest is n = P - i
    static constexpr int deg_group(int n) { return snake(P - n); }
    // position of block n's rows in its group's accumulators (blocks taken largest first)
    static constexpr int deg_pos(int n) {
        int pos = 0;
        for (int q = P; q > n; --q)
            if (deg_group(q) == deg_group(n)) pos += 2 * q + 1;
        return pos;
    }
    static constexpr int group_rows(int g) {
        int r = 0;
        for (int n = 0; n <= P; ++n)
            if (deg_group(n) == g) r += 2 * n + 1;
        return r;
    }
    static constexpr int NACC = group_rows(0) > group_rows(1) ? (group_rows(0) > group_rows(2) ? (group_rows(0) > group_rows(3) ? group_rows(0) : group_rows(3)) : (group_rows(2) > group_rows(3) ? group_rows(2) : group_rows(3)))
                                                               : (group_rows(1) > group_rows(2) ? (group_rows(1) > group_rows(3) ? group_rows(1) : group_rows(3)) : (group_rows(2) > group_rows(3) ? group_rows(2) : group_rows(3)));
    // order blocks: block m has (P+1-m)^2 entries, applied to 1 (m = 0) or 2 (re, im) parts
    static constexpr int ord_work(int m) { return (P + 1 - m) * (P + 1 - m) * (m == 0 ? 1 : 2); }
    static constexpr int ord_group(int m) {
        int rank = 0;
        for (int q = 0; q <= P; ++q)
            if (ord_work(q) > ord_work(m) || (ord_work(q) == ord_work(m) && q < m)) ++rank;
        return snake(rank);
    }
};

// stage A (FWD) or C (!FWD) for degree block N: rows N^2 .. N^2 + 2N of source a
template <int P, int N, bool FWD>
__device__ __forceinline__ void rot_deg_block(const double* F, const double* x_in, double* y_out,
                                              double (&acc)[RotCfg<P>::RB][RotCfg<P>::NACC]) {
    constexpr int w = 2 * N + 1, off = N * (2 * N - 1) * (2 * N + 1) / 3, pos = RotCfg<P>::deg_pos(N);
    constexpr int RB = RotCfg<P>::RB, RS = RotCfg<P>::ROWS * RotCfg<P>::LD;   // row stride of the RB rows
    double x[RB][w];
#pragma unroll
    for (int q = 0; q < RB; ++q)
#pragma unroll
        for (int c = 0; c < w; ++c) x[q][c] = x_in[q * RS + N * N + c];
#pragma unroll
    for (int r = 0; r < w; ++r) {
        double v[RB];
#pragma unroll
        for (int q = 0; q < RB; ++q) v[q] = FWD ? 0.0 : acc[q][pos + r];
#pragma unroll
        for (int c = 0; c < w; ++c) {
            const double f = RotCfg<P>::STAGE ? F[off + r * w + c] : __ldg(F + off + r * w + c);
#pragma unroll
            for (int q = 0; q < RB; ++q) v[q] = fma(f, x[q][c], v[q]);
        }
#pragma unroll
        for (int q = 0; q < RB; ++q) {
            if (FWD) y_out[q * RS + N * N + r] = v[q];
            else acc[q][pos + r] = v[q];
        }
    }
}

// stage B for order block M: z = Z_M y over degrees M..P, re and im parts
template <int P, int M>
__device__ __forceinline__ void rot_ord_block(const double* Z, const double* y_in, double* z_out) {
    constexpr int L = P + 1 - M;
    constexpr int zoff = RotCfg<P>::ZSZ - L * (L + 1) * (2 * L + 1) / 6;
    constexpr int NP = M == 0 ? 1 : 2;                      // parts re, im: same block
    constexpr int RB = RotCfg<P>::RB, RS = RotCfg<P>::ROWS * RotCfg<P>::LD;
    double yv[RB * NP][L];
#pragma unroll
    for (int q = 0; q < RB * NP; ++q)
#pragma unroll
        for (int d = 0; d < L; ++d) {
            const int n = M + d, part = q % NP;
            yv[q][d] = y_in[(q / NP) * RS + (M == 0 ? n * n : n * n + 2 * M - 1 + part)];
        }
#pragma unroll
    for (int jr = 0; jr < L; ++jr) {
        double v[RB * NP];
#pragma unroll
        for (int q = 0; q < RB * NP; ++q) v[q] = 0.0;
#pragma unroll
        for (int d = 0; d < L; ++d) {
            const double f = RotCfg<P>::STAGE ? Z[zoff + jr * L + d] : __ldg(Z + zoff + jr * L + d);
#pragma unroll
            for (int q = 0; q < RB * NP; ++q) v[q] = fma(f, yv[q][d], v[q]);
        }
        const int j = M + jr;
#pragma unroll
        for (int q = 0; q < RB * NP; ++q)
            z_out[(q / NP) * RS + (M == 0 ? j * j : j * j + 2 * M - 1 + q % NP)] = v[q];
    }
}

template <int P, bool FWD, int... Ns>
__device__ __forceinline__ void rot_deg_stage(std::integer_sequence<int, Ns...>, int g, const double* F, const double* x_in,
                                              double* y_out, double (&acc)[RotCfg<P>::RB][RotCfg<P>::NACC]) {
    // largest blocks first, matching deg_pos
    ((RotCfg<P>::deg_group(P - Ns) == g ? rot_deg_block<P, P - Ns, FWD>(F, x_in, y_out, acc) : void()), ...);
}
template <int P, int... Ms>
__device__ __forceinline__ void rot_ord_stage(std::integer_sequence<int, Ms...>, int g, const double* Z, const double* y_in,
                                              double* z_out) {
    ((RotCfg<P>::ord_group(Ms) == g ? rot_ord_block<P, Ms>(Z, y_in, z_out) : void()), ...);
}

// Work items and split sums as in the plain form (ogx_m2l64.cuh): a small tree's tiles are
// cut into ranges of colleague slots so that they fill the SMs.
// Bound: a combination's 64 rows take 2,223 FMAs each at p = 8, 2,200 cycles of the SM's FP64
// pipe; reading every factor and every source row from L2 at the point of use took about ten
// times that.  The next combination's factors and sources now come by cp.async while this one
// runs: its Q once stage A is done with this one's, its Z and its rows (into the buffer that
// stage C does not read) once stage B is, its Q^-1 after stage C.
template <int P>
__global__ void __launch_bounds__(RotCfg<P>::THREADS) k_m2l_rot(TreeView tv, M2L64Args ar, const double* __restrict__ pack,
                                                        const double* __restrict__ mpole, double* lown) {
    using R = RotCfg<P>;
    constexpr int K = R::K, LD = R::LD, RB = R::RB, TH = R::THREADS;
    extern __shared__ __align__(16) double s_rot[];
    double* s_x = s_rot;                    // [64][LD] sources, then z
    double* s_y = s_rot + ROT_TGT * LD;     // [64][LD] y = Q m, then the next sources
    double* s_f = s_rot + 2 * ROT_TGT * LD; // factors (STAGE): Q, Q^-1, Z
    __shared__ int s_Q[27][ROT_TGT];
    __shared__ uint32_t s_mask[7];          // bit 8 D + s: some target of the tile has that source
    __shared__ int s_combo[189];            // present combinations: D | s << 5 | o << 8
    __shared__ int s_tgt[ROT_TGT];
    __shared__ int s_item, s_n;
    const int tid = threadIdx.x, lane = tid & 31;
    const int ga = tid / R::ROWS, ra = tid % R::ROWS;   // block group; rows ra, ra + ROWS, ...
    if (tv_over(tv)) return;
    const int S = ar.gs[GS_SPLIT], tiles = ar.gs[GS_TILES];
    const int ntgt = tv.cnt->ntgt32;
    for (;;) {
        __syncthreads();
        if (tid == 0) s_item = atomicAdd(ar.gs + GS_TICKET, 1);
        if (tid < 7) s_mask[tid] = 0;
        __syncthreads();
        const int item = s_item;
        if (item >= tiles * S) return;
        const int zr = item / tiles, base = (item - zr * tiles) * ROT_TGT;
        const int t = (int)ar.tgt_key[base];
        if (t < 0) continue;
        const int D0 = m2l64_first_slot(zr, S, t), D1 = m2l64_first_slot(zr + 1, S, t);
        if (tid < ROT_TGT) s_tgt[tid] = ((int)ar.tgt_key[base + tid] == t) ? (int)ar.tgt_box[base + tid] : -1;
        __syncthreads();
        const int tx = t & 1, ty = (t >> 1) & 1, tz = (t >> 2) & 1;
        for (int i = tid; i < (D1 - D0) * ROT_TGT; i += TH) {
            const int D = D0 + i / ROT_TGT, r = i % ROT_TGT, b = s_tgt[r];
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
        if (tid < 32) {   // the present combinations in (D, s) order
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
        const int nco = s_n;
        // copies of combination k's factors [f0, f0 + count) and of its source rows (absent: zeros)
        auto factors = [&](int k, int f0, int count) {
            if (!R::STAGE || k >= nco) return;
            const double* src = pack + (size_t)(s_combo[k] >> 8) * R::DPACK + f0;
            for (int i = tid; i < count / 2; i += TH) sm100::cp_async16(s_f + f0 + 2 * i, src + 2 * i);
        };
        auto rows = [&](int k, double* dst) {
            if (k >= nco) return;
            const int code = s_combo[k], lr = tid / (TH / ROT_TGT);   // TH / 64 threads per row
            const int Q = s_Q[code & 31][lr];
            const int b = Q >= 0 ? __ldg(tv.child + 8 * (size_t)Q + ((code >> 5) & 7)) : -1;
            const double* src = mpole + (size_t)max(b, 0) * K;
            for (int kk = tid % (TH / ROT_TGT); kk < K; kk += TH / ROT_TGT)
                sm100::cp_async8_zfill(dst + lr * LD + kk, src + kk, b >= 0 ? 8u : 0u);
        };
        double acc[RB][R::NACC];
#pragma unroll
        for (int q = 0; q < RB; ++q)
#pragma unroll
            for (int i = 0; i < R::NACC; ++i) acc[q][i] = 0.0;
        using Seq = std::make_integer_sequence<int, P + 1>;
        double *x = s_x, *y = s_y;
        factors(0, 0, R::QS);
        factors(0, 2 * R::QS, R::ZS);
        rows(0, x);
        sm100::cp_async_commit();
        sm100::cp_async_wait<0>();
        __syncthreads();
        factors(0, R::QS, R::QS);
        sm100::cp_async_commit();
        for (int k = 0; k < nco; ++k) {
            const double* pk = R::STAGE ? s_f : pack + (size_t)(s_combo[k] >> 8) * R::DPACK;
            rot_deg_stage<P, true>(Seq{}, ga, pk, x + ra * LD, y + ra * LD, acc);              // y = Q m
            __syncthreads();
            factors(k + 1, 0, R::QS);
            sm100::cp_async_commit();
            rot_ord_stage<P>(Seq{}, ga, pk + 2 * R::QS, y + ra * LD, x + ra * LD);            // z = Z y
            sm100::cp_async_wait<1>();                                                       // this combination's Q^-1
            __syncthreads();
            factors(k + 1, 2 * R::QS, R::ZS);
            rows(k + 1, y);
            sm100::cp_async_commit();
            rot_deg_stage<P, false>(Seq{}, ga, pk + R::QS, x + ra * LD, nullptr, acc);         // acc += Q^-1 z
            sm100::cp_async_wait<0>();
            __syncthreads();
            factors(k + 1, R::QS, R::QS);
            sm100::cp_async_commit();
            double* w = x;
            x = y;
            y = w;
        }
        sm100::cp_async_wait_all();
#pragma unroll
        for (int q = 0; q < RB; ++q) {
            const int r0 = ra + q * R::ROWS, b = s_tgt[r0];
            if (b < 0) continue;
            const int pq = base + r0 - ar.gs[9 + t];
            const int64_t j = ar.gs[t] + (int64_t)(pq / 128) * ar.gs[GS_FILL] + pq % 128;   // sorted target
            double* o = S == 1 ? lown + (size_t)b * K : ar.part + ((size_t)zr * ntgt + j) * K;
            const double sc = S == 1 ? 1.0 / (2.0 * tv.center[4 * b + 3]) : 1.0;
#pragma unroll
            for (int n = 0; n <= P; ++n) {
                if (R::deg_group(n) != ga) continue;
                const int pos = R::deg_pos(n);
#pragma unroll
                for (int r = 0; r < 2 * n + 1; ++r) o[n * n + r] = acc[q][pos + r] * sc;
            }
        }
    }
}

// the 343 rotation packs of order P, built once per order in this process
template <int P>
std::shared_ptr<const std::vector<double>> rot_packs() {
    static std::mutex mu;
    static std::shared_ptr<const std::vector<double>> cached;
    std::lock_guard<std::mutex> lk(mu);
    if (cached) return cached;
    using R = RotCfg<P>;
    auto v = std::make_shared<std::vector<double>>((size_t)343 * R::DPACK, 0.0);
    std::vector<double> pk(R::PACK);
    for (int o = 0; o < 343; ++o) {
        std::fill(pk.begin(), pk.end(), 0.0);
        build_rot_pack(P, o, pk.data());
        double* d = v->data() + (size_t)o * R::DPACK;
        std::copy(pk.begin(), pk.begin() + R::QSZ, d);
        std::copy(pk.begin() + R::QSZ, pk.begin() + 2 * R::QSZ, d + R::QS);
        std::copy(pk.begin() + 2 * R::QSZ, pk.end(), d + 2 * R::QS);
    }
    cached = v;
    return cached;
}

template <int P>
int ensure_rot_tables(Handle& h) {
    if (h.rot_ready_p == P) return OGX_OK;
    static_assert(RotCfg<P>::PACK > 0, "pack");
    const auto pk = rot_packs<P>();
    double* d;
    OGX_TRY(arena_get(h.ws, S_ROT_PACK, pk->size(), &d));
    OGX_CUDA(upload_now(d, pk->data(), pk->size() * sizeof(double)));
    h.d_rot = d;
    h.rot_ready_p = P;
    return OGX_OK;
}

template <int P>
int launch_rot(Handle& h, const double* M, double* Lown) {
    OGX_TRY(ensure_rot_tables<P>(h));
    constexpr size_t rsm = RotCfg<P>::SMEM;
    OGX_CUDA(smem_optin((const void*)k_m2l_rot<P>, (int)rsm));
    M2L64Args a;
    OGX_TRY(m2l64_args(h, 0, &a));
    static const int per_sm = [] {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_m2l_rot<P>, RotCfg<P>::THREADS, rsm) != cudaSuccess) {
            cudaGetLastError();
            b = 1;
        }
        return std::max(1, b);
    }();
    const int grid = (int)std::min<int64_t>((int64_t)(h.ntgt_pad / ROT_TGT) * M2L64_MAXSPLIT, (int64_t)per_sm * h.num_sms);
    k_m2l_rot<P><<<grid, RotCfg<P>::THREADS, rsm, h.stream>>>(h.tv, a, h.d_rot, M, Lown);
    ++h.launches;
    return m2l64_sum_launch(h, a, 0, Lown, h.stream);
}

}  // namespace

int m2l_rot_launch(Handle& h, const double* M, double* Lown) {
    switch (h.prm.p) {
        case 1: return launch_rot<1>(h, M, Lown);
        case 2: return launch_rot<2>(h, M, Lown);
        case 3: return launch_rot<3>(h, M, Lown);
        case 4: return launch_rot<4>(h, M, Lown);
        case 5: return launch_rot<5>(h, M, Lown);
        case 6: return launch_rot<6>(h, M, Lown);
        case 7: return launch_rot<7>(h, M, Lown);
        case 8: return launch_rot<8>(h, M, Lown);
        case 9: return launch_rot<9>(h, M, Lown);
        case 10: return launch_rot<10>(h, M, Lown);
        case 11: return launch_rot<11>(h, M, Lown);
        case 12: return launch_rot<12>(h, M, Lown);
        default: return OGX_ERR_INVALID;
    }
}

}  // namespace ogx
