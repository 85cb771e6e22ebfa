// ogx_fmm64.cu -- the passes of an adaptive FMM evaluation, in the plain FP64 form (run_fp64, also
// the third form) and in the mixed form (run_mixed*).
//
// Same passes as AdaptiveFMM3D::computeAccelerations (src3d/AdaptiveFMM3D.hpp:29-110)
// but organised for the GPU:
//   P2M           one-warp block per leaf: a lane takes bodies, adds their terms of one
//                 coefficient at a time to its column of sums (:53-61, ogx_p2x.cuh)
//   M2M           bottom-up in one launch (items of 16 parents taken by ticket, each waiting
//                 for its children) on the FP64 matrix instructions (:62-71, ogx_translate.cu)
//   M2L           all levels in one launch: FP64 matrix instructions (ogx_m2l64.cu), rotations
//                 (ogx_m2l_rot.cu) or the tensor cores (ogx_mixed_kernels.cuh); :78-81, the V
//                 list implicit in the colleague slots
//   P2L           one-warp block per box over its X list (:82, :117-128, ogx_p2x.cuh)
//   L2L           top-down in one launch, the same way as M2M (:75-77)
//   leaf far      L2P and, over the W lists, M2P from coefficient records, a warp per leaf or a
//                 CTA per heavy leaf (:92-93, ogx_far.cuh)
//   leaf near     softened P2P over the U list, j != i, a one-warp block per chunk of at most 32
//                 targets of a leaf (:95-103, ogx_near.cuh)
//   combine       acc[orig] = G (far + near) (:104)
// Potentials (pot = -G Phi) are produced alongside when requested.
#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

#include "ogx_harmonics.cuh"
#include "ogx_p2x.cuh"
#include "ogx_far.cuh"
#include "ogx_near.cuh"
#include "ogx_mixed_kernels.cuh"
#include "ogx_m2l64.cuh"

namespace ogx {

namespace {

// ---- leaf far field (ogx_far.cuh): coefficient records, then M2P over the W lists and L2P.
// The mixed form's M2P part (L2P = false) needs only the multipoles, so it runs on the side
// stream beside the M2L and the downward pass; the plain form takes both parts in one.
template <int P, bool POT, bool L2P, class T>
int launch_m2p(Handle& h, const double* M, const T* grec, double* out, cudaStream_t st) {
    using R = far::Rec<T, P + 1, POT>;
    TreeView& tv = h.tv;
    T* hrec;
    OGX_TRY(arena_get(h.ws, S_EVAL_H, (size_t)tv.nb * R::SIZE, &hrec));
    far::k_far_rec<P, 0, POT, T><<<(tv.nb + 3) / 4, 128, 0, st>>>(tv, tv.nb, M, hrec); ++h.launches;
    int* heavy;
    OGX_TRY(arena_get(h.ws, S_FAR_HEAVY, (size_t)tv.nleaf + 2, &heavy));
    int* ctr = heavy + tv.nleaf;
    OGX_CUDA(cudaMemsetAsync(ctr, 0, 2 * sizeof(int), st));
    far::k_far_heavy_list<T><<<(tv.nleaf + 255) / 256, 256, 0, st>>>(tv, heavy, ctr); ++h.launches;
    constexpr size_t hsmem = far::leaf_far_heavy_smem<P, POT, T>(), smem = far::leaf_far_smem<P, POT, true, T>();
    auto heavyk = far::k_leaf_far_heavy<P, POT, L2P, T>;
    auto lightk = far::k_leaf_far<P, POT, L2P, true, T>;
    OGX_CUDA(smem_optin((const void*)heavyk, (int)hsmem));
    OGX_CUDA(smem_optin((const void*)lightk, (int)smem));
    // two CTAs per SM: a third finishes the 1M merger no sooner (4.03 ms either way) and takes
    // the shared memory that another system's M2L tiles need (three 262,144-body galaxies at
    // p = 4 in turn: 1.51 -> 1.79 ms each)
    heavyk<<<2 * h.num_sms, 32 * far::FAR_HW, hsmem, st>>>(tv, hrec, grec, out, heavy, ctr); ++h.launches;
    lightk<<<tv.nleaf, 32, smem, st>>>(tv, hrec, grec, out); ++h.launches;
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

template <int P, bool POT, class T>
int launch_local_rec(Handle& h, const double* L, T** grec) {
    using R = far::Rec<T, far::rec_degree<P, 1, POT>(), POT>;
    OGX_TRY(arena_get(h.ws, S_EVAL_G, (size_t)h.tv.nleaf * R::SIZE, grec));
    far::k_far_rec<P, 1, POT, T><<<(h.tv.nleaf + 3) / 4, 128, 0, h.stream>>>(h.tv, h.tv.nleaf, L, *grec); ++h.launches;
    return OGX_OK;
}

// plain form: L2P + M2P in FP64, on h.stream
template <int P, bool POT>
int launch_far64(Handle& h, const double* M, const double* L, double* out) {
    double* grec;
    OGX_TRY((launch_local_rec<P, POT, double>(h, L, &grec)));
    return launch_m2p<P, POT, true, double>(h, M, grec, out, h.stream);
}

// mixed form: the L2P, after the downward pass
template <int P, bool POT>
int launch_l2p32(Handle& h, const double* L, double* out) {
    float* grec;
    OGX_TRY((launch_local_rec<P, POT, float>(h, L, &grec)));
    constexpr size_t smem = far::leaf_far_smem<P, POT, false, float>();
    far::k_leaf_far<P, POT, true, false, float><<<h.tv.nleaf, 32, smem, h.stream>>>(h.tv, nullptr, grec, out); ++h.launches;
    return OGX_OK;
}

// ---- work items of the near field (ogx_near.cuh) ----------------------------------------
// the leaf and first target of near-field work item w (leaf, chunk of 32 targets):
// chunk_off[lf] <= w < chunk_off[lf + 1]; false past the last item
__device__ __forceinline__ bool near_item(const TreeView& tv, const int64_t* chunk_off, int64_t w, int& lf, int& j0) {
    if (w >= chunk_off[tv.nleaf]) return false;
    int lo = 0, hi = tv.nleaf;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (chunk_off[mid] <= w) lo = mid;
        else hi = mid;
    }
    lf = lo;
    j0 = 32 * (int)(w - chunk_off[lo]);
    return true;
}

// ---- OGX_SOFT_SPLINE: the far field's pairs within the support ------------------------
// For each leaf b and each leaf c of its S list (not adjacent to b, within the support hs),
// out[4 i] += sum_j m_j (g(r) - r^-3) (r_j - r_i) and, for potentials, m_j (k(r) - 1/r),
// over the pairs closer than hs (the difference is zero beyond).  The far field took these
// pairs with the Newtonian kernel; with this sum they carry the spline kernel's force.
// Warp per near-field work item (a leaf's chunk of 32 targets), a lane per target, FP64 (the
// plain form; the mixed form runs the FP32 near-field kernel over the same lists,
// k_leaf_near<Near32, .., 2>).
template <bool POT>
__global__ void __launch_bounds__(128) k_soft_correct(TreeView tv, const int64_t* __restrict__ chunk_off, double hs, double hinv,
                                                      double* out) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int lf, j0;
    if (tv_over(tv) || !near_item(tv, chunk_off, blockIdx.x * 4 + wid, lf, j0)) return;
    const int64_t e0 = tv.s_off[lf], e1 = tv.s_off[lf + 1];
    if (e0 == e1) return;
    const int b = tv.leafbox[lf];
    const int f0 = tv.pfirst[b], cnt = tv.pcount[b];
    const double hs2 = hs * hs;
    {
        const int jj = j0 + lane;
        const bool act = jj < cnt;
        const int i = f0 + (act ? jj : 0);
        const double x = tv.px[i], y = tv.py[i], z = tv.pz[i];
        double ax = 0, ay = 0, az = 0, ph = 0;
        for (int64_t e = e0; e < e1; ++e) {
            const int c = tv.s_idx[e];
            const int s0 = tv.pfirst[c], sc = tv.pcount[c];
            for (int j = s0; j < s0 + sc; ++j) {
                const double dx = __ldg(tv.px + j) - x, dy = __ldg(tv.py + j) - y, dz = __ldg(tv.pz + j) - z;
                const double r2 = dx * dx + dy * dy + dz * dz;
                if (r2 < hs2 && r2 > 0.0) {
                    double g, k;
                    spline_gk<double>(r2, hs, hinv, g, k);
                    const double ir = rsqrt(r2);
                    const double mj = __ldg(tv.pm + j);
                    const double w = mj * (g - ir * ir * ir);
                    ax = fma(w, dx, ax); ay = fma(w, dy, ay); az = fma(w, dz, az);
                    if (POT) ph = fma(mj, k - ir, ph);
                }
            }
        }
        if (act) {
            out[4 * (size_t)i] += ax;
            out[4 * (size_t)i + 1] += ay;
            out[4 * (size_t)i + 2] += az;
            if (POT) out[4 * (size_t)i + 3] += ph;
        }
    }
}

}  // namespace

// work items of the near field (leaf, chunk of 32 targets), on h.stream; the grid of a
// warp-per-item kernel needs at most nleaf + n / 32 warps
int near_items(Handle& h, int64_t** chunk_off) {
    TreeView& tv = h.tv;
    int* nchunk;
    OGX_TRY(arena_get(h.ws, S_NEAR_CHUNK, (size_t)tv.nleaf, &nchunk));
    OGX_TRY(arena_get(h.ws, S_NEAR_CHUNK_OFF, (size_t)tv.nleaf + 1, chunk_off));
    return scan_i32_to_i64(h, nchunk, *chunk_off, tv.nleaf);
}

int soft_correct_launch(Handle& h, const int64_t* chunk_off, double* out, bool pot, cudaStream_t st) {
    const TreeView& tv = h.tv;
    if (h.soft_pairs == 0 || tv.nleaf == 0) return OGX_OK;
    const double hs = spline_support(h.prm.eps), hinv = 1.0 / hs;
    const int grid = (tv.nleaf + (tv.n + 31) / 32 + 3) / 4;
    if (pot) k_soft_correct<true><<<grid, 128, 0, st>>>(tv, chunk_off, hs, hinv, out);
    else k_soft_correct<false><<<grid, 128, 0, st>>>(tv, chunk_off, hs, hinv, out);
    ++h.launches;
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

namespace {

// ---- dispatch --------------------------------------------------------------------------
template <int P>
int run_fp64(Handle& h, double* d_acc, double* d_pot) {
    constexpr int K = (P + 1) * (P + 1);
    const cudaStream_t st = h.stream;
    TreeView& tv = h.tv;
    OGX_TRY(harm_tables_ready(h.device));
    double *M, *L, *Lown, *far;
    OGX_TRY(arena_get(h.ws, S_MPOLE, (size_t)tv.nb * K, &M));
    OGX_TRY(arena_get(h.ws, S_LOCAL, (size_t)tv.nb * K, &L));
    OGX_TRY(arena_get(h.ws, S_LOWN, (size_t)tv.nb * K, &Lown));
    OGX_TRY(arena_get(h.ws, S_FAR, 4 * (size_t)tv.n, &far));
    OGX_CUDA(timing_record(h, h.ev[2], st));
    // upward
    p2x::k_p2x<P, 0, double><<<tv.nleaf, 32, p2x::p2x_smem<P, double>(), st>>>(tv, tv.nleaf, M); ++h.launches;
    OGX_TRY(m2m_launch(h, M));
    OGX_CUDA(timing_record(h, h.ev[3], st));
    // M2L
    OGX_CUDA(cudaMemsetAsync(Lown, 0, sizeof(double) * (size_t)tv.nb * K, st));
    if (h.ntgt > 0 && h.prm.precision == OGX_PREC_FP64_ROT) {
        // third form: the same V pairs through the rotation-factored operators (ogx_m2l_rot.cu)
        OGX_TRY(m2l_rot_launch(h, M, Lown));
    } else if (h.ntgt > 0) {
        OGX_TRY(m2l_fp64_launch(h, M, Lown));   // ogx_m2l64.cu
    }
    OGX_CUDA(timing_record(h, h.ev[4], st));
    // P2L
    p2x::k_p2x<P, 1, double><<<tv.nb, 32, p2x::p2x_smem<P, double>(), st>>>(tv, tv.nb, Lown); ++h.launches;
    OGX_CUDA(timing_record(h, h.ev[5], st));
    // L2L top-down
    OGX_TRY(l2l_launch(h, L, Lown));
    OGX_CUDA(timing_record(h, h.ev[6], st));
    // leaves
    const bool pot = d_pot != nullptr;
    if (pot) OGX_TRY((launch_far64<P, true>(h, M, L, far)));
    else OGX_TRY((launch_far64<P, false>(h, M, L, far)));
    const double G = h.prm.G, eps2 = h.prm.eps * h.prm.eps;
    int64_t* chunk_off;
    OGX_TRY(near_items(h, &chunk_off));
    double* nearb;
    OGX_TRY(arena_get(h.ws, S_NEAR32, 4 * (size_t)tv.n, &nearb));
    const bool soft = h.prm.softening == OGX_SOFT_SPLINE;
    // the far field's pairs within the support, then the spline kernel in the near field
    if (soft) OGX_TRY(soft_correct_launch(h, chunk_off, far, pot, st));
    using near_field::Near64;
    const double hs = soft ? spline_support(h.prm.eps) : 0.0;
    const near_field::NearPrm<double> npr{eps2, hs, hs > 0.0 ? 1.0 / hs : 0.0};
    const Near64::Bodies bod{tv.px, tv.py, tv.pz, tv.pm};
    auto near = pot ? (soft ? near_field::k_leaf_near<Near64, true, 64, 1> : near_field::k_leaf_near<Near64, true, 64>)
                    : (soft ? near_field::k_leaf_near<Near64, false, 64, 1> : near_field::k_leaf_near<Near64, false, 64>);
    near<<<tv.nleaf + (tv.n + 31) / 32, 32, 0, st>>>(tv, chunk_off, bod, npr, nearb); ++h.launches;
    auto combine = pot ? mixed::k_combine<true> : mixed::k_combine<false>;
    combine<<<(tv.n + 255) / 256, 256, 0, st>>>(tv.n, tv.perm, G, far, nullptr, nearb, d_acc, d_pot, tv.cnt); ++h.launches;
    OGX_CUDA(timing_record(h, h.ev[7], st));
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

// ---- mixed form ---------------------------------------------------------------------

// Operator images for the tensor-core M2L, per offset o, column slice z, K-chunk c
// and part (hi, lo): rows = the slice's output dofs (all of 1..K-1 when there is one
// slice), K-major in the 128-byte-swizzle layout, exactly the bytes one pipeline
// stage holds, so one bulk copy moves a chunk.
// Also row 0 of every T_o (for the degree-0 local coefficient of potentials).
struct MixedImages {
    std::vector<uint8_t> img;
    std::vector<double> row0;
    std::vector<float> ounscale;
};

// built once per order in this process and shared by every handle
template <int P>
std::shared_ptr<const MixedImages> mixed_images() {
    using C = mixed::TcCfg<P>;
    static std::mutex mu;
    static std::shared_ptr<const MixedImages> cached;
    std::lock_guard<std::mutex> lk(mu);
    if (cached) return cached;
    const int K = C::K;
    std::vector<double> T((size_t)K * K);
    auto mi = std::make_shared<MixedImages>();
    std::vector<uint8_t>& img = mi->img;
    std::vector<double>& row0 = mi->row0;
    std::vector<float>& ounscale = mi->ounscale;
    img.assign((size_t)343 * C::NSPLIT * C::NCH * 2 * C::B_BYTES, 0);
    row0.assign((size_t)343 * K, 0.0);
    ounscale.assign(343, 0.f);
    for (int o = 0; o < 343; ++o) {
        const int ox = o % 7 - 3, oy = (o / 7) % 7 - 3, oz = o / 49 - 3;
        if (std::max(std::abs(ox), std::max(std::abs(oy), std::abs(oz))) <= 1) continue;
        build_operator(2, P, o, T.data());
        for (int k = 0; k < K; ++k) row0[(size_t)o * K + k] = T[k];
        // FP16 images of T_o * 2^-e, largest used entry in [0.5, 1); 2^e undoes it
        double mx = 0.0;
        for (int jr = 0; jr < C::NFULL; ++jr)
            for (int k = 0; k < K; ++k) mx = std::max(mx, std::fabs(T[(size_t)(jr + 1) * K + k]));
        int e = 0;
        if (mx > 0.0) std::frexp(mx, &e);
        const double scale = std::ldexp(1.0, -e);
        ounscale[o] = std::ldexp(1.0f, e);
        // slice z, row jr holds output dof 1 + z N + jr
        for (int z = 0; z < C::NSPLIT; ++z)
        for (int c = 0; c < C::NCH; ++c) {
            uint8_t* hi = img.data() + ((size_t)((o * C::NSPLIT + z) * C::NCH + c) * 2) * C::B_BYTES;
            uint8_t* lo = hi + C::B_BYTES;
            for (int jr = 0; jr < C::N; ++jr)
                for (int kk = 0; kk < C::CH * 16; ++kk) {
                    const int k = c * C::CH * 16 + kk, dof = 1 + z * C::N + jr;
                    if (k >= K || dof >= K) continue;
                    const double x = T[(size_t)dof * K + k] * scale;
                    const __half vh = __double2half(x);
                    const __half vl = __double2half(x - (double)__half2float(vh));
                    const int off = mixed::tile_off(jr, kk);
                    std::memcpy(hi + off, &vh, 2);
                    std::memcpy(lo + off, &vl, 2);
                }
        }
    }
    cached = mi;
    return cached;
}

template <int P>
int ensure_mixed_tables(Handle& h) {
    if (h.mix_ready_p == P) return OGX_OK;
    const auto mi = mixed_images<P>();
    const std::vector<uint8_t>& img = mi->img;
    const std::vector<double>& row0 = mi->row0;
    const std::vector<float>& ounscale = mi->ounscale;
    uint8_t* d_img;
    double* d_row0;
    float* d_ous;
    OGX_TRY(arena_get(h.ws, S_MIX_TOPS, img.size(), &d_img));
    OGX_TRY(arena_get(h.ws, S_MIX_ROW0, row0.size(), &d_row0));
    OGX_TRY(arena_get(h.ws, S_MIX_OUNSCALE, ounscale.size(), &d_ous));
    OGX_CUDA(upload_now(d_img, img.data(), img.size()));
    OGX_CUDA(upload_now(d_row0, row0.data(), row0.size() * sizeof(double)));
    OGX_CUDA(upload_now(d_ous, ounscale.data(), ounscale.size() * sizeof(float)));
    h.d_tc_img = d_img;
    h.d_tc_row0 = d_row0;
    h.d_tc_ounscale = d_ous;
    h.mix_ready_p = P;
    return OGX_OK;
}

// Mixed-form upward pass (P2M, M2M, FP16 hi/lo split of the multipoles) on h.up, forked
// from the main stream right after the tree build; the main stream joins it
// (h.ev_up) before the M2L.
template <int P>
int run_mixed_upward(Handle& h) {
    using C = mixed::TcCfg<P>;
    constexpr int K = (P + 1) * (P + 1);
    TreeView& tv = h.tv;
    OGX_TRY(harm_tables_ready(h.device));
    if constexpr (C::SUPPORTED) OGX_TRY(ensure_mixed_tables<P>(h));
    double* M;
    __half *mhi, *mlo;
    float* mus;
    OGX_TRY(arena_get(h.ws, S_MPOLE, (size_t)tv.nb * K, &M));
    OGX_TRY(arena_get(h.ws, S_MIX_MHI, (size_t)tv.nb * C::KPAD, &mhi));
    OGX_TRY(arena_get(h.ws, S_MIX_MLO, (size_t)tv.nb * C::KPAD, &mlo));
    OGX_TRY(arena_get(h.ws, S_MIX_MUNSCALE, (size_t)tv.nb, &mus));
    OGX_CUDA(cudaEventRecord(h.ev_tree, h.stream));
    const cudaStream_t main_st = h.stream, su = h.up;
    OGX_CUDA(cudaStreamWaitEvent(su, h.ev_tree, 0));
    h.stream = su;   // m2m_launch issues on h.stream
    OGX_CUDA(timing_record(h, h.ev[2], su));
    p2x::k_p2x<P, 0, float><<<tv.nleaf, 32, p2x::p2x_smem<P, float>(), su>>>(tv, tv.nleaf, M); ++h.launches;
    const int rc = m2m_launch(h, M);
    h.stream = main_st;
    OGX_TRY(rc);
    if constexpr (C::SUPPORTED) {
        mixed::k_split_mpole<P><<<(tv.nb + 3) / 4, 128, 0, su>>>(M, tv.nb, mhi, mlo, mus, tv.cnt); ++h.launches;
    }
    OGX_CUDA(timing_record(h, h.ev_up_end, su));
    OGX_CUDA(cudaEventRecord(h.ev_up, su));
    return OGX_OK;
}

// Mixed-form M2L on the tensor cores, on h.m2l: it waits for the FP16 split of the
// multipoles (h.ev_up) and the target tiles (h.ev_tgt) and runs beside the U/W/X list
// build; run_mixed joins it (h.ev_m2l) before the P2L, which adds into the same locals.
template <int P>
int run_mixed_m2l(Handle& h, bool pot) {
    using C = mixed::TcCfg<P>;
    constexpr int K = (P + 1) * (P + 1);
    const cudaStream_t sm = h.m2l;
    TreeView& tv = h.tv;
    double *M, *Lown;
    __half *mhi, *mlo;
    float* mus;
    OGX_TRY(arena_get(h.ws, S_MPOLE, (size_t)tv.nb * K, &M));
    OGX_TRY(arena_get(h.ws, S_LOWN, (size_t)tv.nb * K, &Lown));
    OGX_TRY(arena_get(h.ws, S_MIX_MHI, (size_t)tv.nb * C::KPAD, &mhi));
    OGX_TRY(arena_get(h.ws, S_MIX_MLO, (size_t)tv.nb * C::KPAD, &mlo));
    OGX_TRY(arena_get(h.ws, S_MIX_MUNSCALE, (size_t)tv.nb, &mus));
    OGX_CUDA(cudaStreamWaitEvent(sm, h.ev_up, 0));
    OGX_CUDA(cudaStreamWaitEvent(sm, h.ev_tgt, 0));
    OGX_CUDA(timing_record(h, h.ev[3], sm));
    OGX_CUDA(cudaMemsetAsync(Lown, 0, sizeof(double) * (size_t)tv.nb * K, sm));
    if (h.ntgt > 0) {
        static_assert(C::SUPPORTED, "every order's operand fits TMEM, in slices if need be");
        OGX_CUDA(smem_optin((const void*)mixed::k_m2l_tc<P>, C::SMEM));
        M2L64Args a;
        OGX_TRY(m2l64_args(h, C::NSPLIT, &a));
        const int tiles = h.ntgt_pad / 128;
        // ranges of slots per tile, one CTA each (the kernel's own count is exact; this one
        // comes from a bound and may differ)
        const int ranges = m2l_tc_split((h.ntgt + 127) / 128, C::NSPLIT);
        mixed::k_m2l_tc<P><<<dim3(tiles, C::NSPLIT, ranges), C::THREADS, C::SMEM, sm>>>(tv, a, mhi, mlo, mus, h.d_tc_img,
                                                                                       h.d_tc_ounscale, Lown, h.d_err); ++h.launches;
        OGX_TRY(m2l64_sum_launch(h, a, C::NSPLIT, Lown, sm));
        if (pot) {
            mixed::k_m2l_dof0<P><<<(h.ntgt + 3) / 4, 128, 0, sm>>>(tv, h.ntgt, h.tgt_box, h.d_tc_row0, M, Lown); ++h.launches;
        }
    }
    OGX_CUDA(timing_record(h, h.ev[4], sm));
    OGX_CUDA(cudaEventRecord(h.ev_m2l, sm));
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

template <int P>
int run_mixed(Handle& h, double* d_acc, double* d_pot) {
    constexpr int K = (P + 1) * (P + 1);
    const cudaStream_t st = h.stream;
    TreeView& tv = h.tv;
    double *M, *L, *Lown, *far;
    OGX_TRY(arena_get(h.ws, S_MPOLE, (size_t)tv.nb * K, &M));
    OGX_TRY(arena_get(h.ws, S_LOCAL, (size_t)tv.nb * K, &L));
    OGX_TRY(arena_get(h.ws, S_LOWN, (size_t)tv.nb * K, &Lown));
    OGX_TRY(arena_get(h.ws, S_FAR, 4 * (size_t)tv.n, &far));
    double *nearb, *far_m;
    OGX_TRY(arena_get(h.ws, S_NEAR32, 4 * (size_t)tv.n, &nearb));
    OGX_TRY(arena_get(h.ws, S_FAR_M, 4 * (size_t)tv.n, &far_m));
    // near-field work items (leaf, chunk of 32 targets)
    int64_t* chunk_off;
    OGX_TRY(near_items(h, &chunk_off));
    // join the upward pass (the side stream's M2P reads the multipoles)
    OGX_CUDA(cudaStreamWaitEvent(st, h.ev_up, 0));
    // the far field's M2P part and the near field need the tree, the multipoles and the
    // lists: they start here, beside the M2L (launched on h.m2l before the U/W/X lists)
    OGX_CUDA(cudaEventRecord(h.ev_fork, st));
    // near field on the low-priority side stream, issued after the M2L (which takes
    // whole SMs first): its one-warp blocks fill what the M2L's tiles leave free, the
    // SMs its last wave leaves idle, and then what P2L, L2L and the far field leave idle
    {
        const float eps2 = (float)(h.prm.eps * h.prm.eps);
        OGX_CUDA(cudaStreamWaitEvent(h.side, h.ev_fork, 0));
        // the far field's M2P part (multipoles only) first, then the near field
        if (d_pot) OGX_TRY((launch_m2p<P, true, false, float>(h, M, nullptr, far_m, h.side)));
        else OGX_TRY((launch_m2p<P, false, false, float>(h, M, nullptr, far_m, h.side)));
        // one block per work item: the leaves' chunks number at most nleaf + n / 32 (a
        // bounded grid left the far chain waiting)
        const int ngrid = tv.nleaf + (tv.n + 31) / 32;
        // spline kernel in the near field; the far field's pairs within the support are
        // corrected in FP32 into the M2P part (written above on this stream)
        const bool soft = h.prm.softening == OGX_SOFT_SPLINE, p = d_pot != nullptr, u32 = h.near_units == 32;
        const double hs = soft ? spline_support(h.prm.eps) : 0.0;
        using near_field::Near32;
        const near_field::NearPrm<float> npr{eps2, (float)hs, hs > 0.0 ? (float)(1.0 / hs) : 0.f};
        const Near32::Bodies bod{tv.rhi, tv.rlo};
        auto pick = [&](auto km) {
            constexpr int KM = decltype(km)::value;
            return p ? (u32 ? near_field::k_leaf_near<Near32, true, 32, KM> : near_field::k_leaf_near<Near32, true, 64, KM>)
                     : (u32 ? near_field::k_leaf_near<Near32, false, 32, KM> : near_field::k_leaf_near<Near32, false, 64, KM>);
        };
        auto near = soft ? pick(std::integral_constant<int, 1>{}) : pick(std::integral_constant<int, 0>{});
        near<<<ngrid, 32, 0, h.side>>>(tv, chunk_off, bod, npr, nearb); ++h.launches;
        if (soft && h.soft_pairs > 0) {
            // the same staging over the S lists, the kernel difference added into far_m
            pick(std::integral_constant<int, 2>{})<<<ngrid, 32, 0, h.side>>>(tv, chunk_off, bod, npr, far_m); ++h.launches;
        }
        OGX_CUDA(cudaEventRecord(h.ev_join, h.side));
    }
    // join the M2L (its end is timing event 4, recorded on h.m2l)
    OGX_CUDA(cudaStreamWaitEvent(st, h.ev_m2l, 0));
    p2x::k_p2x<P, 1, float><<<tv.nb, 32, p2x::p2x_smem<P, float>(), st>>>(tv, tv.nb, Lown); ++h.launches;
    OGX_CUDA(timing_record(h, h.ev[5], st));
    OGX_TRY(l2l_launch(h, L, Lown));
    OGX_CUDA(timing_record(h, h.ev[6], st));
    const bool pot = d_pot != nullptr;
    if (pot) OGX_TRY((launch_l2p32<P, true>(h, L, far)));
    else OGX_TRY((launch_l2p32<P, false>(h, L, far)));
    // join the side stream (M2P, near field), then acc = G (far + near) in the caller's order
    OGX_CUDA(cudaStreamWaitEvent(st, h.ev_join, 0));
    const double G = h.prm.G;
    if (pot) { mixed::k_combine<true><<<(tv.n + 255) / 256, 256, 0, st>>>(tv.n, tv.perm, G, far, far_m, nearb, d_acc, d_pot, tv.cnt); ++h.launches; }
    else { mixed::k_combine<false><<<(tv.n + 255) / 256, 256, 0, st>>>(tv.n, tv.perm, G, far, far_m, nearb, d_acc, nullptr, tv.cnt); ++h.launches; }
    OGX_CUDA(timing_record(h, h.ev[7], st));
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

}  // namespace

int fmm_mixed_upward(Handle& h) {
    switch (h.prm.p) {
        case 1: return run_mixed_upward<1>(h);
        case 2: return run_mixed_upward<2>(h);
        case 3: return run_mixed_upward<3>(h);
        case 4: return run_mixed_upward<4>(h);
        case 5: return run_mixed_upward<5>(h);
        case 6: return run_mixed_upward<6>(h);
        case 7: return run_mixed_upward<7>(h);
        case 8: return run_mixed_upward<8>(h);
        case 9: return run_mixed_upward<9>(h);
        case 10: return run_mixed_upward<10>(h);
        case 11: return run_mixed_upward<11>(h);
        case 12: return run_mixed_upward<12>(h);
        default: return OGX_ERR_INVALID;
    }
}

int fmm_mixed_m2l(Handle& h, bool pot) {
    switch (h.prm.p) {
        case 1: return run_mixed_m2l<1>(h, pot);
        case 2: return run_mixed_m2l<2>(h, pot);
        case 3: return run_mixed_m2l<3>(h, pot);
        case 4: return run_mixed_m2l<4>(h, pot);
        case 5: return run_mixed_m2l<5>(h, pot);
        case 6: return run_mixed_m2l<6>(h, pot);
        case 7: return run_mixed_m2l<7>(h, pot);
        case 8: return run_mixed_m2l<8>(h, pot);
        case 9: return run_mixed_m2l<9>(h, pot);
        case 10: return run_mixed_m2l<10>(h, pot);
        case 11: return run_mixed_m2l<11>(h, pot);
        case 12: return run_mixed_m2l<12>(h, pot);
        default: return OGX_ERR_INVALID;
    }
}

int fmm_mixed(Handle& h, double* d_acc, double* d_pot) {
    switch (h.prm.p) {
        case 1: return run_mixed<1>(h, d_acc, d_pot);
        case 2: return run_mixed<2>(h, d_acc, d_pot);
        case 3: return run_mixed<3>(h, d_acc, d_pot);
        case 4: return run_mixed<4>(h, d_acc, d_pot);
        case 5: return run_mixed<5>(h, d_acc, d_pot);
        case 6: return run_mixed<6>(h, d_acc, d_pot);
        case 7: return run_mixed<7>(h, d_acc, d_pot);
        case 8: return run_mixed<8>(h, d_acc, d_pot);
        case 9: return run_mixed<9>(h, d_acc, d_pot);
        case 10: return run_mixed<10>(h, d_acc, d_pot);
        case 11: return run_mixed<11>(h, d_acc, d_pot);
        case 12: return run_mixed<12>(h, d_acc, d_pot);
        default: return OGX_ERR_INVALID;
    }
}

int fmm_fp64(Handle& h, double* d_acc, double* d_pot) {
    switch (h.prm.p) {
        case 1: return run_fp64<1>(h, d_acc, d_pot);
        case 2: return run_fp64<2>(h, d_acc, d_pot);
        case 3: return run_fp64<3>(h, d_acc, d_pot);
        case 4: return run_fp64<4>(h, d_acc, d_pot);
        case 5: return run_fp64<5>(h, d_acc, d_pot);
        case 6: return run_fp64<6>(h, d_acc, d_pot);
        case 7: return run_fp64<7>(h, d_acc, d_pot);
        case 8: return run_fp64<8>(h, d_acc, d_pot);
        case 9: return run_fp64<9>(h, d_acc, d_pot);
        case 10: return run_fp64<10>(h, d_acc, d_pot);
        case 11: return run_fp64<11>(h, d_acc, d_pot);
        case 12: return run_fp64<12>(h, d_acc, d_pot);
        default: return OGX_ERR_INVALID;
    }
}

}  // namespace ogx
