// ogx_translate.cu -- M2M and L2L, one launch per pass, on the FP64 matrix instructions.
//
//   M2M: M'_P = sum_s MM_s M'_{child s}                (src3d/AdaptiveFMM3D.hpp:62-71)
//   L2L: L'_{child s} = L'own_{child s} + LL_s L'_P     (src3d/AdaptiveFMM3D.hpp:75-77)
// The reference walks the levels one after another (its GPU form launches once per level,
// src3d/gpu/AdaptiveFMM3DGPU.cu:274-289).  Here one launch covers every level: CTAs take
// work items by ticket (an atomic counter) in level order, root level first for L2L, deepest
// level first for M2M, and an item waits until its inputs are final.  Those items hold
// earlier tickets, so the item with the smallest unfinished ticket never waits and every wait
// ends; each is bounded all the same (one that runs out sets *err).  An item publishes its
// boxes with a fence and a release; data written in this launch is read through L2.
//
// An item is 16 parents: their vectors are the rows of mma.sync m16n8k4 (FP64), the operator
// its columns.  Bound: a narrow level is a chain of latencies (flag, operands, product,
// publish) and a wide one the operator's L2 traffic, 52 KB per octant at p = 8 and 228 KB at
// p = 12.  With 4 parents (2 at p > 8) per CTA and all operator rows read by every CTA the
// passes took 166 + 199 us on the 1M merger and 597 us on 200,003 bodies at p = 12, and a
// small tree took one launch per level, 14 us each.  Now an item reads a quarter of the
// operator's columns per warp (L2L: one octant, the quarters on four warps; M2M: one quarter,
// the octants on eight warps), its first rows while it waits, and only the rows that are not
// zero (M2M raises the degree, L2L lowers it).  A box's result does not depend on the order.
#include <algorithm>

#include "ogx_m2l64.cuh"
#include "ogx_sm100.cuh"

namespace ogx {
namespace {

constexpr int TR_ROWS = 16;       // parents of an item

template <int P>
struct Tr {
    static constexpr int K = (P + 1) * (P + 1);
    static constexpr int K4 = (K + 3) / 4 * 4, STEPS = K4 / 4;
    static constexpr int NT = (K + 7) / 8;                    // 8-column tiles of the output
    static constexpr int PARTS = NT > 20 ? 6 : 4;             // column parts (6: M2M's sums fit 48 KB at p = 12)
    static constexpr int NTW = (NT + PARTS - 1) / PARTS;      // tiles of one part
    static constexpr int LDN = 8 * NT + 4;                    // operator rows (m2l64_pad_cols)
    static constexpr int LDA = (K4 % 16 == 4 || K4 % 16 == 12) ? K4 : K4 + 4;
    static constexpr int UB = 4;                              // steps of operator rows in flight
};

__device__ __forceinline__ int deg_of(int dof) {
    int n = 0;
    while ((n + 1) * (n + 1) <= dof) ++n;
    return n;
}

__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// bounded wait until *flag >= want; false when it ran out (*err is then set) or when
// another wait already gave up
__device__ bool wait_ready(const int* flag, int want, int* err, uint32_t limit = sm100::kSpinLimit) {
    for (uint32_t it = 0; it < limit; ++it) {
        if (ld_acquire_gpu(flag) >= want) return true;
        if (*(volatile int*)err) return false;
        if (it > 16) __nanosleep(64);
    }
    atomicExch(err, 1);
    return false;
}
__device__ __forceinline__ void publish(int* flag) {
    asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(flag) : "memory");
}

// one column part of a product: steps [k0, k1) of A (callable: step -> a0, a1) times the
// operator rows T (this lane's element of step 0, column 0 of the part); `tiles` of its
// column tiles exist.  `first`: the rows of the first block, loaded by tr_load.
template <int P>
__device__ __forceinline__ void tr_load(double (&b)[Tr<P>::UB][Tr<P>::NTW], const double* __restrict__ T, int k0, int k1, int tiles) {
    using C = Tr<P>;
#pragma unroll
    for (int u = 0; u < C::UB; ++u)
#pragma unroll
        for (int i = 0; i < C::NTW; ++i)
            b[u][i] = (k0 + u < k1 && i < tiles) ? __ldg(T + (size_t)(k0 + u) * 4 * C::LDN + 8 * i) : 0.0;
}
template <int P, class A>
__device__ __forceinline__ void tr_product(double (&acc)[Tr<P>::NTW][4], double (&first)[Tr<P>::UB][Tr<P>::NTW],
                                           const double* __restrict__ T, int k0, int k1, int tiles, A&& a_of) {
    using C = Tr<P>;
    for (int k = k0; k < k1; k += C::UB) {
        double next[C::UB][C::NTW];
        tr_load<P>(next, T, k + C::UB, k1, tiles);
        double a0[C::UB], a1[C::UB];
#pragma unroll
        for (int u = 0; u < C::UB; ++u) {
            a0[u] = a1[u] = 0.0;
            if (k + u < k1) a_of(k + u, a0[u], a1[u]);
        }
#pragma unroll
        for (int u = 0; u < C::UB; ++u)
#pragma unroll
            for (int i = 0; i < C::NTW; ++i) sm100::dmma(acc[i], a0[u], a1[u], first[u][i]);
#pragma unroll
        for (int u = 0; u < C::UB; ++u)
#pragma unroll
            for (int i = 0; i < C::NTW; ++i) first[u][i] = next[u][i];
    }
}

// items of the pass's first i + 1 levels into gend (PER items per group of parents)
template <int PER>
__device__ __forceinline__ void level_items(const int* __restrict__ nl_off, int nlev, bool down, int* gend) {
    const int lane = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        int v = 0;
        if (lane < nlev) {
            const int l = down ? lane : nlev - 1 - lane;
            v = (nl_off[l + 1] - nl_off[l] + TR_ROWS - 1) / TR_ROWS * PER;
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane < nlev) gend[lane] = v;
    }
}

// item = (level, group of 16 parents, octant); warp = column part
template <int P>
__global__ void __launch_bounds__(32 * Tr<P>::PARTS, Tr<P>::NTW <= 3 ? 4 : 2) k_l2l(TreeView tv, const int* __restrict__ nonleaf, const int* __restrict__ nl_off,
                                                      int nlev, const double* __restrict__ ops, double* local,
                                                      const double* __restrict__ lown, int* ready, int* ticket, int* err) {
    using C = Tr<P>;
    constexpr int K = C::K;
    __shared__ double s_a[TR_ROWS][C::LDA];
    __shared__ int s_gend[32], s_par[TR_ROWS], s_ch[TR_ROWS];
    __shared__ int s_t[2];
    const int tid = threadIdx.x, lane = tid & 31, part = tid >> 5;
    if (tv_over(tv) || nlev <= 0) return;
    level_items<8>(nl_off, nlev, true, s_gend);
    if (tid == 0) s_t[0] = atomicAdd(ticket, 1);
    const int c0 = part * C::NTW * 8, tiles = min(C::NTW, C::NT - part * C::NTW);
    // rows of degree below the part's first column are zero
    const int k0 = c0 < K ? (deg_of(c0) * deg_of(c0)) / 4 : C::STEPS, k1 = C::STEPS;
    for (int round = 0;; ++round) {
        __syncthreads();
        const int t = s_t[round & 1];
        if (t >= s_gend[nlev - 1]) break;
        if (tid == 0) s_t[(round & 1) ^ 1] = atomicAdd(ticket, 1);   // the next item, fetched beside this one
        int l = 0;
        while (t >= s_gend[l]) ++l;
        const int q = t - (l > 0 ? s_gend[l - 1] : 0), p0 = (q >> 3) * TR_ROWS, s = q & 7;
        const int first = nl_off[l], count = nl_off[l + 1] - first;
        int ch = -1;
        if (tid < TR_ROWS) {
            const int b = p0 + tid < count ? nonleaf[first + p0 + tid] : -1;
            ch = b >= 0 ? tv.child[8 * (size_t)b + s] : -1;
            s_par[tid] = b;
            s_ch[tid] = ch;
        }
        const double* T = ops + ((size_t)s * C::K4 + (lane & 3)) * C::LDN + c0 + (lane >> 2);
        double b0[C::UB][C::NTW];
        tr_load<P>(b0, T, k0, k1, tiles);
        if (tid < TR_ROWS && l > 0 && ch >= 0) wait_ready(ready + s_par[tid], 1, err);   // published by its parent's item
        if (!__syncthreads_or(ch >= 0)) continue;
        for (int i = tid; i < TR_ROWS * C::K4; i += 32 * Tr<P>::PARTS) {
            const int r = i / C::K4, k = i - r * C::K4;
            s_a[r][k] = (k < K && s_ch[r] >= 0) ? __ldcg(local + (size_t)s_par[r] * K + k) : 0.0;
        }
        // own parts of the children, in the accumulators' layout
        double own[C::NTW][4];
#pragma unroll
        for (int i = 0; i < C::NTW; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int d = c0 + 8 * i + 2 * (lane & 3) + (v & 1), c = s_ch[(lane >> 2) + 8 * (v >> 1)];
                own[i][v] = (i < tiles && d < K && c >= 0) ? __ldg(lown + (size_t)c * K + d) : 0.0;
            }
        __syncthreads();
        double acc[C::NTW][4];
#pragma unroll
        for (int i = 0; i < C::NTW; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[i][v] = 0.0;
        tr_product<P>(acc, b0, T, k0, k1, tiles, [&](int k, double& a0, double& a1) {
            a0 = s_a[lane >> 2][4 * k + (lane & 3)];
            a1 = s_a[(lane >> 2) + 8][4 * k + (lane & 3)];
        });
#pragma unroll
        for (int i = 0; i < C::NTW; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int d = c0 + 8 * i + 2 * (lane & 3) + (v & 1), c = s_ch[(lane >> 2) + 8 * (v >> 1)];
                if (i < tiles && d < K && c >= 0) local[(size_t)c * K + d] = own[i][v] + acc[i][v];
            }
        __threadfence();
        __syncthreads();
        if (ch >= 0) publish(ready + ch);
    }
}

// item = (level, group of 16 parents, column part); warp = octant
template <int P>
__global__ void __launch_bounds__(256, 2) k_m2m(TreeView tv, const int* __restrict__ nonleaf, const int* __restrict__ nl_off, int nlev,
                                             const double* __restrict__ ops, double* mpole, int* ready, int* ticket, int* err) {
    using C = Tr<P>;
    constexpr int K = C::K, W = 8 * C::NTW;
    __shared__ double s_part[8][TR_ROWS][W];
    __shared__ int s_gend[32], s_par[TR_ROWS];
    __shared__ int s_t[2];
    const int tid = threadIdx.x, lane = tid & 31, s = tid >> 5;
    if (tv_over(tv) || nlev <= 0) return;
    level_items<Tr<P>::PARTS>(nl_off, nlev, false, s_gend);
    if (tid == 0) s_t[0] = atomicAdd(ticket, 1);
    for (int round = 0;; ++round) {
        __syncthreads();
        const int t = s_t[round & 1];
        if (t >= s_gend[nlev - 1]) break;
        if (tid == 0) s_t[(round & 1) ^ 1] = atomicAdd(ticket, 1);
        int i0 = 0;
        while (t >= s_gend[i0]) ++i0;
        const int l = nlev - 1 - i0, q = t - (i0 > 0 ? s_gend[i0 - 1] : 0);
        const int p0 = (q / Tr<P>::PARTS) * TR_ROWS, part = q % Tr<P>::PARTS;
        const int first = nl_off[l], count = nl_off[l + 1] - first;
        const int c0 = part * W, tiles = min(C::NTW, C::NT - part * C::NTW);
        // rows of degree above the part's last column are zero
        const int dl = c0 < K ? deg_of(min(K, c0 + 8 * tiles) - 1) + 1 : 0;
        const int k1 = tiles > 0 ? min(C::STEPS, (dl * dl + 3) / 4) : 0;
        int b = -1, ch = -1;
        if (lane < TR_ROWS) {
            b = p0 + lane < count ? nonleaf[first + p0 + lane] : -1;
            ch = b >= 0 ? tv.child[8 * (size_t)b + s] : -1;
            if (s == 0) s_par[lane] = b;
        }
        const bool any = __any_sync(0xffffffffu, ch >= 0);
        const double* T = ops + ((size_t)s * C::K4 + (lane & 3)) * C::LDN + c0 + (lane >> 2);
        double acc[C::NTW][4];
#pragma unroll
        for (int i = 0; i < C::NTW; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) acc[i][v] = 0.0;
        if (any) {
            double b0[C::UB][C::NTW];
            tr_load<P>(b0, T, 0, k1, tiles);
            if (ch >= 0 && tv.leafid[ch] < 0) wait_ready(ready + ch, Tr<P>::PARTS, err);   // every part of a non-leaf child
            __syncwarp();
            const int ra = __shfl_sync(0xffffffffu, ch, lane >> 2), rb = __shfl_sync(0xffffffffu, ch, (lane >> 2) + 8);
            const double* pa = mpole + (size_t)max(ra, 0) * K;
            const double* pb = mpole + (size_t)max(rb, 0) * K;
            tr_product<P>(acc, b0, T, 0, k1, tiles, [&](int k, double& a0, double& a1) {
                const int kk = 4 * k + (lane & 3);
                a0 = (ra >= 0 && kk < K) ? __ldcg(pa + kk) : 0.0;
                a1 = (rb >= 0 && kk < K) ? __ldcg(pb + kk) : 0.0;
            });
        }
#pragma unroll
        for (int i = 0; i < C::NTW; ++i)
#pragma unroll
            for (int v = 0; v < 4; ++v) s_part[s][(lane >> 2) + 8 * (v >> 1)][8 * i + 2 * (lane & 3) + (v & 1)] = acc[i][v];
        __syncthreads();
        for (int i = tid; i < TR_ROWS * W; i += 256) {
            const int r = i / W, d = c0 + i % W;
            if (s_par[r] < 0 || d >= K) continue;
            double v = 0.0;
#pragma unroll
            for (int o = 0; o < 8; ++o) v += s_part[o][r][i % W];
            mpole[(size_t)s_par[r] * K + d] = v;
        }
        __threadfence();
        __syncthreads();
        if (s == 0 && b >= 0) publish(ready + b);
    }
}

// boxes of level l: exact in an eager evaluation, the capacity in capacity mode
int level_boxes(const Handle& h, int l) {
    if (h.cap_mode) return h.cap.level_boxes[l];
    return l <= h.max_level ? h.level_off[l + 1] - h.level_off[l] : 0;
}

// One launch: CTAs for the widest level's items (taking a quarter of the next level's boxes
// for a level's parents), at most four (M2M, of eight warps: two) per SM.  Any number is
// correct; more would only wait and hold the SMs that other systems need.
template <int P>
int translate(Handle& h, bool down, Slot slot, double* M, double* L, const double* Lown) {
    const int nlev = h.max_level;   // parent levels 0 .. max_level-1
    if (nlev <= 0) return OGX_OK;
    int items = 1;
    for (int l = 0; l < nlev; ++l) {
        const int parents = std::min(level_boxes(h, l), std::max(1, level_boxes(h, l + 1) / 4));
        items = std::max(items, (parents + TR_ROWS - 1) / TR_ROWS * (down ? 8 : Tr<P>::PARTS));
    }
    int* ready;
    const size_t nready = (size_t)h.tv.nb + 1;
    OGX_TRY(arena_get(h.ws, slot, nready, &ready));
    OGX_CUDA(cudaMemsetAsync(ready, 0, sizeof(int) * nready, h.stream));
    int* ticket = ready + h.tv.nb;
    const int grid = std::min(items, (down ? 4 : 2) * h.num_sms);
    if (down)
        k_l2l<P><<<grid, 32 * Tr<P>::PARTS, 0, h.stream>>>(h.tv, h.d_nonleaf, h.d_nonleaf_off, nlev, h.d_l2l, L, Lown, ready, ticket,
                                                           h.d_err);
    else
        k_m2m<P><<<grid, 256, 0, h.stream>>>(h.tv, h.d_nonleaf, h.d_nonleaf_off, nlev, h.d_m2m, M, ready, ticket, h.d_err);
    ++h.launches;
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

template <int P>
int l2l(Handle& h, double* L, const double* Lown) {
    // root (no parent): its local is its own M2L/P2L part; box 0 is the root
    OGX_CUDA(cudaMemcpyAsync(L, Lown, sizeof(double) * Tr<P>::K, cudaMemcpyDeviceToDevice, h.stream));
    return translate<P>(h, true, S_TR_READY_L, nullptr, L, Lown);
}

}  // namespace

// One thread runs the passes' bounded flag wait, with a limit of `polls`, on a flag that
// nothing sets: the wait runs out and sets *err as in the passes.
__global__ void k_flag_wait_probe(const int* flag, int* err, uint32_t polls) {
    if (threadIdx.x == 0) wait_ready(flag, 1, err, polls);
}

int flag_wait_probe(Handle& h, uint32_t polls, const int* flag, int* err) {
    k_flag_wait_probe<<<1, 32, 0, h.stream>>>(flag, err, polls);
    ++h.launches;
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

int m2m_launch(Handle& h, double* M) {
    switch (h.prm.p) {
        case 1: return translate<1>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 2: return translate<2>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 3: return translate<3>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 4: return translate<4>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 5: return translate<5>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 6: return translate<6>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 7: return translate<7>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 8: return translate<8>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 9: return translate<9>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 10: return translate<10>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 11: return translate<11>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        case 12: return translate<12>(h, false, S_TR_READY_M, M, nullptr, nullptr);
        default: return OGX_ERR_INVALID;
    }
}

int l2l_launch(Handle& h, double* L, const double* Lown) {
    switch (h.prm.p) {
        case 1: return l2l<1>(h, L, Lown);
        case 2: return l2l<2>(h, L, Lown);
        case 3: return l2l<3>(h, L, Lown);
        case 4: return l2l<4>(h, L, Lown);
        case 5: return l2l<5>(h, L, Lown);
        case 6: return l2l<6>(h, L, Lown);
        case 7: return l2l<7>(h, L, Lown);
        case 8: return l2l<8>(h, L, Lown);
        case 9: return l2l<9>(h, L, Lown);
        case 10: return l2l<10>(h, L, Lown);
        case 11: return l2l<11>(h, L, Lown);
        case 12: return l2l<12>(h, L, Lown);
        default: return OGX_ERR_INVALID;
    }
}

}  // namespace ogx
