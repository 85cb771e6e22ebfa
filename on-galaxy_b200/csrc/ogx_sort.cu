// ogx_sort.cu -- stable LSD radix sort and exclusive scans.
//
// The tree build needs two stable sorts (the reference gets the same order
// from its recursive stable counting sort, src3d/AdaptiveOctree.hpp:114-118):
//   1. bodies by their 72-bit octant path (9 passes of 8 bits),
//   2. bodies by leaf id, starting from the original order, so that inside a
//      leaf the bodies keep their original index order (2-3 passes).
// Ranking is the same everywhere: a warp ranks 32 keys by votes (digit_peers),
// keeps per-warp digit counters in shared memory and warps are ordered by their
// contiguous sub-tiles, so a pass is stable.
//
// Up to 65,536 items, all passes run in ONE launch of a thread-block cluster: every CTA
// keeps its items in registers and shared memory, digit counts are exchanged and items
// scattered through distributed shared memory, with two cluster barriers per pass.  These
// sizes are bound by latency, not by memory: as four launches per pass (histogram, two
// scans, scatter) a pass took 35-40 us whatever its size, and an evaluation runs 15 passes.
// Above, each pass is three launches: per-tile digit histogram -> scan over the tiles of
// every digit -> scatter (which scans the 256 digit totals itself).
#include <cooperative_groups.h>

#include "ogx_internal.cuh"

namespace ogx {
namespace {

namespace cg = cooperative_groups;
constexpr unsigned FULL = 0xffffffffu;

// lanes of the warp whose digit equals this lane's (8 bits; 0xFFFFFFFF: no item), by a vote
// per bit: nine votes, where __match_any_sync takes a turn per distinct digit
__device__ __forceinline__ unsigned digit_peers(uint32_t d) {
    unsigned m = __ballot_sync(FULL, d <= 0xFFu);
    if (d > 0xFFu) m = ~m;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const bool one = (d >> b) & 1u;
        const unsigned v = __ballot_sync(FULL, one);
        m &= one ? v : ~v;
    }
    return m;
}

struct Key32 {
    uint32_t* k;
    using T = uint32_t;
    __device__ __forceinline__ T load(int64_t i) const { return k[i]; }
    __device__ __forceinline__ void store(int64_t i, T v) const { k[i] = v; }
    __device__ __forceinline__ static uint32_t digit(T v, int pass) { return (v >> (8 * pass)) & 0xFFu; }
    // a tile's keys in shared memory (rs_cluster)
    static constexpr int BYTES = 4;
    using Smem = uint32_t*;
    __device__ __forceinline__ static Smem smem(unsigned char* p, int) { return reinterpret_cast<uint32_t*>(p); }
    __device__ __forceinline__ static void put(Smem s, const cg::cluster_group& cl, unsigned c, unsigned o, T v) {
        cl.map_shared_rank(s, c)[o] = v;
    }
    __device__ __forceinline__ static T get(Smem s, int i) { return s[i]; }
};

struct K72 {
    uint64_t hi;
    uint32_t lo;
};
struct Key72 {
    uint64_t* hi;
    uint32_t* lo;
    using T = K72;
    __device__ __forceinline__ T load(int64_t i) const { return K72{hi[i], lo[i]}; }
    __device__ __forceinline__ void store(int64_t i, T v) const { hi[i] = v.hi; lo[i] = v.lo; }
    // digit `pass` of the 72-bit value (hi << 9) | lo
    __device__ __forceinline__ static uint32_t digit(T v, int pass) {
        if (pass == 0) return v.lo & 0xFFu;
        if (pass == 1) return ((v.lo >> 8) & 1u) | (uint32_t)((v.hi & 0x7Full) << 1);
        return (uint32_t)((v.hi >> (8 * pass - 9)) & 0xFFull);
    }
    static constexpr int BYTES = 12;
    struct Smem {
        uint64_t* hi;
        uint32_t* lo;
    };
    __device__ __forceinline__ static Smem smem(unsigned char* p, int tile) {
        return Smem{reinterpret_cast<uint64_t*>(p), reinterpret_cast<uint32_t*>(p + (size_t)tile * 8)};
    }
    __device__ __forceinline__ static void put(Smem s, const cg::cluster_group& cl, unsigned c, unsigned o, T v) {
        cl.map_shared_rank(s.hi, c)[o] = v.hi;
        cl.map_shared_rank(s.lo, c)[o] = v.lo;
    }
    __device__ __forceinline__ static T get(Smem s, int i) { return K72{s.hi[i], s.lo[i]}; }
};

// ---- one launch, all passes: a cluster of CTAs ------------------------------------------
// A pass is bound by the instructions of one SM (about 700 per warp), so small inputs take
// small CTAs on more SMs: 8,192 bodies (15 passes) 297 -> 257 us per evaluation, 50,000 with
// the spline 670 -> 600 (CTAs of 1,024 threads before).  100,001 bodies (FP64 rotation form)
// alone take 2.12 ms with clusters of 16 x 1,024 x 8 and 2.02 ms with tiles, which spread
// over more SMs: the line is 16 CTAs of 512 threads.
constexpr int RC_MAX = 65536;   // 16 CTAs of 512 threads x 8 items

template <class KO, int RC_THREADS, int IPT>
constexpr int rc_smem() { return RC_THREADS * IPT * (int)(KO::BYTES + 4) + RC_THREADS / 32 * 256 * 4; }

template <class KO, int RC_THREADS, int IPT>
__global__ void __launch_bounds__(RC_THREADS) rs_cluster(KO kin, KO kout, const uint32_t* vin, uint32_t* vout, int n,
                                                         int first_pass, int npasses) {
    constexpr int TILE = RC_THREADS * IPT, RC_WARPS = RC_THREADS / 32, NQ = RC_THREADS / 256;
    extern __shared__ __align__(16) unsigned char rc_raw[];
    __shared__ uint32_t s_cnt[256], s_base[256], s_quarter[NQ][256], s_warp[8];
    typename KO::Smem sk = KO::smem(rc_raw, TILE);
    uint32_t* sv = reinterpret_cast<uint32_t*>(rc_raw + (size_t)TILE * KO::BYTES);
    uint32_t(*wcnt)[256] = reinterpret_cast<uint32_t(*)[256]>(sv + TILE);
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), me = (int)cl.block_rank();
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int local0 = w * 32 * IPT + lane;      // this thread's items: local0 + 32 r
    const int left = min(max(n - me * TILE, 0), TILE);   // items of this CTA
    typename KO::T key[IPT];
    uint32_t val[IPT];
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        const int i = local0 + 32 * r;
        if (i < left) {
            key[r] = kin.load((int64_t)me * TILE + i);
            val[r] = vin[(int64_t)me * TILE + i];
        }
    }
    for (int pass = first_pass; pass < npasses; ++pass) {
        for (int i = t; i < RC_WARPS * 256; i += RC_THREADS) (&wcnt[0][0])[i] = 0;
        __syncthreads();
        uint32_t loc[IPT];
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            const bool valid = local0 + 32 * r < left;
            const uint32_t d = valid ? KO::digit(key[r], pass) : 0xFFFFFFFFu;
            const unsigned peers = digit_peers(d);
            uint32_t c = 0;
            if (valid) c = wcnt[w][d];
            __syncwarp();
            if (valid && lane == __ffs(peers) - 1) wcnt[w][d] = c + __popc(peers);
            __syncwarp();
            loc[r] = c + __popc(peers & lt);
        }
        __syncthreads();
        {   // counters -> offsets inside the CTA's digit, eight warps per thread
            const int d = t & 255, q = t >> 8;
            uint32_t run = 0;
#pragma unroll
            for (int k = 0; k < RC_WARPS / NQ; ++k) {
                const uint32_t c = wcnt[q * (RC_WARPS / NQ) + k][d];
                wcnt[q * (RC_WARPS / NQ) + k][d] = run;
                run += c;
            }
            s_quarter[q][d] = run;
        }
        __syncthreads();
        if (t < 256) {
            uint32_t run = 0;
#pragma unroll
            for (int q = 0; q < NQ; ++q) {
                const uint32_t c = s_quarter[q][t];
                s_quarter[q][t] = run;
                run += c;
            }
            s_cnt[t] = run;
        }
        cl.sync();
        uint32_t tot = 0, before = 0, x = 0;
        if (t < 256) {
            for (int c = 0; c < C; ++c) {
                const uint32_t v = cl.map_shared_rank(s_cnt, c)[t];
                if (c < me) before += v;
                tot += v;
            }
            x = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) s_warp[w] = x;
        }
        __syncthreads();
        if (t < 256) {
            uint32_t pre = 0;
            for (int k = 0; k < w; ++k) pre += s_warp[k];
            s_base[t] = pre + x - tot + before;
        }
        __syncthreads();
        const bool last = pass + 1 == npasses;
#pragma unroll
        for (int r = 0; r < IPT; ++r) {
            if (local0 + 32 * r < left) {
                const uint32_t d = KO::digit(key[r], pass);
                const uint32_t pos = s_base[d] + s_quarter[w / (RC_WARPS / NQ)][d] + wcnt[w][d] + loc[r];
                if (last) {
                    kout.store(pos, key[r]);
                    vout[pos] = val[r];
                } else {
                    const unsigned c = pos / TILE, o = pos % TILE;
                    KO::put(sk, cl, c, o, key[r]);
                    cl.map_shared_rank(sv, c)[o] = val[r];
                }
            }
        }
        cl.sync();   // every item is in place (and, after the last pass, no CTA exits while its counts are read)
        if (!last) {
#pragma unroll
            for (int r = 0; r < IPT; ++r) {
                const int i = local0 + 32 * r;
                if (i < left) {
                    key[r] = KO::get(sk, i);
                    val[r] = sv[i];
                }
            }
        }
    }
}

// ---- three launches per pass ----------------------------------------------------------
constexpr int RS_THREADS = 512;
constexpr int RS_WARPS = RS_THREADS / 32;

template <class KO, int IPT>
__global__ void __launch_bounds__(RS_THREADS) rs_hist(KO keys, int64_t n, int pass, uint32_t* hist, int nblocks) {
    __shared__ uint32_t h[256];
    if (threadIdx.x < 256) h[threadIdx.x] = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t start = (int64_t)blockIdx.x * (RS_THREADS * IPT) + threadIdx.x;
    uint32_t d[IPT];
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        const int64_t i = start + r * RS_THREADS;
        d[r] = i < n ? KO::digit(keys.load(i), pass) : 0xFFFFFFFFu;
    }
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        const unsigned peers = digit_peers(d[r]);
        if (d[r] < 256 && lane == __ffs(peers) - 1) atomicAdd(&h[d[r]], (uint32_t)__popc(peers));
    }
    __syncthreads();
    if (threadIdx.x < 256) hist[(int64_t)threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// Digit-major histogram hist[d * nblocks + b] -> exclusive offsets within each digit
// (one CTA per digit, coalesced over the tiles), digit totals into tot[d].
__global__ void __launch_bounds__(256) rs_scan_digit(uint32_t* hist, int nblocks, uint32_t* tot) {
    __shared__ uint32_t warp_sum[8];
    uint32_t* a = hist + (size_t)blockIdx.x * nblocks;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    uint32_t carry = 0;
    for (int b0 = 0; b0 < nblocks; b0 += 256) {
        const int i = b0 + t;
        const uint32_t v = (i < nblocks) ? a[i] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[w] = x;
        __syncthreads();
        uint32_t pre = 0, all = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const uint32_t s = warp_sum[k];
            if (k < w) pre += s;
            all += s;
        }
        if (i < nblocks) a[i] = carry + pre + x - v;
        carry += all;
        __syncthreads();
    }
    if (t == 0) tot[blockIdx.x] = carry;
}

template <class KO, int IPT>
__global__ void __launch_bounds__(RS_THREADS) rs_scatter(KO kin, KO kout, const uint32_t* vin, uint32_t* vout, int64_t n,
                                                         int pass, const uint32_t* scanned, int nblocks, const uint32_t* tot) {
    __shared__ uint32_t wcnt[RS_WARPS][256];
    __shared__ uint32_t gbase[256], s_warp[8];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int64_t base = (int64_t)blockIdx.x * (RS_THREADS * IPT) + (int64_t)w * 32 * IPT + lane;
    // every load of the tile is in flight before the first rank
    typename KO::T key[IPT];
    uint32_t val[IPT], loc[IPT];
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        const int64_t i = base + r * 32;
        if (i < n) {
            key[r] = kin.load(i);
            val[r] = vin[i];
        }
    }
    uint32_t tv = 0, x = 0, sc = 0;
    if (t < 256) {
        x = tv = tot[t];
        sc = scanned[(int64_t)t * nblocks + blockIdx.x];
    }
    for (int i = t; i < RS_WARPS * 256; i += RS_THREADS) (&wcnt[0][0])[i] = 0;
    if (t < 256) {   // exclusive scan of the 256 digit totals
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_warp[w] = x;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        const bool valid = base + r * 32 < n;
        const uint32_t d = valid ? KO::digit(key[r], pass) : 0xFFFFFFFFu;
        const unsigned peers = digit_peers(d);
        uint32_t c = 0;
        if (valid) c = wcnt[w][d];
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) wcnt[w][d] = c + __popc(peers);
        __syncwarp();
        loc[r] = c + __popc(peers & lt);
    }
    __syncthreads();
    if (t < 256) {
        uint32_t run = 0;
#pragma unroll
        for (int k = 0; k < RS_WARPS; ++k) {
            const uint32_t c = wcnt[k][t];
            wcnt[k][t] = run;
            run += c;
        }
        uint32_t pre = 0;
        for (int k = 0; k < w; ++k) pre += s_warp[k];
        gbase[t] = pre + x - tv + sc;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < IPT; ++r) {
        if (base + r * 32 < n) {
            const uint32_t d = KO::digit(key[r], pass);
            const int64_t pos = (int64_t)gbase[d] + wcnt[w][d] + loc[r];
            kout.store(pos, key[r]);
            vout[pos] = val[r];
        }
    }
}

// ---- generic exclusive scan int32 -> int64 (out has n+1 entries) --------------
// Two arrays of one length at a time (grid y); up to SC_ONE entries in one launch, in
// which every tile's CTA sums the entries before it itself (one CTA walking eight tiles in
// turn took 9 us, a barrier chain per tile; 8 steps of 30,011 bodies 4.27 -> 4.18 ms); else per-tile sums and a second launch in which
// every tile adds the sums before it.
constexpr int SC_THREADS = 1024;
constexpr int SC_IPT = 4;
constexpr int SC_TILE = SC_THREADS * SC_IPT;
constexpr int64_t SC_ONE = 32 * SC_TILE;

struct ScanPair {
    const int* in[2];
    int64_t* out[2];
    int64_t* part[2];
};

__device__ __forceinline__ int64_t block_excl_scan_i64(int64_t v, int64_t* sh, int64_t* total) {
    // sh: 32 int64 scratch
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        int64_t s = (lane < nw) ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(FULL, s, o);
            if (lane >= o) s += y;
        }
        if (lane < nw) sh[lane] = s;
    }
    __syncthreads();
    const int64_t wpre = (w > 0) ? sh[w - 1] : 0;
    if (total) *total = sh[(blockDim.x >> 5) - 1];
    __syncthreads();
    return wpre + x - v;
}

__device__ __forceinline__ void sc_load(const int* in, int64_t b, int64_t n, int (&v)[SC_IPT]) {
#pragma unroll
    for (int k = 0; k < SC_IPT; ++k) v[k] = b + k < n ? in[b + k] : 0;
}

__global__ void __launch_bounds__(SC_THREADS) sc_one(ScanPair sp, int64_t n) {
    __shared__ int64_t sh[32], s_before[32];
    const int* in = sp.in[blockIdx.y];
    int64_t* out = sp.out[blockIdx.y];
    const int64_t t0 = (int64_t)blockIdx.x * SC_TILE, b = t0 + (int64_t)threadIdx.x * SC_IPT;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int v[SC_IPT];
    sc_load(in, b, n, v);
    int64_t before = 0, s = 0, tot;
#pragma unroll 16
    for (int64_t i = threadIdx.x; i < t0; i += SC_THREADS) before += in[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(FULL, before, o);
    if (lane == 0) s_before[w] = before;
#pragma unroll
    for (int k = 0; k < SC_IPT; ++k) s += v[k];
    const int64_t mine = block_excl_scan_i64(s, sh, &tot);
    int64_t carry = s_before[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) carry += __shfl_xor_sync(FULL, carry, o);
    int64_t run = carry + mine;
#pragma unroll
    for (int k = 0; k < SC_IPT; ++k) {
        if (b + k < n) out[b + k] = run;
        run += v[k];
    }
    if (blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) out[n] = carry + tot;
}

__global__ void __launch_bounds__(SC_THREADS) sc_partials(ScanPair sp, int64_t n) {
    __shared__ int64_t sh[32];
    int v[SC_IPT];
    sc_load(sp.in[blockIdx.y], (int64_t)blockIdx.x * SC_TILE + (int64_t)threadIdx.x * SC_IPT, n, v);
    int64_t s = 0, tot;
#pragma unroll
    for (int k = 0; k < SC_IPT; ++k) s += v[k];
    block_excl_scan_i64(s, sh, &tot);
    if (threadIdx.x == 0) sp.part[blockIdx.y][blockIdx.x] = tot;
}

__global__ void __launch_bounds__(SC_THREADS) sc_finish(ScanPair sp, int64_t n) {
    __shared__ int64_t sh[32];
    const int64_t* part = sp.part[blockIdx.y];
    int64_t* out = sp.out[blockIdx.y];
    const int64_t b = (int64_t)blockIdx.x * SC_TILE + (int64_t)threadIdx.x * SC_IPT;
    int v[SC_IPT];
    sc_load(sp.in[blockIdx.y], b, n, v);
    int64_t pre = 0, base;
    for (int k = threadIdx.x; k < (int)blockIdx.x; k += SC_THREADS) pre += part[k];
    block_excl_scan_i64(pre, sh, &base);   // the sum of the tiles before this one
    int64_t s = 0, tot;
#pragma unroll
    for (int k = 0; k < SC_IPT; ++k) s += v[k];
    int64_t run = base + block_excl_scan_i64(s, sh, &tot);
#pragma unroll
    for (int k = 0; k < SC_IPT; ++k) {
        if (b + k < n) out[b + k] = run;
        run += v[k];
    }
    if (blockIdx.x + 1 == gridDim.x && threadIdx.x == 0) out[n] = base + tot;
}

}  // namespace

static int scan_arrays(Handle& h, ScanPair sp, int count, int64_t n) {
    if (n == 0) {
        for (int a = 0; a < count; ++a) OGX_CUDA(cudaMemsetAsync(sp.out[a], 0, sizeof(int64_t), h.stream));
        return OGX_OK;
    }
    if (n <= SC_ONE) {
        sc_one<<<dim3((unsigned)((n + SC_TILE - 1) / SC_TILE), count), SC_THREADS, 0, h.stream>>>(sp, n); ++h.launches;
    } else {
        const int nparts = (int)((n + SC_TILE - 1) / SC_TILE);
        OGX_TRY(arena_get(h.ws, S_SCAN_TMP, 2 * (size_t)nparts, &sp.part[0]));
        sp.part[1] = sp.part[0] + nparts;
        sc_partials<<<dim3(nparts, count), SC_THREADS, 0, h.stream>>>(sp, n); ++h.launches;
        sc_finish<<<dim3(nparts, count), SC_THREADS, 0, h.stream>>>(sp, n); ++h.launches;
    }
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

int scan_i32_to_i64(Handle& h, const int* in, int64_t* out, int64_t n) {
    ScanPair sp{};
    sp.in[0] = in;
    sp.out[0] = out;
    return scan_arrays(h, sp, 1, n);
}

int scan2_i32_to_i64(Handle& h, const int* in_a, int64_t* out_a, const int* in_b, int64_t* out_b, int64_t n) {
    ScanPair sp{};
    sp.in[0] = in_a; sp.in[1] = in_b;
    sp.out[0] = out_a; sp.out[1] = out_b;
    return scan_arrays(h, sp, 2, n);
}

// The cluster sort with the fewest CTAs (a power of two) that hold n.
template <class KO, int RC_THREADS, int IPT>
static int cluster_sort(Handle& h, KO a, KO b, const uint32_t* va, uint32_t* vb, int64_t n, int npasses, int first_pass) {
    auto kern = rs_cluster<KO, RC_THREADS, IPT>;
    constexpr int smem = rc_smem<KO, RC_THREADS, IPT>();
    OGX_CUDA(smem_optin((const void*)kern, smem));
    int ctas = 1;
    while ((int64_t)ctas * RC_THREADS * IPT < n) ctas *= 2;
    if (ctas > 8) OGX_CUDA(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(RC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = h.stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    OGX_CUDA(cudaLaunchKernelEx(&cfg, kern, a, b, va, vb, (int)n, first_pass, npasses)); ++h.launches;
    return OGX_OK;
}

template <class KO, int IPT>
static int tile_sort(Handle& h, KO src, KO dst, uint32_t* vs, uint32_t* vd, int64_t n, int npasses, int first_pass) {
    const int nblocks = (int)((n + RS_THREADS * IPT - 1) / (RS_THREADS * IPT));
    uint32_t* hist;
    OGX_TRY(arena_get(h.ws, S_RS_HIST, (size_t)256 * nblocks + 256, &hist));
    uint32_t* tot = hist + (size_t)256 * nblocks;
    for (int pass = first_pass; pass < npasses; ++pass) {
        rs_hist<KO, IPT><<<nblocks, RS_THREADS, 0, h.stream>>>(src, n, pass, hist, nblocks); ++h.launches;
        rs_scan_digit<<<256, 256, 0, h.stream>>>(hist, nblocks, tot); ++h.launches;
        rs_scatter<KO, IPT><<<nblocks, RS_THREADS, 0, h.stream>>>(src, dst, vs, vd, n, pass, hist, nblocks, tot); ++h.launches;
        std::swap(src, dst);
        std::swap(vs, vd);
    }
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

template <class KO>
static int radix_passes(Handle& h, KO a, KO b, uint32_t* va, uint32_t* vb, int64_t n, int npasses, int* which,
                        int first_pass = 0) {
    if (n <= RC_MAX) {
        *which = 1;
        if (n <= 8 * 256 * 4) return cluster_sort<KO, 256, 4>(h, a, b, va, vb, n, npasses, first_pass);
        if (n <= 16 * 256 * 8) return cluster_sort<KO, 256, 8>(h, a, b, va, vb, n, npasses, first_pass);
        return cluster_sort<KO, 512, 8>(h, a, b, va, vb, n, npasses, first_pass);
    }
    *which = (npasses - first_pass) & 1;  // 0: result in a, 1: result in b
    // tiles of 2,048 while 4,096 would leave SMs without one
    if (n <= (int64_t)RS_THREADS * 8 * h.num_sms) return tile_sort<KO, 4>(h, a, b, va, vb, n, npasses, first_pass);
    return tile_sort<KO, 8>(h, a, b, va, vb, n, npasses, first_pass);
}

int radix_sort_u32(Handle& h, Slot kin, Slot vin, Slot kalt, Slot valt, int64_t n, int bits, uint32_t** kout,
                   uint32_t** vout) {
    uint32_t *k0, *v0, *k1, *v1;
    OGX_TRY(arena_get(h.ws, kin, n, &k0));
    OGX_TRY(arena_get(h.ws, vin, n, &v0));
    OGX_TRY(arena_get(h.ws, kalt, n, &k1));
    OGX_TRY(arena_get(h.ws, valt, n, &v1));
    int npasses = (bits + 7) / 8;
    if (npasses < 1) npasses = 1;
    int which = 0;
    if (n > 0) OGX_TRY(radix_passes(h, Key32{k0}, Key32{k1}, v0, v1, n, npasses, &which));
    *kout = which ? k1 : k0;
    *vout = which ? v1 : v0;
    return OGX_OK;
}

int radix_sort_key72(Handle& h, int64_t n, int first_pass, uint64_t** khi, uint32_t** klo, uint32_t** idx) {
    uint64_t *h0, *h1;
    uint32_t *l0, *l1, *i0, *i1;
    OGX_TRY(arena_get(h.ws, S_KHI, n, &h0));
    OGX_TRY(arena_get(h.ws, S_KLO, n, &l0));
    OGX_TRY(arena_get(h.ws, S_IDX, n, &i0));
    OGX_TRY(arena_get(h.ws, S_KHI2, n, &h1));
    OGX_TRY(arena_get(h.ws, S_KLO2, n, &l1));
    OGX_TRY(arena_get(h.ws, S_IDX2, n, &i1));
    int which = 0;
    if (n > 0) OGX_TRY(radix_passes(h, Key72{h0, l0}, Key72{h1, l1}, i0, i1, n, 9, &which, first_pass));
    *khi = which ? h1 : h0;
    *klo = which ? l1 : l0;
    *idx = which ? i1 : i0;
    return OGX_OK;
}

}  // namespace ogx
