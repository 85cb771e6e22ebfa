// ogx_near.cuh -- the near field (softened P2P over the U lists) of both forms.
//
// Replaces the pair loop of AdaptiveFMM3D::computeAccelerations (src3d/AdaptiveFMM3D.hpp:95-103).
// A one-warp block takes one work item (leaf, chunk of at most 32 targets; k_leaf_occupancy), so
// a leaf of many bodies (the eps floor stops splitting in dense cores) spreads over many
// blocks.  In a chunk of T targets, unit u = lane + 32 r is target u mod T with source part
// u / T, which takes every G-th source of each staged round.  The leaf itself is one
// round (with the self pair skipped); the bodies of all other U-list entries are
// concatenated and staged NEAR_CAP at a time.  The G parts of each target are added in part
// order in FP64 through shared memory (deterministic).
//
// FP32 (mixed form): double-float coordinates.  Every sorted body's position relative to the
// root centre is held as hi + lo FP32 (k_gather_bodies).  For a close pair
// the two hi parts lie within a factor of two of each other, so s_hi - t_hi is exact
// (Sterbenz) and d = (s_hi - t_hi) + (s_lo - t_lo) carries the FP32 relative accuracy of |d|
// itself (absolute error ~2^-48 of the root box), however small |d| is.  Bound: issue slots
// (the FMA pipe was 45% busy at 75% issue); two sources of a part go together in packed
// f32x2 operations up to the pair's weight, and a part's staged sources lie one after another
// in separate x, y, z, m arrays so that one 16-byte load brings a coordinate of four.  The
// sums take the sources one by one: another order of the sums is as exact, but unsoftened
// close pairs amplify its rounding over a few steps.  (Two targets per operation leave half
// the lanes of a 32-target chunk idle: 1.5 ms.)  Every round's sum goes into a compensated
// (Kahan) accumulator.
// FP64 (plain form): the same items and rounds on pair64 (ogx_pair64.cuh); one warp per
// chunk walked the list source by source before, half its lanes idle on a 17-body leaf.
#pragma once

#include "ogx_internal.cuh"
#include "ogx_pair64.cuh"
#include "ogx_packed.cuh"
#include "ogx_softening.cuh"

namespace ogx {
namespace near_field {

__device__ __forceinline__ void kahan_add(float& s, float& c, float v) {
    const float y = v - c;
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

constexpr int NEAR_CAP = 128;    // source bodies staged per round (several U-list entries)

// Number of source parts G for a chunk of T targets: units (target, part) = T G,
// at most NU, are spread over the 32 lanes in R = ceil(T G / 32) rounds; G maximises
// the busy fraction T G / (32 R) (ties: the smaller G).  With NU = 64 a 17-body leaf
// gets G = 3 (80% busy; one target per lane would leave 47% of the lanes idle), a
// 5-body leaf G = 6 (94%).
struct PartTable {
    unsigned char g[2][33];   // [units 32, 64][targets]
    constexpr PartTable() : g() {
        for (int w = 0; w < 2; ++w)
            for (int T = 1; T <= 32; ++T) {
                int best = 1, bu = 0;
                for (int G = 1; G <= 32 && T * G <= 32 * (w + 1); ++G) {
                    const int U = T * G;
                    const int u = (U << 10) / (32 * ((U + 31) >> 5));   // busy fraction, fixed point
                    if (u > bu) { bu = u; best = G; }
                }
                g[w][T] = (unsigned char)best;
            }
    }
};
static __constant__ const PartTable c_parts{};

// KM (kernel): 0 Plummer's (eps2); 1 the spline of support hs (ogx_softening.cuh);
// 2 (FP32) the spline minus the Newtonian kernel, zero from hs on (the far field's pairs
// inside the support, OGX_SOFT_SPLINE)
// The G parts of a staged round: part p holds sources p, p + G, ...; S slots per part (4 mod 8,
// so that the 16-byte loads of up to eight parts meet different banks)
struct Parts {
    int G, S;
    unsigned inv;   // x / G = x * inv >> 16 for x < NEAR_CAP
    __device__ __forceinline__ explicit Parts(int g) : G(g), S((((NEAR_CAP + g - 1) / g + 3) & ~7) + 4), inv((65536u + g - 1) / g) {}
    __device__ __forceinline__ int div(int q) const { return (int)((unsigned)q * inv >> 16); }
    __device__ __forceinline__ int count(int p, int n) const { return n > p ? div(n - p - 1) + 1 : 0; }
};

template <class T>
struct NearPrm {
    T eps2, hs, hinv;
};

// ---- FP32 ----
struct Near32 {
    using T = float;
    struct Bodies { const float4 *hi, *lo; };
    // hi x, y, z, lo x, y, z, mass; a part's sources lie one after another (G S <= 252 slots for the G of the table)
    struct alignas(16) Stage { float v[7][256]; };
    struct Target { float h[3], l[3]; };
    struct Acc { float s[4], c[4]; };

    __device__ static __forceinline__ void put(Stage& st, const Parts& pa, const Bodies& b, int q, int j) {
        const float4 h = b.hi[j], l = b.lo[j];
        const int i = pa.div(q), e = (q - i * pa.G) * pa.S + i;
        st.v[0][e] = h.x; st.v[1][e] = h.y; st.v[2][e] = h.z;
        st.v[3][e] = l.x; st.v[4][e] = l.y; st.v[5][e] = l.z;
        st.v[6][e] = h.w;
    }
    // every part up to a multiple of 4: no mass, far away on every axis.  (A target at exactly that
    // point would make 0 / 0 of it; on the x axis alone a pair at +-float(1e18) did.)
    __device__ static __forceinline__ void pad(Stage& st, const Parts& pa, int n, int lane) {
        for (int i = lane; i < 4 * pa.G; i += 32) {
            const int p = i >> 2, c = pa.count(p, n), k = (c & ~3) + (i & 3);
            if ((c & 3) && k >= c) {
#pragma unroll
                for (int a = 0; a < 7; ++a) st.v[a][p * pa.S + k] = a == 0 ? 1.0e18f : a == 1 ? 1.1e18f : a == 2 ? 1.3e18f : 0.f;
            }
        }
    }
    __device__ static __forceinline__ Target target(const Bodies& b, int i) {
        const float4 h = b.hi[i], l = b.lo[i];
        return Target{{h.x, h.y, h.z}, {l.x, l.y, l.z}};
    }
    __device__ static __forceinline__ void clear(Acc& a) {
#pragma unroll
        for (int k = 0; k < 4; ++k) a.s[k] = a.c[k] = 0.f;
    }
    __device__ static __forceinline__ double total(const Acc& a, int k) { return (double)a.s[k] - (double)a.c[k]; }

    // the sources of one part of a round of n, in order; SELF: staged position self_q is the target
    template <bool SELF, bool POT, int KM>
    __device__ static __forceinline__ void round(const Stage& st, const Parts& pa, int part, int n, int self_q, const Target& t,
                                                 const NearPrm<float>& pr, Acc& acc) {
        float a[4] = {0.f, 0.f, 0.f, 0.f};
        const int quads = (pa.count(part, n) + 3) >> 2, first = part * pa.S >> 2;
        int self = -1;   // the target's place in this part
        if (SELF && self_q >= 0 && self_q < n) {
            const int i = pa.div(self_q);
            if (self_q - i * pa.G == part) self = i;
        }
        if constexpr (KM == 0) {
            f2 nh[3], nl[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                nh[k] = pack2(-t.h[k], -t.h[k]);
                nl[k] = pack2(-t.l[k], -t.l[k]);
            }
            const f2 e2 = pack2(pr.eps2, pr.eps2);
            for (int i = 0; i < quads; ++i) {
                ulonglong2 s[7];
#pragma unroll
                for (int k = 0; k < 7; ++k) s[k] = reinterpret_cast<const ulonglong2*>(st.v[k])[first + i];
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    f2 d[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        d[k] = add2(add2(f2{p ? s[k].y : s[k].x}, nh[k]), add2(f2{p ? s[k + 3].y : s[k + 3].x}, nl[k]));
                    const f2 r2 = fma2(d[0], d[0], fma2(d[1], d[1], fma2(d[2], d[2], e2)));
                    // rsqrtf alone (within 2 ulp): its error, ~1e-7 per pair in random directions,
                    // stays far below the form's budget
                    float y0, y1, w0, w1, m0, m1;
                    unpack2(r2, y0, y1);
                    y0 = rsqrtf(y0);
                    y1 = rsqrtf(y1);
                    if (SELF) {
                        if (4 * i + 2 * p == self) y0 = 0.f;
                        if (4 * i + 2 * p + 1 == self) y1 = 0.f;
                    }
                    const f2 y = pack2(y0, y1);
                    const f2 my = mul2(f2{p ? s[6].y : s[6].x}, y);
                    unpack2(mul2(mul2(my, y), y), w0, w1);
                    // the sums take the sources one by one, in order
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        float d0, d1;
                        unpack2(d[k], d0, d1);
                        a[k] = fmaf(w1, d1, fmaf(w0, d0, a[k]));
                    }
                    if (POT) {
                        unpack2(my, m0, m1);
                        a[3] = (a[3] + m0) + m1;
                    }
                }
            }
        } else {
            for (int i = 0; i < quads; ++i) {
                float4 s[7];
#pragma unroll
                for (int k = 0; k < 7; ++k) s[k] = reinterpret_cast<const float4*>(st.v[k])[first + i];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    auto el = [&](int k) { return u == 0 ? s[k].x : u == 1 ? s[k].y : u == 2 ? s[k].z : s[k].w; };
                    const float dx = (el(0) - t.h[0]) + (el(3) - t.l[0]);
                    const float dy = (el(1) - t.h[1]) + (el(4) - t.l[1]);
                    const float dz = (el(2) - t.h[2]) + (el(5) - t.l[2]);
                    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
                    const float mq = el(6);
                    if constexpr (KM == 1) {
                        const bool me = SELF && 4 * i + u == self;
                        float g, k;
                        spline_gk<float>(me ? 1.0f : r2, pr.hs, pr.hinv, g, k);
                        const float m = me ? 0.0f : mq;
                        const float w = m * g;
                        a[0] = fmaf(w, dx, a[0]);
                        a[1] = fmaf(w, dy, a[1]);
                        a[2] = fmaf(w, dz, a[2]);
                        if (POT) a[3] = fmaf(m, k, a[3]);
                    } else if (r2 < pr.hs * pr.hs && r2 > 0.0f) {
                        float g, k;
                        spline_gk<float>(r2, pr.hs, pr.hinv, g, k);
                        const float y = rsqrtf(r2);
                        const float w = mq * (g - y * y * y);
                        a[0] = fmaf(w, dx, a[0]);
                        a[1] = fmaf(w, dy, a[1]);
                        a[2] = fmaf(w, dz, a[2]);
                        if (POT) a[3] = fmaf(mq, k - y, a[3]);
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < 3 || POT) kahan_add(acc.s[k], acc.c[k], a[k]);
    }
};

// ---- FP64 ----
struct Near64 {
    using T = double;
    struct Bodies { const double *x, *y, *z, *m; };
    struct alignas(16) Stage { double2 xy[NEAR_CAP], zm[NEAR_CAP]; };
    struct Target { double x, y, z; };
    struct Acc { double s[4]; };

    __device__ static __forceinline__ void put(Stage& st, const Parts&, const Bodies& b, int q, int j) {
        st.xy[q] = make_double2(__ldg(b.x + j), __ldg(b.y + j));
        st.zm[q] = make_double2(__ldg(b.z + j), __ldg(b.m + j));
    }
    __device__ static __forceinline__ void pad(Stage&, const Parts&, int, int) {}
    __device__ static __forceinline__ Target target(const Bodies& b, int i) { return Target{b.x[i], b.y[i], b.z[i]}; }
    __device__ static __forceinline__ void clear(Acc& a) {
#pragma unroll
        for (int k = 0; k < 4; ++k) a.s[k] = 0.0;
    }
    __device__ static __forceinline__ double total(const Acc& a, int k) { return a.s[k]; }

    template <bool SELF, bool POT, int KM>
    __device__ static __forceinline__ void round(const Stage& st, const Parts& pa, int part, int n, int self_q, const Target& t,
                                                 const NearPrm<double>& pr, Acc& acc) {
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        if constexpr (KM == 0) {
#pragma unroll 4
            for (int q = part; q < n; q += pa.G) {
                if (SELF && q == self_q) continue;
                const double2 p = st.xy[q], r = st.zm[q];
                pair64<POT>(p.x - t.x, p.y - t.y, r.x - t.z, r.y, pr.eps2, a);
            }
            if (!sums_finite<POT>(a)) {
                a[0] = a[1] = a[2] = a[3] = 0.0;
                for (int q = part; q < n; q += pa.G) {
                    if (SELF && q == self_q) continue;
                    const double2 p = st.xy[q], r = st.zm[q];
                    pair64_exact<POT>(p.x - t.x, p.y - t.y, r.x - t.z, r.y, pr.eps2, a);
                }
            }
        } else {
            static_assert(KM == 1, "the plain form corrects the far field in k_soft_correct");
            for (int q = part; q < n; q += pa.G) {
                if (SELF && q == self_q) continue;
                const double2 p = st.xy[q], r = st.zm[q];
                const double dx = p.x - t.x, dy = p.y - t.y, dz = r.x - t.z;
                double g, k;
                spline_gk<double>(dx * dx + dy * dy + dz * dz, pr.hs, pr.hinv, g, k);
                const double w = r.y * g;
                a[0] = fma(w, dx, a[0]);
                a[1] = fma(w, dy, a[1]);
                a[2] = fma(w, dz, a[2]);
                if (POT) a[3] = fma(r.y, k, a[3]);
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) acc.s[k] += a[k];
    }
};

// KM = 2: the leaf's S list in place of its U list (no self round), the result added to
// near[] rather than stored.  Output: near[4 i] = (sum m d / r^3 xyz, sum m / r) of sorted
// body i, FP64.  The kernel needs only the tree and the lists, so in the mixed form it runs
// beside the far-field chain.
template <class N, bool POT, int NU, int KM = 0>
__global__ void __launch_bounds__(32, sizeof(typename N::T) == 4 ? 28 : 20)
    k_leaf_near(TreeView tv, const int64_t* __restrict__ chunk_off, typename N::Bodies bod, NearPrm<typename N::T> pr,
                double* __restrict__ near) {
    constexpr int R = NU / 32;
    static_assert(R * 32 == NU && R >= 1 && R <= 2, "near-field units: 32 or 64");
    __shared__ typename N::Stage st;
    __shared__ double s_red[NU][4];
    const int lane = threadIdx.x & 31;
    if (tv_over(tv)) return;
    const int64_t items = chunk_off[tv.nleaf];
    for (int64_t w = blockIdx.x; w < items; w += gridDim.x) {
        // the leaf of item w: chunk_off[lf] <= w < chunk_off[lf + 1] (warp-uniform search)
        int lo = 0, hi = tv.nleaf;
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (chunk_off[mid] <= w) lo = mid;
            else hi = mid;
        }
        const int lf = lo;
        const int b = tv.leafbox[lf];
        const int f0 = tv.pfirst[b], cnt = tv.pcount[b];
        const int64_t u0 = KM == 2 ? tv.s_off[lf] : tv.u_off[lf], u1 = KM == 2 ? tv.s_off[lf + 1] : tv.u_off[lf + 1];
        if (KM == 2 && u0 == u1) continue;
        const int j0 = 32 * (int)(w - chunk_off[lf]);
        const int T = min(32, cnt - j0);
        const int G = c_parts.g[NU / 32 - 1][T];
        const int U = T * G;
        const Parts pa(G);
        // the lane's units: target tt[r] (index in the leaf), source part pp[r]
        int tt[R], pp[R];
        bool act[R];
        typename N::Target tg[R];
        typename N::Acc acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int u = lane + 32 * r;
            act[r] = u < U;
            tt[r] = act[r] ? u % T : 0;
            pp[r] = act[r] ? u / T : 0;
            tg[r] = N::target(bod, f0 + j0 + tt[r]);
            N::clear(acc[r]);
        }
        // round 0: the leaf itself
        for (int k0 = 0; k0 < (KM == 2 ? 0 : cnt); k0 += NEAR_CAP) {
            const int n = min(NEAR_CAP, cnt - k0);
            __syncwarp();
            for (int q = lane; q < n; q += 32) N::put(st, pa, bod, q, f0 + k0 + q);
            N::pad(st, pa, n, lane);
            __syncwarp();
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (act[r]) N::template round<true, POT, KM>(st, pa, pp[r], n, j0 + tt[r] - k0, tg[r], pr, acc[r]);
        }
        // the other U-list entries, 32 at a time: lane e holds entry e's first body and
        // count; an inclusive scan of the counts maps a flat source position to its entry
        for (int64_t eb = u0; eb < u1; eb += 32) {
            const int64_t e = eb + lane;
            int pf = 0, pc = 0;
            if (e < u1) {
                const int c = KM == 2 ? tv.s_idx[e] : tv.u_idx[e];
                if (c != b) { pf = tv.pfirst[c]; pc = tv.pcount[c]; }
            }
            int pre = pc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, pre, o);
                if (lane >= o) pre += v;
            }
            const int total = __shfl_sync(0xffffffffu, pre, 31);
            for (int base = 0; base < total; base += NEAR_CAP) {
                const int n = min(NEAR_CAP, total - base);
                __syncwarp();
                // warp-uniform trip count: every lane takes part in every shuffle
                for (int q0 = 0; q0 < n; q0 += 32) {
                    const int q = q0 + lane;
                    const int f = base + q;
                    // entry of flat position f: the number of entries whose inclusive
                    // prefix is <= f (five halving steps over the 32 prefixes)
                    int pos = 0;
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1)
                        if (__shfl_sync(0xffffffffu, pre, pos + step - 1) <= f) pos += step;
                    const int ep = __shfl_sync(0xffffffffu, pre, pos), ec = __shfl_sync(0xffffffffu, pc, pos);
                    const int j = __shfl_sync(0xffffffffu, pf, pos) + f - (ep - ec);
                    if (q < n) N::put(st, pa, bod, q, j);
                }
                N::pad(st, pa, n, lane);
                __syncwarp();
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if (act[r]) N::template round<false, POT, KM>(st, pa, pp[r], n, -1, tg[r], pr, acc[r]);
            }
        }
        // the parts of every target, in part order, in FP64
        __syncwarp();
#pragma unroll
        for (int r = 0; r < R; ++r)
            if (act[r])
#pragma unroll
                for (int k = 0; k < 4; ++k) s_red[lane + 32 * r][k] = N::total(acc[r], k);
        __syncwarp();
        if (lane < T) {
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            for (int p = 0; p < G; ++p)
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] += s_red[p * T + lane][k];
            double2* o = reinterpret_cast<double2*>(near + 4 * (size_t)(f0 + j0 + lane));
            if (KM == 2) {
                const double2 o0 = o[0], o1 = o[1];
                o[0] = make_double2(o0.x + v[0], o0.y + v[1]);
                o[1] = make_double2(o1.x + v[2], o1.y + (POT ? v[3] : 0.0));
            } else {
                o[0] = make_double2(v[0], v[1]);
                o[1] = make_double2(v[2], POT ? v[3] : 0.0);
            }
        }
        __syncwarp();
    }
}

}  // namespace near_field
}  // namespace ogx
