// ogx_p2x.cuh -- particle -> expansion: P2M of the leaves and P2L over the X lists, float in
// the mixed form and double in the plain form.
//
// P2M (fmm::P2M, src3d/FmmExpansions3D.hpp:148-163):  M'_n^m  = sum q conj(R_n^m(u)), u = (x - c) / side
// P2L (AdaptiveFMM3D::p2lAccum, src3d/AdaptiveFMM3D.hpp:117-128):
//                                                     L'_n^m += sum (q / side) conj(S_n^m(u))
// A harmonic of order m is s_nm D^m T_nm with a complex D and a real polynomial T_nm (the
// recurrences of ogx_far.cuh), so a body adds (q D^m).re T_nm and -(q D^m).im T_nm: five
// operations per (n, m) with the recurrence, where complex harmonics took eight; the
// constants s_nm are applied once to the sums.  Warp per box (one warp per block).  A lane
// holds NB bodies of a chunk at a time (FP32: in f32x2 pairs), walks the columns m and adds
// its bodies' terms of one (n, m) at once, so no lane keeps the K sums (81 registers a lane
// at p = 8, and another kernel that staged whole rows above p = 9); the lanes' sums meet in
// FP64 through shared memory, in FP32 after every 32 bodies of a lane at the latest.
// The bodies of the X list's leaves form one flat sequence (lane e of a group of 32 entries
// holds entry e; a scan of the counts maps positions to entries), so all lanes are busy
// however the leaves are sized and a chunk's loads are in flight together.
#pragma once

#include "ogx_harmonics.cuh"
#include "ogx_packed.cuh"

namespace ogx {
namespace p2x {

__host__ __device__ constexpr double rec_b(int n, int m) {
    return (double)((n - 1) * (n - 1) - m * m) / (double)((2 * n - 1) * (2 * n - 3));
}

// columns of partial sums in shared memory (FP64: the lanes are folded to 8 first; folding the
// FP32 lanes to 16 costs more than the occupancy it buys, 410 -> 471 us on the 1M merger)
template <class T> constexpr int sums() { return sizeof(T) == 4 ? 32 : 8; }

__device__ __forceinline__ f2 vmul(f2 a, f2 b) { return mul2(a, b); }
__device__ __forceinline__ f2 vfma(f2 a, f2 b, f2 c) { return fma2(a, b, c); }
__device__ __forceinline__ double vmul(double a, double b) { return a * b; }
__device__ __forceinline__ double vfma(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ f2 vset(float a, f2*) { return pack2(a, a); }
__device__ __forceinline__ double vset(double a, double*) { return a; }
__device__ __forceinline__ float vsum(f2 a) { return sum2(a); }
__device__ __forceinline__ double vsum(double a) { return a; }
__device__ __forceinline__ f2 vadd(f2 a, f2 b) { return add2(a, b); }
__device__ __forceinline__ double vadd(double a, double b) { return a + b; }

template <class T> struct Vec;
template <> struct Vec<float> { using V = f2; static constexpr int W = 2; };
template <> struct Vec<double> { using V = double; static constexpr int W = 1; };

// A body's offset from the box centre is one FP64 difference, scaled in FP64 and rounded to T
// once: taken from the near field's hi + lo FP32 pairs it carried three FP32 roundings.
template <class T>
struct Center {
    double c[3], inv;
    __device__ __forceinline__ Center(const TreeView& tv, int b) {
#pragma unroll
        for (int a = 0; a < 3; ++a) c[a] = tv.center[4 * (size_t)b + a];
        inv = 1.0 / (2.0 * tv.center[4 * (size_t)b + 3]);
    }
    __device__ __forceinline__ void body(const TreeView& tv, int i, T& x, T& y, T& z, T& q) const {
        x = (T)((tv.px[i] - c[0]) * inv);
        y = (T)((tv.py[i] - c[1]) * inv);
        z = (T)((tv.pz[i] - c[2]) * inv);
        q = (T)tv.pm[i];
    }
};

template <int NV> __device__ __forceinline__ void gather(const float (&x)[2 * NV], f2 (&v)[NV]) {
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = pack2(x[2 * i], x[2 * i + 1]);
}
template <int NV> __device__ __forceinline__ void gather(const double (&x)[NV], double (&v)[NV]) {
#pragma unroll
    for (int i = 0; i < NV; ++i) v[i] = x[i];
}

// adds the terms of this lane's NB bodies (scaled offsets x, y, z, weights q) to its column of
// s_red [K][sums + 1]; FIRST: the first chunk stores instead
template <int P, bool SING, class T, int NB>
__device__ __forceinline__ void add_chunk(const T (&x)[NB], const T (&y)[NB], const T (&z)[NB], const T (&q)[NB], T* s_red, int lane,
                                          bool first) {
    using V = typename Vec<T>::V;
    constexpr int NV = NB / Vec<T>::W, LD = sums<T>() + 1;
    V X[NV], Y[NV], nY[NV], Z[NV], nk[NV], dr[NV], di[NV];
    {
        T a[NB], b[NB], nb[NB], c[NB], k[NB], d[NB];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            T r2 = x[i] * x[i] + y[i] * y[i] + z[i] * z[i], w = q[i];
            a[i] = x[i]; b[i] = y[i]; c[i] = z[i];
            if (SING) {
                T ir;
                if constexpr (sizeof(T) == 4) ir = rsqrtf(r2); else ir = rsqrt(r2);
                w *= ir;
                const T k2 = ir * ir;
                // FP64: 1 / r2 to half an ulp, as in ogx_far.cuh
                if constexpr (sizeof(T) == 8) r2 = fma(k2, fma(-r2, k2, T(1)), k2); else r2 = k2;
                a[i] *= r2; b[i] *= r2; c[i] *= r2;
            }
            nb[i] = -b[i];
            k[i] = -r2;
            d[i] = w;
        }
        gather<NV>(a, X); gather<NV>(b, Y); gather<NV>(nb, nY); gather<NV>(c, Z); gather<NV>(k, nk); gather<NV>(d, dr);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) di[i] = vset(T(0), (V*)nullptr);
    auto put = [&](int dof, V s) {
        T v = vsum(s);
        if constexpr (sizeof(T) == 8) {
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            if (lane >= 8) return;
        }
        T* o = s_red + dof * LD + lane;
        *o = first ? v : *o + v;
    };
#pragma unroll
    for (int m = 0; m <= P; ++m) {
        V t0[NV], t1[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) t1[i] = Z[i];
#pragma unroll
        for (int n = m; n <= P; ++n) {
            V re, im;
            if (n == m) {
                re = dr[0];
                im = di[0];
#pragma unroll
                for (int i = 1; i < NV; ++i) {
                    re = vadd(re, dr[i]);
                    im = vadd(im, di[i]);
                }
            } else {
                if (n >= m + 2) {
                    const V b = vset((T)rec_b(n, m), (V*)nullptr);
#pragma unroll
                    for (int i = 0; i < NV; ++i) {
                        const V bk = vmul(b, nk[i]);
                        const V t = n == m + 2 ? vfma(Z[i], t1[i], bk) : vfma(Z[i], t1[i], vmul(bk, t0[i]));
                        t0[i] = t1[i];
                        t1[i] = t;
                    }
                }
                re = vmul(dr[0], t1[0]);
                im = vmul(di[0], t1[0]);
#pragma unroll
                for (int i = 1; i < NV; ++i) {
                    re = vfma(dr[i], t1[i], re);
                    im = vfma(di[i], t1[i], im);
                }
            }
            put(dof_re(n, m), re);
            if (m > 0) put(dof_re(n, m) + 1, im);
        }
        if (m < P) {
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const V nr = vfma(dr[i], X[i], vmul(di[i], nY[i]));
                di[i] = vfma(dr[i], Y[i], vmul(di[i], X[i]));
                dr[i] = nr;
            }
        }
    }
}

// MODE 0: P2M of leaf t (stored); MODE 1: P2L of box t over its X list (added)
template <int P, int MODE, class T>
__global__ void __launch_bounds__(32) k_p2x(TreeView tv, int ntargets, double* __restrict__ out) {
    constexpr int K = (P + 1) * (P + 1), LD = sums<T>() + 1;
    // bodies of a chunk per lane: leaves hold tens, X lists some hundred
    constexpr int NB = MODE == 0 ? Vec<T>::W : 4 * Vec<T>::W;
    extern __shared__ __align__(16) unsigned char s_p2x[];
    T* s_red = reinterpret_cast<T*>(s_p2x);
    const int lane = threadIdx.x, t = blockIdx.x;
    if (t >= ntargets || t >= (MODE == 0 ? tv_nleaf(tv) : tv_nb(tv)) || tv_over(tv)) return;
    const int b = MODE == 0 ? tv.leafbox[t] : t;
    int64_t e0 = 0, e1 = 1;
    if (MODE == 1) {
        e0 = tv.x_off[b];
        e1 = tv.x_off[b + 1];
        if (e0 == e1) return;
    }
    const Center<T> cen(tv, b);
    bool first = true;
    int cols = sums<T>();   // columns of s_red in use
    // The columns' sums, in FP64: added up at the end, and in FP32 after every 32 bodies of a
    // column too (lane = coefficients lane, lane + 32, ...), so that a chain of FP32 additions
    // is no longer in a leaf of thousands of bodies than in one of a thousand.
    constexpr int NPL = (K + 31) / 32, FLUSH = 32 / NB;
    double sum[NPL];
#pragma unroll
    for (int u = 0; u < NPL; ++u) sum[u] = 0.0;
    auto flush = [&]() {
        __syncwarp();
#pragma unroll
        for (int u = 0; u < NPL; ++u) {
            const int d = lane + 32 * u;
            if (d < K) {
#pragma unroll 8
                for (int r = 0; r < cols; ++r) sum[u] += (double)s_red[d * LD + r];
            }
        }
        __syncwarp();   // the next chunk overwrites the columns
        first = true;
    };
    int held = 0;           // chunks in the columns
    for (int64_t eb = e0; eb < e1; eb += 32) {
        int pf = 0, pc = 0;
        if (MODE == 0) {
            if (lane == 0) { pf = tv.pfirst[b]; pc = tv.pcount[b]; }
        } else if (eb + lane < e1) {
            const int c = tv.x_idx[eb + lane];
            pf = tv.pfirst[c];
            pc = tv.pcount[c];
        }
        int pre = pc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += v;
        }
        const int total = __shfl_sync(0xffffffffu, pre, 31);
        const int f00 = __shfl_sync(0xffffffffu, pf, 0);
        for (int base = 0; base < total; base += 32 * NB) {
            T x[NB], y[NB], z[NB], q[NB];
#pragma unroll
            for (int i = 0; i < NB; ++i) {
                // MODE 0: neighbouring bodies share a lane, so a small leaf uses few columns
                const int f = base + (MODE == 0 ? NB * lane + i : lane + 32 * i);
                int j = f00 + f;
                if (MODE == 1) {
                    // entry of flat position f: the number of entries whose inclusive prefix is <= f
                    int pos = 0;
#pragma unroll
                    for (int step = 16; step > 0; step >>= 1)
                        if (__shfl_sync(0xffffffffu, pre, pos + step - 1) <= f) pos += step;
                    const int ep = __shfl_sync(0xffffffffu, pre, pos), ec = __shfl_sync(0xffffffffu, pc, pos);
                    j = __shfl_sync(0xffffffffu, pf, pos) + f - (ep - ec);
                }
                x[i] = T(1); y[i] = z[i] = q[i] = T(0);
                if (f < total) cen.body(tv, j, x[i], y[i], z[i], q[i]);
            }
            if (MODE == 0 && sizeof(T) == 4 && first) cols = min(sums<T>(), (total + NB - 1) / NB);
            add_chunk<P, MODE == 1, T, NB>(x, y, z, q, s_red, lane, first);
            first = false;
            if (sizeof(T) == 4 && ++held == FLUSH) {
                flush();
                held = 0;
            }
        }
    }
    if (!first) flush();
    const double scale = MODE == 1 ? 1.0 / (2.0 * tv.center[4 * (size_t)b + 3]) : 1.0;
#pragma unroll
    for (int u = 0; u < NPL; ++u) {
        const int d = lane + 32 * u;
        if (d >= K) continue;
        const double v = sum[u] * __ldg(&g_harm.sd[d]);   // s_nm, negative for the imaginary part (the conjugate)
        if (MODE == 0) out[(size_t)b * K + d] = v;
        else out[(size_t)b * K + d] += v * scale;
    }
}
template <int P, class T>
constexpr int p2x_smem() { return (P + 1) * (P + 1) * (sums<T>() + 1) * (int)sizeof(T); }

}  // namespace p2x
}  // namespace ogx
