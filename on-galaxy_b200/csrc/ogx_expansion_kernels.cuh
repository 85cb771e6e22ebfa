// ogx_expansion_kernels.cuh -- particle <-> expansion kernels, templated on the
// arithmetic type T (double for the plain form, float for the mixed form).
// Global-to-box-centre shifts (x - c) are always taken in FP64 and only the
// scaled box-relative coordinate u = (x - c) / side is rounded to T.
#pragma once

#include "ogx_harmonics.cuh"

namespace ogx {

// ---- P2M / P2L: particle -> expansion --------------------------------------------
// MODE 0: P2M for leaf t (fmm::P2M, src3d/FmmExpansions3D.hpp:148-163): store
//         M'_n^m = sum q conj(R_n^m(u)),  u = (x - c)/side.
// MODE 1: P2L for box t over X(t) (AdaptiveFMM3D::p2lAccum, src3d/AdaptiveFMM3D.hpp:117-128):
//         L'_n^m += sum (q/side) conj(S_n^m(u)).
// Warp per target: lanes build the harmonics of 32 sources into shared memory
// (one row each), then every lane sums a few coefficient columns.
template <int P, int MODE, class T>
__global__ void __launch_bounds__(128) k_p2x(TreeView tv, int ntargets, double* out) {
    constexpr int K = (P + 1) * (P + 1);
    constexpr int LD = K | 1;
    extern __shared__ __align__(16) unsigned char s_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int t = blockIdx.x * 4 + wid;
    if (t >= ntargets || t >= (MODE == 0 ? tv_nleaf(tv) : tv_nb(tv)) || tv_over(tv)) return;
    T* buf = reinterpret_cast<T*>(s_raw) + (size_t)wid * 32 * LD;
    const int b = (MODE == 0) ? tv.leafbox[t] : t;
    int64_t e0, e1;
    if (MODE == 0) { e0 = 0; e1 = 1; }
    else { e0 = tv.x_off[b]; e1 = tv.x_off[b + 1]; if (e0 == e1) return; }
    const double cx = tv.center[4 * b], cy = tv.center[4 * b + 1], cz = tv.center[4 * b + 2];
    const double side = 2.0 * tv.center[4 * b + 3], inv = 1.0 / side;
    constexpr int NPL = (K + 31) / 32;
    double acc[NPL];
#pragma unroll
    for (int q = 0; q < NPL; ++q) acc[q] = 0.0;
    for (int64_t e = e0; e < e1; ++e) {
        const int src = (MODE == 0) ? b : tv.x_idx[e];
        const int f0 = tv.pfirst[src], cnt = tv.pcount[src];
        for (int j0 = 0; j0 < cnt; j0 += 32) {
            const int j = j0 + lane;
            T* row = buf + (size_t)lane * LD;
            if (j < cnt) {
                const int i = f0 + j;
                const T q = (T)tv.pm[i];
                const T ux = (T)((tv.px[i] - cx) * inv), uy = (T)((tv.py[i] - cy) * inv), uz = (T)((tv.pz[i] - cz) * inv);
                auto put = [&](int n, int m, T re, T im) {
                    if (m == 0) row[n * n] = q * re;
                    else { row[n * n + 2 * m - 1] = q * re; row[n * n + 2 * m] = -q * im; }
                };
                if (MODE == 0) for_regular<P>(ux, uy, uz, put);
                else for_singular<P>(ux, uy, uz, put);
            } else {
                for (int d = 0; d < K; ++d) row[d] = T(0);
            }
            __syncwarp();
#pragma unroll
            for (int q = 0; q < NPL; ++q) {
                const int d = lane + 32 * q;
                if (d < K) {
                    T s = 0;
#pragma unroll 8
                    for (int r = 0; r < 32; ++r) s += buf[(size_t)r * LD + d];
                    acc[q] += (double)s;
                }
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int q = 0; q < NPL; ++q) {
        const int d = lane + 32 * q;
        if (d < K) {
            if (MODE == 0) out[(size_t)b * K + d] = acc[q];
            else out[(size_t)b * K + d] += acc[q] * inv;
        }
    }
}

template <int P, class T>
constexpr size_t p2x_smem_bytes() {
    return (size_t)4 * 32 * ((P + 1) * (P + 1) | 1) * sizeof(T);
}

}  // namespace ogx
