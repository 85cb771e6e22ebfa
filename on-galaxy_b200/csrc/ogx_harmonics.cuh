// ogx_harmonics.cuh -- solid-harmonic constants and the layout of expansion coefficients.
//
// The reference evaluates Y_n^m through cos/sin/atan2 and the seminormalised
// Legendre recurrence (src3d/FmmExpansions3D.hpp:75-107) and multiplies by
// rho^n or rho^-(n+1) afterwards.  As solid harmonics in Cartesian form the same
// functions are
//   R_n^m = rho^n Y_n^m:           R_m^m = (x+iy) a_m R_{m-1}^{m-1}
//                                  R_{m+1}^m = z b_m R_m^m
//                                  R_n^m = z A_nm R_{n-1}^m - r^2 B_nm R_{n-2}^m
//   S_n^m = Y_n^m / rho^{n+1}:     same recurrences with a factor 1/r^2 per step
// with a_m = sqrt((2m-1)/2m), b_m = sqrt(2m+1), A_nm = (2n-1)/sqrt(n^2-m^2),
// B_nm = sqrt((n-1)^2-m^2)/sqrt(n^2-m^2): the reference's Q recurrence
// multiplied through by rho^n e^{i m phi} (no trigonometric calls).  The kernels take them
// as R_n^m = s_nm (x+iy)^m T_nm with real polynomials T_nm of leading coefficient 1
// (ogx_far.cuh, ogx_p2x.cuh); only the products s_nm of a, b and A are kept here.
//
// Real coefficient layout (K = (p+1)^2 doubles): dof(n,0) = n^2,
// dof(n,m>0) = n^2 + 2m - 1 (real part), n^2 + 2m (imaginary part).
// Negative orders follow from c_n^{-m} = conj(c_n^m) for real sources.
#pragma once

#include <cmath>
#include <mutex>

#include "ogx_internal.cuh"

namespace ogx {

constexpr int kTab = kDegMax + 2;

struct HarmTables {
    // gradient-coefficient constants (derivative recurrences of FmmExpansions3D.hpp:111-129)
    double gz[kTab][kTab], gp[kTab][kTab], gm[kTab][kTab];  // local  -> degree n (from degree n+1)
    double hz[kTab][kTab], hp[kTab][kTab], hm[kTab][kTab];  // mpole  -> degree n (from degree n-1)
    // R_n^m = s[n][m] (x+iy)^m T_nm: the product of the recurrence constants a, b, A (ogx_far.cuh)
    double s[kTab][kTab];
    // the same per real dof, negative for imaginary parts (conjugate sums, ogx_p2x.cuh)
    double sd[(kPMax + 1) * (kPMax + 1)];
};

// the reference's derivative coefficients (FmmExpansions3D.hpp:111-129)
inline double ref_cz_R(int n, int m) { return std::sqrt(double(n * n - m * m)); }
inline double ref_cp_R(int n, int m) { return ((m >= 0) ? -1.0 : 1.0) * std::sqrt(double((n - m) * (n - m - 1))); }
inline double ref_cm_R(int n, int m) { return ((m > 0) ? 1.0 : -1.0) * std::sqrt(double((n + m) * (n + m - 1))); }
inline double ref_dz_S(int n, int m) { return -std::sqrt(double((n + 1) * (n + 1) - m * m)); }
inline double ref_dp_S(int n, int m) { return ((m >= 0) ? -1.0 : 1.0) * std::sqrt(double((n + m + 1) * (n + m + 2))); }
inline double ref_dm_S(int n, int m) { return ((m > 0) ? 1.0 : -1.0) * std::sqrt(double((n - m + 1) * (n - m + 2))); }

// One copy per translation unit (whole-program compilation, no device linking);
// every unit that launches harmonic kernels calls harm_tables_ready() first.
// In global memory: the kernels' lanes index them divergently (the constant cache serialises
// lanes that read different addresses).
static __device__ HarmTables g_harm;

static inline void fill_harm_tables(HarmTables& t) {
    t = HarmTables{};
    for (int n = 0; n < kTab; ++n)
        for (int m = 0; m < kTab; ++m) {
            if (m <= n) {
                // G_n^m from L_{n+1}^{m}, L_{n+1}^{m-1}, L_{n+1}^{m+1}
                t.gz[n][m] = ref_cz_R(n + 1, m);
                t.gp[n][m] = ref_cp_R(n + 1, m - 1);
                t.gm[n][m] = ref_cm_R(n + 1, m + 1);
                // H_n^m from M_{n-1}^{m}, M_{n-1}^{m-1}, M_{n-1}^{m+1} (zero where the source order is absent)
                if (n >= 1) {
                    t.hz[n][m] = (m <= n - 1) ? ref_dz_S(n - 1, m) : 0.0;
                    t.hp[n][m] = (std::abs(m - 1) <= n - 1) ? ref_dp_S(n - 1, m - 1) : 0.0;
                    t.hm[n][m] = (m + 1 <= n - 1) ? ref_dm_S(n - 1, m + 1) : 0.0;
                }
            }
        }
    double am = 1.0;
    for (int m = 0; m < kTab; ++m) {
        am *= m > 0 ? std::sqrt((2.0 * m - 1.0) / (2.0 * m)) : 1.0;
        double v = am;
        for (int n = m; n < kTab; ++n) {
            if (n == m + 1) v *= std::sqrt(2.0 * m + 1.0);
            else if (n > m + 1) v *= (2.0 * n - 1.0) / std::sqrt((double)(n * n - m * m));
            t.s[n][m] = v;
        }
    }
    for (int n = 0; n <= kPMax; ++n)
        for (int m = 0; m <= n; ++m) {
            const int d = m == 0 ? n * n : n * n + 2 * m - 1;
            t.sd[d] = t.s[n][m];
            if (m > 0) t.sd[d + 1] = -t.s[n][m];
        }
}

static inline int harm_tables_ready(int device) {
    static std::mutex mu;
    static bool done[64] = {};
    std::lock_guard<std::mutex> lk(mu);
    if (device < 0 || device >= 64) return OGX_ERR_INVALID;
    if (done[device]) return OGX_OK;
    HarmTables t;
    fill_harm_tables(t);
    cudaError_t e = cudaMemcpyToSymbol(g_harm, &t, sizeof(t));
    // the copy from the pageable t may still be in flight on the legacy stream,
    // which the library's non-blocking streams do not wait for
    if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
    if (e != cudaSuccess) {
        set_last_error(OGX_ERR_CUDA, std::string("harmonic tables: ") + cudaGetErrorString(e));
        return OGX_ERR_CUDA;
    }
    done[device] = true;
    return OGX_OK;
}

__host__ __device__ __forceinline__ constexpr int dof_re(int n, int m) { return m == 0 ? n * n : n * n + 2 * m - 1; }

// complex coefficient c_n^m from a real layout (m may be negative)
template <class T>
__device__ __forceinline__ void coef_get(const T* c, int n, int m, T& re, T& im) {
    if (m < -n || m > n || n < 0) { re = 0; im = 0; return; }
    if (m == 0) { re = c[n * n]; im = 0; return; }
    const int am = m < 0 ? -m : m;
    re = c[n * n + 2 * am - 1];
    im = c[n * n + 2 * am];
    if (m < 0) im = -im;
}

}  // namespace ogx
