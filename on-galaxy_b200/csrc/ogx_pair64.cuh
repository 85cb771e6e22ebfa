// ogx_pair64.cuh -- the FP64 Plummer pair and its inverse square root.
//
// CUDA's rsqrt(double) costs as much as ten FMAs (1.77e12/s against 18.4e12 FMA/s measured
// on the whole GPU) and was 40% of a pair.  Here y0 = rsqrt.approx.ftz.f64(r2) (the MUFU
// seed, |1 - r2 y0^2| <= 1.9e-6 measured) is refined by the series of (1 - e)^{-1/2} and
// (1 - e)^{-3/2} in e = 1 - r2 y0^2 (binomial series; the first term left out is 5/16 e^3
// and 35/16 e^3, 1.5e-17): 16 FP64 operations per pair instead of about 24.
//
// The series has no special cases: r2 = 0, subnormal or infinite, or an overflow of y^3,
// gives a NaN or an infinity.  Callers sum a tile of sources, and a tile whose sums are not
// all finite is summed again with pair64_exact, which is the previous arithmetic.
#pragma once

namespace ogx {

// acc += m y^3 d, ph += m y with y = (dx^2 + dy^2 + dz^2 + eps2)^{-1/2}
template <bool POT>
__device__ __forceinline__ void pair64(double dx, double dy, double dz, double m, double eps2, double (&a)[4]) {
    const double r2 = fma(dx, dx, fma(dy, dy, fma(dz, dz, eps2)));
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(r2));
    const double s = y0 * y0;
    const double e = fma(-r2, s, 1.0);
    double w;
    if (POT) {
        const double y = fma(y0 * e, fma(e, 0.375, 0.5), y0);
        const double my = m * y;
        w = my * (y * y);
        a[3] += my;
    } else {
        const double u = (m * y0) * s;
        w = fma(u * e, fma(e, 1.875, 1.5), u);
    }
    a[0] = fma(w, dx, a[0]);
    a[1] = fma(w, dy, a[1]);
    a[2] = fma(w, dz, a[2]);
}

template <bool POT>
__device__ __forceinline__ void pair64_exact(double dx, double dy, double dz, double m, double eps2, double (&a)[4]) {
    const double r2 = (dx * dx + dy * dy + dz * dz) + eps2;
    const double ir = rsqrt(r2);
    const double w = m * ir * ir * ir;
    a[0] = fma(w, dx, a[0]);
    a[1] = fma(w, dy, a[1]);
    a[2] = fma(w, dz, a[2]);
    if (POT) a[3] = fma(m, ir, a[3]);
}

// false when some sum is infinite or NaN (x - x is NaN for those)
template <bool POT>
__device__ __forceinline__ bool sums_finite(const double (&a)[4]) {
    double t = (a[0] - a[0]) + (a[1] - a[1]) + (a[2] - a[2]);
    if (POT) t += a[3] - a[3];
    return t == 0.0;
}

}  // namespace ogx
