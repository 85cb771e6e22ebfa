// ogx_direct.cu -- all-pairs direct summation on the GPU (the FP64 oracle path).
//
// Replaces DirectSolver3D::computeAccelerations (src3d/DirectSolver3D.hpp:15-34):
//   a_i = G sum_{j != i} m_j (r_j - r_i) / (|r_j - r_i|^2 + eps^2)^{3/2}
// The reference walks unique pairs i<j and applies Newton's third law; on the
// GPU every target sums its own row (no write conflicts).  The optional potential is
// pot_i = -G sum_{j != i} m_j / sqrt(|d|^2 + eps^2) (Kernel3D.hpp:39-42 per body, without
// the m_i factor).  With OGX_SOFT_SPLINE every pair takes the spline kernel
// (ogx_softening.cuh) instead.
//
// Bound: the FP64 pipe, 16 operations per pair (ogx_pair64.cuh): 16,384 bodies cannot take
// less than 0.23 ms.  One thread per target over all sources (as before) filled 64 of 148
// SMs at 16,384 bodies and 4 at 1,000.  Now a CTA holds 32 targets (lane = target) and its
// 8 warps share the sources; a cluster of up to 8 CTAs shares them further while the
// targets alone do not make DT_CTAS CTAs.  The parts' sums meet in warp and CTA order
// through (distributed) shared memory, so no workspace is needed and the result depends on
// n only.
#include <cooperative_groups.h>

#include "ogx_internal.cuh"
#include "ogx_pair64.cuh"
#include "ogx_softening.cuh"

namespace ogx {
namespace {

namespace cg = cooperative_groups;
constexpr int DT_WARPS = 8;
constexpr int DT_CTAS = 16 * SPLIT_SMS;    // CTAs wanted: 4 waves of 4 per SM

// SOFT: the spline kernel of support hs (ogx_softening.cuh) instead of Plummer's eps2
template <bool POT, bool SOFT>
__global__ void __launch_bounds__(32 * DT_WARPS, 4) k_direct(const double* __restrict__ pos, const double* __restrict__ mass, int64_t n,
                                                            double G, double eps2, double* __restrict__ acc,
                                                            double* __restrict__ pot, double hs, double hinv) {
    __shared__ double2 s_xy[DT_WARPS][32], s_zm[DT_WARPS][32];
    __shared__ double s_part[DT_WARPS][32][4], s_sum[32][4];
    cg::cluster_group cl = cg::this_cluster();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t i = (int64_t)(blockIdx.x / C) * 32 + lane;
    const bool act = i < n;
    const double xi = act ? pos[3 * i] : 0.0, yi = act ? pos[3 * i + 1] : 0.0, zi = act ? pos[3 * i + 2] : 0.0;
    // this warp's sources: whole groups of 32, spread evenly over the cluster's warps
    const int64_t groups = (n + 31) / 32, parts = (int64_t)C * DT_WARPS, me = (int64_t)rank * DT_WARPS + w;
    const int64_t g0 = groups * me / parts, g1 = groups * (me + 1) / parts;
    double sum[4] = {0.0, 0.0, 0.0, 0.0};
    double nx = 0.0, ny = 0.0, nz = 0.0, nm = 0.0;
    auto fetch = [&](int64_t g) {
        const int64_t j = 32 * g + lane;
        const bool ok = g < g1 && j < n;
        nx = ok ? pos[3 * j] : 0.0; ny = ok ? pos[3 * j + 1] : 0.0; nz = ok ? pos[3 * j + 2] : 0.0;
        nm = ok ? mass[j] : 0.0;
    };
    fetch(g0);
    for (int64_t g = g0; g < g1; ++g) {
        __syncwarp();
        s_xy[w][lane] = make_double2(nx, ny);
        s_zm[w][lane] = make_double2(nz, nm);
        __syncwarp();
        fetch(g + 1);
        const int lim = (int)min((int64_t)32, n - 32 * g);
        const int self = (int64_t)(blockIdx.x / C) == g ? lane : -1;   // the group that holds the targets themselves
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        if constexpr (SOFT) {
            for (int k = 0; k < lim; ++k) {
                if (k == self) continue;
                const double2 p = s_xy[w][k], q = s_zm[w][k];
                const double dx = p.x - xi, dy = p.y - yi, dz = q.x - zi;
                double gk, kk;
                spline_gk<double>(dx * dx + dy * dy + dz * dz, hs, hinv, gk, kk);
                const double f = q.y * gk;
                a[0] += f * dx; a[1] += f * dy; a[2] += f * dz;
                if (POT) a[3] += q.y * kk;
            }
        } else {
            if (self < 0) {
#pragma unroll 4
                for (int k = 0; k < lim; ++k) {
                    const double2 p = s_xy[w][k], q = s_zm[w][k];
                    pair64<POT>(p.x - xi, p.y - yi, q.x - zi, q.y, eps2, a);
                }
            } else {
                for (int k = 0; k < lim; ++k) {
                    const double2 p = s_xy[w][k], q = s_zm[w][k];
                    if (k != self) pair64<POT>(p.x - xi, p.y - yi, q.x - zi, q.y, eps2, a);
                }
            }
            if (!sums_finite<POT>(a)) {
                a[0] = a[1] = a[2] = a[3] = 0.0;
                for (int k = 0; k < lim; ++k) {
                    const double2 p = s_xy[w][k], q = s_zm[w][k];
                    if (k != self) pair64_exact<POT>(p.x - xi, p.y - yi, q.x - zi, q.y, eps2, a);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) sum[q] += a[q];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) s_part[w][lane][q] = sum[q];
    __syncthreads();
    const int t = threadIdx.x;
    if (t < 128) {
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < DT_WARPS; ++k) v += (&s_part[k][0][0])[t];
        (&s_sum[0][0])[t] = v;
    }
    cl.sync();
    if (rank == 0 && t < 128) {
        double v = 0.0;
        for (int c = 0; c < C; ++c) v += cl.map_shared_rank(&s_sum[0][0], c)[t];
        const int64_t o = (int64_t)(blockIdx.x / C) * 32 + (t >> 2);
        if (o < n) {
            if ((t & 3) < 3) acc[3 * o + (t & 3)] = G * v;
            else if (POT) pot[o] = -(G * v);
        }
    }
    cl.sync();   // a CTA's sums are read before it exits
}

template <bool POT, bool SOFT>
int launch(const double* d_pos, const double* d_mass, int64_t n, double G, double eps2, double* d_acc, double* d_pot, double hs,
           double hinv, cudaStream_t st) {
    const int64_t blocks = (n + 31) / 32;
    int c = 1;
    while (c < 8 && blocks * c < DT_CTAS && (int64_t)c * DT_WARPS * 2 <= blocks) c *= 2;   // at least one group per warp
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(blocks * c));
    cfg.blockDim = dim3(32 * DT_WARPS);
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = c;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    OGX_CUDA(cudaLaunchKernelEx(&cfg, k_direct<POT, SOFT>, d_pos, d_mass, n, G, eps2, d_acc, d_pot, hs, hinv));
    return OGX_OK;
}

}  // namespace

// FP64 direct sum on caller-provided device buffers and stream (no handle)
int direct_launch(const double* d_pos, const double* d_mass, int64_t n, double G, double eps2, double* d_acc, double* d_pot,
                  cudaStream_t st) {
    if (n == 0) return OGX_OK;
    if (d_pot) return launch<true, false>(d_pos, d_mass, n, G, eps2, d_acc, d_pot, 0.0, 0.0, st);
    return launch<false, false>(d_pos, d_mass, n, G, eps2, d_acc, nullptr, 0.0, 0.0, st);
}

int direct_eval(Handle& h, const double* d_pos, const double* d_mass, int64_t n, double* d_acc, double* d_pot) {
    if (n == 0) return OGX_OK;
    const double eps2 = h.prm.eps * h.prm.eps;
    ++h.launches;
    if (h.prm.softening != OGX_SOFT_SPLINE) return direct_launch(d_pos, d_mass, n, h.prm.G, eps2, d_acc, d_pot, h.stream);
    const double hs = spline_support(h.prm.eps), hinv = hs > 0.0 ? 1.0 / hs : 0.0;
    if (d_pot) return launch<true, true>(d_pos, d_mass, n, h.prm.G, eps2, d_acc, d_pot, hs, hinv, h.stream);
    return launch<false, true>(d_pos, d_mass, n, h.prm.G, eps2, d_acc, nullptr, hs, hinv, h.stream);
}

}  // namespace ogx
