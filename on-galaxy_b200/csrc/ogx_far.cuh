// ogx_far.cuh -- the leaf far field: L2P and, over the W lists, M2P (float in the mixed
// form, double in the plain form).
//
// Replaces fmm::localField / fmm::multipoleField per body (src3d/FmmExpansions3D.hpp:180-235,
// called in src3d/AdaptiveFMM3D.hpp:92-93).  The gradient of an expansion is a sum of solid
// harmonics with three coefficient sets H^x, H^y, H^z, and a solid harmonic of order m is a
// complex factor of m alone times a REAL polynomial of z and r^2:
//   R_n^m = s_nm (x+iy)^m T_nm(z, r^2)             S_n^m(u) = R_n^m(u / r^2) / r
//   T_mm = 1, T_{m+1,m} = z, T_nm = z T_{n-1,m} - b_nm r^2 T_{n-2,m},
//   b_nm = ((n-1)^2 - m^2) / ((2n-1)(2n-3))        (the recurrences of ogx_harmonics.cuh
// with the constants A_nm collected in s_nm).  The constants s_nm are folded into the
// coefficient records, so per (n, m) an evaluation takes three operations for T_nm and two
// per axis (real and imaginary coefficient); the complex factor is applied once per m.
// With complex harmonics it took six, and an M2P evaluation at p = 8 about 800 instructions.
// In FP32 two columns m, m + 1 go together in packed pairs (f32x2: the FMA pipe's rate at
// half the issue slots): step i of the pair is T_{m+i,m} and T_{m+1+i,m+1}.
// Bound: FP32 issue slots (the records come from shared memory as warp-wide broadcasts).
// M2P + L2P of the 1M merger (p = 8, 14.4M evaluations, serialised): 1.33 -> 0.72 ms; in
// FP64 the 262,144-body galaxy: 1.30 -> 0.41 ms (one warp per leaf had walked the W list
// of a leaf in turn, 199 boxes at most).
#pragma once

#include "ogx_harmonics.cuh"
#include "ogx_packed.cuh"
#include "ogx_sm100.cuh"

namespace ogx {
namespace far {

// largest degree of a record: M2P gradients reach P + 1, L2P gradients P - 1 (potential P)
template <int P, int MODE, bool POT>
constexpr int rec_degree() { return MODE == 0 ? P + 1 : (POT ? P : P - 1); }

// values of a record: FP32 steps of column pairs (12 or 16 floats), FP64 entries per (n, m)
// column by column (6 or 8 doubles): {gx.re, gx.im, gy.re, gy.im, gz.re, gz.im(, phi.re, phi.im)}
template <class T, int L, bool POT>
struct Rec {
    static constexpr bool PAIR = sizeof(T) == 4;
    static constexpr int V = POT ? 8 : 6;
    static constexpr int entries() {
        if (!PAIR) return (L + 1) * (L + 2) / 2;
        int s = 0;
        for (int m = 0; m <= L; m += 2) s += L - m + 1;
        return s;
    }
    static constexpr int STEPS = entries();
    static constexpr int SIZE = STEPS * V * (PAIR ? 2 : 1);      // values of T
    static constexpr int F4 = SIZE * (int)sizeof(T) / 16;        // 16-byte pieces
    static_assert(SIZE * sizeof(T) % 16 == 0, "records are copied in 16-byte pieces");
};

// Both parts (re, im) of entry (n, m) of a gradient coefficient set (FmmExpansions3D.hpp:111-129)
//   MODE 0: multipole set H from M_{n-1} (dz_S / dp_S / dm_S)
//   MODE 1: local set G from L_{n+1}     (cz_R / cp_R / cm_R)
// (constants from global memory: the lanes hold different (n, m))
template <int MODE>
__device__ __forceinline__ void grad_entry(const double* c, int n, int m, double gr[3], double gi[3]) {
    if (MODE == 0 && n == 0) return;
    const int N = MODE == 0 ? n - 1 : n + 1;
    double lr, li, pr, pi, mr, mi;
    coef_get(c, N, m, lr, li);
    coef_get(c, N, m - 1, mr, mi);
    coef_get(c, N, m + 1, pr, pi);
    const double cz = __ldg(MODE == 0 ? &g_harm.hz[n][m] : &g_harm.gz[n][m]);
    const double cp = __ldg(MODE == 0 ? &g_harm.hp[n][m] : &g_harm.gp[n][m]);
    const double cm = __ldg(MODE == 0 ? &g_harm.hm[n][m] : &g_harm.gm[n][m]);
    const double xr = 0.5 * (cp * mr + cm * pr), xi = 0.5 * (cp * mi + cm * pi);
    const double dr = cp * mr - cm * pr, di = cp * mi - cm * pi;
    gr[0] = xr; gr[1] = 0.5 * di; gr[2] = cz * lr;
    if (m > 0) { gi[0] = xi; gi[1] = -0.5 * dr; gi[2] = cz * li; }
}

// Coefficient records, warp per box (MODE 0, boxes of some W list) or leaf (MODE 1).  The
// weights are folded in (m = 0: (c.re, 0); m > 0: (2 c.re, -2 c.im)), so that
// sum_nm Re(c_nm z_nm) = sum re' z.re + im' z.im.
template <int P, int MODE, bool POT, class T>
__global__ void __launch_bounds__(128) k_far_rec(TreeView tv, int count, const double* __restrict__ coef, T* __restrict__ rec) {
    constexpr int K = (P + 1) * (P + 1), L = rec_degree<P, MODE, POT>();
    using R = Rec<T, L, POT>;
    const int lane = threadIdx.x & 31;
    const int k = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (k >= count || k >= (MODE == 0 ? tv_nb(tv) : tv_nleaf(tv)) || tv_over(tv)) return;
    const int b = (MODE == 0) ? k : tv.leafbox[k];
    if (MODE == 0 && tv.x_off[b] == tv.x_off[b + 1]) return;   // never an M2P source
    const double* c = coef + (size_t)b * K;
    T* o = rec + (size_t)k * R::SIZE;
    for (int e = lane; e < R::STEPS * (R::PAIR ? 2 : 1); e += 32) {
        // entry e: column m, step i (n = m + i); FP32: half of column pair m0
        const int half = R::PAIR ? (e & 1) : 0;
        int i = R::PAIR ? (e >> 1) : e, m = 0;
        while (i > L - m) { i -= L - m + 1; m += R::PAIR ? 2 : 1; }
        m += half;
        const int n = m + i;
        double gr[3] = {0.0, 0.0, 0.0}, gi[3] = {0.0, 0.0, 0.0}, pr = 0.0, pi = 0.0;
        if (n <= L) {
            if (MODE == 0 || n < P) grad_entry<MODE>(c, n, m, gr, gi);
            if (POT && n <= P) {
                pr = c[dof_re(n, m)];
                if (m > 0) pi = c[dof_re(n, m) + 1];
            }
        }
        const double s = n <= L ? __ldg(&g_harm.s[n][m]) : 0.0;
        const double wr = m == 0 ? s : 2.0 * s, wi = m == 0 ? 0.0 : -2.0 * s;
        const double v[8] = {wr * gr[0], wi * gi[0], wr * gr[1], wi * gi[1], wr * gr[2], wi * gi[2], wr * pr, wi * pi};
        constexpr int ST = R::PAIR ? 2 : 1;
        T* q = o + (size_t)(R::PAIR ? (e >> 1) : e) * R::V * ST + half;
#pragma unroll
        for (int a = 0; a < R::V; ++a) q[a * ST] = (T)v[a];
    }
}

__host__ __device__ constexpr double rec_b(int n, int m) {
    return (double)((n - 1) * (n - 1) - m * m) / (double)((2 * n - 1) * (2 * n - 3));
}

// out[k] = {sum_axis x, y, z(, phi)} of NB bodies at scaled offsets (x, y, z)[k] for a record
// in shared memory, read once for all of them; SING: singular harmonics (M2P), else regular
// (L2P)
template <int L, bool POT, bool SING, int NB>
__device__ __forceinline__ void eval(const float4* rec, float (&x)[NB], float (&y)[NB], float (&z)[NB], float (&out)[NB][4]) {
    using R = Rec<float, L, POT>;
    f2 z2[NB], nk2[NB], qr2[NB], qi2[NB], nqi2[NB], dr[NB], di[NB], o[NB][4];
#pragma unroll
    for (int k = 0; k < NB; ++k) {
        float kap = x[k] * x[k] + y[k] * y[k] + z[k] * z[k], d0 = 1.f;
        if (SING) {
            d0 = rsqrtf(kap);
            kap = d0 * d0;
            x[k] *= kap; y[k] *= kap; z[k] *= kap;
        }
        z2[k] = pack2(z[k], z[k]);
        nk2[k] = pack2(-kap, -kap);
        // (x + iy)^2 carries a column pair to the next
        const float qr = x[k] * x[k] - y[k] * y[k], qi = 2.f * x[k] * y[k];
        qr2[k] = pack2(qr, qr);
        qi2[k] = pack2(qi, qi);
        nqi2[k] = pack2(-qi, -qi);
        dr[k] = pack2(d0, d0 * x[k]);
        di[k] = pack2(0.f, d0 * y[k]);
#pragma unroll
        for (int a = 0; a < 4; ++a) o[k][a].v = 0ull;
    }
    const ulonglong2* r = reinterpret_cast<const ulonglong2*>(rec);
    int e = 0;
#pragma unroll
    for (int m = 0; m <= L; m += 2) {
        f2 s[NB][R::V], t0[NB], t1[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) {
            t0[k] = pack2(1.f, 1.f);
            t1[k] = z2[k];
        }
#pragma unroll
        for (int i = 0; i <= L - m; ++i, ++e) {
            f2 c[R::V];
#pragma unroll
            for (int a = 0; a < R::V / 2; ++a) {
                const ulonglong2 w = r[e * (R::V / 2) + a];
                c[2 * a].v = w.x;
                c[2 * a + 1].v = w.y;
            }
#pragma unroll
            for (int k = 0; k < NB; ++k) {
                if (i == 0) {
#pragma unroll
                    for (int a = 0; a < R::V; ++a) s[k][a] = c[a];
                    continue;
                }
                f2 t = t1[k];
                if (i >= 2) {
                    const f2 b = pack2((float)rec_b(m + i, m), (float)rec_b(m + 1 + i, m + 1));
                    t = fma2(z2[k], t1[k], mul2(mul2(b, nk2[k]), t0[k]));
                    t0[k] = t1[k];
                    t1[k] = t;
                }
#pragma unroll
                for (int a = 0; a < R::V; ++a) s[k][a] = fma2(c[a], t, s[k][a]);
            }
        }
#pragma unroll
        for (int k = 0; k < NB; ++k) {
#pragma unroll
            for (int a = 0; a < R::V / 2; ++a) o[k][a] = fma2(s[k][2 * a], dr[k], fma2(s[k][2 * a + 1], di[k], o[k][a]));
            if (m + 2 <= L) {
                const f2 nr = fma2(dr[k], qr2[k], mul2(di[k], nqi2[k]));
                di[k] = fma2(dr[k], qi2[k], mul2(di[k], qr2[k]));
                dr[k] = nr;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NB; ++k)
#pragma unroll
        for (int a = 0; a < 4; ++a) out[k][a] = a < R::V / 2 ? sum2(o[k][a]) : 0.f;
}

template <int L, bool POT, bool SING, int NB>
__device__ __forceinline__ void eval(const float4* rec, double (&xs)[NB], double (&ys)[NB], double (&zs)[NB], double (&outs)[NB][4]) {
    static_assert(NB == 1, "the FP64 pipe, not the records' reads, bounds this form");
    using R = Rec<double, L, POT>;
    double x = xs[0], y = ys[0], z = zs[0], (&out)[4] = outs[0];
    double kap = x * x + y * y + z * z, dr = 1.0, di = 0.0;
    if (SING) {
        const double r2 = kap;
        dr = rsqrt(r2);
        kap = dr * dr;
        kap = fma(kap, fma(-r2, kap, 1.0), kap);   // 1 / r2 to half an ulp: degree n carries its n-th power
        x *= kap; y *= kap; z *= kap;
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) out[a] = 0.0;
    const double2* r = reinterpret_cast<const double2*>(rec);
    int e = 0;
#pragma unroll
    for (int m = 0; m <= L; ++m) {
        double s[R::V], t0 = 1.0, t1 = z;
#pragma unroll
        for (int i = 0; i <= L - m; ++i, ++e) {
            double c[R::V], t = t1;
#pragma unroll
            for (int a = 0; a < R::V / 2; ++a) {
                const double2 w = r[e * (R::V / 2) + a];
                c[2 * a] = w.x;
                c[2 * a + 1] = w.y;
            }
            if (i == 0) {
#pragma unroll
                for (int a = 0; a < R::V; ++a) s[a] = c[a];
                continue;
            }
            if (i >= 2) {
                t = fma(z, t1, -(rec_b(m + i, m) * kap) * t0);
                t0 = t1;
                t1 = t;
            }
#pragma unroll
            for (int a = 0; a < R::V; ++a)
                if (m > 0 || !(a & 1)) s[a] = fma(c[a], t, s[a]);   // order 0 is real
        }
#pragma unroll
        for (int a = 0; a < R::V / 2; ++a) out[a] = fma(s[2 * a], dr, m > 0 ? fma(s[2 * a + 1], di, out[a]) : out[a]);
        if (m < L) {
            const double nr = dr * x - di * y;
            di = dr * y + di * x;
            dr = nr;
        }
    }
}

// ---- tasks: the (NB bodies, W box) pairs of a block of at most 64 bodies, W-major, taken in
// rounds of at most 32 (lane = task).  Heavy
// leaves in FP32 take NB = 2: one read of a record's coefficients serves two bodies (with one
// the shared-memory pipe was 76% busy, the FMA pipe 39%; 1M merger 547 -> 388 us).  A light
// leaf's few tasks then fill 20 lanes of 32 instead of 25 (230 -> 275 us): NB = 1.  A round covers at most RW W boxes, whose records
// one warp stages in shared memory.
template <class T> struct Res;
template <> struct Res<float> { using V = float4; };
template <> struct Res<double> { using V = double4; };

template <class T> constexpr int FAR_HEAVY_NB = sizeof(T) == 4 ? 2 : 1;   // bodies of a heavy leaf's task
constexpr int FAR_RW = 3;          // boxes of a round: 32 tasks, 16 and more per box, span at most 3
constexpr int FAR_HW = 8;          // warps of a heavy leaf's CTA

// Leaves with more M2P tasks (bodies x W boxes) than this are taken by a CTA of FAR_HW
// warps (k_leaf_far_heavy), so that one leaf with a long W list does not decide the
// kernel's length.  That matters while the leaves are fewer than the warps the GPU holds, and
// more in FP64, where a task takes longer.  One evaluation alone, lines 1,024 / 512 / 256 / 128
// (us): 8,192 bodies (516 leaves) 403 / 381 / 373 / 373, 30,011 (1,855) 520 / 513 / 510 / 501;
// FP64, 16,384 bodies (1,009) 964 / 933 / 917 / 913, 60,000 (3,480) 1,532 / 1,510 / 1,490 / 1,478.
// In larger trees the lines 1,024, 512 and 256 lie within 1% of one another (1M merger 3.92 / 3.88 /
// 3.91 ms, 262,144 bodies in FP64 3.31 ms each), and systems that share the GPU do better with
// fewer heavy CTAs (three of 262,144 bodies, order 4: 1.06 ms at 1,024, 1.08 at 512).
template <class T>
__device__ __forceinline__ int64_t heavy_line(const TreeView& tv) { return sizeof(T) == 8 || tv_nleaf(tv) < 4096 ? 256 : 1024; }

// shared memory of one warp
template <int P, bool POT, class T, int NB>
struct alignas(16) WarpSmem {
    static constexpr int RF4 = Rec<T, P + 1, POT>::F4;
    float4 rec[FAR_RW * RF4];
    typename Res<T>::V res[32 * NB];
    double hdr[FAR_RW][4];       // box centre, 1 / side
};

// Positions of a block's bodies.  An offset from a box is one FP64 difference, scaled in FP64
// and rounded to T once: through the leaf's centre it took two roundings, the first
// magnified by the ratio of the sides for a W box many levels below its leaf.
struct Bodies { double x[3][64]; };

// 1 / side of a W box `up` levels below one of 1 / side = v: v * 2^up, exact (a division takes
// thirty operations)
__device__ __forceinline__ double scale2(double v, int up) { return v * __hiloint2double((1023 + up) << 20, 0); }

// results of the bodies j[k] for a W box
template <class T, int L, bool POT, int NB>
__device__ __forceinline__ void m2p_task(const float4* rec, const double (&h)[4], const Bodies& s, const int (&j)[NB],
                                         typename Res<T>::V (&res)[NB]) {
    const T w = (T)h[3], w2 = w * w;
    T u[3][NB], o[NB][4];
#pragma unroll
    for (int k = 0; k < NB; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a) u[a][k] = (T)((s.x[a][j[k]] - h[a]) * h[3]);
    eval<L, POT, true, NB>(rec, u[0], u[1], u[2], o);
#pragma unroll
    for (int k = 0; k < NB; ++k) res[k] = typename Res<T>::V{o[k][0] * w2, o[k][1] * w2, o[k][2] * w2, POT ? o[k][3] * w : T(0)};
}

// The rounds first, first + stride, ... of a block of nbk bodies and nw W boxes; every body
// sums its own task results in task order into acc (FP64; lane owns bodies lane, lane + 32).
template <int P, bool POT, int NB, class T>
__device__ __forceinline__ void m2p_rounds(const TreeView& tv, const T* __restrict__ hrec, int64_t w0, int nw, int nbk, int first,
                                           int stride, const Bodies& sb, double inv, int level,
                                           WarpSmem<P, POT, T, NB>& sm, int lane, double (&acc)[2][4]) {
    using R = Rec<T, P + 1, POT>;
    constexpr int RF4 = R::F4;
    const int nt1 = (nbk + NB - 1) / NB;   // tasks of a box: bodies j, j + nt1, ...
    const int total = nt1 * nw;
    // tasks of a round: at most FAR_RW boxes (whole ones where a box has fewer than 16)
    const int Q = nt1 >= 16 ? 32 : (FAR_RW * nt1 <= 32 ? FAR_RW : FAR_RW - 1) * nt1;
    int b0 = first * Q;
    // this lane's task: box w, first body j
    int w = (b0 + lane) / nt1, j = b0 + lane - w * nt1;
    const int dq = stride * Q / nt1, dr = stride * Q - dq * nt1;
    // the round's boxes wa .. wa + nrec - 1, box index c of lane's one: known a round ahead, so
    // a round waits for its records only
    int nt = min(Q, total - b0), wa = 0, nrec = 0, c = 0;
    auto boxes = [&]() {
        wa = __shfl_sync(0xffffffffu, w, 0);
        nrec = __shfl_sync(0xffffffffu, w, max(nt, 1) - 1) - wa + 1;
        c = (nt > 0 && lane < nrec) ? tv.w_idx[w0 + wa + lane] : 0;
    };
    boxes();
    while (b0 < total) {
        for (int q = 0; q < nrec; ++q) {
            const float4* src = reinterpret_cast<const float4*>(hrec + (size_t)__shfl_sync(0xffffffffu, c, q) * R::SIZE);
#pragma unroll
            for (int i = 0; i < (RF4 + 31) / 32; ++i)
                if (32 * i + lane < RF4) sm100::cp_async16(sm.rec + q * RF4 + 32 * i + lane, src + 32 * i + lane);
        }
        if (lane < nrec) {
            const double2 c01 = __ldg(reinterpret_cast<const double2*>(tv.center) + 2 * (size_t)c);
            const double2 c23 = __ldg(reinterpret_cast<const double2*>(tv.center) + 2 * (size_t)c + 1);
            const int up = __ldg(tv.level + c) - level;
            double* hd = sm.hdr[lane];
            hd[0] = c01.x; hd[1] = c01.y; hd[2] = c23.x; hd[3] = scale2(inv, up);
        }
        const int wr = w - wa, jr = j, ja = __shfl_sync(0xffffffffu, j, 0), ntr = nt;
        b0 += stride * Q;
        w += dq;
        j += dr;
        if (j >= nt1) { j -= nt1; ++w; }
        nt = min(Q, total - b0);
        boxes();   // of the next round
        sm100::cp_async_wait_all();
        __syncwarp();
        if (lane < ntr) {
            int jb[NB];
            typename Res<T>::V v[NB];
#pragma unroll
            for (int k = 0; k < NB; ++k) jb[k] = jr + k * nt1 < nbk ? jr + k * nt1 : jr;
            m2p_task<T, P + 1, POT, NB>(sm.rec + wr * RF4, sm.hdr[wr], sb, jb, v);
#pragma unroll
            for (int k = 0; k < NB; ++k) sm.res[32 * k + lane] = v[k];
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int jo = lane + 32 * q;
            if (jo < nbk) {
                const int half = NB > 1 && jo >= nt1, jt = jo - half * nt1;
                for (int k = jt >= ja ? jt - ja : jt - ja + nt1; k < ntr; k += nt1) {
                    const auto v = sm.res[32 * half + k];
                    acc[q][0] += v.x; acc[q][1] += v.y; acc[q][2] += v.z;
                    if (POT) acc[q][3] += v.w;
                }
            }
        }
        __syncwarp();   // the next round's copies overwrite the records and results
    }
}

// L2P of the block's bodies (lane owns bodies lane and lane + 32)
template <int P, bool POT, class T>
__device__ __forceinline__ void l2p_block(const T* __restrict__ g, int nbk, const Bodies& sb, double cx, double cy, double cz,
                                          double inv, float4* srec, int lane,
                                          double (&acc)[2][4]) {
    constexpr int L = rec_degree<P, 1, POT>();
    using R = Rec<T, L, POT>;
    __syncwarp();
    for (int i = lane; i < R::F4; i += 32) srec[i] = __ldg(reinterpret_cast<const float4*>(g) + i);
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        const int j = lane + 32 * q;
        if (j < nbk) {
            T u[3][1] = {{(T)((sb.x[0][j] - cx) * inv)}, {(T)((sb.x[1][j] - cy) * inv)}, {(T)((sb.x[2][j] - cz) * inv)}}, o[1][4];
            eval<L, POT, false, 1>(srec, u[0], u[1], u[2], o);
            acc[q][0] += (double)o[0][0] * inv;
            acc[q][1] += (double)o[0][1] * inv;
            acc[q][2] += (double)o[0][2] * inv;
            if (POT) acc[q][3] += (double)o[0][3];
        }
    }
    __syncwarp();
}

// Warp per leaf (one warp per block, so a block's resources return as soon as its leaf is
// done), bodies in blocks of 64.  The mixed form runs the two parts apart: M2P (DO_M2P,
// multipoles only) beside the M2L and the downward pass, L2P (DO_L2P) after it.  With
// DO_M2P, heavy leaves are left to k_leaf_far_heavy.
template <int P, bool POT, bool DO_L2P, bool DO_M2P, class T>
__global__ void __launch_bounds__(32, sizeof(T) == 4 ? 20 : 12) k_leaf_far(TreeView tv, const T* __restrict__ hrec,
                                                                           const T* __restrict__ grec, double* __restrict__ far) {
    using GR = Rec<T, rec_degree<P, 1, POT>(), POT>;
    extern __shared__ __align__(16) unsigned char s_far_dyn[];
    __shared__ Bodies sb;
    const int lane = threadIdx.x;
    const int lf = blockIdx.x;
    if (lf >= tv.nleaf || lf >= tv_nleaf(tv) || tv_over(tv)) return;
    const int b = tv.leafbox[lf];
    const int f0 = tv.pfirst[b], cnt = tv.pcount[b];
    const int64_t w0 = DO_M2P ? tv.w_off[lf] : 0;
    const int nw = DO_M2P ? (int)(tv.w_off[lf + 1] - w0) : 0;
    if (DO_M2P && (int64_t)cnt * nw > heavy_line<T>(tv)) return;
    const double cx = tv.center[4 * b], cy = tv.center[4 * b + 1], cz = tv.center[4 * b + 2];
    const double inv = 1.0 / (2.0 * tv.center[4 * b + 3]);
    for (int jb = 0; jb < cnt; jb += 64) {
        const int nbk = min(64, cnt - jb);
        double acc[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
        if (DO_L2P || nw > 0) {
            __syncwarp();
            for (int j = lane; j < nbk; j += 32) {
                const int i = f0 + jb + j;
                sb.x[0][j] = tv.px[i]; sb.x[1][j] = tv.py[i]; sb.x[2][j] = tv.pz[i];
            }
            __syncwarp();
        }
        if constexpr (DO_L2P)
            l2p_block<P, POT, T>(grec + (size_t)lf * GR::SIZE, nbk, sb, cx, cy, cz, inv, reinterpret_cast<float4*>(s_far_dyn), lane, acc);
        if constexpr (DO_M2P)
            if (nw > 0)
                m2p_rounds<P, POT, 1, T>(tv, hrec, w0, nw, nbk, 0, 1, sb, inv, tv.level[b],
                                         *reinterpret_cast<WarpSmem<P, POT, T, 1>*>(s_far_dyn), lane, acc);
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int j = lane + 32 * q;
            if (j < nbk) {
                double2* o = reinterpret_cast<double2*>(far + 4 * (size_t)(f0 + jb + j));
                o[0] = make_double2(acc[q][0], acc[q][1]);
                o[1] = make_double2(acc[q][2], acc[q][3]);
            }
        }
    }
}
// shared memory of k_leaf_far: the M2P stage, or the L2P record
template <int P, bool POT, bool DO_M2P, class T>
constexpr size_t leaf_far_smem() {
    constexpr size_t a = sizeof(float4) * Rec<T, rec_degree<P, 1, POT>(), POT>::F4;
    return DO_M2P ? (sizeof(WarpSmem<P, POT, T, 1>) > a ? sizeof(WarpSmem<P, POT, T, 1>) : a) : a;
}

// list of the heavy leaves (order irrelevant: every leaf's result is computed
// independently); *count zero before the launch
template <class T>
__global__ void k_far_heavy_list(TreeView tv, int* __restrict__ list, int* count) {
    const int lf = blockIdx.x * blockDim.x + threadIdx.x;
    if (lf >= tv.nleaf || lf >= tv_nleaf(tv) || tv_over(tv)) return;
    if ((int64_t)tv.pcount[tv.leafbox[lf]] * (tv.w_off[lf + 1] - tv.w_off[lf]) > heavy_line<T>(tv)) list[atomicAdd(count, 1)] = lf;
}

// Heavy leaves: a CTA of FAR_HW warps per leaf, leaves taken from the list through a shared
// counter (ctr[1], zero before the launch; ctr[0] = list length) so the CTAs balance
// themselves.  Warp w runs the rounds w, w + FAR_HW, ...; warp 0 also the L2P; the warps'
// per-body partial sums are added in warp order through shared memory (deterministic).
template <int P, bool POT, bool DO_L2P, class T>
__global__ void __launch_bounds__(32 * FAR_HW, 2) k_leaf_far_heavy(TreeView tv, const T* __restrict__ hrec,
                                                                                       const T* __restrict__ grec,
                                                                                       double* __restrict__ far,
                                                                                       const int* __restrict__ list, int* ctr) {
    using GR = Rec<T, rec_degree<P, 1, POT>(), POT>;
    extern __shared__ __align__(16) unsigned char s_far_dyn[];
    __shared__ Bodies sb;
    __shared__ int s_lf;
    double* s_part = reinterpret_cast<double*>(s_far_dyn);   // [FAR_HW][64][4], over the records once the rounds are done
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    using Smem = WarpSmem<P, POT, T, FAR_HEAVY_NB<T>>;
    Smem& sm = reinterpret_cast<Smem*>(s_far_dyn)[wid];
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            const int k = atomicAdd(&ctr[1], 1);
            s_lf = (k < ctr[0]) ? list[k] : -1;
        }
        __syncthreads();
        const int lf = s_lf;
        if (lf < 0) return;
        const int b = tv.leafbox[lf];
        const int f0 = tv.pfirst[b], cnt = tv.pcount[b];
        const int64_t w0 = tv.w_off[lf];
        const int nw = (int)(tv.w_off[lf + 1] - w0);
        const double cx = tv.center[4 * b], cy = tv.center[4 * b + 1], cz = tv.center[4 * b + 2];
        const double inv = 1.0 / (2.0 * tv.center[4 * b + 3]);
        for (int jb = 0; jb < cnt; jb += 64) {
            const int nbk = min(64, cnt - jb);
            __syncthreads();
            for (int j = threadIdx.x; j < nbk; j += blockDim.x) {
                const int i = f0 + jb + j;
                sb.x[0][j] = tv.px[i]; sb.x[1][j] = tv.py[i]; sb.x[2][j] = tv.pz[i];
            }
            __syncthreads();
            double acc[2][4] = {{0.0, 0.0, 0.0, 0.0}, {0.0, 0.0, 0.0, 0.0}};
            if constexpr (DO_L2P)
                if (wid == 0) l2p_block<P, POT, T>(grec + (size_t)lf * GR::SIZE, nbk, sb, cx, cy, cz, inv, sm.rec, lane, acc);
            m2p_rounds<P, POT, FAR_HEAVY_NB<T>, T>(tv, hrec, w0, nw, nbk, wid, FAR_HW, sb, inv, tv.level[b], sm, lane, acc);
            __syncthreads();
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int j = lane + 32 * q;
                if (j < nbk) {
#pragma unroll
                    for (int a = 0; a < 4; ++a) s_part[(wid * 64 + j) * 4 + a] = acc[q][a];
                }
            }
            __syncthreads();
            for (int t = threadIdx.x; t < 4 * nbk; t += blockDim.x) {
                double v = 0.0;
#pragma unroll
                for (int w = 0; w < FAR_HW; ++w) v += s_part[w * 256 + t];
                far[4 * (size_t)(f0 + jb) + t] = v;
            }
        }
    }
}
template <int P, bool POT, class T>
constexpr size_t leaf_far_heavy_smem() {
    constexpr size_t a = FAR_HW * sizeof(WarpSmem<P, POT, T, FAR_HEAVY_NB<T>>), b = sizeof(double) * FAR_HW * 64 * 4;
    return a > b ? a : b;
}

}  // namespace far
}  // namespace ogx
