// ogx_lists.cu -- Carrier-Greengard-Rokhlin interaction lists on the GPU.
//
// Replaces AdaptiveOctree::buildLists (src3d/AdaptiveOctree.hpp:137-189):
//  - colleagues: same-level adjacent boxes, the children of the parent's
//    colleagues that pass `adjacent` (:143-151).  Box centres are exact binary
//    fractions of the root box, so for same-level boxes that test holds exactly
//    for integer offsets in [-1,1]^3: every (box, slot) finds its colleague in
//    one launch through the tree's pointers.  A second launch replays the reference's recursion over
//    the children of each parent's colleagues with the FP64 predicate and counts
//    every disagreement (expected 0);
//  - V is implicit: children of the parent's colleagues at integer offset
//    max|o| >= 2 (:154-161); every candidate is also classified with the
//    reference's FP64 predicate and disagreements are counted (expected 0);
//  - U/W per leaf (:164-169 with collectAdjLeaves :176-180 and descendW
//    :181-189): warp per leaf, lane d owns colleague slot d: the slot's leaf
//    (same level), the slot of every ancestor (coarser adjacent leaves) and a
//    bounded explicit-stack descent of the slot's non-leaf colleague (finer U
//    members and the W boxes).  A count pass sizes the CSR, a fill pass writes
//    each lane's items at its warp-scan offset, so the order is deterministic;
//  - X = transpose of W through a stable sort by W member (:171-173).
#include <algorithm>

#include "ogx_tree_common.cuh"
#include "ogx_softening.cuh"
#include "ogx_m2l64.cuh"

namespace ogx {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int UW_STACK = 192;

// colleague slot d of box b: the box of b's level at integer offset (d % 3 - 1, ...), found by
// climbing to the first ancestor that contains both and descending by the other's octants
// (two or three steps each way on average; a binary search of the level took a dozen steps
// of three loads: 47 -> 20 us on the 1M merger)
__global__ void k_colleagues(int nb_cap, const int* __restrict__ level, const int* __restrict__ coord,
                             const int* __restrict__ parent, const int* __restrict__ child, int* __restrict__ col,
                             const DevCounts* counts) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= 27 * (int64_t)nb_cap || counts->overflow) return;
    const int b = (int)(t / 27), d = (int)(t - 27 * (int64_t)b);
    if (b >= counts->nb32) { col[t] = -1; return; }
    if (d == 13) { col[t] = b; return; }
    const int l = level[b];
    const int side = 1 << l;
    const int x = coord[3 * b], y = coord[3 * b + 1], z = coord[3 * b + 2];
    const int nx = x + d % 3 - 1, ny = y + (d / 3) % 3 - 1, nz = z + d / 9 - 1;
    int found = -1;
    if (nx >= 0 && ny >= 0 && nz >= 0 && nx < side && ny < side && nz < side) {
        const int up = 32 - __clz((x ^ nx) | (y ^ ny) | (z ^ nz));   // levels to the common ancestor
        found = b;
        for (int i = 0; i < up; ++i) found = parent[found];
        for (int i = up - 1; i >= 0 && found >= 0; --i)
            found = child[8 * (size_t)found + (((nx >> i) & 1) | (((ny >> i) & 1) << 1) | (((nz >> i) & 1) << 2))];
    }
    col[t] = found;
}

// the reference's recursion (children of the parent's colleagues, FP64 `adjacent`)
// checked against the searched colleagues; also counts the V-list pairs
__global__ void __launch_bounds__(128) k_colleagues_check(int first, int count, const int* __restrict__ leafid,
                                                          const int* __restrict__ child, const double* __restrict__ ctr,
                                                          const RootInfo* root, const int* __restrict__ col,
                                                          DevCounts* counts) {
    __shared__ double s_kc[4][8][4];   // centres (x, y, z, half) of each warp's parent's children
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int k = blockIdx.x * 4 + wid;
    if (k >= count || first + k >= counts->nb32 || counts->overflow) return;
    const int P = first + k;
    if (leafid[P] >= 0) return;
    int kids[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) kids[t] = child[8 * P + t];
    if (lane < 32) {
        const int t = lane >> 2, q = lane & 3;
        s_kc[wid][t][q] = (kids[t] >= 0) ? ctr[4 * kids[t] + q] : 0.0;
    }
    __syncwarp();
    const double tol = root->tol;
    int mism = 0, nv = 0;
    if (lane < 27) {
        const int D = lane;
        const int Q = col[27 * P + D];
        if (Q >= 0) {
            const int Dx = D % 3 - 1, Dy = (D / 3) % 3 - 1, Dz = D / 9 - 1;
            for (int s = 0; s < 8; ++s) {
                const int c = child[8 * Q + s];
                if (c < 0) continue;
                const double cx = ctr[4 * c], cy = ctr[4 * c + 1], cz = ctr[4 * c + 2], ch = ctr[4 * c + 3];
#pragma unroll
                for (int t = 0; t < 8; ++t) {
                    const int b = kids[t];
                    if (b < 0) continue;
                    const int ox = 2 * Dx + (s & 1) - (t & 1), oy = 2 * Dy + ((s >> 1) & 1) - ((t >> 1) & 1),
                              oz = 2 * Dz + ((s >> 2) & 1) - ((t >> 2) & 1);
                    const bool adj_i = max(abs(ox), max(abs(oy), abs(oz))) <= 1;
                    // adjacent64(ctr, b, c, tol) with both centres already in hand
                    const double* kb = s_kc[wid][t];
                    const double lim = __dadd_rn(__dadd_rn(kb[3], ch), tol);
                    const bool adj_f = fabs(__dsub_rn(kb[0], cx)) <= lim && fabs(__dsub_rn(kb[1], cy)) <= lim &&
                                       fabs(__dsub_rn(kb[2], cz)) <= lim;
                    if (adj_i != adj_f) ++mism;
                    if (adj_i) { if (col[27 * b + colleague_slot(ox, oy, oz)] != c) ++mism; }
                    else ++nv;
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mism += __shfl_xor_sync(FULL, mism, o);
        nv += __shfl_xor_sync(FULL, nv, o);
    }
    if (lane == 0) {
        if (mism) atomicAdd((unsigned long long*)&counts->adj_mismatch, (unsigned long long)mism);
        if (nv) atomicAdd((unsigned long long*)&counts->v_total, (unsigned long long)nv);
    }
}

__device__ __forceinline__ int warp_excl_scan(int v, int lane) {
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, x, o);
        if (lane >= o) x += y;
    }
    return x - v;
}

// A node's descent step takes two rounds of loads: its children and centre, then the leaf
// ids of the adjacent children (a child's centre is its parent's shifted by half the child's
// edge, the operation k_boxes formed it with); one child after another, with its centre
// loaded, took some twenty.  FILL also emits the transposed W pairs (X lists) and counts them.
template <bool FILL>
__global__ void __launch_bounds__(128) k_uw_warp(int nleaf, const int* __restrict__ leafbox, const int* __restrict__ parent,
                                                 const int* __restrict__ child, const int* __restrict__ leafid,
                                                 const int* __restrict__ col, const double* __restrict__ ctr,
                                                 const int* __restrict__ pcount, const RootInfo* root, int* lane_u, int* lane_w,
                                                 int* ucnt, int* wcnt, const int64_t* uoff, const int64_t* woff, int* uidx,
                                                 int* widx, uint32_t* xkey, uint32_t* xval, int* xcnt, DevCounts* counts) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int lf = blockIdx.x * 4 + wid;
    __shared__ unsigned long long s_tot[2];
    if (!FILL) {
        if (threadIdx.x < 2) s_tot[threadIdx.x] = 0;
        __syncthreads();
    }
    auto leaf_lists = [&]() {
    if (lf >= nleaf || lf >= counts->nleaf32 || counts->overflow) return;
    const int b = leafbox[lf];
    const double tol = root->tol;
    // adjacent64(ctr, a, b, tol) with b's centre held in registers
    const double bx = ctr[4 * b], by = ctr[4 * b + 1], bz = ctr[4 * b + 2], bh = ctr[4 * b + 3];
    auto adj = [&](double x, double y, double z, double h) {
        const double lim = __dadd_rn(__dadd_rn(h, bh), tol);
        return fabs(__dsub_rn(x, bx)) <= lim && fabs(__dsub_rn(y, by)) <= lim && fabs(__dsub_rn(z, bz)) <= lim;
    };
    auto centre = [&](int a, double2& c01, double2& c23) {
        c01 = __ldg(reinterpret_cast<const double2*>(ctr) + 2 * (size_t)a);
        c23 = __ldg(reinterpret_cast<const double2*>(ctr) + 2 * (size_t)a + 1);
    };
    int nu = 0, nw = 0;
    int64_t upairs = 0, ub = 0, wb = 0;
    bool overflow = false;
    if (FILL) {
        ub = uoff[lf] + warp_excl_scan(lane_u[32 * lf + lane], lane);
        wb = woff[lf] + warp_excl_scan(lane_w[32 * lf + lane], lane);
    }
    auto addU = [&](int c) {
        if (FILL) uidx[ub + nu] = c;
        else upairs += pcount[c];
        ++nu;
    };
    if (lane < 27) {
        const int d = lane;
        const int c = col[27 * (size_t)b + d];
        const int lc = c >= 0 ? leafid[c] : -1;
        if (c >= 0 && lc >= 0) addU(c);  // same-level adjacent leaves (b itself in slot 13)
        for (int A = parent[b]; A >= 0;) {  // coarser adjacent leaves
            const int up = parent[A], a2 = col[27 * (size_t)A + d];
            if (a2 >= 0 && leafid[a2] >= 0) {
                double2 c01, c23;
                centre(a2, c01, c23);
                if (adj(c01.x, c01.y, c23.x, c23.y)) addU(a2);
            }
            A = up;
        }
        if (c >= 0 && c != b && lc < 0) {  // finer: descend the non-leaf colleague
            int stk[UW_STACK];
            int sp = 0;
            stk[sp++] = c;
            while (sp > 0) {
                const int node = stk[--sp];
                const int4 k0 = __ldg(reinterpret_cast<const int4*>(child + 8 * (size_t)node));
                const int4 k1 = __ldg(reinterpret_cast<const int4*>(child + 8 * (size_t)node) + 1);
                double2 c01, c23;
                centre(node, c01, c23);
                const int ch[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
                const double h2 = __dmul_rn(0.5, c23.y);
                // per axis: the lower and the upper child's coordinate (k_boxes' operations)
                const double xs[2] = {__dadd_rn(c01.x, -h2), __dadd_rn(c01.x, h2)}, ys[2] = {__dadd_rn(c01.y, -h2), __dadd_rn(c01.y, h2)},
                             zs[2] = {__dadd_rn(c23.x, -h2), __dadd_rn(c23.x, h2)};
                int leaf[8];
                unsigned near = 0;
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const bool a = ch[s] >= 0 && adj(xs[s & 1], ys[(s >> 1) & 1], zs[s >> 2], h2);
                    leaf[s] = a ? __ldg(leafid + ch[s]) : -1;
                    if (a) near |= 1u << s;
                }
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    if (ch[s] < 0) continue;
                    if (!(near >> s & 1u)) {
                        if (FILL) {
                            widx[wb + nw] = ch[s];
                            xkey[wb + nw] = (uint32_t)ch[s];
                            xval[wb + nw] = (uint32_t)b;
                            atomicAdd(&xcnt[ch[s]], 1);
                        }
                        ++nw;
                    } else if (leaf[s] >= 0) {
                        addU(ch[s]);
                    } else if (sp < UW_STACK) {
                        stk[sp++] = ch[s];
                    } else {
                        overflow = true;
                    }
                }
            }
        }
    }
    if (!FILL) {
        lane_u[32 * lf + lane] = nu;
        lane_w[32 * lf + lane] = nw;
        int tu = nu, tw = nw;
        int64_t tp = upairs;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            tu += __shfl_xor_sync(FULL, tu, o);
            tw += __shfl_xor_sync(FULL, tw, o);
            tp += __shfl_xor_sync(FULL, tp, o);
        }
        const bool any_over = __any_sync(FULL, overflow);
        // totals: one addition per block (one per leaf to the same words took 70 us on the 1M merger)
        if (lane == 0) {
            ucnt[lf] = tu;
            wcnt[lf] = tw;
            const unsigned long long pb = (unsigned long long)pcount[b];
            atomicAdd(&s_tot[0], pb * (unsigned long long)tp - pb);
            atomicAdd(&s_tot[1], pb * (unsigned long long)tw);
            if (any_over) atomicAdd((unsigned long long*)&counts->adj_mismatch, 1ull << 40);
        }
    }
    };
    leaf_lists();
    if (!FILL) {
        __syncthreads();
        if (threadIdx.x == 0 && s_tot[0] + s_tot[1] > 0) {
            atomicAdd((unsigned long long*)&counts->p2p_pairs, s_tot[0]);
            atomicAdd((unsigned long long*)&counts->m2p_evals, s_tot[1]);
            atomicAdd((unsigned long long*)&counts->p2l_evals, s_tot[1]);
        }
    }
}

// M2L targets: boxes of level >= 2 keyed by their child octant
// Sort key of an M2L target: its octant t inside the parent (bits 27-29; a tensor-core
// tile holds targets of one octant) and, below it, which of the parent's 27 colleague
// slots D give the target any V-list source (bit 26 - D).  Targets with the same slot
// pattern then share tiles, so a tile runs fewer (colleague, child) combinations and
// fewer of its operand rows are empty (on the 1M merger: 17% fewer combinations).  The
// order of a tile's targets does not change any target's result.
// Launched over the capacity of boxes: the targets are boxes level_off[2] .. nb - 1
// (device counts); slots behind them get key 1 << 30 and sort after every target.
// Warp per target, lane = colleague slot.
__global__ void __launch_bounds__(128) k_tgt_keys(int cap, const int* __restrict__ level_off, const int* __restrict__ coord,
                                                  const int* __restrict__ parent, const int* __restrict__ col,
                                                  const int* __restrict__ child, uint32_t* key, uint32_t* val, DevCounts* counts) {
    const int lane = threadIdx.x & 31;
    const int k = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (k >= cap || counts->overflow) return;
    const int first = level_off[2], ntgt = counts->nb32 - first;
    if (k == 0 && lane == 0) counts->ntgt32 = ntgt;
    if (k >= ntgt) {
        if (lane == 0) {
            key[k] = 1u << 30;
            val[k] = 0xFFFFFFFFu;
        }
        return;
    }
    const int b = first + k;
    const int tx = coord[3 * b] & 1, ty = coord[3 * b + 1] & 1, tz = coord[3 * b + 2] & 1;
    const int Q = lane < 27 ? col[27 * (size_t)parent[b] + lane] : -1;
    bool any = false;
    if (Q >= 0) {
        const int4 c0 = __ldg(reinterpret_cast<const int4*>(child + 8 * (size_t)Q));
        const int4 c1 = __ldg(reinterpret_cast<const int4*>(child + 8 * (size_t)Q) + 1);
        const int ch[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        const int Dx = lane % 3 - 1, Dy = (lane / 3) % 3 - 1, Dz = lane / 9 - 1;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const int ox = 2 * Dx + (s & 1) - tx, oy = 2 * Dy + ((s >> 1) & 1) - ty, oz = 2 * Dz + ((s >> 2) & 1) - tz;
            any |= ch[s] >= 0 && max(abs(ox), max(abs(oy), abs(oz))) > 1;
        }
    }
    const unsigned slots = __ballot_sync(FULL, any);   // bit D
    if (lane == 0) {
        key[k] = ((uint32_t)(tx | (ty << 1) | (tz << 2)) << 27) | (__brev(slots) >> 5);   // slot D in bit 26 - D
        val[k] = (uint32_t)b;
    }
}

// padded per-octant layout of the M2L targets (sorted by k_tgt_keys' key, octant in
// bits 27-29): every octant group starts on a multiple of `tile`, so a tile never
// mixes octants.  gs[0..8] = group starts,
// gs[9..17] = padded group starts, then the FP64 M2L's work split (ogx_m2l64.cuh).
__global__ void k_target_groups(const uint32_t* key, const DevCounts* counts, int tile, int fill, int* gs) {
    __shared__ int lo_s[9];
    const int g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ntgt = counts->overflow ? 0 : counts->ntgt32;
    if (g <= 8) {   // warp g: the first index with key octant >= g, 32 probes at a time
        int lo = 0, hi = ntgt;
        while (hi > lo) {
            const int step = (hi - lo + 31) / 32, i = lo + lane * step;
            const bool below = i < hi && (int)(key[i] >> 27) < g;
            const int c = __popc(__ballot_sync(FULL, below));   // probes below: a prefix
            if (c == 0) { hi = lo; break; }
            const int last = lo + (c - 1) * step;
            hi = min(hi, last + step);
            lo = last + 1;
        }
        if (lane == 0) {
            lo_s[g] = lo;
            gs[g] = lo;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int pad = 0;
        for (int q = 0; q <= 8; ++q) {
            gs[9 + q] = pad;
            if (q < 8) pad += ((lo_s[q + 1] - lo_s[q] + fill - 1) / fill) * tile;
        }
        int tiles64 = 0, tiles128 = 0;
        for (int q = 0; q < 8; ++q) {
            tiles64 += (lo_s[q + 1] - lo_s[q] + M2L64_TGT - 1) / M2L64_TGT;
            tiles128 += (lo_s[q + 1] - lo_s[q] + 127) / 128;
        }
        gs[GS_TILES128] = tiles128;
        for (int sl = 1; sl <= 3; ++sl) gs[GS_TC_SPLIT + sl - 1] = m2l_tc_split(tiles128, sl);
        gs[GS_SPLIT] = max(1, min(M2L64_MAXSPLIT, (M2L64_ITEMS + tiles64 - 1) / max(tiles64, 1)));
        gs[GS_TILES] = pad / M2L64_TGT;
        gs[GS_TICKET] = 0;
        gs[GS_FILL] = fill;
    }
}
// slot q of a padded group holds target (q - start) / tile * fill + (q - start) % tile
// when that slot index is below `fill` (the batch width) and the target exists
__global__ void k_target_pad(const uint32_t* box, const int* gs, int npad, int tile, int fill, uint32_t* pkey,
                             uint32_t* pbox) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= npad) return;
    uint32_t k = 0xFFFFFFFFu, b = 0xFFFFFFFFu;
    for (int g = 0; g < 8; ++g) {
        const int ps = gs[9 + g], pe = gs[9 + g + 1];
        if (q >= ps && q < pe) {
            const int slot = (q - ps) % tile;
            const int local = (q - ps) / tile * fill + slot;
            if (slot < fill && local < gs[g + 1] - gs[g]) { k = (uint32_t)g; b = box[gs[g] + local]; }
            break;
        }
    }
    pkey[q] = k;
    pbox[q] = b;
}


// list totals (the last entry of each exclusive scan over the leaf capacity, whose
// padding counts are zero), checked against the capacities of the index arrays
__global__ void k_check_lists(DevCounts* counts, const int64_t* utot, const int64_t* wtot, int64_t cap_u, int64_t cap_w) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    counts->u_total = *utot;
    counts->w_total = *wtot;
    if (*utot > cap_u || *wtot > cap_w) counts->overflow = 1;
}

// X-list keys behind the W total (device) get `v` and sort last
__global__ void k_fill_tail_x(uint32_t* a, const DevCounts* counts, int64_t cap, uint32_t v) {
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k < cap && k >= counts->w_total) a[k] = v;
}

inline int grid_for(int64_t n, int b) { return (int)((n + b - 1) / b); }
inline int bits_for(int64_t v) {
    int b = 1;
    while ((1ll << b) <= v) ++b;
    return b;
}

// OGX_SOFT_SPLINE: for each leaf b, the leaves c that are not adjacent to b (the far
// field takes their pairs) and whose box lies within the spline's support `hs` of b's
// box, found by a depth-first walk from the root that skips every box farther than hs.
// Adjacency is the U-list predicate (AdaptiveOctree::adjacent, same FP64 operations), so
// every leaf pair is either in b's U list or a candidate here.  Pass 1 counts, pass 2 writes
// in the same order.
//
// Warp per leaf: the 32 boxes on top of a stack in shared memory are tested together, their
// children pushed, so a walk takes a dozen rounds of loads (a thread per leaf took one box
// after another, 24 blocks' worth of threads for the 50k merger, 200 us a pass).  A round
// takes at most 32 boxes and pushes at most 256, and what it pushes is taken first, so at
// most 224 boxes wait per level.
constexpr int kSoftStack = 256 * (kMaxDepth + 1);
constexpr int kSoftSmem = 2 * kSoftStack * (int)sizeof(int);   // two warps per block
template <bool EMIT>
__global__ void __launch_bounds__(64) k_soft_lists(int nleaf, const int* __restrict__ leafbox, const int* __restrict__ child,
                                                   const int* __restrict__ leafid, const double* __restrict__ ctr,
                                                   const RootInfo* __restrict__ root, double hs, int* cnt,
                                                   const int64_t* __restrict__ off, int* idx, const DevCounts* counts) {
    extern __shared__ int s_soft[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int lf = blockIdx.x * 2 + wid;
    if (lf >= nleaf) return;
    if (lf >= counts->nleaf32 || counts->overflow) {
        if (!EMIT && lane == 0) cnt[lf] = 0;
        return;
    }
    int* stack = s_soft + wid * kSoftStack;
    const int b = leafbox[lf];
    const double tol = root->tol;
    const double bx = ctr[4 * b], by = ctr[4 * b + 1], bz = ctr[4 * b + 2], bh = ctr[4 * b + 3];
    const double hs2 = hs * hs;
    const unsigned lt = (1u << lane) - 1u;
    int sp = 1, n = 0;
    const int64_t o = EMIT ? off[lf] : 0;
    if (lane == 0) stack[0] = 0;   // the root
    __syncwarp();
    while (sp > 0) {
        const int take = min(32, sp);
        const int c = lane < take ? stack[sp - 1 - lane] : -1;
        __syncwarp();   // read before the pushes below overwrite
        sp -= take;
        int leaf = -1;
        int4 k0 = make_int4(-1, -1, -1, -1), k1 = k0;
        bool in = false, adj = false;
        if (c >= 0) {
            const double2 c01 = __ldg(reinterpret_cast<const double2*>(ctr) + 2 * (size_t)c);
            const double2 c23 = __ldg(reinterpret_cast<const double2*>(ctr) + 2 * (size_t)c + 1);
            leaf = __ldg(leafid + c);
            k0 = __ldg(reinterpret_cast<const int4*>(child + 8 * (size_t)c));
            k1 = __ldg(reinterpret_cast<const int4*>(child + 8 * (size_t)c) + 1);
            const double ch = c23.y;
            // gap between the two boxes along each axis (0 where they overlap)
            const double gx = fmax(0.0, fabs(c01.x - bx) - (ch + bh));
            const double gy = fmax(0.0, fabs(c01.y - by) - (ch + bh));
            const double gz = fmax(0.0, fabs(c23.x - bz) - (ch + bh));
            in = !(gx * gx + gy * gy + gz * gz >= hs2);
            const double lim = __dadd_rn(__dadd_rn(ch, bh), tol);
            adj = fabs(__dsub_rn(c01.x, bx)) <= lim && fabs(__dsub_rn(c01.y, by)) <= lim && fabs(__dsub_rn(c23.x, bz)) <= lim;
        }
        const bool found = in && leaf >= 0 && !adj;
        const unsigned mf = __ballot_sync(FULL, found);
        if (EMIT && found) idx[o + n + __popc(mf & lt)] = c;
        n += __popc(mf);
        const bool open = in && leaf < 0;
        const int kid[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
        for (int s = 0; s < 8; ++s) {
            const bool push = open && kid[s] >= 0;
            const unsigned m = __ballot_sync(FULL, push);
            if (push) stack[sp + __popc(m & lt)] = kid[s];
            sp += __popc(m);
        }
        __syncwarp();
    }
    if (!EMIT && lane == 0) cnt[lf] = n;
}

}  // namespace

// Built after the U/W/X lists of an eager evaluation (one more count read-back).
int soft_lists_build(Handle& h) {
    const cudaStream_t st = h.stream;
    TreeView& tv = h.tv;
    const int nleaf = tv.nleaf;
    int* cnt;
    int64_t* off;
    OGX_TRY(arena_get(h.ws, S_SOFT_CNT, nleaf, &cnt));
    OGX_TRY(arena_get(h.ws, S_SOFT_OFF, nleaf + 1, &off));
    const double hs = spline_support(h.prm.eps);
    OGX_CUDA(smem_optin((const void*)k_soft_lists<false>, kSoftSmem));
    OGX_CUDA(smem_optin((const void*)k_soft_lists<true>, kSoftSmem));
    k_soft_lists<false><<<grid_for(nleaf, 2), 64, kSoftSmem, st>>>(nleaf, tv.leafbox, tv.child, tv.leafid, tv.center, tv.root, hs,
                                                              cnt, nullptr, nullptr, h.d_counts); ++h.launches;
    OGX_TRY(scan_i32_to_i64(h, cnt, off, nleaf));
    int64_t ns = 0;
    OGX_CUDA(cudaMemcpyAsync(&ns, off + nleaf, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    OGX_CUDA(cudaStreamSynchronize(st));
    int* idx;
    OGX_TRY(arena_get(h.ws, S_SOFT_IDX, ns + 1, &idx));
    k_soft_lists<true><<<grid_for(nleaf, 2), 64, kSoftSmem, st>>>(nleaf, tv.leafbox, tv.child, tv.leafid, tv.center, tv.root, hs,
                                                             nullptr, off, idx, h.d_counts); ++h.launches;
    tv.s_off = off;
    tv.s_idx = idx;
    h.soft_pairs = ns;
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

int lists_build(Handle& h) {
    OGX_TRY(lists_build_targets(h));
    return lists_build_uwx(h);
}

int lists_build_targets(Handle& h) {
    const cudaStream_t st = h.stream;
    TreeView& tv = h.tv;
    const int nb = tv.nb;   // launch size (the capacity in capacity mode)
    DevCounts* dc = h.d_counts;
    int* col;
    OGX_TRY(arena_get(h.ws, S_BOX_COL, 27 * (size_t)nb, &col));
    k_colleagues<<<grid_for(27 * (int64_t)nb, 256), 256, 0, st>>>(nb, tv.level, tv.coord, tv.parent, tv.child, col, dc); ++h.launches;
    tv.col = col;

    // M2L targets (levels >= 2) grouped by child octant, then by the slot pattern of
    // their V lists; launched over the box capacity, the padding sorts last.  They need
    // only the colleagues, so they are built on the aux stream beside the U/W passes
    // (which use the scan scratch, not the radix-sort scratch); the main stream joins
    // before the X-list sort, which uses the radix-sort scratch again.
    OGX_CUDA(cudaEventRecord(h.ev_col, st));
    // nothing of the evaluation waits for the check and the V-pair count: on the side stream
    // (joined at the evaluation's end)
    OGX_CUDA(cudaStreamWaitEvent(h.side, h.ev_col, 0));
    k_colleagues_check<<<grid_for(nb, 4), 128, 0, h.side>>>(0, nb, tv.leafid, tv.child, tv.center, tv.root, col, dc); ++h.launches;
    OGX_CUDA(cudaEventRecord(h.ev_check, h.side));
    OGX_CUDA(cudaStreamWaitEvent(h.aux, h.ev_col, 0));
    h.stream = h.aux;   // radix_sort_u32 issues on h.stream
    const int tcap = std::max(nb, 1);
    uint32_t *tk, *tb;
    OGX_TRY(arena_get(h.ws, S_TGT_KEY, tcap + 1, &tk));
    OGX_TRY(arena_get(h.ws, S_TGT_BOX, tcap + 1, &tb));
    k_tgt_keys<<<grid_for(tcap, 4), 128, 0, h.aux>>>(tcap, h.d_level_off, tv.coord, tv.parent, col, tv.child, tk, tb, dc); ++h.launches;
    uint32_t *tk_s, *tb_s;
    const int rc_t = radix_sort_u32(h, S_TGT_KEY, S_TGT_BOX, S_TGT_KEY2, S_TGT_BOX2, tcap, 31, &tk_s, &tb_s);
    h.stream = st;
    OGX_TRY(rc_t);
    h.tgt_key = tk_s;
    h.tgt_box = tb_s;
    const int tile = 128;  // tensor-core M2L tile; a multiple of the FP64 kernel's 64
    const int fill = h.tile_fill;   // targets per tile (the M2L batch width)
    const int ntgt_bound = h.cap_mode ? tcap : std::max(0, nb - (h.max_level >= 2 ? h.level_off[2] : nb));
    const int npad = ((ntgt_bound + fill - 1) / fill + 8) * tile;
    int* gs;
    uint32_t *pk, *pb;
    OGX_TRY(arena_get(h.ws, S_TGT_TILE, 32, &gs));
    OGX_TRY(arena_get(h.ws, S_TGT_PKEY, npad, &pk));
    OGX_TRY(arena_get(h.ws, S_TGT_PBOX, npad, &pb));
    k_target_groups<<<1, 288, 0, h.aux>>>(tk_s, dc, tile, fill, gs); ++h.launches;
    k_target_pad<<<grid_for(npad, 256), 256, 0, h.aux>>>(tb_s, gs, npad, tile, fill, pk, pb); ++h.launches;
    h.tgt_groups = gs;
    h.tgt_tile_key = pk;
    h.tgt_tile_box = pb;
    h.ntgt_pad = npad;
    h.ntgt = ntgt_bound;
    OGX_CUDA(cudaEventRecord(h.ev_tgt, h.aux));
    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

int lists_build_uwx(Handle& h) {
    const cudaStream_t st = h.stream;
    TreeView& tv = h.tv;
    const int nb = tv.nb, nleaf = tv.nleaf;   // launch sizes (capacities in capacity mode)
    DevCounts* dc = h.d_counts;
    const int* col = tv.col;
    int *ucnt, *wcnt, *lane_uw;
    int64_t *uoff, *woff;
    OGX_TRY(arena_get(h.ws, S_U_CNT, nleaf, &ucnt));
    OGX_TRY(arena_get(h.ws, S_W_CNT, nleaf, &wcnt));
    OGX_TRY(arena_get(h.ws, S_UW_LANE, 64 * (size_t)nleaf, &lane_uw));
    OGX_TRY(arena_get(h.ws, S_U_OFF, nleaf + 1, &uoff));
    OGX_TRY(arena_get(h.ws, S_W_OFF, nleaf + 1, &woff));
    if (h.cap_mode) {   // padding leaves count nothing
        OGX_CUDA(cudaMemsetAsync(ucnt, 0, sizeof(int) * (size_t)nleaf, st));
        OGX_CUDA(cudaMemsetAsync(wcnt, 0, sizeof(int) * (size_t)nleaf, st));
    }
    int* lane_u = lane_uw;
    int* lane_w = lane_uw + 32 * (size_t)nleaf;
    k_uw_warp<false><<<grid_for(nleaf, 4), 128, 0, st>>>(nleaf, tv.leafbox, tv.parent, tv.child, tv.leafid, col, tv.center,
                                                         tv.pcount, tv.root, lane_u, lane_w, ucnt, wcnt, nullptr, nullptr,
                                                         nullptr, nullptr, nullptr, nullptr, nullptr, dc); ++h.launches;
    OGX_TRY(scan2_i32_to_i64(h, ucnt, uoff, wcnt, woff, nleaf));
    int64_t nu, nw;
    if (h.cap_mode) {
        nu = h.cap.u;
        nw = h.cap.w;
        k_check_lists<<<1, 32, 0, st>>>(dc, uoff + nleaf, woff + nleaf, nu, nw); ++h.launches;
    } else {
        // sync point 2: list sizes
        k_check_lists<<<1, 32, 0, st>>>(dc, uoff + nleaf, woff + nleaf, INT64_MAX, INT64_MAX); ++h.launches;
        OGX_CUDA(cudaMemcpyAsync(h.h_counts, dc, sizeof(DevCounts), cudaMemcpyDeviceToHost, st));
        OGX_CUDA(cudaStreamSynchronize(st));
        nu = h.h_counts->u_total;
        nw = h.h_counts->w_total;
    }
    int *uidx, *widx;
    OGX_TRY(arena_get(h.ws, S_U_IDX, nu + 1, &uidx));
    OGX_TRY(arena_get(h.ws, S_W_IDX, nw + 1, &widx));
    // X lists: W transposed by a stable sort on the W member; keys behind the W total
    // (capacity padding) sort last and are never referenced by x_off
    const int xbits = bits_for(nb);
    uint32_t *xk, *xv;
    int* xcnt;
    int64_t* xoff;
    OGX_TRY(arena_get(h.ws, S_X_KEY, nw + 1, &xk));
    OGX_TRY(arena_get(h.ws, S_X_VAL, nw + 1, &xv));
    OGX_TRY(arena_get(h.ws, S_X_CNT, nb, &xcnt));
    OGX_TRY(arena_get(h.ws, S_X_OFF, nb + 1, &xoff));
    OGX_CUDA(cudaMemsetAsync(xcnt, 0, sizeof(int) * (size_t)nb, st));
    k_uw_warp<true><<<grid_for(nleaf, 4), 128, 0, st>>>(nleaf, tv.leafbox, tv.parent, tv.child, tv.leafid, col, tv.center,
                                                        tv.pcount, tv.root, lane_u, lane_w, nullptr, nullptr, uoff, woff, uidx,
                                                        widx, xk, xv, xcnt, dc); ++h.launches;
    tv.u_off = uoff; tv.w_off = woff; tv.u_idx = uidx; tv.w_idx = widx;
    OGX_CUDA(cudaStreamWaitEvent(st, h.ev_tgt, 0));   // target sort done with the radix scratch
    if (h.cap_mode) { k_fill_tail_x<<<grid_for(nw, 256), 256, 0, st>>>(xk, dc, nw, (1u << xbits) - 1u); ++h.launches; }
    uint32_t *xk_s, *xv_s;
    OGX_TRY(radix_sort_u32(h, S_X_KEY, S_X_VAL, S_X_KEY2, S_X_VAL2, nw, xbits, &xk_s, &xv_s));
    OGX_TRY(scan_i32_to_i64(h, xcnt, xoff, nb));
    tv.x_off = xoff;
    tv.x_idx = (const int*)xv_s;

    OGX_CUDA(cudaGetLastError());
    return OGX_OK;
}

}  // namespace ogx
