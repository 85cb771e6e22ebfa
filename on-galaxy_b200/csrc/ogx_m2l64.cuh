// ogx_m2l64.cuh -- how the FP64 M2L (plain and rotation form) is cut into work items.
//
// A work item is (64-target tile, range of colleague slots D): a small tree has too few
// tiles for the SMs (16,384 bodies: about 20), so its tiles are cut into up to 27 ranges
// of slots, whose sums are added in range order by k_m2l64_sum.  The number of ranges
// depends only on the targets per octant, so a target's result does not depend on the
// launch's capacities, on the batch width or on which targets share its tile.
#pragma once

#include "ogx_internal.cuh"

namespace ogx {

constexpr int M2L64_TGT = 64;        // targets per tile; the target layout is padded to 128
constexpr int M2L64_ITEMS = 6 * SPLIT_SMS;   // items wanted: 3 per CTA slot of 2 per SM (2.5: 0.2 ms more of tail at 262,144 bodies)
constexpr int M2L64_MAXSPLIT = 27;
constexpr int TC_ITEMS = 6 * SPLIT_SMS;      // most items (tile, slice, range) a split of the tensor-core M2L makes
// k_target_groups' words behind the group starts gs[0..17]
constexpr int GS_SPLIT = 18, GS_TILES = 19, GS_TICKET = 20, GS_FILL = 21, GS_TILES128 = 22, GS_TC_SPLIT = 23 /* for 1, 2, 3 slices */;

// V children that slot D offers a target of octant t: the 8 children less the adjacent ones
__host__ __device__ __forceinline__ int m2l64_slot_count(int D, int t) {
    const int d[3] = {D % 3 - 1, (D / 3) % 3 - 1, D / 9 - 1};
    int adj = 1;
    for (int a = 0; a < 3; ++a) {
        const int ta = (t >> a) & 1;
        adj *= d[a] == 0 ? 2 : (d[a] > 0 ? ta : 1 - ta);
    }
    return 8 - adj;
}

// first slot of range z of S (about 189 / S combinations each); range z ends where z + 1 starts
__host__ __device__ __forceinline__ int m2l64_first_slot(int z, int S, int t) {
    if (z >= S) return 27;
    const int want = 189 * z;
    int c = 0, D = 0;
    while (D < 27 && c * S < want) c += m2l64_slot_count(D++, t);
    return D;
}

// partial rows (of K doubles) that any tree of at most ntgt targets can need (a captured
// step's tree may be smaller than its capacity): S <= 27, S < M2L64_ITEMS / tiles + 1, and
// S = 1 (none) from M2L64_ITEMS tiles on
inline size_t m2l64_partial_rows(int64_t ntgt) {
    const int64_t full = (int64_t)M2L64_TGT * M2L64_ITEMS;
    const int64_t a = M2L64_MAXSPLIT * ntgt, b = full + (ntgt < full ? ntgt : full);
    return (size_t)(a < b ? a : b);
}

// Ranges of the tensor-core M2L for `tiles` 128-target tiles of `slices` column slices each
// (one CTA per SM): the fewest waves of work, where a CTA costs 1 / S of a tile and 0.045 of
// one for its set-up and partial sums (17,000 of 500,000 cycles at p = 8, and the rows).
__host__ __device__ __forceinline__ int m2l_tc_split(int tiles, int slices) {
    const int n = tiles * slices;
    int best = 1;
    float cost = 1e30f;
    for (int s = 1; s <= M2L64_MAXSPLIT && (s == 1 || n * s <= TC_ITEMS); ++s) {
        const float c = (float)((n * s + SPLIT_SMS - 1) / SPLIT_SMS) * (1.0f / (float)s + 0.045f);
        if (c < cost * 0.999f) { cost = c; best = s; }
    }
    return best;
}
// partial rows (of K doubles) that any tree of at most ntgt targets can need
inline size_t m2l_tc_partial_rows(int64_t ntgt, int slices) {
    size_t rows = 0;
    const int64_t most = (ntgt + 127) / 128 + 8;
    for (int64_t n = 1; n <= most && n * slices * 2 <= TC_ITEMS; ++n) {   // more are not split
        const int s = m2l_tc_split((int)n, slices);
        if (s > 1) {
            const size_t r = (size_t)s * (size_t)(128 * n < ntgt ? 128 * n : ntgt);
            if (r > rows) rows = r;
        }
    }
    return rows;
}

struct M2L64Args {
    const uint32_t *tgt_key, *tgt_box;   // padded tiles
    const uint32_t* sorted_box;          // targets in sorted order, without padding
    int* gs;                             // group starts, split, tiles, ticket
    double* part;                        // [range][target][K], used when the split is above 1
};

int m2l_fp64_launch(Handle& h, const double* M, double* Lown);   // the plain form's M2L, on h.stream
// the ranges' sums (split above 1) into Lown; slices > 0: those of the tensor-core M2L (dofs
// 1 .. K - 1)
int m2l64_sum_launch(Handle& h, const M2L64Args& a, int slices, double* Lown, cudaStream_t st);
int m2l64_args(Handle& h, int slices, M2L64Args* a);
// operators [343][K padded to 4][NP + 4] of the plain form, zero padded, for d_m2l
int m2l64_pad_rows(int p);
int m2l64_pad_cols(int p);

}  // namespace ogx
