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
constexpr int M2L64_ITEMS = 1184;    // items wanted: 4 per CTA slot of 2 x 148
constexpr int M2L64_MAXSPLIT = 27;
// k_target_groups' words behind the group starts gs[0..17]
constexpr int GS_SPLIT = 18, GS_TILES = 19, GS_TICKET = 20, GS_FILL = 21;

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

// partial rows (of K doubles) that S ranges of at most ntgt targets can need: S <= 27,
// S < M2L64_ITEMS / tiles + 1, and S = 1 (no partial rows) from M2L64_ITEMS tiles on (a
// capacity is at most twice the targets it was taken from)
inline size_t m2l64_partial_rows(int64_t ntgt) {
    if (ntgt >= 2ll * M2L64_TGT * M2L64_ITEMS) return 0;
    const int64_t a = M2L64_MAXSPLIT * ntgt, b = (int64_t)M2L64_TGT * M2L64_ITEMS + ntgt;
    return (size_t)(a < b ? a : b);
}

struct M2L64Args {
    const uint32_t *tgt_key, *tgt_box;   // padded tiles
    const uint32_t* sorted_box;          // targets in sorted order, without padding
    int* gs;                             // group starts, split, tiles, ticket
    double* part;                        // [range][target][K], used when the split is above 1
};

int m2l_fp64_launch(Handle& h, const double* M, double* Lown);   // the plain form's M2L, on h.stream
// adds the ranges' sums (split above 1) into Lown
int m2l64_sum_launch(Handle& h, const M2L64Args& a, double* Lown, cudaStream_t st);
int m2l64_args(Handle& h, M2L64Args* a);
// operators [343][K padded to 4][NP + 4] of the plain form, zero padded, for d_m2l
int m2l64_pad_rows(int p);
int m2l64_pad_cols(int p);

}  // namespace ogx
