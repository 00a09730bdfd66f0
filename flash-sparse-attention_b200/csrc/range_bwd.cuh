// Shared by the range-attention backward's kernels (range_bwd_dkdv.cu) and their callers (fsa_api.cu, sel_bwd.cu).
#pragma once
#include "sel_launch.cuh"

namespace fsa {

inline int range_kv_items() { return 8 * sm_count(); }       // work items (all heads) that the plan aims at
constexpr int kRkMinTiles = 8;          // shortest stretch that a K/V tile's tokens are cut into, in row tiles

struct RangeKvPlan {
    const int32_t* cu_q;
    const int32_t* cu_k;
    const int32_t* kv_lo;
    const int32_t* kv_hi;
    int64_t N, Nk;
    int B, Hk, TPT, max_tiles;
    int aim;            // range_kv_items()
    int* counts;        // [0] items, [1] tiles cut into several items
    int4* tiles;        // [max_tiles] first K/V row, rows, first and last token that see one of them
    int4* items;        // tile, first row tile of its stretch, row tiles, slab (-1: written in place)
    int4* multi;        // first K/V row, rows, first slab, slabs
};

// Sizes of the plan and the slabs: ceil(n / C) <= 2 n / C for a tile that is cut, so the cut tiles have at most 2 aim / Hk items.
inline int64_t range_kv_max_tiles(const SelShape& s) { return (s.Nk + kTileRows - 1) / kTileRows + s.B; }
inline int64_t range_kv_max_cut(const SelShape& s) {
    const int64_t row_tiles = range_kv_max_tiles(s) * ((s.N + s.TPT - 1) / s.TPT);
    const int64_t a = 2 * (int64_t)range_kv_items() / s.Hk + 1, b = 2 * row_tiles / kRkMinTiles + 1;
    return a < b ? a : b;
}
inline int64_t range_kv_plan_bytes(const SelShape& s) { return 256 + 16 * (3 * range_kv_max_tiles(s) + range_kv_max_cut(s)); }
inline int64_t range_kv_slab_bytes(const SelShape& s) { return range_kv_max_cut(s) * s.Hk * (2 * 128 * 128 * 4); }

cudaError_t launch_range_bwd_plan(const RangeKvPlan& p, const SelBwdArgs& a, int* status, cudaStream_t stream);
cudaError_t launch_range_bwd_dkdv(int dtype, const RangeKvPlan& p, const SelBwdArgs& a, const SelShape& s, const CUtensorMap& kmap,
                                  const CUtensorMap& vmap, int* status, cudaStream_t stream);

}  // namespace fsa
