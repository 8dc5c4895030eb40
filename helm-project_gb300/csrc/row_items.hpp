// Work of the FP64 apply's warps (k_f64_fused in apply.cu), as the kernel and
// its launch take it: the long-row warps come first, then the short rows'
// warps, tile after tile of fields, a slice of 32 rows each. The grid is
// whole blocks of eight warps, so up to seven warps have no item: on is false
// for them, and they must not touch the row order, which holds 32 * n_slices
// rows.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define AXGB_HD __host__ __device__ __forceinline__
#else
#define AXGB_HD inline
#endif

namespace axgb {

struct RowItem {
    std::int64_t tile, slice;
    bool on;
};

// Item of the w-th warp after the long rows'. One tile is found without the
// division.
AXGB_HD RowItem row_item(std::int64_t w, std::int64_t n_slices, std::int64_t nrhs, std::int64_t tile) {
    const std::int64_t t = nrhs <= tile ? 0 : w / n_slices, slice = w - t * n_slices;
    return {t, slice, slice < n_slices && t * tile < nrhs};
}

// Warps of a launch: a long row for each chunk of F fields, a slice for each tile.
AXGB_HD std::int64_t row_item_warps(std::int64_t n_long, std::int64_t F, std::int64_t n_slices, std::int64_t nrhs,
                                    std::int64_t tile) {
    return n_long * ((nrhs + F - 1) / F) + n_slices * ((nrhs + tile - 1) / tile);
}

}  // namespace axgb
