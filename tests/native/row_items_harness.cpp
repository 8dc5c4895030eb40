// Test harness: the FP64 apply's map from warps to work (row_items.hpp)
// through a C entry point, compiled by tests/test_cpu_row_items.py.
#include "row_items.hpp"

extern "C" {

// Walks every warp of the launch's whole blocks of eight as the kernel does.
// Long-row warps are counted in long_hits[n_long * chunks]; a short-row warp
// that is on adds one to hits[tile * n_slices + slice] when that lies in
// range. Returns the warps that would read the row order out of range.
long long row_items_walk(long long n_long, long long F, long long n_slices, long long nrhs, long long tile,
                         int *long_hits, int *hits) {
    const long long warps = axgb::row_item_warps(n_long, F, n_slices, nrhs, tile);
    const long long first = n_long * ((nrhs + F - 1) / F), tiles = (nrhs + tile - 1) / tile;
    long long bad = 0;
    for (long long w = 0; w < (warps + 7) / 8 * 8; ++w) {
        if (w < first) {
            ++long_hits[w];
            continue;
        }
        const axgb::RowItem it = axgb::row_item(w - first, n_slices, nrhs, tile);
        if (!it.on) continue;
        if (it.slice < 0 || it.slice >= n_slices || it.tile < 0 || it.tile >= tiles)
            ++bad;
        else
            ++hits[it.tile * n_slices + it.slice];
    }
    return bad;
}

}
