// Tile order and split of K shared by the fully connected layer's kernels.
#pragma once
#include "common.h"

namespace ttk {

// Tiles in bands of 16 tile rows, so that the CTAs of one wave share their operand panels in L2.
constexpr int kBandRows = 16;
__device__ __forceinline__ void fc_tile_coords(int t, int tiles_m, int tiles_n, int& mb, int& nb) {
    const int per_band = kBandRows * tiles_n;
    const int band = t / per_band;
    const int first = band * kBandRows;
    const int rows = min(kBandRows, tiles_m - first);
    const int r = t - band * per_band;
    mb = first + r % rows;
    nb = r / rows;
}

// CTAs of a cluster that share a tile's sum over K: as many as the SMs that the tiles leave idle, up to 8 (the portable
// cluster size), each with at least four of the `blocks` steps of 64 along K (the exchange costs about as much as those).
// bf16 forward [256,8192]x[8192,512] (4 tiles, 128 blocks) 46.5 -> 18.3 us, [2048,4096]x[4096,1024] (64 tiles) 30.1 -> 21.1;
// with 75 tiles and more every CTA keeps a tile of its own.  A cluster lies inside one GPC, so the largest counts of a size
// do not all run at once: [128 t,8192]x[8192,256] with t = 16, 18, 19 35.1, 36.4, 23.3 us, 33, 37, 38 23.8, 43.3, 30.2 (one CTA
// per tile 43 to 47).
inline int fc_k_ctas(long long tiles, int blocks) {
    int n = 1;
    while (n < 8 && tiles * n * 2 <= sm_count() && blocks >= n * 2 * 4) n *= 2;
    return n;
}

}  // namespace ttk
