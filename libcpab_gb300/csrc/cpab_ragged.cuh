// Device pieces shared by the ragged kernels (cpab_ragged.cu: 1D series;
// cpab_ragged_points.cu: point sets of any dimension).
//
// Work is cut into warp tiles of consecutive points of one set.  k_ragged_plan
// builds the tile prefix tile_off[S+1] on the device; a warp of a persistent
// grid owns the contiguous tile range [w K, (w+1) K), K = ceil(tiles / warps),
// so set s is touched exactly by warps tile_off[s]/K .. (tile_off[s+1]-1)/K and
// each (warp, set) pair writes its own partial slot w + s: the finalize sums a
// set's slots in warp order (deterministic, no atomics).
#pragma once
#include "cpab_adjoint.cuh"

namespace cpab {

__device__ __forceinline__ bool series_ok(long long a, long long b, long long total) {
    return a >= 0 && b >= a && b <= total && b - a < kRaggedMaxLen;
}

// Largest s with tile_off[s] <= t (tile_off[0] = 0 <= t < tile_off[S]).
__device__ __forceinline__ int find_series(const int *tile_off, int S, int t) {
    int lo = 0, hi = S;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(tile_off + mid) <= t) lo = mid;
        else hi = mid;
    }
    return lo;
}


// Warp-tile prefix over sets (one block): tile_off[s] = sum_{s'<s} tiles(s'),
// tile_off[S] = total tiles (tpw points per tile).  Invalid sets count as
// empty and raise kErrBadOffsets.  Defined in cpab_ragged.cu.
cudaError_t launch_ragged_plan(int S, const long long *off, long long total, int tpw,
                               int *tile_off, unsigned *err, cudaStream_t s);

}  // namespace cpab
