// Device pieces shared by the ragged kernels (cpab_ragged.cu: 1D series;
// cpab_ragged_points.cu: point sets of any dimension).
//
// Work is cut into warp tiles of consecutive points of one set.  k_ragged_plan
// builds the tile prefix tile_off[S+1] on the device.  The forward kernels give a
// warp of a persistent grid the contiguous tile range [w K, (w+1) K), K =
// ceil(tiles / warps).  The adjoints cut the tiles into the chunks of tile_chunks:
// warp w takes chunk w, then the next one that nobody has (a counter in
// tile_off[S+1], which the plan sets to zero).  Set s is touched exactly by the
// chunks of its tiles and each (chunk, set) pair writes its own partial slot
// v + s, whichever warp ran it: the finalize sums a set's slots in chunk order
// (deterministic, no atomics).
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


// Chunks of the adjoints' tiles per SM (24 to 32 warps are resident; twice as many
// chunks made the sums and the finalize longer than it saved).
constexpr int kChunksPerSM = 64;
// Chunks per warp of the forward kernel of point sets (it keeps no sums): 1,024
// sets 0.60 -> 0.59 ms, 24 mixed images 0.141 -> 0.107 ms (0.62 and 0.116 with 3).
constexpr int kForwardChunks = 8;

// The next chunk for a warp that has done one (called by all its lanes).
__device__ __forceinline__ int next_chunk(int *counter, int warps) {
    int v = 0;
    if ((threadIdx.x & 31) == 0) v = warps + atomicAdd(counter, 1);
    return __shfl_sync(0xffffffffu, v, 0);
}

// Bytes of tile_off: the prefix and the counter.
inline size_t tile_off_bytes(int S) { return (((size_t)S + 2) * 4 + 255) & ~(size_t)255; }

// Warp-tile prefix over sets (one block): tile_off[s] = sum_{s'<s} tiles(s'),
// tile_off[S] = total tiles (tpw points per tile).  Invalid sets count as
// empty and raise kErrBadOffsets.  Defined in cpab_ragged.cu.
cudaError_t launch_ragged_plan(int S, const long long *off, long long total, int tpw,
                               int *tile_off, unsigned *err, cudaStream_t s);

}  // namespace cpab
