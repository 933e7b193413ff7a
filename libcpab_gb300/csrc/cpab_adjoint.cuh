// Device helpers shared by the adjoint kernels (cpab_adjoint.cu) and the
// fused transform_data backward (cpab_fused.cu).  The scheme is described at
// the top of cpab_adjoint.cu.
#pragma once
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "cpab_launch.h"
#include "cpab_midpoint.cuh"

namespace cpab {

constexpr int kSeg = 10;

// The per-cell adjoint table (build_dtab) is two arrays: the N x N
// propagators D (row stride dtab_stride, 16-byte aligned rows for the vector
// loads in 2D and 3D), then the N-float translations of the midpoint maps
// (row stride mtab_stride) starting at mtab_of.
template <int N>
__host__ __device__ constexpr int dtab_stride() { return N == 1 ? 1 : (N == 2 ? 4 : 12); }
template <int N>
__host__ __device__ constexpr int mtab_stride() { return N == 1 ? 1 : (N == 2 ? 2 : 4); }

__host__ __device__ inline int round4(int x) { return (x + 3) & ~3; }

template <int N>
__host__ __device__ inline int dtab_floats(int nC) {
    return round4(nC * dtab_stride<N>()) + round4(nC * mtab_stride<N>());
}
template <int N>
__host__ __device__ inline float *mtab_of(float *dtab, int nC) {
    return dtab + round4(nC * dtab_stride<N>());
}

// The midpoint step of an affine field is itself affine,
// p + h A~(p~ + h/2 A~ p~) = p + (h A~ + h^2/2 A~^2) p~ (A~ = [A; 0]): one map
// per cell.  The reverse sweep rebuilds segment positions with it (from the
// exactly stepped checkpoints of the forward sweep: positions within a few
// ulp of the reference's, which only the sums of lambda p~^T see).
template <int N>
__device__ __forceinline__ void load_dtab(const float *dtab, int c, float (&D)[N * N]);

template <int N>
__device__ __forceinline__ void mid_map_step(const float *dtab, const float *mtab, int c,
                                             float (&p)[N]) {
    float D[N * N], m[N];
    load_dtab<N>(dtab, c, D);
    const float *ms = mtab + c * mtab_stride<N>();
    if constexpr (N == 1) {
        m[0] = ms[0];
    } else if constexpr (N == 2) {
        const float2 b = *reinterpret_cast<const float2 *>(ms);
        m[0] = b.x; m[1] = b.y;
    } else {
        const float4 b = *reinterpret_cast<const float4 *>(ms);
        m[0] = b.x; m[1] = b.y; m[2] = b.z;
    }
    float y[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
        float acc = m[r];
#pragma unroll
        for (int k = 0; k < N; ++k) acc = fmaf(D[r * N + k], p[k], acc);
        y[r] = acc;
    }
#pragma unroll
    for (int r = 0; r < N; ++r) p[r] += y[r];
}

// One forward step of the trajectory that the adjoint differentiates: the
// reference's midpoint rule in modes 0 and 2 (tab holds A), the compensated
// step p += E [p; 1] of k_integrate in mode 1 (tab holds E).  Mode 2's
// logged forward takes the collapsed midpoint map instead (forward_step).
template <int N, int MODE>
__device__ __forceinline__ void traj_step(const float *tab, int c, const Steps &st,
                                          float (&p)[N]) {
    if constexpr (MODE == 0) {
        float A[N * (N + 1)];
        load_cell<N>(tab, c, A);
        ref_mid_step<N>(A, st, p);
    } else {
        constexpr int P = N * (N + 1);
        float M[P], y[N];
        load_cell<N>(tab, c, M);
        affine_apply<N>(M, p, y);
#pragma unroll
        for (int r = 0; r < N; ++r) p[r] += y[r];
    }
}

// The step the reverse sweep uses to rebuild a segment from its checkpoint:
// the midpoint map from dtab in mode 0, the compensated step in mode 1.
template <int N, int MODE>
__device__ __forceinline__ void rebuild_step(const float *tab, const float *dtab,
                                             const float *mtab, int c, const Steps &st,
                                             float (&p)[N]) {
    if constexpr (MODE != 1) mid_map_step<N>(dtab, mtab, c, p);
    else traj_step<N, 1>(tab, c, st, p);
}

// Per-cell adjoint table: row c of D at dtab[c * dtab_stride<N>()], the N x N
// propagator (row-major) with lambda_n = lambda_{n+1} + D^T lambda_{n+1}:
//     modes 0, 2: D = h A_lin + h^2/2 A_lin^2  (M - I of the midpoint sensitivity)
//     mode 1:     D = E_lin                     (the linear part of T - I)
// and, in modes 0 and 2, row c of mtab = mtab_of(dtab, nC), the translation of the
// midpoint map h a + h^2/2 A_lin a (a = the cell's translation column;
// mid_map_step).  tab keeps A (modes 0, 2) or E (mode 1).  Cells are split over
// the calling threads (first, first + stride, ...); the caller synchronises.
template <int N, int MODE>
__device__ __forceinline__ void build_dtab(const float *tab, float *dtab, int nC, const Steps &st,
                                           int first, int stride) {
    float *mtab = mtab_of<N>(dtab, nC);
    for (int c = first; c < nC; c += stride) {
        const float *a = tab + c * (N * (N + 1));
        float *d = dtab + c * dtab_stride<N>();
        float *m = mtab + c * mtab_stride<N>();
        if constexpr (MODE == 1) {
#pragma unroll
            for (int r = 0; r < N; ++r)
#pragma unroll
                for (int k = 0; k < N; ++k) d[r * N + k] = a[r * (N + 1) + k];
        } else {
#pragma unroll
            for (int r = 0; r < N; ++r)
#pragma unroll
                for (int k = 0; k <= N; ++k) {
                    float s = 0.f;
#pragma unroll
                    for (int q = 0; q < N; ++q) s = fmaf(a[r * (N + 1) + q], a[q * (N + 1) + k], s);
                    const float v = fmaf(st.h, a[r * (N + 1) + k], st.hh2 * s);
                    if (k < N) d[r * N + k] = v;
                    else m[r] = v;
                }
            if constexpr (N == 3) m[3] = 0.f;
        }
    }
}

template <int N>
__device__ __forceinline__ void load_dtab(const float *dtab, int c, float (&D)[N * N]) {
    const float *src = dtab + c * dtab_stride<N>();
    if constexpr (N == 1) {
        D[0] = src[0];
    } else if constexpr (N == 2) {
        const float4 a = *reinterpret_cast<const float4 *>(src);
        D[0] = a.x; D[1] = a.y; D[2] = a.z; D[3] = a.w;
    } else {
        const float4 a = reinterpret_cast<const float4 *>(src)[0];
        const float4 b = reinterpret_cast<const float4 *>(src)[1];
        D[0] = a.x; D[1] = a.y; D[2] = a.z; D[3] = a.w;
        D[4] = b.x; D[5] = b.y; D[6] = b.z; D[7] = b.w;
        D[8] = src[8];
    }
}

// One reverse step: S_c += lambda_{n+1} [p_n;1]^T, then lambda_n from
// lambda_{n+1}.  Both modes accumulate the same outer product; the mode-0
// cell gradient G_c is a fixed linear map of S_c applied in k_finalize.
template <int N>
__device__ __forceinline__ void adjoint_step(const float (&D)[N * N], const float (&p)[N],
                                             float (&lam)[N], float (&acc)[N * (N + 1)]) {
#pragma unroll
    for (int r = 0; r < N; ++r) {
#pragma unroll
        for (int k = 0; k < N; ++k) acc[r * (N + 1) + k] = fmaf(lam[r], p[k], acc[r * (N + 1) + k]);
        acc[r * (N + 1) + N] += lam[r];
    }
    float nl[N];
#pragma unroll
    for (int k = 0; k < N; ++k) {
        float s = lam[k];
#pragma unroll
        for (int r = 0; r < N; ++r) s = fmaf(D[r * N + k], lam[r], s);
        nl[k] = s;
    }
#pragma unroll
    for (int k = 0; k < N; ++k) lam[k] = nl[k];
}

// Shared memory carve-up for the adjoint kernels (floats unless noted):
//   tab   [round4(G)]            cell table of this theta (TMA destination)
//   dtab  [dtab_floats(nC)]      per-cell propagators D and midpoint-map translations
//   gw    [W][round4(G)]         per-warp cell-gradient tables (or in global memory, see
//                                carve_adjoint)
//   ck    [nseg][N][block]       checkpoints (position every kSeg steps)
//   pb    [kSeg][N][block]       positions of the segment being reversed
//   cl    [nsteps][block] (CT)   per-step cells
// Per-thread arrays are indexed [...][block] by thread, so warps access
// consecutive words (no bank conflicts).
template <int N, typename CT>
__host__ __device__ inline size_t adjoint_smem_bytes(int nC, int nsteps, int block,
                                                     bool gw_in_smem = true) {
    constexpr int P = N * (N + 1);
    const int G = round4(nC * P);
    const int Dn = dtab_floats<N>(nC);
    const int W = gw_in_smem ? block / 32 : 0;
    const int nseg = (nsteps + kSeg - 1) / kSeg;
    size_t b = (size_t)G * 4 + (size_t)Dn * 4 + (size_t)W * G * 4 +
               (size_t)nseg * N * block * 4 + (size_t)kSeg * N * block * 4 +
               (size_t)nsteps * block * sizeof(CT);
    return (b + 15) & ~(size_t)15;
}

// Host: the launch shape of an adjoint kernel with the most resident warps per
// SM among 256/128/64 threads per CTA and per-warp tables in shared memory
// (kern_shared) or in global memory (kern_global, may be nullptr; see
// carve_adjoint), where a warp counts seven eighths: its flushes wait for L2.
// [4,4], 64 x 224^2: 0.99 ms with 28 warps in shared memory, 1.04 ms with 32 in
// global memory; 13 x 151 x 203, exact mode, 0.139 and 0.155 ms; [4,5] 1.34
// (shared, 24 warps) and 1.32 ms, [5,5] 1.05 (24) and 1.04 ms.  Ties keep shared
// memory and the larger CTA.  force_block
// (> 0) and force_staging (0 shared, 1 global; -1 either) restrict the
// candidates (the autotuner's shapes).
template <int N, typename CT, typename K>
inline bool adjoint_shape(K kern_shared, K kern_global, int nC, int nsteps, int *block,
                          bool *global_gw, size_t *smem, int *per_sm, int force_block = 0,
                          int force_staging = -1) {
    const bool allow_global = kern_global != nullptr;
    int dev = 0, max_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (max_optin <= 0) max_optin = 48 * 1024;
    const int cands[3] = {256, 128, 64};
    int best = 0;
    for (int g = 0; g < (allow_global ? 2 : 1); ++g) {
        if (force_staging >= 0 && g != force_staging) continue;
        for (int ci = 0; ci < 3; ++ci) {
            const int b = cands[ci];
            if (force_block > 0 && b != force_block) continue;
            const size_t sm = adjoint_smem_bytes<N, CT>(nC, nsteps, b, g == 0) + 64;
            if (sm > (size_t)max_optin) continue;
            const K kern = g == 0 ? kern_shared : kern_global;
            if (allow_smem((const void *)kern, sm) != cudaSuccess) return false;
            const int n = resident_blocks((const void *)kern, b, sm);
            const int worth = n * (b / 32) * (g == 0 ? 8 : 7);
            if (worth > best) {
                best = worth;
                *block = b;
                *global_gw = g == 1;
                *smem = sm;
                *per_sm = n;
            }
        }
    }
    return best > 0;
}

// Host: CTAs per theta (or image), each taking every parts-th of its `tiles`
// tiles, for n of them on a GPU that holds `resident` CTAs.  In units of a
// tile the launch lasts about the average load of a resident slot (or, within
// one wave, one CTA, `own` tiles), plus 0.17 own for the uneven end (fitted to
// 9 .. 196 CTAs per image of 64 x 224^2), plus the setup of each CTA's tables of
// G floats.  Small tables are cheap, so most launches take one tile per CTA: 16
// images of 196 tiles 258 us, against 336 us with two waves of CTAs of up to 3
// tiles (the earlier rule), 64 images 921 against 1,003 us.
// max_waves bounds the CTAs (tables in global memory take space for each).
inline long long adjoint_parts(long long tiles, long long n, long long resident, int G,
                               double max_waves) {
    const double setup = 1e-4 * G;
    const long long most =
        std::max(1ll, std::min(tiles, (long long)(max_waves * (double)resident / (double)n) + 1));
    long long best = 1;
    double least = 0.0;
    for (long long p = 1; p <= most; p = p < 512 ? p + 1 : p + p / 64) {
        const double own = (double)((tiles + p - 1) / p), waves = (double)(n * p) / (double)resident;
        const double load = (double)(n * tiles) / (double)resident;
        const double cost = std::max(load, waves <= 1.0 ? own : 0.0) + 0.17 * own + waves * setup;
        if (p == 1 || cost < least) {
            best = p;
            least = cost;
        }
    }
    return best;
}

// Host: launch plans are computed once per problem shape and device (the
// occupancy queries behind a plan cost tens of microseconds, on the critical
// path of an eager training step).
struct PlanCache {
    using Key = std::tuple<int, int, int, int, int, int, int, long long, int, int, int>;
    std::mutex mu;
    std::map<Key, AdjointPlan> plans;

    template <typename F>
    bool get(int kind, const Tess &t, int nsteps, int mode, long long nP, int n, int flag,
             AdjointPlan *plan, F compute) {
        int dev = 0;
        cudaGetDevice(&dev);
        const Key key(dev, kind, t.ndim, t.nc[0], t.nc[1], t.nc[2], nsteps, nP, n, mode, flag);
        {
            std::lock_guard<std::mutex> lock(mu);
            auto it = plans.find(key);
            if (it != plans.end()) {
                *plan = it->second;
                return true;
            }
        }
        if (!compute(plan)) return false;
        std::lock_guard<std::mutex> lock(mu);
        if (plans.size() > 4096) plans.clear();
        plans[key] = *plan;
        return true;
    }
};

template <int N, typename CT>
struct AdjSmem {
    float *tab, *dtab, *mtab, *gw, *ck, *pb;
    CT *cl;
};

// GWG: gw_ext is this CTA's W per-warp tables in global memory (L2-resident; each
// warp owns its table and adds to it by reductions, see table_add), else the tables
// are in shared memory and the flush is a read, an addition and a write.  Global
// tables free shared memory for more resident warps when the tables are large (3D,
// hundreds of cells).
template <int N, typename CT, bool GWG = false>
__device__ __forceinline__ AdjSmem<N, CT> carve_adjoint(float *base, int nC, int nsteps,
                                                        float *gw_ext = nullptr) {
    constexpr int P = N * (N + 1);
    const int B = blockDim.x, W = B / 32;
    const int Gr = round4(nC * P);
    const int nseg = (nsteps + kSeg - 1) / kSeg;
    AdjSmem<N, CT> s;
    s.tab = base;
    s.dtab = s.tab + Gr;
    s.mtab = mtab_of<N>(s.dtab, nC);
    float *after = s.dtab + dtab_floats<N>(nC);
    if constexpr (GWG) {   // a template choice keeps the shared-memory path's
        s.gw = gw_ext;     // flushes on shared-memory instructions
        s.ck = after;
    } else {
        s.gw = after;
        s.ck = after + (size_t)W * Gr;
    }
    s.pb = s.ck + (size_t)nseg * N * B;
    s.cl = reinterpret_cast<CT *>(s.pb + (size_t)kSeg * N * B);
    return s;
}

// dst += v in the warp's table.  In global memory a fire-and-forget reduction:
// its element gets one addition per flush, flushes are ordered by __syncwarp,
// so the order of the sum is fixed all the same and nobody waits for a load.
template <bool GWG>
__device__ __forceinline__ void table_add(float *dst, float v) {
    if constexpr (GWG) atomicAdd(dst, v);
    else *dst += v;
}

// Sums of v[0..P) over the warp by recursive halving: at each round a lane
// keeps half of the values it holds and gives the other half to its partner,
// so P = 6 (padded to 8) takes 9 shuffles instead of 30.  Afterwards lane l
// holds, in v[0], the sum of value sum_index(l), the same in each lane that
// shares the index; the order of the additions is fixed.
template <int W, int P>
__device__ __forceinline__ void halve(float (&v)[P], int xor_lane, bool up) {
#pragma unroll
    for (int i = 0; i < W; ++i) {
        const float send = up ? v[i] : v[i + W], keep = up ? v[i + W] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, xor_lane);
    }
}

__host__ __device__ constexpr int pad_pow2(int P) { return P <= 2 ? 2 : P <= 8 ? 8 : 16; }

// Index of the value whose sum lane l holds (>= P: padding).
template <int P>
__device__ __forceinline__ int sum_index(int lane) {
    if constexpr (pad_pow2(P) == 16) return lane >> 1;
    else if constexpr (pad_pow2(P) == 8) return lane >> 2;
    else return lane >> 4;
}

template <int P>
__device__ __forceinline__ float warp_sums(const float (&acc)[P], bool in) {
    constexpr int W = pad_pow2(P);
    const int lane = threadIdx.x & 31;
    float v[W];
#pragma unroll
    for (int i = 0; i < W; ++i) v[i] = (i < P && in) ? acc[i < P ? i : 0] : 0.f;
    halve<W / 2>(v, 16, lane & 16);
    if constexpr (W >= 8) {
        halve<W / 4>(v, 8, lane & 8);
        halve<W / 8>(v, 4, lane & 4);
    }
    if constexpr (W >= 16) halve<1>(v, 2, lane & 2);
#pragma unroll
    for (int d = 16 / W; d > 0; d >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], d);
    return v[0];
}

// Add the accumulators of the lanes that leave their cell at this step into
// the warp's cell table, for warps of neighbouring points (called by all lanes
// of the warp).  A lane that leaves its cell alone adds its sums itself.  Lanes
// that leave the same cell together, as neighbours that cross a face do, are
// summed first: up to four of a kind one after the other into their lowest
// lane, all cells at once (15 instructions per lane of the largest group),
// else one cell after the other by warp_sums (50 instructions per cell).  Every
// table element so receives at most one addition per step, in step order, and
// the summation order depends only on the inputs: the sums are reproducible.
// [8,8] on a 512^2 meshgrid, adjoint kernel: 7.1 ms with flush_scattered, 6.4 ms
// with this, 5.1 ms on patches (PointOrder).
constexpr int kChainLanes = 4;

template <int P, bool GWG>
__device__ __forceinline__ void flush_neighbours(bool change, int cell, const float (&acc)[P],
                                                 float *warp_tab) {
    const int lane = threadIdx.x & 31;
    const unsigned grp = __match_any_sync(0xffffffffu, change ? cell : -1 - lane);
    const int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)__popc(grp));
    if (most <= kChainLanes) {
        float sum[P];
#pragma unroll
        for (int i = 0; i < P; ++i) sum[i] = acc[i];
        unsigned rest = grp & (grp - 1u);        // the other members, lowest first
#pragma unroll 1
        for (int k = 1; k < most; ++k) {
            const int src = rest ? __ffs(rest) - 1 : lane;
#pragma unroll
            for (int i = 0; i < P; ++i) {
                const float u = __shfl_sync(0xffffffffu, acc[i], src);
                if (rest) sum[i] += u;
            }
            rest &= rest - 1u;
        }
        if (change && lane == __ffs(grp) - 1) {
            float *dst = warp_tab + cell * P;
#pragma unroll
            for (int i = 0; i < P; ++i) table_add<GWG>(dst + i, sum[i]);
        }
    } else {
        const bool alone = (grp & (grp - 1u)) == 0u;
        unsigned todo = __ballot_sync(0xffffffffu, change && !alone);
        if (change && alone) {
            float *dst = warp_tab + cell * P;
#pragma unroll
            for (int i = 0; i < P; ++i) table_add<GWG>(dst + i, acc[i]);
        }
#pragma unroll 1
        while (todo) {
            const int first = __ffs(todo) - 1;
            const unsigned g = __shfl_sync(0xffffffffu, grp, first);
            const int c = __shfl_sync(0xffffffffu, cell, first);
            const float v = warp_sums<P>(acc, (g >> lane) & 1u);
            const int i = sum_index<P>(lane);
            if (i < P && (lane & (32 / pad_pow2(P) - 1)) == 0)
                table_add<GWG>(warp_tab + c * P + i, v);
            todo &= ~g;
        }
    }
    __syncwarp();
}

// Sum each contiguous lane run [lo, hi] of sum[] into lane lo (five fixed
// shuffle rounds) and add it there.  All lanes of m call it; runs lie in m.
template <int P>
__device__ __forceinline__ void add_runs(unsigned m, int lo, int hi, float (&sum)[P], float *dst) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const float u = __shfl_down_sync(m, sum[i], off);
            if (lane + off <= hi) sum[i] += u;
        }
    }
    if (lane == lo) {
#pragma unroll
        for (int i = 0; i < P; ++i) dst[i] += sum[i];
    }
}

// The same for warps of scattered points, called by exactly the lanes in m that
// leave a cell at this step: the largest group decides how all are summed, which
// is cheaper where groups are few and small (1,024 sets of random points 2.54
// against 2.65 ms).  Lanes that
// leave the same cell at the same step are first summed into their lowest
// lane (a fixed shuffle tree when every group is a contiguous run of more than
// four lanes, else a lane-order chain), so every table element receives at
// most one add per step, in step order, and the summation order depends only
// on the inputs: the sums are reproducible.  In the common case (no two lanes
// share a cell) all lanes add in one pass.
template <int P>
__device__ __forceinline__ void flush_scattered(unsigned m, int cell, const float (&acc)[P],
                                            float *warp_tab) {
    const int lane = threadIdx.x & 31;
    float *dst = warp_tab + cell * P;
    const unsigned grp = __match_any_sync(m, cell);
    const unsigned gmax = __reduce_max_sync(m, (unsigned)__popc(grp));
    if (gmax == 1u) {
#pragma unroll
        for (int i = 0; i < P; ++i) dst[i] += acc[i];
        return;
    }
    float sum[P];
#pragma unroll
    for (int i = 0; i < P; ++i) sum[i] = acc[i];
    const int lo = __ffs(grp) - 1;
    const unsigned run = grp >> lo;
    if (gmax > 4u && __all_sync(m, (run & (run + 1u)) == 0u)) {
        // Every group is a contiguous run of lanes [lo, hi] (typical when
        // neighbouring points cross a face together): tree reduction towards
        // the lowest lane in five fixed shuffle rounds.
        add_runs<P>(m, lo, 31 - __clz(grp), sum, dst);
        return;
    }
    unsigned rest = grp & (grp - 1u);        // the other members, lowest first
    for (unsigned k = 1; k < gmax; ++k) {
        const int src = rest ? __ffs(rest) - 1 : lane;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const float u = __shfl_sync(m, acc[i], src);
            if (rest) sum[i] += u;
        }
        rest &= rest - 1u;
    }
    if (lane == __ffs(grp) - 1) {
#pragma unroll
        for (int i = 0; i < P; ++i) dst[i] += sum[i];
    }
}

// Warp-level flush: lanes with flush = true add their accumulators for
// `cell`.  Called by all lanes of the warp.
template <int P>
__device__ __forceinline__ void warp_flush(bool flush, int cell, const float (&acc)[P],
                                           float *warp_tab) {
    const unsigned m = __ballot_sync(0xffffffffu, flush);
    if (m) {
        if (flush) flush_scattered<P>(m, cell, acc, warp_tab);
        __syncwarp();
    }
}

// 1D variant of warp_flush.  A 1D flow keeps the order of points, so the
// lanes of a warp holding consecutive points of a sorted grid (the ragged
// series) sit in non-decreasing cells: equal cells form contiguous lane runs.
// Then every lane takes part in a fixed five-round shuffle tree over its run
// (non-flushing lanes add zeros) and the run's lowest lane adds the sum if
// any lane of the run flushes: the same one-add-per-element-per-step
// discipline as flush_scattered, without match.any.  Unsorted warps use
// warp_flush.  Called by all lanes of the warp.
template <int P>
__device__ __forceinline__ void warp_flush_1d(bool flush, int cell, const float (&acc)[P],
                                              float *warp_tab) {
    const unsigned fm = __ballot_sync(0xffffffffu, flush);
    if (!fm) return;
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(0xffffffffu, cell, 1);
    if (__any_sync(0xffffffffu, lane > 0 && prev > cell)) {
        warp_flush<P>(flush, cell, acc, warp_tab);
        return;
    }
    const unsigned heads = __ballot_sync(0xffffffffu, lane == 0 || prev != cell);
    const unsigned le = 0xffffffffu >> (31 - lane);            // lanes <= lane
    const int lo = 31 - __clz(heads & le);
    const unsigned above = heads & ~le;
    const int hi = above ? __ffs(above) - 2 : 31;
    float sum[P];
#pragma unroll
    for (int i = 0; i < P; ++i) sum[i] = flush ? acc[i] : 0.f;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const float u = __shfl_down_sync(0xffffffffu, sum[i], off);
            if (lane + off <= hi) sum[i] += u;
        }
    }
    const unsigned run = (hi == 31 ? 0xffffffffu : ((1u << (hi + 1)) - 1u)) & ~((1u << lo) - 1u);
    if (lane == lo && (fm & run)) {
        float *dst = warp_tab + cell * P;
#pragma unroll
        for (int i = 0; i < P; ++i) dst[i] += sum[i];
    }
    __syncwarp();
}

// Where reverse_sweep puts a lane's accumulated dL/dA of a cell when the lane
// leaves it: the warp's cell table.  changed() is called by all lanes of the
// warp with the ballot of the lanes that leave their cell, not zero.
// SCATTERED: the warp's points are in no order that this code knows of.
template <int N, bool GWG, bool SCATTERED>
struct WarpTabSink {
    static constexpr bool kWarp = true;   // changed() is a warp-wide call
    float *warp_tab;
    template <int P>
    __device__ __forceinline__ void changed(unsigned m, bool change, int cell,
                                            const float (&acc)[P]) const {
        if constexpr (N == 1) {
            warp_flush_1d<P>(change, cell, acc, warp_tab);
        } else if constexpr (SCATTERED) {
            if (change) flush_scattered<P>(m, cell, acc, warp_tab);
            __syncwarp();
        } else {
            flush_neighbours<P, GWG>(change, cell, acc, warp_tab);
        }
    }
};

// Reverse sweep of one trajectory whose cells are logged in cl and whose
// checkpoints are in ck; lam holds dL/dp_N on entry and dL/dp_0 on exit.  A lane
// without a point walks with lam = 0 from a point that another lane of the theta
// has: its sums are zeros unless that trajectory overflows (0 * inf is NaN), and
// then that lane's are not finite either.
// Each segment's positions are rebuilt from its checkpoint with the logged
// cells (no lookups) into pb, then walked backwards.  The loops are not
// unrolled: the body stays small enough for the instruction cache (unrolled by
// five, with the positions in registers, it ran 18 % fewer instructions and
// took 35 % longer at [8,8], 18 % at [4,4,4]).  A lane reloads the propagator
// only where it enters another cell.
// Executed by all lanes of the warp (uniform trip counts); sink receives each
// lane's sum over a run of steps in one cell.
template <int N, int MODE, typename CT, typename Sink>
__device__ __forceinline__ void reverse_sweep_to(const AdjSmem<N, CT> &sm, int nsteps,
                                                 const Steps &st, float (&lam)[N], Sink &sink) {
    constexpr int P = N * (N + 1);
    const int B = blockDim.x, tid = threadIdx.x;
    const int nseg = (nsteps + kSeg - 1) / kSeg;
    float acc[P], D[N * N];
#pragma unroll
    for (int i = 0; i < P; ++i) acc[i] = 0.f;
    int gcell = (int)sm.cl[(nsteps - 1) * B + tid];
    load_dtab<N>(sm.dtab, gcell, D);
    for (int seg = nseg - 1; seg >= 0; --seg) {
        const int n0 = seg * kSeg;
        const int len = min(kSeg, nsteps - n0);
        float x[N];
#pragma unroll
        for (int r = 0; r < N; ++r) x[r] = sm.ck[(seg * N + r) * B + tid];
#pragma unroll 1
        for (int s = 0; s < len; ++s) {
#pragma unroll
            for (int r = 0; r < N; ++r) sm.pb[(s * N + r) * B + tid] = x[r];
            rebuild_step<N, MODE>(sm.tab, sm.dtab, sm.mtab, (int)sm.cl[(n0 + s) * B + tid], st,
                                  x);
        }
#pragma unroll 1
        for (int s = len - 1; s >= 0; --s) {
            const int c = (int)sm.cl[(n0 + s) * B + tid];
            const bool change = c != gcell;
            const unsigned m = Sink::kWarp ? __ballot_sync(0xffffffffu, change) : change;
            if (m) {
                sink.changed(m, change, gcell, acc);
                if (change) {
                    gcell = c;
#pragma unroll
                    for (int i = 0; i < P; ++i) acc[i] = 0.f;
                    load_dtab<N>(sm.dtab, c, D);
                }
            }
            float p[N];
#pragma unroll
            for (int r = 0; r < N; ++r) p[r] = sm.pb[(s * N + r) * B + tid];
            adjoint_step<N>(D, p, lam, acc);
        }
    }
    sink.changed(0xffffffffu, true, gcell, acc);
}

template <int N, int MODE, typename CT, bool GWG, bool SCATTERED>
__device__ __forceinline__ void reverse_sweep(const AdjSmem<N, CT> &sm, int nsteps,
                                              const Steps &st, float (&lam)[N],
                                              float *warp_tab) {
    WarpTabSink<N, GWG, SCATTERED> sink{warp_tab};
    reverse_sweep_to<N, MODE, CT>(sm, nsteps, st, lam, sink);
}

template <int N>
__device__ __forceinline__ void e_step(const float *tabE, const Tess &t, float (&p)[N],
                                       unsigned long long *ties) {
    constexpr int P = N * (N + 1);
    const int c = find_cell<N>(p, t, ties);
    float M[P], y[N];
    load_cell<N>(tabE, c, M);
    affine_apply<N>(M, p, y);
#pragma unroll
    for (int r = 0; r < N; ++r) p[r] += y[r];
}

// Sweep with the arithmetic of k_integrate's compensated path,
// p <- p + E_c [p;1], nsteps times.  tabE may be in shared or global memory.
template <int N>
__device__ __forceinline__ void e_sweep(const float *tabE, const Tess &t, int nsteps,
                                        float (&p)[N], unsigned long long *ties, unsigned *err) {
    for (int s = 0; s < nsteps; ++s) e_step<N>(tabE, t, p, ties);
}

// Forward sweep that logs cells and checkpoints; p holds p_0 on entry and
// p_N on exit.
// beside: another trajectory's step, taken at each of these.
struct NoStep {
    __device__ __forceinline__ void operator()() const {}
};

template <int N, int MODE, typename CT, typename Step = NoStep>
__device__ __forceinline__ void logged_forward(const AdjSmem<N, CT> &sm, const Tess &t,
                                               int nsteps, const Steps &st, float (&p)[N],
                                               unsigned long long *ties, unsigned *err,
                                               const Step &beside = Step()) {
    const int B = blockDim.x, tid = threadIdx.x;
    for (int n0 = 0, seg = 0; n0 < nsteps; n0 += kSeg, ++seg) {
#pragma unroll
        for (int r = 0; r < N; ++r) sm.ck[(seg * N + r) * B + tid] = p[r];
        const int end = min(n0 + kSeg, nsteps);
        for (int n = n0; n < end; ++n) {
            int c = find_cell<N>(p, t, ties);
            sm.cl[n * B + tid] = (CT)c;
            if constexpr (MODE == 2) mid_map_step<N>(sm.dtab, sm.mtab, c, p);
            else traj_step<N, MODE>(sm.tab, c, st, p);
            beside();
        }
    }
}

// Order of a theta's points over the threads of the adjoint.  The points of a
// meshgrid (the first axis fastest, uniform_meshgrid's order) are taken in
// patches of 8 x 4, 4 x 8 or 16 x 2 points per warp instead of 32 along a row:
// the lanes then cross a cell boundary at nearly the same step, so the warp
// flushes its cell sums at fewer steps (flush_neighbours).  The length of a row
// is read off the points: it is the number of leading points that share their
// second coordinate.  Any points may be passed, this is a permutation of them
// whatever they are.
struct PointOrder {
    int row, wide, shift;   // row length (0: in order), patch width and log2 of it
};

constexpr int kMaxRow = 1024;   // rows looked for (four reads of a 256-thread block)

// Called by all threads of the block; `found` is shared.
// MOVED: the points are a meshgrid that a transformation has moved; its rows are
// told by the jump back of the first coordinate instead.
template <int N, bool MOVED = false>
__device__ __forceinline__ PointOrder point_order(const float *points, long long nP, int *found) {
    PointOrder o = {0, 32, 5};
    if constexpr (N >= 2) {
        if (nP < 64 || nP >= (1ll << 31)) return o;
        if (threadIdx.x == 0) *found = kMaxRow + 1;
        __syncthreads();
        const float *y = points + (MOVED ? 0 : nP);
        const float y0 = __ldg(y);
        const int most = (int)min(nP, (long long)kMaxRow + 1);
        int row = kMaxRow + 1;
        for (int i = 1 + threadIdx.x; i - (int)threadIdx.x < most; i += blockDim.x) {
            if (i < most && (MOVED ? __ldg(y + i) < __ldg(y + i - 1) - 0.25f : __ldg(y + i) != y0))
                atomicMin(found, i);
            __syncthreads();
            row = *found;
            __syncthreads();
            if (row <= kMaxRow) break;
        }
        if (row > kMaxRow || nP % row) return o;
        const int rows = (int)(nP / row);
        if (row % 8 == 0 && rows % 4 == 0) o.shift = 3;
        else if (row % 4 == 0 && rows % 8 == 0) o.shift = 2;
        else if (row % 16 == 0 && rows % 2 == 0) o.shift = 4;
        else return o;
        o.row = row;
        o.wide = 1 << o.shift;
    }
    return o;
}

// Index of the point of thread v.
__device__ __forceinline__ long long ordered_point(long long v, const PointOrder &o) {
    if (!o.row) return v;
    const unsigned w = (unsigned)(v >> 5), lane = (unsigned)v & 31u;
    const unsigned per = (unsigned)o.row >> o.shift;
    const unsigned band = w / per, col = w - band * per;
    const unsigned r = band * (32u >> o.shift) + (lane >> o.shift);
    return (long long)r * o.row + col * o.wide + (lane & (o.wide - 1u));
}

// Kernel prologue: stage the cell table, build the propagators and clear the
// per-warp tables.  Returns false (block exits) if staging failed.
template <int N, int MODE, typename CT>
__device__ __forceinline__ bool adjoint_prologue(const AdjSmem<N, CT> &sm, const float *table,
                                                 int nC, const Steps &st, uint64_t *bar,
                                                 unsigned *err) {
    constexpr int P = N * (N + 1);
    const int W = blockDim.x / 32, Gr = round4(nC * P);
    if (!stage_table(sm.tab, table, nC * P, bar, err)) return false;
    build_dtab<N, MODE>(sm.tab, sm.dtab, nC, st, threadIdx.x, blockDim.x);
    for (int i = threadIdx.x; i < W * Gr; i += blockDim.x) sm.gw[i] = 0.f;
    __syncthreads();
    return true;
}

// Kernel epilogue: write this CTA's partial (per-warp tables summed in warp
// order).
template <int N, typename CT, bool GWG>
__device__ __forceinline__ void adjoint_epilogue(const AdjSmem<N, CT> &sm, int nC, float *dst) {
    constexpr int P = N * (N + 1);
    const int B = blockDim.x, W = B / 32, G = nC * P, Gr = round4(G);
    __syncthreads();
    for (int i = threadIdx.x; i < G; i += B) {
        float s = 0.f;
        for (int w = 0; w < W; ++w) {
            const float *q = sm.gw + (size_t)w * Gr + i;
            s += GWG ? __ldcg(q) : *q;   // the reductions are in L2
        }
        dst[i] = s;
    }
}

}  // namespace cpab
