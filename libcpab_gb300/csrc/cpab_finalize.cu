// Per-theta tail of every dtheta backward: sum the partial cell statistics,
// map them to dL/dA and contract with the basis,
// dtheta[k] = sum_i B[i, k] dA[i].
//
// A thread-block cluster of K CTAs works on one theta (or series, or point
// set), each on a contiguous slice of the cells: the CTA sums its columns of
// the partials (the threads of a column split the partials, and their sums are
// added in a fixed order), applies the cell map and contracts its rows of the
// basis; the leading CTA then adds the K partial dtheta rows over distributed
// shared memory in rank order.  One launch, no atomics, fixed summation order:
// the result is reproducible.
//
// The work is a few microseconds of reads, so what bounds it is the length of
// the dependent chain: one CTA per theta (the earlier scheme) walked all
// partials and all basis rows alone and left most SMs idle at small batches
// (51 us for one theta with 196 partials, 548 us for 64 thetas of [8,8] with
// 1536 x 234 basis elements, 211 us for 8 thetas of [4,4,4]; the whole forward
// and backward of the latter two went from 9.78 to 9.30 and from 14.45 to
// 14.27 ms).  K grows (1, 2,
// 4, 8: the portable cluster sizes) while the launch stays within four CTAs
// per SM and a CTA keeps at least four cells: with more, the cluster barrier
// costs more than the shorter chain gives.
#include <cooperative_groups.h>

#include "cpab_frechet.cuh"
#include "cpab_ragged.cuh"

namespace cpab {

namespace cg = cooperative_groups;

constexpr int kFinalizeThreads = 512;
// Columns of dtheta per launch: their share of a CTA is held in 32 KB of shared memory.
// Bases in use have some hundreds; wider ones take a launch for each slice.
constexpr int kFinalizeColumns = 8192;

// Where a theta's partials are: `count` rows of G floats from `first`.
// Dense: [n_theta][parts][G].  Ragged (tile_off != null): set s owns the slots
// v + s of the chunks v that touch it (see cpab_ragged.cuh).
struct Partials {
    const float *base;
    int parts;
    const int *tile_off;   // [S + 1] or null
    int S, warps, chunks;  // tile_chunks
};

__device__ __forceinline__ void partial_rows(const Partials &p, int th, long long *first,
                                             int *count) {
    if (!p.tile_off) {
        *first = (long long)th * p.parts;
        *count = p.parts;
        return;
    }
    const int TT = __ldg(p.tile_off + p.S);
    const TileChunks tc = tile_chunks(TT, p.warps, p.chunks);
    const int a = __ldg(p.tile_off + th), b = __ldg(p.tile_off + th + 1);
    const unsigned v0 = tc.of((unsigned)a);
    *first = (long long)v0 + th;
    *count = b > a ? (int)(tc.of((unsigned)(b - 1)) - v0) + 1 : 0;
}

// Cell statistics g (n cells from A's first row) -> dL/dA in place.
// mode 0: G = h S (I + h/2 [A;0])^T + h^2/2 A_lin^T S, S_c = sum_n
// lambda_{n+1} [p_n;1]^T; mode 1: the adjoint Frechet derivative of expm,
// dL/dA_c = dt [L_exp(X^T, [dL/dT_c; 0])]_{top rows}; mode 3 (exact-flow
// adjoint): already dL/dA.
template <int N, int MODE>
__device__ __forceinline__ void map_cells(float *g, const float *__restrict__ A, int n,
                                          const Steps &st) {
    constexpr int P = N * (N + 1);
    if constexpr (MODE == 3) return;
    for (int c = threadIdx.x; c < n; c += blockDim.x) {
        const float *a = A + (long long)c * P;
        if constexpr (MODE == 1) {
            const float dt = st.h;
            float Y[N + 1][N + 1], E[N + 1][N + 1], L[N + 1][N + 1];
#pragma unroll
            for (int i = 0; i <= N; ++i)
#pragma unroll
                for (int j = 0; j <= N; ++j) {
                    Y[j][i] = (i < N) ? dt * a[i * (N + 1) + j] : 0.f;   // Y = X^T
                    E[i][j] = (i < N) ? g[c * P + i * (N + 1) + j] : 0.f;
                }
            frechet_expm<N + 1>(Y, E, L);
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = 0; j <= N; ++j) g[c * P + i * (N + 1) + j] = dt * L[i][j];
        } else {
            float S[N][N + 1], Gc[N][N + 1];
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = 0; j <= N; ++j) S[i][j] = g[c * P + i * (N + 1) + j];
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = 0; j <= N; ++j) {
                    float x = 0.f, y = 0.f;
                    if (j < N) {
#pragma unroll
                        for (int k = 0; k <= N; ++k) x = fmaf(S[i][k], a[j * (N + 1) + k], x);
                    }
#pragma unroll
                    for (int r = 0; r < N; ++r) y = fmaf(a[r * (N + 1) + i], S[r][j], y);
                    Gc[i][j] = fmaf(st.h, fmaf(st.hh, x, S[i][j]), st.hh2 * y);
                }
#pragma unroll
            for (int i = 0; i < N; ++i)
#pragma unroll
                for (int j = 0; j <= N; ++j) g[c * P + i * (N + 1) + j] = Gc[i][j];
        }
    }
    __syncthreads();
}

// sum_{q = q0, q0 + step, ... < n} src[q * stride]: eight loads in flight, in
// eight interleaved sums combined in a fixed order.
__device__ __forceinline__ float strided_sum(const float *__restrict__ src, int q0, int step, int n,
                                             long long stride) {
    float s[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) s[u] = 0.f;
    int q = q0;
    for (; q + 7 * step < n; q += 8 * step)
#pragma unroll
        for (int u = 0; u < 8; ++u) s[u] += __ldg(src + (long long)(q + u * step) * stride);
    for (; q < n; q += step) s[0] += __ldg(src + (long long)q * stride);
    return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}

// d columns from basis and dtheta on, of rows of ld.
template <int N, int MODE>
__global__ void __launch_bounds__(kFinalizeThreads)
    k_finalize(int nC, int cells, Steps st, Partials ps, const float *__restrict__ A,
               const float *__restrict__ basis, int d, int ld, float *__restrict__ dtheta,
               const float *__restrict__ sse_partials, float *__restrict__ sse) {
    constexpr int P = N * (N + 1);
    extern __shared__ float4 smem4[];
    __shared__ float sse_s[kFinalizeThreads / 32];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), K = (int)cluster.num_blocks();
    const int th = blockIdx.x / K, tid = threadIdx.x, B = blockDim.x;
    const int G = nC * P;
    const int c0 = min(rank * cells, nC), c1 = min(c0 + cells, nC);
    const int rows = (c1 - c0) * P;
    float *g = reinterpret_cast<float *>(smem4);   // [cells * P] this slice's statistics
    float *red = g + round4(cells * P);            // [B] partial sums of a column
    float *dth = red + B;                          // [d] this slice's share of dtheta
    long long first;
    int count;
    partial_rows(ps, th, &first, &count);
    const float *src = ps.base + first * G + c0 * P;
    // the squared error: the chunks' sums over the whole block, in a fixed order (one
    // thread took up to 10,000 of them one after the other where a series is long)
    const bool squared = sse && rank == 0;
    if (squared) {
        float v = strided_sum(sse_partials + first, tid, B, count, 1);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (!(tid & 31)) sse_s[tid >> 5] = v;
    }
    auto store_sse = [&] {   // after a barrier
        if (!squared || tid) return;
        float acc = 0.f;
        for (int q = 0; q < kFinalizeThreads / 32; ++q) acc += sse_s[q];
        sse[th] = acc;
    };
    if (!dtheta || d <= 0) {   // uniform over the cluster
        __syncthreads();
        store_sse();
        return;
    }
    // columns of the partials, `split` threads on each
    if (rows > 0 && 2 * rows <= B) {
        const int split = B / rows, i = tid % rows, q0 = tid / rows;
        if (q0 < split) red[tid] = strided_sum(src + i, q0, split, count, G);
        __syncthreads();
        if (tid < rows) {
            float acc = red[tid];
            for (int q = 1; q < split; ++q) acc += red[q * rows + tid];
            g[tid] = acc;
        }
    } else {
        for (int i = tid; i < rows; i += B) g[i] = strided_sum(src + i, 0, 1, count, G);
    }
    __syncthreads();
    store_sse();
    map_cells<N, MODE>(g, A + (long long)th * G + c0 * P, c1 - c0, st);
    // rows of the basis, `split` threads on each column of dtheta
    const float *b = basis + (long long)c0 * P * ld;
    const int split = d <= B ? B / d : 1;
    for (int k0 = 0; k0 < d; k0 += B) {
        const int k = k0 + (d <= B ? tid % d : tid), r0 = d <= B ? tid / d : 0;
        float s[4] = {0.f, 0.f, 0.f, 0.f};
        if (k < d && r0 < split) {
            int i = r0;
            // 16 loads in flight, added in the same order as four by four
            for (; i + 15 * split < rows; i += 16 * split) {
                float v[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) v[u] = __ldg(b + (long long)(i + u * split) * ld + k);
#pragma unroll
                for (int u = 0; u < 16; ++u) s[u & 3] = fmaf(v[u], g[i + u * split], s[u & 3]);
            }
            for (; i + 3 * split < rows; i += 4 * split)
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    s[u] = fmaf(__ldg(b + (long long)(i + u * split) * ld + k), g[i + u * split],
                                s[u]);
            for (; i < rows; i += split)
                s[0] = fmaf(__ldg(b + (long long)i * ld + k), g[i], s[0]);
        }
        const float v = (s[0] + s[1]) + (s[2] + s[3]);
        if (split == 1) {
            if (k < d && r0 < split) dth[k] = v;
        } else {
            red[tid] = v;
            __syncthreads();
            if (tid < d) {
                float acc = red[tid];
                for (int q = 1; q < split; ++q) acc += red[q * d + tid];
                dth[tid] = acc;
            }
        }
    }
    if (K == 1) {   // each thread wrote the entries it stores
        for (int k = tid; k < d; k += B) dtheta[(long long)th * ld + k] = dth[k];
        return;
    }
    cluster.sync();   // every slice's share is in place
    for (int k = rank * B + tid; k < d; k += K * B) {
        float acc = 0.f;
        for (int q = 0; q < K; ++q) acc += cluster.map_shared_rank(dth, q)[k];
        dtheta[(long long)th * ld + k] = acc;
    }
    cluster.sync();   // no CTA leaves while its shared memory is read
}

template <int N, int MODE>
static cudaError_t launch_columns(int nC, const Steps &st, const Partials &ps, const float *A,
                                  const float *basis, int d, int ld, int n, float *dtheta,
                                  const float *sse_partials, float *sse, cudaStream_t s) {
    constexpr int P = N * (N + 1);
    int K = 1, max_optin = 48 * 1024;
    auto bytes = [&](int k) {
        return ((size_t)round4((nC + k - 1) / k * P) + kFinalizeThreads + (d > 0 ? d : 0)) *
               sizeof(float);
    };
    if (bytes(1) > 48 * 1024) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&max_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) !=
                cudaSuccess)
            return cudaErrorInvalidDevice;
    }
    while (K < 8 && (((long long)n * 2 * K <= 4ll * num_sms() && nC >= 8 * K) ||
                     bytes(K) > (size_t)max_optin))
        K *= 2;
    const size_t smem = bytes(K);
    auto kern = k_finalize<N, MODE>;
    if (const cudaError_t e = allow_smem((const void *)kern, smem)) return e;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = K;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n * K);
    cfg.blockDim = dim3(kFinalizeThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, nC, (nC + K - 1) / K, st, ps, A, basis, d, ld, dtheta,
                              sse_partials, sse);
}

template <int N, int MODE>
static cudaError_t launch_finalize_t(int nC, const Steps &st, const Partials &ps, const float *A,
                                     const float *basis, int d, int n, float *dtheta,
                                     const float *sse_partials, float *sse, cudaStream_t s) {
    for (int k = 0;;) {
        const cudaError_t e = launch_columns<N, MODE>(
            nC, st, ps, A, basis + k, std::min(d - k, kFinalizeColumns), d, n,
            dtheta ? dtheta + k : nullptr, sse_partials, k ? nullptr : sse, s);
        k += kFinalizeColumns;
        if (e != cudaSuccess || !dtheta || k >= d) return e;
    }
}

static cudaError_t dispatch(const Tess &t, int nsteps, int mode, const Partials &ps,
                            const float *A, const float *basis, int d, int n, float *dtheta,
                            const float *sse_partials, float *sse, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const Steps st = make_steps(nsteps);
#define CPAB_FIN(N)                                                                              \
    if (mode == kFinalizeDirect) /* the partials are dL/dA (exact-flow adjoint) */               \
        return launch_finalize_t<N, 3>(t.nC, st, ps, A, basis, d, n, dtheta, sse_partials, sse, s); \
    if (mode == 1)                                                                               \
        return launch_finalize_t<N, 1>(t.nC, st, ps, A, basis, d, n, dtheta, sse_partials, sse, s); \
    return launch_finalize_t<N, 0>(t.nC, st, ps, A, basis, d, n, dtheta, sse_partials, sse, s);
    switch (t.ndim) {
        case 1: { CPAB_FIN(1) }
        case 2: { CPAB_FIN(2) }
        default: { CPAB_FIN(3) }
    }
#undef CPAB_FIN
}

cudaError_t launch_finalize(const Tess &t, int nsteps, int mode, const float *partials, int parts,
                            const float *A, const float *basis, int d, int n_theta,
                            float *dtheta, cudaStream_t s) {
    const Partials ps = {partials, parts, nullptr, 0, 0};
    return dispatch(t, nsteps, mode, ps, A, basis, d, n_theta, dtheta, nullptr, nullptr, s);
}

cudaError_t launch_ragged_finalize(const Tess &t, int nsteps, int mode, const float *partials,
                                   const int *tile_off, int S, int warps, int chunks, const float *A,
                                   const float *basis, int d, float *dtheta,
                                   const float *sse_partials, float *sse, cudaStream_t s) {
    const Partials ps = {partials, 0, tile_off, S, warps, chunks};
    return dispatch(t, nsteps, mode, ps, A, basis, d, S, dtheta, sse_partials, sse, s);
}

}  // namespace cpab
