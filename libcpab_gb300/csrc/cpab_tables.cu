// theta -> per-cell velocity maps A and step maps T / E = T - I.
//
// Replaces the host-side chain of the reference (libcpab/pytorch/transformer.py:146-155:
// B = torch.Tensor(basis) copied to the device on every call, As = B theta,
// Trels = expm(dT [A;0]) as ~15 small launches with a device->host sync in
// libcpab/pytorch/expm.py:30-32) with one launch.
//
// The exponential is computed in compensated form.  With X = dT [A;0] =
// [[M, v],[0, 0]] one has expm(X) - I = [[M phi(M), phi(M) v],[0, 0]] where
// phi(M) = sum_k M^k/(k+1)!.  phi is evaluated by Taylor series on M/2^s
// (||M/2^s||_1 <= 1/2, degree 10, truncation < 1e-11) and scaled back with
// the identity phi(2Y) = phi(Y) (I + Y phi(Y) / 2), which never forms
// I + (small) and so keeps the increment E to full FP32 relative precision.
// The integrator then advances p <- p + E [p;1]; with T stored directly the
// per-step increment would carry an absolute error of ~1 ulp of 1.
//
// A block takes a tile of cells and TB thetas.  The rows of the basis that belong
// to the tile go through shared memory in chunks of kChunk columns (coalesced
// loads, an odd pitch), one thread forms one entry of A = B theta for the TB
// thetas, in the order of the columns, and then one thread per (theta, cell) the
// exponential.  (One thread per (theta, cell) for all of it read the basis with a
// stride of P d between lanes, and waited on the queue of the load unit for nine
// cycles in ten.)  64 thetas, [8,8], d = 234: 95 -> 12 us (54 us with one theta per
// block and no chunk in flight); 4,096 thetas, [100]: 104 -> 24 us; 16 thetas of
// [50], d = 50, back to back 4.4 -> 3.2 us.  Small bases keep the one thread
// (k_cell_tables_small).
#include "cpab_expm.cuh"

namespace cpab {

constexpr int kChunk = 32;
template <int N>
__host__ __device__ constexpr int tile_cells() { return N == 1 ? 64 : N == 2 ? 32 : 16; }
template <int N>
__host__ __device__ constexpr int tile_rows() { return tile_cells<N>() * N * (N + 1); }

// T = expm(dt [A;0]) and E = T - I (either may be null) of one cell, from its rows a
// of A, to element off.
template <int N>
__device__ __forceinline__ void store_exp(const float *a, float dt, long long off,
                                          float *__restrict__ T, float *__restrict__ E) {
    float M[N][N], v[N], El[N][N], Et[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
#pragma unroll
        for (int j = 0; j < N; ++j) M[r][j] = a[r * (N + 1) + j] * dt;
        v[r] = a[r * (N + 1) + N] * dt;
    }
    expm1_affine<N>(M, v, El, Et);
#pragma unroll
    for (int r = 0; r < N; ++r) {
#pragma unroll
        for (int j = 0; j < N; ++j) {
            if (E) E[off + r * (N + 1) + j] = El[r][j];
            if (T) T[off + r * (N + 1) + j] = El[r][j] + ((r == j) ? 1.f : 0.f);
        }
        if (E) E[off + r * (N + 1) + N] = Et[r];
        if (T) T[off + r * (N + 1) + N] = Et[r];
    }
}

template <int N, int TB>
__global__ void __launch_bounds__(tile_rows<N>())
    k_cell_tables(int nC, int cells, int tiles, float dt, const float *__restrict__ theta,
                  int n_theta, int d, const float *__restrict__ basis, float *__restrict__ A,
                  float *__restrict__ T, float *__restrict__ E) {
    constexpr int P = N * (N + 1), R = tile_rows<N>(), W = R / 32;
    __shared__ float rows_s[R * (kChunk + 1)];
    __shared__ float theta_s[kChunk * TB];
    __shared__ float a_s[TB * R];
    const int tid = threadIdx.x, lane = tid & 31, wib = tid >> 5;
    const int c0 = (int)(blockIdx.x % (unsigned)tiles) * cells;
    const int th0 = (int)(blockIdx.x / (unsigned)tiles) * TB;
    const int nc = min(cells, nC - c0), rows = nc * P, nt = min(TB, n_theta - th0);
    const float *b0 = basis + (long long)c0 * P * d;
    float acc[TB];
#pragma unroll
    for (int q = 0; q < TB; ++q) acc[q] = 0.f;
    float next[32], next_t[(TB + W - 1) / W];   // the chunk after this one, in flight
    auto load = [&](int k) {
        const bool in = k + lane < d;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const int r = wib + i * W;
            next[i] = in && r < rows ? __ldg(b0 + (long long)r * d + k + lane) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < (TB + W - 1) / W; ++i) {
            const int q = wib + i * W;
            next_t[i] = in && q < nt ? __ldg(theta + (long long)(th0 + q) * d + k + lane) : 0.f;
        }
    };
    load(0);
    for (int k0 = 0; k0 < d; k0 += kChunk) {
        const int kc = min(kChunk, d - k0);
        if (k0) __syncthreads();
#pragma unroll
        for (int i = 0; i < 32; ++i) rows_s[(wib + i * W) * (kChunk + 1) + lane] = next[i];
#pragma unroll
        for (int i = 0; i < (TB + W - 1) / W; ++i)
            if (wib + i * W < TB) theta_s[lane * TB + wib + i * W] = next_t[i];
        __syncthreads();
        if (k0 + kChunk < d) load(k0 + kChunk);
        if (tid < rows) {
            const float *mine = rows_s + tid * (kChunk + 1);
#pragma unroll 8
            for (int k = 0; k < kc; ++k) {
                const float b = mine[k];
#pragma unroll
                for (int q = 0; q < TB; ++q) acc[q] = fmaf(b, theta_s[k * TB + q], acc[q]);
            }
        }
    }
    if (tid < rows) {
#pragma unroll
        for (int q = 0; q < TB; ++q) {
            a_s[q * R + tid] = acc[q];
            if (A && q < nt) A[((long long)(th0 + q) * nC + c0) * P + tid] = acc[q];
        }
    }
    if (!T && !E) return;
    __syncthreads();
    for (int i = tid; i < nt * nc; i += R) {
        const int q = i / nc, c = i - q * nc;
        store_exp<N>(a_s + q * R + c * P, dt, ((long long)(th0 + q) * nC + c0 + c) * P, T, E);
    }
}

// Small bases (see small_basis): one thread per (theta, cell) does all of it.  The
// basis stays in L1, and no lane waits for a tile to fill: 100,000 thetas of [2],
// d = 1, 6 us against 55 us on tiles, 65,536 of [20], d = 10, 16 against 41 us, 16 of
// [10], d = 5, 1.7 against 2.2 us.
template <int N>
__global__ void __launch_bounds__(128)
    k_cell_tables_small(int nC, float dt, const float *__restrict__ theta, int n_theta, int d,
                        const float *__restrict__ basis, float *__restrict__ A,
                        float *__restrict__ T, float *__restrict__ E) {
    constexpr int P = N * (N + 1);
    const long long gid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (long long)n_theta * nC) return;
    const long long th = gid / nC;
    const float *tv = theta + th * d, *rows = basis + (gid - th * nC) * P * d;
    float a[P];
#pragma unroll
    for (int i = 0; i < P; ++i) a[i] = 0.f;
    for (int k = 0; k < d; ++k) {
        const float tk = __ldg(tv + k);
#pragma unroll
        for (int i = 0; i < P; ++i) a[i] = fmaf(__ldg(rows + i * d + k), tk, a[i]);
    }
    if (A) {
#pragma unroll
        for (int i = 0; i < P; ++i) A[gid * P + i] = a[i];
    }
    if (T || E) store_exp<N>(a, dt, gid * P, T, E);
}

// Where one thread per (theta, cell) is the faster way, from both ways measured over
// [1] .. [16,16] and [4,4,4], d from a tenth to half of the rows, 1 to 500,000 thetas:
// 4 KB of basis or less, with up to 50 loads per thread (from there on its chain of
// loads is longer than the tile's barriers: [2,2], d = 9, 54 loads, equal; [20], d =
// 20, 40 loads, equal) or with thousands of thetas, which hide the chain ([1,1],
// d = 12, 65,536 thetas 8 against 103 us, 1,024 thetas 2.4 against 2.8 us).  With those also
// 8 KB, where the cells fill a third of a tile at most ([1,1,1], d = 30: 43 against
// 127 us).  Above, tiles: [50], d = 25, 65,536 thetas 60 us against 180 us.
template <int N>
static bool small_basis(int nC, int d, int n_theta) {
    constexpr int P = N * (N + 1);
    const long long floats = (long long)nC * P * d;
    if (floats <= 1024) return P * d <= 50 || n_theta >= 4096;
    return floats <= 2048 && n_theta >= 4096 && 3 * nC <= tile_cells<N>();
}

// Eight or four thetas per block (the basis is then read once for them) as long
// as that gives every other SM a block; else one, on smaller tiles of cells while
// there are SMs without one.
template <int N>
static cudaError_t launch_tables(int nC, float dt, const float *theta, int n_theta, int d,
                                 const float *basis, float *A, float *T, float *E,
                                 cudaStream_t s) {
    if (small_basis<N>(nC, d, n_theta)) {
        const long long grid = ((long long)n_theta * nC + 127) / 128;
        if (grid >= (1ll << 31)) return cudaErrorInvalidConfiguration;
        k_cell_tables_small<N><<<(unsigned)grid, 128, 0, s>>>(nC, dt, theta, n_theta, d, basis, A,
                                                              T, E);
        return cudaGetLastError();
    }
    int tiles = (nC + tile_cells<N>() - 1) / tile_cells<N>(), tb = 8;
    auto blocks = [&] { return (n_theta + tb - 1ll) / tb * tiles; };
    if (2 * blocks() < num_sms()) tb = 4;
    if (2 * blocks() < num_sms()) tb = 1;
    while (blocks() < num_sms() && tb == 1 && nC > 4 * tiles) tiles *= 2;
    const int cells = (nC + tiles - 1) / tiles;
    tiles = (nC + cells - 1) / cells;
    if (blocks() >= (1ll << 31)) return cudaErrorInvalidConfiguration;
    auto kern = tb == 8 ? k_cell_tables<N, 8> : tb == 4 ? k_cell_tables<N, 4> : k_cell_tables<N, 1>;
    kern<<<(unsigned)blocks(), tile_rows<N>(), 0, s>>>(nC, cells, tiles, dt, theta, n_theta, d,
                                                       basis, A, T, E);
    return cudaGetLastError();
}

cudaError_t launch_cell_tables(const Tess &t, int nsteps, const float *theta, int n_theta, int d,
                               const float *basis, float *A, float *T, float *E,
                               cudaStream_t s) {
    if ((long long)n_theta * t.nC == 0) return cudaSuccess;
    const float dt = (float)(1.0 / nsteps);
    switch (t.ndim) {
        case 1: return launch_tables<1>(t.nC, dt, theta, n_theta, d, basis, A, T, E, s);
        case 2: return launch_tables<2>(t.nC, dt, theta, n_theta, d, basis, A, T, E, s);
        default: return launch_tables<3>(t.nC, dt, theta, n_theta, d, basis, A, T, E, s);
    }
}

}  // namespace cpab
