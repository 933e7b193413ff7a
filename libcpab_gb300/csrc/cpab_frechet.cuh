// Frechet derivative of the matrix exponential, for the finalize kernel
// (cpab_finalize.cu).
#pragma once
#include "cpab_launch.h"

namespace cpab {

// Frechet derivative of expm at Y in direction E, by a truncated Horner
// recursion on Y/2^s, E/2^s followed by s squarings:
//   R_{k-1} = I + (Y/k) R_k,  dR_{k-1} = (E/k) R_k + (Y/k) dR_k,
//   then  L <- L R + R L,  R <- R R.
template <int K>
__device__ __forceinline__ void frechet_expm(const float (&Y0)[K][K], const float (&E0)[K][K],
                                             float (&L)[K][K]) {
    float norm = 0.f;
#pragma unroll
    for (int j = 0; j < K; ++j) {
        float s = 0.f;
#pragma unroll
        for (int i = 0; i < K; ++i) s += fabsf(Y0[i][j]);
        norm = fmaxf(norm, s);
    }
    int sq = 0;
    if (norm > 0.5f) sq = min(64, (int)ceilf(log2f(norm / 0.5f)));
    const float sc = ldexpf(1.f, -sq);
    float Y[K][K], E[K][K], R[K][K], D[K][K];
#pragma unroll
    for (int i = 0; i < K; ++i)
#pragma unroll
        for (int j = 0; j < K; ++j) {
            Y[i][j] = Y0[i][j] * sc;
            E[i][j] = E0[i][j] * sc;
            R[i][j] = (i == j) ? 1.f : 0.f;
            D[i][j] = 0.f;
        }
    for (int k = 12; k >= 1; --k) {
        const float r = 1.f / (float)k;
        float nR[K][K], nD[K][K];
#pragma unroll
        for (int i = 0; i < K; ++i)
#pragma unroll
            for (int j = 0; j < K; ++j) {
                float a = 0.f, b = 0.f;
#pragma unroll
                for (int m = 0; m < K; ++m) {
                    a = fmaf(Y[i][m], R[m][j], a);
                    b = fmaf(E[i][m], R[m][j], fmaf(Y[i][m], D[m][j], b));
                }
                nR[i][j] = fmaf(a, r, (i == j) ? 1.f : 0.f);
                nD[i][j] = b * r;
            }
#pragma unroll
        for (int i = 0; i < K; ++i)
#pragma unroll
            for (int j = 0; j < K; ++j) { R[i][j] = nR[i][j]; D[i][j] = nD[i][j]; }
    }
    for (int s = 0; s < sq; ++s) {
        float nR[K][K], nD[K][K];
#pragma unroll
        for (int i = 0; i < K; ++i)
#pragma unroll
            for (int j = 0; j < K; ++j) {
                float a = 0.f, b = 0.f;
#pragma unroll
                for (int m = 0; m < K; ++m) {
                    a = fmaf(R[i][m], R[m][j], a);
                    b = fmaf(D[i][m], R[m][j], fmaf(R[i][m], D[m][j], b));
                }
                nR[i][j] = a;
                nD[i][j] = b;
            }
#pragma unroll
        for (int i = 0; i < K; ++i)
#pragma unroll
            for (int j = 0; j < K; ++j) { R[i][j] = nR[i][j]; D[i][j] = nD[i][j]; }
    }
#pragma unroll
    for (int i = 0; i < K; ++i)
#pragma unroll
        for (int j = 0; j < K; ++j) L[i][j] = D[i][j];
}

}  // namespace cpab
