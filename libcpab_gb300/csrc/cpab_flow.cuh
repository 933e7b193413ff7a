// One sub-step of the exact flow and of its adjoint inside a cell (cpab_exact.cu),
// host and device: the host test checks the step's certificate and both series
// against 64 bits.
#pragma once
#include <cmath>

#include "cpab_common.cuh"

namespace cpab {

// How far a sub-step may pass a face of its cell (domain units).
constexpr float kOvershoot = 1e-5f;

// Conservative distance (domain units) from p to the face lines of its
// cell's square/cube and to the sub-cell diagonals/planes; the domain
// boundary is excluded (edge cells extend past it).  A single cell in 1D has no
// face: 1e15 stands for that, so that a step is bounded by 1 / |A| all the same,
// which the series and the quadrature of a step rest on.
template <int N>
CPAB_HD inline float face_distance(const float (&p)[N], const Tess &t) {
    float sub[N];
    float d = 1e15f;
    float imin = t.inc[0];
#pragma unroll
    for (int j = 0; j < N; ++j) {
        float fi, r;
        split_exact(p[j], t.inc[j], t.rinc[j], fi, r);
        const float ci = fminf(fmaxf(fi, 0.f), t.ncf[j] - 1.f);
        const float x = fmaf(r, t.rinc[j], fi - ci);
        sub[j] = x;
        if (ci > 0.f) d = fminf(d, fabsf(x) * t.inc[j]);
        if (ci < t.ncf[j] - 1.f) d = fminf(d, fabsf(1.f - x) * t.inc[j]);
        imin = fminf(imin, t.inc[j]);
    }
    if constexpr (N == 2) {
        const float s = imin * 0.70710678f;
        d = fminf(d, fabsf(sub[0] - sub[1]) * s);
        d = fminf(d, fabsf((sub[0] + sub[1]) - 1.f) * s);
    } else if constexpr (N == 3) {
        // the tetrahedron planes of both parities: z - x - y, x + y + z - 2,
        // y - x - z, x - y - z and their images under x <-> y, y -> 1 - x
        const float s = imin * 0.57735027f;
        const float x = sub[0], y = sub[1], z = sub[2];
        const float xf = y, yf = 1.f - x;
        d = fminf(d, fabsf((z - x) - y) * s);
        d = fminf(d, fabsf(((x + y) + z) - 2.f) * s);
        d = fminf(d, fabsf((y - x) - z) * s);
        d = fminf(d, fabsf((x - y) - z) * s);
        d = fminf(d, fabsf((z - xf) - yf) * s);
        d = fminf(d, fabsf(((xf + yf) + z) - 2.f) * s);
        d = fminf(d, fabsf((yf - xf) - z) * s);
        d = fminf(d, fabsf((xf - yf) - z) * s);
    }
    // rounding of the sub-cell coordinates (< 2^-22 of a cell)
    return fmaxf(d - 4e-7f * imin, 0.f);
}

// Root and quotient of a step's bound, approximate on the GPU: within 2^-22 of the exact
// ones (the rounded ones were a fifth of a step's dependent chain, and a trajectory
// that slides along a face takes thousands of steps one after the other: 64 x 224^2,
// forward and gradient, 3.96 ms, rounded 4.14).  With five roundings of 2^-24 a step
// is at most 2^-20 longer than the exact rule's, so it passes a face by at most
// kOvershoot + 2^-20.  (Taken off the step instead, that changes which steps a
// trajectory takes that ends at the limit of their number, and its result with them
// by up to 1e-3.)  The quotient is 0 for a bound above 2^126, which no finite speed
// gives: its square has overflowed at 2^64.  On the host the rounded ones, off by
// CPAB_FLOW_ERROR, which the test sets to the ends of the range.
#ifndef CPAB_FLOW_ERROR
#define CPAB_FLOW_ERROR 0.f
#endif
CPAB_HD inline float bound_root(float x) {
#if defined(__CUDA_ARCH__)
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return sqrtf(x) * (1.f + CPAB_FLOW_ERROR);
#endif
}
CPAB_HD inline float bound_quotient(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fdividef(a, b);
#else
    return (a / b) * (1.f - CPAB_FLOW_ERROR);
#endif
}

// Velocity at p in cell map M, and the certified step there; negative for a
// field that vanishes at p and has no linear part, or NaN input.
template <int N>
CPAB_HD inline float certified_step(const float (&M)[N * (N + 1)], const float (&p)[N],
                                    float (&v)[N], float &norm, const Tess &t) {
    float speed2 = 0.f, anorm2 = 0.f;
    affine_apply<N>(M, p, v);
#pragma unroll
    for (int r = 0; r < N; ++r) {
        speed2 = fmaf(v[r], v[r], speed2);
#pragma unroll
        for (int k = 0; k < N; ++k) anorm2 = fmaf(M[r * (N + 1) + k], M[r * (N + 1) + k], anorm2);
    }
    const float reach = face_distance<N>(p, t) + kOvershoot;
    norm = bound_root(anorm2);
    const float bound = bound_root(speed2) + norm * reach;
    return bound > 0.f ? bound_quotient(reach, bound) : -1.f;
}

// Terms of the in-cell flow's series: with |A| dt < 1 the first one left out is
// below 1 / 12! = 2e-9 of the step; below kShortStep (steps shrink towards a
// face), kShortTerms leave less than that.  Each lane decides for itself, so its
// result does not depend on its neighbours.
constexpr int kFlowTerms = 11, kShortTerms = 5;
constexpr float kShortStep = 0.06f;

// p + sum_{k=1..K} term_k, term_1 = dt v, term_{k+1} = dt A_lin term_k / (k + 1)
template <int N, int K>
CPAB_HD inline void flow_step(const float (&M)[N * (N + 1)], const float (&v)[N], float dt,
                              float (&p)[N]) {
    float term[N], sum[N];
#pragma unroll
    for (int r = 0; r < N; ++r) sum[r] = term[r] = dt * v[r];
#pragma unroll
    for (int k = 2; k <= K; ++k) {
        float nt[N];
        const float f = dt * (1.f / (float)k);
#pragma unroll
        for (int r = 0; r < N; ++r) {
            float q = 0.f;
#pragma unroll
            for (int j = 0; j < N; ++j) q = fmaf(M[r * (N + 1) + j], term[j], q);
            nt[r] = f * q;
        }
#pragma unroll
        for (int r = 0; r < N; ++r) {
            term[r] = nt[r];
            sum[r] += nt[r];
        }
    }
#pragma unroll
    for (int r = 0; r < N; ++r) p[r] += sum[r];
}

// Gauss-Legendre nodes and weights on [0, 1].
template <int G>
CPAB_HD constexpr float gauss_node(int n) {
    if (G == 2) return n == 0 ? 0.21132486540518711775f : 0.78867513459481288225f;
    return n == 0   ? 0.06943184420297371239f
           : n == 1 ? 0.33000947820757186760f
           : n == 2 ? 0.66999052179242813240f
                    : 0.93056815579702628761f;
}
template <int G>
CPAB_HD constexpr float gauss_weight(int n) {
    if (G == 2) return 0.5f;
    return n == 0 || n == 3 ? 0.17392742256872692869f : 0.32607257743127307131f;
}

// One sub-step back over dt from p (velocity v of the forward field M) with the
// cotangent lam: q [p_prev; 1], nl = lambda_prev, and acc += the integral of
// lambda [p; 1]^T.  K terms of the series of both at G nodes and at the end: for
// |A| dt < 1, 11 terms and 4 nodes (error below 6e-10 (2 |A| dt)^8 <= 1.5e-7 of
// the integrand), below kShortStep 5 and 2 ((2 |A| dt)^4 / 4320 <= 5e-8).
template <int N, int K, int G>
CPAB_HD inline void back_step(const float (&M)[N * (N + 1)], const float (&p)[N],
                              const float (&v)[N], const float (&lam)[N], float dt,
                              float (&acc)[N * (N + 1)], float (&q)[N + 1], float (&nl)[N]) {
    float tp[N], tl[N], sp[G + 1][N], sl[G + 1][N], power[G];
#pragma unroll
    for (int r = 0; r < N; ++r) {
        tp[r] = -dt * v[r];
        tl[r] = lam[r];
        sp[G][r] = tp[r];
        sl[G][r] = lam[r];
    }
#pragma unroll
    for (int n = 0; n < G; ++n) {
        power[n] = gauss_node<G>(n);
#pragma unroll
        for (int r = 0; r < N; ++r) {
            sp[n][r] = power[n] * tp[r];
            sl[n][r] = lam[r];
        }
    }
#pragma unroll
    for (int k = 1; k <= K; ++k) {
        const float fl = dt * (1.f / (float)k), fp = -dt * (1.f / (float)(k + 1));
        float np[N], nt[N];
#pragma unroll
        for (int r = 0; r < N; ++r) {
            float a = 0.f, b = 0.f;
#pragma unroll
            for (int j = 0; j < N; ++j) {
                a = fmaf(M[r * (N + 1) + j], tp[j], a);
                b = fmaf(M[j * (N + 1) + r], tl[j], b);
            }
            np[r] = fp * a;
            nt[r] = fl * b;
        }
#pragma unroll
        for (int r = 0; r < N; ++r) {
            tp[r] = np[r];
            tl[r] = nt[r];
            sl[G][r] += tl[r];
            sp[G][r] += tp[r];
        }
#pragma unroll
        for (int n = 0; n < G; ++n) {   // node^k for the cotangent, node^(k+1) for the point
#pragma unroll
            for (int r = 0; r < N; ++r) sl[n][r] = fmaf(power[n], tl[r], sl[n][r]);
            power[n] *= gauss_node<G>(n);
#pragma unroll
            for (int r = 0; r < N; ++r) sp[n][r] = fmaf(power[n], tp[r], sp[n][r]);
        }
    }
#pragma unroll
    for (int n = 0; n < G; ++n) {
        const float w = gauss_weight<G>(n) * dt;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float l = w * sl[n][i];
#pragma unroll
            for (int j = 0; j < N; ++j)
                acc[i * (N + 1) + j] = fmaf(l, p[j] + sp[n][j], acc[i * (N + 1) + j]);
            acc[i * (N + 1) + N] += l;
        }
    }
#pragma unroll
    for (int r = 0; r < N; ++r) {
        q[r] = p[r] + sp[G][r];
        nl[r] = sl[G][r];
    }
    q[N] = 1.f;
}

}  // namespace cpab
