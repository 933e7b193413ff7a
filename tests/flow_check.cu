// Host harness for one sub-step of the exact flow and of its adjoint
// (libcpab_gb300/csrc/cpab_flow.cuh; compiled by tests/test_exact_substep_host.py
// with nvcc and -ffp-contract=off; runs on the CPU).
//
// usage: flow_check <in.bin> <out.bin>
//   in:  int32 ndim, int32 nc[3], int64 n, float A[n][ndim][ndim+1], float p[n][ndim],
//        float lam[n][ndim], float time[n]
//   out: per point: float step, norm, reach, dt, end[ndim], start[ndim], lam_start[ndim],
//        grad[ndim][ndim+1]
// dt = min(time, step) (time where there is no step) as in the kernels: `end` is the
// flow over dt, the rest the adjoint's sub-step back over dt.
#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <vector>

#include "../libcpab_gb300/csrc/cpab_flow.cuh"

template <int N>
static void run(const cpab::Tess &t, int64_t n, const float *A, const float *p, const float *lam,
                const float *time, std::vector<float> &out) {
    constexpr int P = N * (N + 1);
    for (int64_t i = 0; i < n; ++i) {
        float M[P], x[N], l[N], v[N], norm, end[N], acc[P], q[N + 1], nl[N];
        std::copy(A + i * P, A + (i + 1) * P, M);
        std::copy(p + i * N, p + (i + 1) * N, x);
        std::copy(lam + i * N, lam + (i + 1) * N, l);
        const float step = cpab::certified_step<N>(M, x, v, norm, t);
        const float dt = step >= 0.f ? fminf(time[i], step) : time[i];
        std::copy(x, x + N, end);
        std::fill(acc, acc + P, 0.f);
        if (norm * dt < cpab::kShortStep) {
            cpab::flow_step<N, cpab::kShortTerms>(M, v, dt, end);
            cpab::back_step<N, cpab::kShortTerms, 2>(M, x, v, l, dt, acc, q, nl);
        } else {
            cpab::flow_step<N, cpab::kFlowTerms>(M, v, dt, end);
            cpab::back_step<N, cpab::kFlowTerms, 4>(M, x, v, l, dt, acc, q, nl);
        }
        const float head[4] = {step, norm, cpab::face_distance<N>(x, t) + cpab::kOvershoot, dt};
        out.insert(out.end(), head, head + 4);
        out.insert(out.end(), end, end + N);
        out.insert(out.end(), q, q + N);
        out.insert(out.end(), nl, nl + N);
        out.insert(out.end(), acc, acc + P);
    }
}

int main(int argc, char **argv) {
    if (argc != 3) return 2;
    FILE *f = fopen(argv[1], "rb");
    if (!f) return 3;
    int32_t hdr[4];
    int64_t n = 0;
    if (fread(hdr, 4, 4, f) != 4 || fread(&n, 8, 1, f) != 1) return 4;
    const int ndim = hdr[0];
    cpab::Tess t;
    cpab::tess_init(ndim, hdr + 1, &t);
    std::vector<float> A((size_t)n * ndim * (ndim + 1)), p((size_t)n * ndim), lam(p.size()), time(n);
    for (auto *v : {&A, &p, &lam, &time})
        if (fread(v->data(), 4, v->size(), f) != v->size()) return 5;
    fclose(f);
    std::vector<float> out;
    if (ndim == 1) run<1>(t, n, A.data(), p.data(), lam.data(), time.data(), out);
    else if (ndim == 2) run<2>(t, n, A.data(), p.data(), lam.data(), time.data(), out);
    else run<3>(t, n, A.data(), p.data(), lam.data(), time.data(), out);
    FILE *o = fopen(argv[2], "wb");
    if (!o) return 6;
    fwrite(out.data(), 4, out.size(), o);
    fclose(o);
    return 0;
}
