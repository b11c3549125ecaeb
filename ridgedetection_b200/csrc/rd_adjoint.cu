// rd_adjoint.cu -- reverse pass of `iters` evolve passes (no reference
// counterpart; the reference is forward-only).
//
// Forward, on the engine with the movement test switched off: A^t is the exact
// assignment of the cloud to S^{t-1} (the engine's pass kernels, which touch only
// what the last pass changed), and
// S^t_k = (FP32 sum of A^t_k in index order) / |A^t_k| for |A^t_k| > 0, else
// S^{t-1}_k.  Loss L = sum_k <W_k, S^iters_k>.
// Reverse, assignments frozen, FP64: g = W; for t = iters..1 every member i of
// a non-empty cluster k gets g_k / |A^t_k| added to dL/dP_i and g_k is reset;
// empty clusters carry g_k to S^{t-1}.  What is left of g is dL/dS^0.
// Memory: all assignments are kept (iters x N ints) when checkpoint_every = 0;
// otherwise S is checkpointed every `checkpoint_every` passes and the
// assignments of one segment at a time are recomputed during the reverse pass
// (the last segment's are kept as the forward makes them).
//
// The reverse of a segment is two kernels: g before every pass of it, one
// thread per chosen coordinate (a pass with members resets it), then one thread
// per point that adds its terms in the order of the passes, so that dL/dP is
// read and written once per segment instead of once per pass.  g before every pass
// is ns x dim doubles a pass, more than the kept assignments where nearly every
// point is chosen: passes are taken in blocks of at most ADJ_G_BYTES of it.  262,144 points,
// 20 passes in segments of 5: 40 kernel pairs and 256 us before, 4 and 64 us now.
#include "rd_adjoint.hpp"

#include <algorithm>
#include <cstring>

namespace rdb {

namespace {

// G[q] = g before (in reverse) pass t1 - 1 - q of the segment, q < len; g ends as
// what is left of it.  cnt: the segment's counts, pass t0 first.
__global__ void k_adj_carry(const int32_t* __restrict__ cnt, int64_t ns, int dim, int len,
                            double* __restrict__ g, double* __restrict__ G)
{
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, n = ns * dim;
    if (e >= n) return;
    const int64_t k = e / dim;
    double x = g[e];
    for (int q = 0; q < len; ++q) {
        G[q * n + e] = x;
        if (cnt[(len - 1 - q) * ns + k] > 0) x = 0.0;
    }
    g[e] = x;
}

template <int DIM>
__global__ void __launch_bounds__(256) k_adj_members(const int32_t* __restrict__ keys,
                                                     const int32_t* __restrict__ cnt,
                                                     const double* __restrict__ G, int64_t n,
                                                     int64_t ns, int len, double* __restrict__ gP)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x) {
        double x[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) x[d] = gP[i * DIM + d];
        for (int q = 0; q < len; ++q) {
            const int k = keys[(len - 1 - q) * n + i];
            if (k < 0) continue;
            const double inv = 1.0 / (double)cnt[(len - 1 - q) * ns + k];
#pragma unroll
            for (int d = 0; d < DIM; ++d) x[d] += G[(q * ns + k) * DIM + d] * inv;
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d) gP[i * DIM + d] = x[d];
    }
}

constexpr int64_t ADJ_G_BYTES = int64_t(64) << 20;

int grid_for(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 148 * 16)); }

}  // namespace

int AdjointRunner::fail(const char* what, cudaError_t e)
{
    last_error = std::string(what) + ": " + cudaGetErrorString(e);
    return 2;
}

#define AK(call)                                      \
    do {                                              \
        cudaError_t e_ = (call);                      \
        if (e_ != cudaSuccess) return fail(#call, e_); \
    } while (0)

int AdjointRunner::run(int dim, const float* d_P, int64_t np, const float* d_S0, int64_t ns,
                       float r1, int iters, int ckpt, const double* d_W, float* d_S_final,
                       double* d_gP, double* d_gS0, cudaStream_t st)
{
    if (!dim_supported(dim)) { last_error = "dim must be 1 to 4"; return 6; }
    if (np < 1 || ns < 1 || ns > np || iters < 0 || ckpt < 0) { last_error = "bad sizes"; return 1; }
    CloudDesc cd;
    std::memset(&cd, 0, sizeof(cd));
    cd.n_all = (int32_t)np;
    cd.n_own = (int32_t)np;
    cd.r1 = r1;
    cd.r2 = r1;
    GroupDesc gd;
    std::memset(&gd, 0, sizeof(gd));
    gd.n_clouds = 1;
    if (int rc = eng_.setup(dim, {cd}, {gd}, np)) { last_error = eng_.last_error; return rc; }
    AK(cudaMemcpyAsync(eng_.points(), d_P, sizeof(float) * np * dim, cudaMemcpyDeviceToDevice, st));
    AK(cudaMemcpyAsync(eng_.chosen_mut(), d_S0, sizeof(float) * ns * dim, cudaMemcpyDeviceToDevice, st));
    eng_.given_ns.assign(1, (int32_t)ns);
    if (int rc = eng_.adjoint_setup(st)) { last_error = eng_.last_error; return rc; }
    const int seg = ckpt > 0 ? std::min(ckpt, std::max(iters, 1)) : std::max(iters, 1);
    const int nseg = (iters + seg - 1) / seg;
    const bool reverse = d_gP != nullptr;
    float* S = eng_.chosen_mut();
    const size_t sbytes = sizeof(float) * ns * dim;
    const int64_t nk = ns * dim;
    // passes reversed by one pair of kernels
    const int block = (int)std::max<int64_t>(1, std::min<int64_t>(seg, ADJ_G_BYTES / (8 * nk)));
    if (reverse) {
        AK(bKeys_.ensure(sizeof(int32_t) * (size_t)np * seg + 16));
        AK(bCnt_.ensure(sizeof(int32_t) * (size_t)ns * seg + 16));
        AK(bCkpt_.ensure(sizeof(float) * (size_t)nk * (nseg + 1) + 16));
        AK(bG_.ensure(sizeof(double) * (size_t)nk * (block + 1) + 16));
    }
    double* g = bG_.as<double>();
    double* G = g + nk;
    auto keep = [&](int slot) -> int {
        AK(cudaMemcpyAsync(bKeys_.as<int32_t>() + (size_t)slot * np, eng_.keys(),
                           sizeof(int32_t) * np, cudaMemcpyDeviceToDevice, st));
        AK(cudaMemcpyAsync(bCnt_.as<int32_t>() + (size_t)slot * ns, eng_.counts(),
                           sizeof(int32_t) * ns, cudaMemcpyDeviceToDevice, st));
        return 0;
    };
    // forward, checkpointing S at the start of every segment
    for (int t = 0; t < iters; ++t) {
        if (reverse && t % seg == 0)
            AK(cudaMemcpyAsync(bCkpt_.as<float>() + (size_t)(t / seg) * nk, S, sbytes,
                               cudaMemcpyDeviceToDevice, st));
        if (int rc = eng_.adjoint_step(st)) { last_error = eng_.last_error; return rc; }
        if (reverse && t / seg == nseg - 1)
            if (int rc = keep(t % seg)) return rc;
    }
    if (d_S_final) AK(cudaMemcpyAsync(d_S_final, S, sbytes, cudaMemcpyDeviceToDevice, st));
    if (!reverse) {
        AK(cudaStreamSynchronize(st));
        return 0;
    }
    AK(cudaMemcpyAsync(g, d_W, sizeof(double) * nk, cudaMemcpyDeviceToDevice, st));
    AK(cudaMemsetAsync(d_gP, 0, sizeof(double) * np * dim, st));
    for (int s = nseg - 1; s >= 0; --s) {
        const int t0 = s * seg, len = std::min(iters, t0 + seg) - t0;
        if (s < nseg - 1) {  // recompute the segment's assignments from its checkpoint
            AK(cudaMemcpyAsync(S, bCkpt_.as<float>() + (size_t)s * nk, sbytes,
                               cudaMemcpyDeviceToDevice, st));
            if (int rc = eng_.adjoint_restart(st)) { last_error = eng_.last_error; return rc; }
            for (int q = 0; q < len; ++q) {
                if (int rc = eng_.adjoint_step(st)) { last_error = eng_.last_error; return rc; }
                if (int rc = keep(q)) return rc;
            }
        }
        for (int q1 = len; q1 > 0; q1 -= block) {
            const int q0 = std::max(0, q1 - block);
            const int32_t* kt = bKeys_.as<int32_t>() + (size_t)q0 * np;
            const int32_t* ct = bCnt_.as<int32_t>() + (size_t)q0 * ns;
            k_adj_carry<<<(int)((nk + 255) / 256), 256, 0, st>>>(ct, ns, dim, q1 - q0, g, G);
            AK(with_dim(dim, [&](auto D) {
                constexpr int DIM = decltype(D)::value;
                k_adj_members<DIM><<<grid_for(np), 256, 0, st>>>(kt, ct, G, np, ns, q1 - q0, d_gP);
                return cudaGetLastError();
            }));
        }
    }
    if (d_gS0) AK(cudaMemcpyAsync(d_gS0, bG_.p, sizeof(double) * ns * dim, cudaMemcpyDeviceToDevice, st));
    AK(cudaStreamSynchronize(st));
    return 0;
}

}  // namespace rdb
