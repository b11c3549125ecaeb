// rd_quality.cu -- quality metrics of a ridge on the device
// (rd/utils/assessment_quality.hpp), with the reference's float arithmetic:
//   distance(p, B)  = sqrt(min over B of the squared distance p - b)
//   Hausdorff(T, I) = max(max over T of distance(t, I), max over I of distance(i, T))
//   stats(S, I)     = min, max, median (sorted[n/2]) and mean (float sum in
//                     sorted order / n) of distance(s, I)
//   segment(T)      = max over T of sqrt(sum over d >= 1 of t_d^2)
// The min-distance search is all pairs, threads holding points of one set
// against shared-memory tiles of a slice of the other; the mean's ordered sum uses the exact
// parallel fold (rd_fold.cuh), so it equals the sequential float sum.
#include "rd_engine.cuh"
#include "rd_fold.cuh"

#include <algorithm>
#include <cfloat>
#include <cub/cub.cuh>
#include <cuda_runtime.h>

namespace rdb {
namespace {

constexpr int Q_TILE = 1024;

// one row of the staged tile (PadDim<DIM> floats, one vector load)
template <int DIM>
__device__ __forceinline__ void load_tile_row(const float* sB, int k, float* s)
{
    constexpr int DP = PadDim<DIM>::v;
    if constexpr (DP == 4) {
        const float4 t = reinterpret_cast<const float4*>(sB)[k];
        s[0] = t.x; s[1] = t.y; s[2] = t.z;
        if constexpr (DIM == 4) s[3] = t.w;
    } else if constexpr (DP == 2) {
        const float2 t = reinterpret_cast<const float2*>(sB)[k];
        s[0] = t.x; s[1] = t.y;
    } else {
        s[0] = sB[k];
    }
}

// Smallest squared distance of each point of A to the slice blockIdx.y of B
// (slices of `per` points), merged over the slices with an integer minimum:
// the values are sums of squares, so their bit patterns order as they do, and
// a minimum does not depend on the order it is taken in.  out holds FLT_MAX
// before; a NaN distance never passes the strict '<'.
// Bound by the FP32 pipe once enough CTAs are in flight: 3 DIM - 1 rounded
// operations and a minimum per pair.  The slices are what fills the chip when
// A is a ridge of a few hundred points: 300 points against 100,000 in 3D took
// 5,770 us as one CTA over all of B, 21 us in 148 x 4 CTAs (whose floor by
// operations is 8 us: each slice re-reads its points through L2).
template <int DIM, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK) k_min_dist(const float* __restrict__ A, int na,
                                                    const float* __restrict__ B, int nb, int per,
                                                    unsigned* __restrict__ out)
{
    constexpr int DP = PadDim<DIM>::v;
    __shared__ __align__(16) float sB[Q_TILE * DP];
    const int tid = threadIdx.x;
    const int i0 = blockIdx.x * BLOCK * ITEMS + tid;
    const int b0 = (int)min((int64_t)nb, (int64_t)blockIdx.y * per);
    const int b1 = (int)min((int64_t)nb, (int64_t)b0 + per);
    float p[ITEMS][DIM], best[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int64_t i = i0 + (int64_t)j * BLOCK;
#pragma unroll
        for (int d = 0; d < DIM; ++d) p[j][d] = (i < na) ? A[i * DIM + d] : 0.0f;
        best[j] = FLT_MAX;
    }
    for (int t0 = b0; t0 < b1; t0 += Q_TILE) {
        const int tl = min(Q_TILE, b1 - t0);
        __syncthreads();
        for (int e = tid; e < tl * DIM; e += BLOCK)
            sB[(e / DIM) * DP + e % DIM] = B[(int64_t)t0 * DIM + e];
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < tl; ++k) {
            float s[DIM];
            load_tile_row<DIM>(sB, k, s);
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const float dd = sqdist_exact<DIM>(p[j], s);
                if (dd < best[j]) best[j] = dd;
            }
        }
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
        const int64_t i = i0 + (int64_t)j * BLOCK;
        if (i < na) atomicMin(&out[i], __float_as_uint(best[j]));
    }
}

__global__ void __launch_bounds__(256) k_fill_far(float* out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = FLT_MAX;
}

__global__ void __launch_bounds__(256) k_sqrt(float* d, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) d[i] = sqrtf(d[i]);
}

template <int DIM>
__global__ void __launch_bounds__(256) k_axis_dist(const float* __restrict__ T, int n,
                                                  float* __restrict__ out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = 0.0f;
#pragma unroll
    for (int k = 1; k < DIM; ++k) {
        const float x = T[(int64_t)i * DIM + k];
        s = __fadd_rn(s, __fmul_rn(x, x));
    }
    out[i] = (s > 0.0f) ? sqrtf(s) : 0.0f;
}

// largest value of a[0..na) and b[0..nb) (one CTA)
__global__ void __launch_bounds__(1024) k_max2(const float* a, int na, const float* b, int nb,
                                               float* out)
{
    __shared__ float s_w[32];
    float m = -FLT_MAX;
    for (int i = threadIdx.x; i < na; i += 1024) m = fmaxf(m, a[i]);
    for (int i = threadIdx.x; i < nb; i += 1024) m = fmaxf(m, b[i]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) s_w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = s_w[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0) *out = m;
    }
}

__global__ void k_iota(int32_t* idx, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) idx[i] = i;
}

// {median, mean, min, max} of the sorted distances (one CTA of 256 threads)
__global__ void __launch_bounds__(256) k_stats(const float* sorted, const int32_t* iota, int n,
                                              float* out)
{
    __shared__ FoldCtaSmem<8, 1> sm;
    fold_members_cta<8, 1>(iota, n, sorted, sm);
    if (threadIdx.x == 0) {
        out[0] = sorted[n / 2];
        out[1] = __fdiv_rn(sm.s[0], (float)n);
        out[2] = sorted[0];
        out[3] = sorted[n - 1];
    }
}

// Slices of B so that the grid holds at least Q_CTAS CTAs (four per SM), each
// slice of at least Q_MIN_SLICE points (a shorter one spends more on its
// start than on its pairs).
constexpr int Q_CTAS = 148 * 4, Q_MIN_SLICE = 128;

template <int DIM, int BLOCK, int ITEMS>
cudaError_t min_dist_grid(const float* A, int na, const float* B, int nb, unsigned* out,
                          cudaStream_t st)
{
    const int64_t gx = ((int64_t)na + BLOCK * ITEMS - 1) / (BLOCK * ITEMS);
    const int64_t want = (Q_CTAS + gx - 1) / gx;
    const int64_t most = std::max<int64_t>(1, ((int64_t)nb + Q_MIN_SLICE - 1) / Q_MIN_SLICE);
    const int64_t gy = std::max<int64_t>(1, std::min(want, most));
    const int per = (int)(((int64_t)nb + gy - 1) / gy);
    k_min_dist<DIM, BLOCK, ITEMS><<<dim3((unsigned)gx, (unsigned)gy), BLOCK, 0, st>>>(A, na, B, nb, per, out);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_min_dist(int dim, const float* A, int na, const float* B, int nb, float* out,
                            cudaStream_t st)
{
    if (na <= 0) return cudaSuccess;
    // a small A takes one point per thread: fewer idle lanes in the last CTA
    // (300 points fill 384 slots, not 1,024)
    const int g = (na + 255) / 256;
    k_fill_far<<<g, 256, 0, st>>>(out, na);
    unsigned* bits = reinterpret_cast<unsigned*>(out);
    cudaError_t e = with_dim(dim, [&](auto D) {
        constexpr int DIM = decltype(D)::value;
        return (na <= 4096) ? min_dist_grid<DIM, 128, 1>(A, na, B, nb, bits, st)
                            : min_dist_grid<DIM, 256, 4>(A, na, B, nb, bits, st);
    });
    if (e != cudaSuccess) return e;
    k_sqrt<<<g, 256, 0, st>>>(out, na);
    return cudaGetLastError();
}

cudaError_t launch_axis_dist(int dim, const float* T, int n, float* out, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    return with_dim(dim, [&](auto D) {
        k_axis_dist<decltype(D)::value><<<(n + 255) / 256, 256, 0, st>>>(T, n, out);
        return cudaGetLastError();
    });
}

cudaError_t launch_max2(const float* a, int na, const float* b, int nb, float* out, cudaStream_t st)
{
    k_max2<<<1, 1024, 0, st>>>(a, na, b, nb, out);
    return cudaGetLastError();
}

// sorts d (n floats, all >= 0) through the scratch and writes {median, mean,
// min, max} to out (device); scratch: 2n floats + n ints + cub storage
cudaError_t launch_dist_stats(float* d, int n, float* sorted, int32_t* iota, void* temp,
                              size_t temp_bytes, float* out, cudaStream_t st)
{
    cudaError_t e = cub::DeviceRadixSort::SortKeys(temp, temp_bytes, d, sorted, n, 0, 32, st);
    if (e != cudaSuccess) return e;
    k_iota<<<(n + 255) / 256, 256, 0, st>>>(iota, n);
    k_stats<<<1, 256, 0, st>>>(sorted, iota, n, out);
    return cudaGetLastError();
}

size_t dist_stats_temp_bytes(int n)
{
    size_t bytes = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, bytes, (float*)nullptr, (float*)nullptr, n, 0, 32);
    return bytes;
}

}  // namespace rdb
