// rd_spatial.cu -- spatial order of the evolve points for the culled
// assignment (k_assign_cull in rd_kernels.cu).
//
// The brute-force assignment of rd/cpu/brute_force/evolve.hpp:43-66 keeps a
// point's nearest chosen point only when it lies within r1.  A group of points
// that are close together in space therefore needs only the chosen points
// within r1 of the group's bounding box (of the nearer of its two: the order is cut
// where it jumps from one occupied place to another).  This file builds, once per run (the
// evolve points never move), a copy of every cloud's points in a spatial
// order -- cells of edge r1/4, Morton order of the cells, the packed slot
// order inside a cell.  The copy pads DIM 3 to four floats per point, so that
// a point is one 16-byte load.
#include "rd_engine.cuh"

#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstdint>

namespace rdb {
namespace {

// x's low 16 bits moved to the even bit positions
__device__ __forceinline__ uint32_t spread_by_1(uint32_t x)
{
    x &= 0xffffu;
    x = (x | (x << 8)) & 0x00ff00ffu;
    x = (x | (x << 4)) & 0x0f0f0f0fu;
    x = (x | (x << 2)) & 0x33333333u;
    x = (x | (x << 1)) & 0x55555555u;
    return x;
}

// x's low 10 bits moved to every third bit position
__device__ __forceinline__ uint32_t spread_by_2(uint32_t x)
{
    x &= 0x3ffu;
    x = (x | (x << 16)) & 0x030000ffu;
    x = (x | (x << 8)) & 0x0300f00fu;
    x = (x | (x << 4)) & 0x030c30c3u;
    x = (x | (x << 2)) & 0x09249249u;
    return x;
}

template <int DIM>
__device__ __forceinline__ uint32_t morton_code(const float* p, float inv)
{
    // the order only affects how tight the culling boxes are: one dimension
    // sorts by its cell, four and more interleave the first three
    if constexpr (DIM == 1) {
        return spatial_cell(p[0], inv);
    } else if constexpr (DIM == 2) {
        return spread_by_1(spatial_cell(p[0], inv)) | (spread_by_1(spatial_cell(p[1], inv)) << 1);
    } else {
        return spread_by_2(spatial_cell(p[0], inv)) | (spread_by_2(spatial_cell(p[1], inv)) << 1) |
               (spread_by_2(spatial_cell(p[2], inv)) << 2);
    }
}

// chunk lc of cloud cd covers positions [lo, hi) of the cloud
__device__ __forceinline__ void chunk_range(const CloudDesc& cd, int lc, int& lo, int& hi)
{
    lo = (int)(((int64_t)lc * cd.n_all) / cd.n_chunks);
    hi = (int)(((int64_t)(lc + 1) * cd.n_all) / cd.n_chunks);
}

// sort keys: (cloud << 32) | Morton code, of one cloud the code alone (half the
// bytes of the sort's passes); values: packed slot
template <int DIM, class Key>
__global__ void __launch_bounds__(256) k_morton(EngineView v, Key* key, int32_t* val)
{
    for (int ch = blockIdx.x; ch < v.n_chunks; ch += gridDim.x) {
        const int c = v.chunk_cloud[ch];
        const CloudDesc cd = v.cl[c];
        int lo, hi;
        chunk_range(cd, (int)(ch - cd.chunk_begin), lo, hi);
        const float inv = spatial_cell_inv(cd.r1);
        for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
            const int64_t s = cd.p_off + i;
            float p[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) p[d] = v.P[s * DIM + d];
            if constexpr (sizeof(Key) == 8) key[s] = ((uint64_t)(uint32_t)c << 32) | morton_code<DIM>(p, inv);
            else key[s] = morton_code<DIM>(p, inv);
            val[s] = (int32_t)s;
            v.keys[s] = -1;   // no point has a key before the first pass
        }
    }
}

// Ps, sorder, (second half of sorder) each position's histogram row -- the
// chunk of its slot inside its cloud -- and the two bounding boxes of every
// block of 32 x items positions of a cloud, one warp per block: the order is
// cut where consecutive points are furthest apart, which is where it leaves one
// occupied place for another (a block over such a jump as one box would span
// the space between, and the culled assignment would look at every chosen
// point there: on the 1M helix a handful of such blocks took 50 us each, as
// long as all the others together).  A part without points has an empty box.
template <int DIM>
__global__ void __launch_bounds__(256) k_gather_spatial(EngineView v, int items, int64_t n,
                                                        const int32_t* val, float* Ps,
                                                        int32_t* sorder, float* bbox)
{
    constexpr int DP = PadDim<DIM>::v;
    const int lane = threadIdx.x & 31;
    const int wpc = v.chunk_pts / (32 * items);
    const int64_t blocks = (int64_t)v.n_chunks * wpc;
    for (int64_t wb = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); wb < blocks;
         wb += (int64_t)gridDim.x * 8) {
        const int chunk = (int)(wb / wpc);
        const CloudDesc cd = v.cl[v.chunk_cloud[chunk]];
        const int64_t i0 = ((chunk - cd.chunk_begin) * wpc + wb % wpc) * 32 * items;
        const float ratio = (float)cd.n_chunks / (float)cd.n_all;
        float far = -1.0f;      // longest step of this lane's points from their predecessors
        int cut = 0;            // and the position it leads to
        float last[DIM];        // the previous row's last point
        for (int j = 0; j < items; ++j) {
            const int64_t i = i0 + j * 32 + lane;
            const bool in = i < cd.n_all;
            float x[DIM], step = 0.0f;
            const int64_t pos = cd.p_off + i;
            const int32_t s = in ? val[pos] : 0;
            if (in) {
                sorder[n + pos] = slot_chunk((int)(s - cd.p_off), cd.n_all, cd.n_chunks, ratio);
                sorder[pos] = s;
                v.ksp[pos] = -1;
            }
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                x[d] = in ? v.P[(int64_t)s * DIM + d] : 0.0f;
                if (in) Ps[pos * DP + d] = x[d];
                float prev = __shfl_up_sync(0xffffffffu, x[d], 1);
                if (lane == 0) prev = (j > 0) ? last[d] : x[d];
                step = fmaxf(step, fabsf(x[d] - prev));
                last[d] = __shfl_sync(0xffffffffu, x[d], 31);
            }
            if (in)
#pragma unroll
                for (int d = DIM; d < DP; ++d) Ps[pos * DP + d] = 0.0f;
            if (in && step > far) {
                far = step;
                cut = j * 32 + lane;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float f = __shfl_xor_sync(0xffffffffu, far, o);
            const int q = __shfl_xor_sync(0xffffffffu, cut, o);
            if (f > far || (f == far && q < cut)) {
                far = f;
                cut = q;
            }
        }
        float lo[2][DIM], hi[2][DIM];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                lo[h][d] = INFINITY;
                hi[h][d] = -INFINITY;
            }
        for (int j = 0; j < items; ++j) {
            const int64_t i = i0 + j * 32 + lane;
            if (i >= cd.n_all) break;
            const bool second = j * 32 + lane >= cut;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const float x = Ps[(cd.p_off + i) * DP + d];   // this lane's own writes
                lo[0][d] = fminf(lo[0][d], second ? INFINITY : x);
                hi[0][d] = fmaxf(hi[0][d], second ? -INFINITY : x);
                lo[1][d] = fminf(lo[1][d], second ? x : INFINITY);
                hi[1][d] = fmaxf(hi[1][d], second ? x : -INFINITY);
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    lo[h][d] = fminf(lo[h][d], __shfl_xor_sync(0xffffffffu, lo[h][d], o));
                    hi[h][d] = fmaxf(hi[h][d], __shfl_xor_sync(0xffffffffu, hi[h][d], o));
                }
                if (lane == 0) {
                    bbox[(wb * 2 + h) * 2 * DIM + d] = lo[h][d];
                    bbox[(wb * 2 + h) * 2 * DIM + DIM + d] = hi[h][d];
                }
            }
    }
}

size_t sort_temp_bytes(int64_t n)
{
    size_t bytes = 0, bytes32 = 0;
    cub::DoubleBuffer<uint64_t> k(nullptr, nullptr);
    cub::DoubleBuffer<uint32_t> k32(nullptr, nullptr);
    cub::DoubleBuffer<int32_t> v(nullptr, nullptr);
    cub::DeviceRadixSort::SortPairs(nullptr, bytes, k, v, (int)n, 0, 64);
    cub::DeviceRadixSort::SortPairs(nullptr, bytes32, k32, v, (int)n, 0, 32);
    return std::max(bytes, bytes32);
}

size_t align256(size_t x) { return (x + 255) / 256 * 256; }

template <int DIM>
cudaError_t spatial_prep_dim(const EngineView& v, int items, int64_t n, void* scratch,
                             size_t scratch_bytes, float* Ps, int32_t* sorder, float* bbox,
                             cudaStream_t st)
{
    if (n <= 0 || v.n_chunks <= 0) return cudaSuccess;
    unsigned char* p = static_cast<unsigned char*>(scratch);
    int32_t* v0 = reinterpret_cast<int32_t*>(p + 2 * align256(8 * (size_t)n));
    int32_t* v1 = reinterpret_cast<int32_t*>(p + 2 * align256(8 * (size_t)n) + align256(4 * (size_t)n));
    unsigned char* tmp = p + 2 * align256(8 * (size_t)n) + 2 * align256(4 * (size_t)n);
    const size_t used = (size_t)(tmp - p);
    if (scratch_bytes < used) return cudaErrorInvalidValue;
    size_t tmp_bytes = scratch_bytes - used;
    const int sms = v.n_sms > 0 ? v.n_sms : 148;
    const int cgrid = std::max(1, std::min(v.n_chunks, sms * 8));
    cub::DoubleBuffer<int32_t> vb(v0, v1);
    auto sort = [&](auto kind, int end_bit) -> cudaError_t {
        using Key = decltype(kind);
        Key* k0 = reinterpret_cast<Key*>(p);
        Key* k1 = reinterpret_cast<Key*>(p + align256(8 * (size_t)n));
        k_morton<DIM, Key><<<cgrid, 256, 0, st>>>(v, k0, v0);
        cub::DoubleBuffer<Key> kb(k0, k1);
        return cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, kb, vb, (int)n, 0, end_bit, st);
    };
    // 10 bits of three cell coordinates, 16 of two, 32 of one
    const int code_bits = DIM >= 3 ? 30 : 32;
    int cloud_bits = 0;
    while (cloud_bits < 32 && (int64_t(1) << cloud_bits) < v.n_clouds) ++cloud_bits;
    const cudaError_t e = v.n_clouds == 1 ? sort(uint32_t(0), code_bits) : sort(uint64_t(0), 32 + cloud_bits);
    if (e != cudaSuccess) return e;
    const int64_t blocks = (int64_t)v.n_chunks * (v.chunk_pts / (32 * items));
    const int ggrid = (int)std::max<int64_t>(1, std::min<int64_t>((blocks + 7) / 8, (int64_t)sms * 16));
    k_gather_spatial<DIM><<<ggrid, 256, 0, st>>>(v, items, n, vb.Current(), Ps, sorder, bbox);
    return cudaGetLastError();
}

}  // namespace

size_t spatial_prep_scratch_bytes(int64_t n)
{
    if (n <= 0) return 256;
    return 2 * align256(8 * (size_t)n) + 2 * align256(4 * (size_t)n) + align256(sort_temp_bytes(n));
}

cudaError_t launch_spatial_prep(int dim, const EngineView& v, int items, int64_t n, void* scratch,
                                size_t scratch_bytes, float* Ps, int32_t* sorder, float* bbox,
                                cudaStream_t st)
{
    return with_dim(dim, [&](auto D) {
        return spatial_prep_dim<decltype(D)::value>(v, items, n, scratch, scratch_bytes, Ps, sorder,
                                                    bbox, st);
    });
}

}  // namespace rdb
