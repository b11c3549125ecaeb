// rd_decbits.cuh -- in-order decimation of a small set over bit matrices, by one
// CTA (included by rd_kernels.cu).
//
// Same decimation, by the same argument for resolving a pass in parallel rounds,
// as decimate_scan_lists (rd_grid.cuh), for sets of up to DEC_BITS_MAX points:
// "within r2" and "within 2 r2" are written down once as bit rows by all pairs,
// and a point's earlier removed / undecided neighbours are population counts of
// its row against bit masks, one word per lane.  Buckets, list lengths, lists
// and their walks -- chains of dependent loads, one point per thread -- took 735 us
// for the 790 points of the 1M helix and 271 us for those of a 77,777-point one, now
// 61 us; a batch of 2,048 clouds 699 -> 635 ms.  Bound by the instructions of the
// all-pairs test and by two barriers per round.
#pragma once

#include "rd_grid.cuh"

namespace rdb {
namespace {

// pitch of a bit row in words: odd, so that rows start in different banks
__host__ __device__ inline int dec_bits_pitch(int total) { return ((total + 31) / 32) | 1; }
// shared memory besides the matrices: two counts per point, five masks
__host__ __device__ inline int dec_bits_fixed(int total)
{
    return 8 * total + 5 * 4 * ((total + 31) / 32) + 16;
}
__host__ __device__ inline int64_t dec_bits_matrix(int total)
{
    return (int64_t)8 * total * dec_bits_pitch(total);
}

// both in shared memory
__host__ __device__ inline int64_t dec_matrix_bytes(int total)
{
    return (dec_bits_fixed(total) + 15) / 16 * 16 + dec_bits_matrix(total);
}

// Pairs of DEC_SAMPLES points of a set, spread over its order, with a point of it
// within 2 r2 (themselves included), by the whole CTA, the same in every thread.
// coord(i, d): coordinate d of point i.
template <int DIM, int BLOCK, class F>
__device__ int dec_near_samples(F&& coord, const int total, const float r2)
{
    __shared__ int s_near;
    __syncthreads();   // coordinates are there, the last reader of s_near is done
    if (threadIdx.x == 0) s_near = 0;
    __syncthreads();
    const float rsq4 = __fmul_rn(4.0f, sqr_rn(r2));
    int near = 0;
    for (int t = threadIdx.x; t < DEC_SAMPLES * total; t += BLOCK) {
        const int i = (int)((int64_t)(t / total) * total / DEC_SAMPLES), j = t % total;
        float p[DIM], q[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            p[d] = coord(i, d);
            q[d] = coord(j, d);
        }
        near += sqdist_exact<DIM>(p, q) <= rsq4;
    }
    near = __reduce_add_sync(FULL, near);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_near, near);
    __syncthreads();
    return s_near;
}

// mat: two matrices of total x dec_bits_pitch(total) words (shared or global
// memory); smem: dec_bits_fixed(total) bytes.  alive[i] = 1 for the survivors.
template <int DIM, int BLOCK>
__device__ void decimate_bits(const float* X, const int total, const float r2, const int nocopy,
                              int32_t* alive, uint32_t* mat, unsigned char* smem, int32_t* err,
                              int32_t* tally)
{
    constexpr int NW = BLOCK / 32;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float rsq = sqr_rn(r2);
    const float rsq4 = __fmul_rn(4.0f, rsq);
    const int W = (total + 31) / 32, pitch = dec_bits_pitch(total);
    uint32_t* a1 = mat;                                // within r2 (not the point itself)
    uint32_t* a2 = mat + (int64_t)total * pitch;       // within 2 r2
    int* c1 = reinterpret_cast<int*>(smem);            // alive ones among them, itself included
    int* c2 = c1 + total;
    uint32_t* al = reinterpret_cast<uint32_t*>(c2 + total);
    uint32_t* und = al + W;    // undecided in this pass
    uint32_t* rem = und + W;   // removed in this pass
    uint32_t* nrem = rem + W;  // decided in this round
    uint32_t* nkept = nrem + W;
    for (int t = tid; t < total * W; t += BLOCK) {
        const int w = t / total, i = t - w * total;   // a warp shares the word: broadcast reads
        float p[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) p[d] = X[(int64_t)i * DIM + d];
        uint32_t m1 = 0, m2 = 0;
        const int n = min(32, total - w * 32);
#pragma unroll 8
        for (int b = 0; b < n; ++b) {
            float q[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) q[d] = X[(int64_t)(w * 32 + b) * DIM + d];
            const float sq = sqdist_exact<DIM>(p, q);
            m1 |= (sq <= rsq) ? (1u << b) : 0u;
            m2 |= (sq <= rsq4) ? (1u << b) : 0u;
        }
        const uint32_t self = (i >> 5) == w ? (1u << (i & 31)) : 0u;
        a1[(int64_t)i * pitch + w] = m1 & m2 & ~self;
        a2[(int64_t)i * pitch + w] = m2 & ~self;
    }
    for (int w = tid; w < W; w += BLOCK) {
        const int left = total - w * 32;
        al[w] = und[w] = left >= 32 ? 0xffffffffu : (1u << left) - 1u;
        rem[w] = nrem[w] = nkept[w] = 0;
    }
    __syncthreads();
    auto has = [](const uint32_t* m, int i) { return (m[i >> 5] >> (i & 31)) & 1u; };
    auto recount = [&]() {
        for (int i = warp; i < total; i += NW) {
            if (!has(al, i)) continue;
            unsigned n = 0;
            for (int w = lane; w < W; w += 32)
                n += __popc(a1[(int64_t)i * pitch + w] & al[w]) |
                     (__popc(a2[(int64_t)i * pitch + w] & al[w]) << 16);
            n = __reduce_add_sync(FULL, n);
            if (lane == 0) {
                c1[i] = 1 + (int)(n & 0xffffu);
                c2[i] = 1 + (int)(n >> 16);
            }
        }
    };
    recount();
    __syncthreads();
    int cnt = total, guard = 0;
    bool fallback = false;
    while (cnt > 3) {
        if (++guard > total + 2) {
            if (tid == 0) atomicOr(err, ERRB_DEC_CAP);
            break;
        }
        for (int round = 0;; ++round) {
            for (int i = warp; i < total; i += NW) {
                if (!has(und, i)) continue;
                unsigned n1 = 0, n2 = 0;   // removed, undecided << 16
                for (int w = lane; w <= (i >> 5); w += 32) {
                    const uint32_t earlier = w == (i >> 5) ? (1u << (i & 31)) - 1u : 0xffffffffu;
                    const uint32_t x1 = a1[(int64_t)i * pitch + w] & earlier;
                    const uint32_t x2 = a2[(int64_t)i * pitch + w] & earlier;
                    n1 += __popc(x1 & rem[w]) | (__popc(x1 & und[w]) << 16);
                    n2 += __popc(x2 & rem[w]) | (__popc(x2 & und[w]) << 16);
                }
                n1 = __reduce_add_sync(FULL, n1);
                n2 = __reduce_add_sync(FULL, n2);
                const int a = c1[i] - (int)(n1 & 0xffffu), b = c2[i] - (int)(n2 & 0xffffu);
                if (lane == 0) {
                    if (a - (int)(n1 >> 16) >= 4 || b < 3) atomicOr(&nrem[i >> 5], 1u << (i & 31));
                    else if (a < 4 && b - (int)(n2 >> 16) >= 3) atomicOr(&nkept[i >> 5], 1u << (i & 31));
                }
            }
            __syncthreads();
            int left = 0;
            for (int w = tid; w < W; w += BLOCK) {
                rem[w] |= nrem[w];
                und[w] &= ~(nrem[w] | nkept[w]);
                nrem[w] = nkept[w] = 0;
                left |= und[w] != 0;
            }
            if (tally && tid == 0) atomicAdd(&tally[1], 1);
            if (!__syncthreads_or(left)) break;
            if (round > total) {   // cannot happen: every round decides a point
                if (tid == 0) atomicOr(err, ERRB_DEC_CAP);
                break;
            }
        }
        if (tally && tid == 0) atomicAdd(&tally[0], 1);
        unsigned removed = 0;   // the same in every warp
        for (int w = lane; w < W; w += 32) removed += __popc(rem[w]);
        removed = __reduce_add_sync(FULL, removed);
        const bool apply = removed > 0 && cnt - (int)removed >= 3;
        __syncthreads();
        for (int w = tid; w < W; w += BLOCK) {
            if (apply) al[w] &= ~rem[w];
            und[w] = al[w];
            rem[w] = 0;
        }
        __syncthreads();
        if (removed == 0) break;       // a pass that changed nothing ends the loop
        if (!apply) {                  // the minimum-count rule may act
            fallback = true;
            break;
        }
        cnt -= (int)removed;
        recount();
        __syncthreads();
    }
    if (fallback && warp == 0) {
        // in order, one removal at a time (decimate.hpp:58-81, :104-127)
        int left = -1;
        bool stop = false;
        guard = 0;
        while (left != cnt && cnt > 3 && !stop) {
            if (++guard > total + 2) {
                if (lane == 0) atomicOr(err, ERRB_DEC_CAP);
                break;
            }
            left = cnt;
            int i = 0;
            while (i < total) {
                const int q = i + lane;
                const unsigned bal =
                    __ballot_sync(FULL, q < total && has(al, q) && (c1[q] >= 4 || c2[q] < 3));
                if (bal == 0) { i += 32; continue; }
                const int j = i + __ffs(bal) - 1;
                if (nocopy && cnt - 1 < 3) { stop = true; break; }
                __syncwarp();
                if (lane == 0) al[j >> 5] &= ~(1u << (j & 31));
                --cnt;
                for (int w = lane; w < W; w += 32) {   // distinct neighbours per lane
                    const uint32_t x1 = a1[(int64_t)j * pitch + w];
                    for (uint32_t x2 = a2[(int64_t)j * pitch + w]; x2; x2 &= x2 - 1) {
                        const int b = __ffs(x2) - 1;
                        c2[w * 32 + b] -= 1;
                        c1[w * 32 + b] -= (x1 >> b) & 1u;
                    }
                }
                __syncwarp();
                if (!nocopy && cnt < 3) break;
                i = j + 1;
            }
            if (!nocopy && cnt < 3) break;
        }
    }
    __syncthreads();
    for (int i = tid; i < total; i += BLOCK) alive[i] = (int)has(al, i);
    __syncthreads();
}

}  // namespace
}  // namespace rdb
