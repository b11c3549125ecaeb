// rd_order.cu -- ordering of a ridge into chains (rd/cpu/brute_force/order.hpp:45-141,
// with the condition the brute-force class passes, ridge_detection.inl:148-168).
//
// Every remaining point, in index order, seeds a chain.  The chain then takes,
// again and again, the first later remaining point (lowest index) that is
// within r2 of its front -- tested first -- or of its back, until none is
// left.  Each step depends on the last, but "the first remaining point within
// r2 of either end" is a min-index search over all later points, which one
// CTA does in parallel: every thread scans its stride of candidates up to its
// first hit, then a block-wide min picks the winner.  The chain grows in a
// deque (front and back indices around the middle of a 2*ns+1 buffer) and is
// written out front to back.
//
// Ridges of up to ORDER_BITS_MAX points (those a solve ends with) take
// k_order_bits instead: the "within r2" relation is symmetric and does not
// change, so the CTA first writes it down as a bit matrix in shared memory, and
// one warp then grows the chains with a word of the alive mask per lane.  The
// serial chain of steps is what bounds either kernel; a step of the bit walk
// is one shared-memory load, a ballot and a shuffle instead of three barriers
// of 1,024 threads: a call with 300 points in 3D 284 us -> 127 us, 1,000 points 811 -> 274.
#include "rd_engine.cuh"

#include <climits>
#include <cuda_runtime.h>

namespace rdb {
namespace {

constexpr int ORDER_BLOCK = 1024;

template <int DIM>
__global__ void __launch_bounds__(ORDER_BLOCK)
    k_order_chains(const float* __restrict__ S, int ns, float rsq, unsigned char* alive,
                   int32_t* deq, int32_t* order, int32_t* chain_start, int32_t* n_chains)
{
    __shared__ int s_min[ORDER_BLOCK / 32];
    __shared__ int s_hit, s_head, s_tail;
    __shared__ float s_f[DIM], s_b[DIM];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < ns; i += ORDER_BLOCK) alive[i] = 1;
    __syncthreads();
    int out = 0, nch = 0;  // the same in every thread
    for (int p = 0; p < ns; ++p) {
        if (!alive[p]) continue;  // written by thread 0 before a barrier: uniform
        __syncthreads();
        if (tid == 0) {
            alive[p] = 0;
            deq[ns] = p;
            s_head = ns;
            s_tail = ns;
#pragma unroll
            for (int d = 0; d < DIM; ++d) s_f[d] = s_b[d] = S[(int64_t)p * DIM + d];
        }
        __syncthreads();
        for (;;) {
            float f[DIM], b[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                f[d] = s_f[d];
                b[d] = s_b[d];
            }
            int best = INT_MAX;
            for (int j = p + 1 + tid; j < ns; j += ORDER_BLOCK) {
                if (!alive[j]) continue;
                float q[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d) q[d] = S[(int64_t)j * DIM + d];
                if (sqdist_exact<DIM>(q, f) <= rsq || sqdist_exact<DIM>(q, b) <= rsq) {
                    best = j;
                    break;
                }
            }
            const int m = __reduce_min_sync(0xffffffffu, best);
            if (lane == 0) s_min[warp] = m;
            __syncthreads();
            if (warp == 0) {
                const int v = __reduce_min_sync(0xffffffffu, (lane < ORDER_BLOCK / 32) ? s_min[lane] : INT_MAX);
                if (lane == 0) s_hit = v;
            }
            __syncthreads();
            const int hit = s_hit;
            if (hit == INT_MAX) break;
            if (tid == 0) {
                alive[hit] = 0;
                float q[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d) q[d] = S[(int64_t)hit * DIM + d];
                if (sqdist_exact<DIM>(q, f) <= rsq) {
                    deq[--s_head] = hit;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) s_f[d] = q[d];
                } else {
                    deq[++s_tail] = hit;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) s_b[d] = q[d];
                }
            }
            __syncthreads();
        }
        const int head = s_head, tail = s_tail;
        for (int k = head + tid; k <= tail; k += ORDER_BLOCK) order[out + (k - head)] = deq[k];
        if (tid == 0) chain_start[nch] = out;
        out += tail - head + 1;
        ++nch;
        __syncthreads();  // the deque is reused by the next chain
    }
    if (tid == 0) {
        chain_start[nch] = out;
        *n_chains = nch;
    }
}

constexpr int ORDER_BITS_MAX = 1024;   // one alive word per lane
// words of a bit row: odd, so that rows start in different banks
__host__ __device__ constexpr int order_pitch(int ns) { return ((ns + 31) / 32) | 1; }

// chains by one warp over the bit matrix adj[i * order_pitch(ns) + w]:
// bit j of row i = points i and j within r2.  Every alive point is later than
// the seed (earlier ones are in a chain already), so the first alive neighbour
// of either end is the lowest set bit of (row(front) | row(back)) & alive.
template <int DIM>
__global__ void __launch_bounds__(ORDER_BLOCK)
    k_order_bits(const float* __restrict__ S, int ns, float rsq, int32_t* deq, int32_t* order,
                 int32_t* chain_start, int32_t* n_chains)
{
    extern __shared__ uint32_t adj[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int words = (ns + 31) / 32, pitch = order_pitch(ns);
    // a warp shares the word, its points are broadcast reads (with lanes on words of one
    // row every read touched 32 lines: 1,000 points 1,713 us, the serial search 811)
    for (int t = tid; t < ns * words; t += ORDER_BLOCK) {
        const int w = t / ns, i = t - w * ns;
        float f[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) f[d] = S[i * DIM + d];
        uint32_t m = 0;
        const int j1 = min(32, ns - w * 32);
        for (int b = 0; b < j1; ++b) {
            float q[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) q[d] = S[(w * 32 + b) * DIM + d];
            m |= (sqdist_exact<DIM>(q, f) <= rsq) ? (1u << b) : 0u;
        }
        adj[i * pitch + w] = m;
    }
    __syncthreads();
    if (warp != 0) return;
    const bool on = lane < words;
    uint32_t alive = 0;
    if (on) alive = (lane == words - 1 && (ns & 31)) ? ((1u << (ns & 31)) - 1u) : 0xffffffffu;
    int out = 0, nch = 0;
    for (;;) {
        const unsigned left = __ballot_sync(0xffffffffu, alive != 0);
        if (!left) break;
        const int sl = __ffs(left) - 1;
        const int p = sl * 32 + __ffs(__shfl_sync(0xffffffffu, alive, sl)) - 1;
        if (lane == sl) alive &= alive - 1;
        uint32_t af = on ? adj[p * pitch + lane] : 0u, ab = af;
        int head = ns, tail = ns;
        if (lane == 0) deq[ns] = p;
        for (;;) {
            const uint32_t m = (af | ab) & alive;
            const unsigned any = __ballot_sync(0xffffffffu, m != 0);
            if (!any) break;
            const int hl = __ffs(any) - 1;
            // the hit's bit, whether the front reaches it (tested first)
            const int bit = __ffs(m) - 1;
            const int code = (bit & 31) | (((af >> (bit & 31)) & 1u) << 5);
            const int c = __shfl_sync(0xffffffffu, code, hl);
            const int hit = hl * 32 + (c & 31);
            const bool front = (c >> 5) & 1;
            if (lane == hl) alive &= ~(1u << (c & 31));
            const uint32_t a = on ? adj[hit * pitch + lane] : 0u;
            if (front) { af = a; --head; }
            else { ab = a; ++tail; }
            if (lane == 0) deq[front ? head : tail] = hit;
        }
        __syncwarp();
        for (int k = head + lane; k <= tail; k += 32) order[out + (k - head)] = deq[k];
        if (lane == 0) chain_start[nch] = out;
        out += tail - head + 1;
        ++nch;
        __syncwarp();  // the deque is reused by the next chain
    }
    if (lane == 0) {
        chain_start[nch] = out;
        *n_chains = nch;
    }
}

}  // namespace

cudaError_t launch_order_chains(int dim, const float* S, int ns, float rsq, unsigned char* alive,
                                int32_t* deq, int32_t* order, int32_t* chain_start,
                                int32_t* n_chains, cudaStream_t st)
{
    return with_dim(dim, [&](auto D) {
        // up to 132 KB of shared memory for the bit matrix; larger ridges search
        // their candidates in every step
        if (ns <= ORDER_BITS_MAX) {
            const int bytes = ns * order_pitch(ns) * 4;
            const cudaError_t e = cudaFuncSetAttribute(
                k_order_bits<decltype(D)::value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                ORDER_BITS_MAX * order_pitch(ORDER_BITS_MAX) * 4);
            if (e != cudaSuccess) return e;
            k_order_bits<decltype(D)::value><<<1, ORDER_BLOCK, bytes, st>>>(S, ns, rsq, deq, order,
                                                                         chain_start, n_chains);
            return cudaGetLastError();
        }
        k_order_chains<decltype(D)::value><<<1, ORDER_BLOCK, 0, st>>>(S, ns, rsq, alive, deq, order,
                                                                     chain_start, n_chains);
        return cudaGetLastError();
    });
}

}  // namespace rdb
