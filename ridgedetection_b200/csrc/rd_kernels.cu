// rd_kernels.cu -- sm_100a kernels of the batch engine (see rd_engine.cuh).
//
// All arithmetic is FP32 on the CUDA cores.  The point/chosen contraction has
// K = DIM <= 3, far too thin for tcgen05 tiles, and the reference's rounding
// (sub, mul, add, each rounded) rules out the |p|^2 - 2 p.c + |c|^2 expansion a
// tensor-core formulation would need, so the hot loop is a register-blocked
// SIMT kernel instead: each thread holds ITEMS cloud points, the chosen set
// streams through shared memory, and every pair costs DIM sub + DIM mul +
// (DIM-1) add + compare + 2 selects, all explicitly rounded.
#include "rd_engine.cuh"
#include "rd_grid.cuh"
#include "rd_decbits.cuh"
#include "rd_fold.cuh"
#include "rd_segfold.cuh"

#include <cooperative_groups.h>

#include <cuda_runtime.h>
#include <cub/cub.cuh>

#include <algorithm>
#include <atomic>
#include <cstring>

namespace rdb {

namespace {

// Long member lists.  The fold by a whole CTA (the warp-segmented exact fold of
// rd_segfold.cuh) needs more than 128 registers a thread; the merge of k_merge_fold
// wants four CTAs per SM, and with the 64 registers those leave the fold spills and
// takes twice as long (lists of 500,000 members: 2,850 us, 1,350 with its registers).
// And a CTA merges the edits of a list at about 4.5 ns a row, while a regrouping of
// the cloud scatters over the whole GPU.  So runs of few chosen points (LONG_AVG points
// for each) take a variant of k_merge_fold that has the registers, folds lists of
// SUM_BIG_MIN members that way -- while the pass has no more keys to fold than CTAs;
// with more every key is folded by a chain, which does less work in all -- and
// regroups when such a list has an edit.  Others do so from larger lengths on, as the
// slower fold and the cost of regrouping everybody ask for.  1M-point helix, evolve
// from the chosen set, one variant for all / this, ms: r1 0.6 (35 chosen points) 18.8 /
// 11.1, 0.4 (55) 17.9 / 12.4, 3 (2) 10.7 / 5.3.  What it does not reach: a list of most
// of a cloud's points beside thousands of short ones (900,000 of 1M points beside
// 4,714: one pass 3.9 ms, 1.9 if its fold had the registers).
constexpr int LONG_AVG = 8192;
constexpr int SUM_BIG_MIN = 16384, SUM_BIG_MIN_SLOW = 65536;
// regions of 16,384 and 32,768 members
constexpr int MERGE_CAP_LONG = list_room(16384), MERGE_CAP = list_room(32768);

// Programmatic dependent launch: the loop-body kernels are launched with
// programmatic stream serialisation, so a kernel's CTAs may become resident
// while the previous kernel drains. Each waits here, before its first access
// to memory, until the previous grid has completed and its writes are
// visible, then lets the next kernel launch. Launched without the attribute,
// both instructions return at once.
__device__ __forceinline__ void pdl_enter()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Cloud c's descriptor: a run of one cloud has it in the launch parameters, one
// memory round trip less in each of a pass's latency-bound kernels.
__device__ __forceinline__ CloudDesc cloud_desc(const EngineView& v, const int c)
{
    return v.single ? v.one : v.cl[c];
}

// Work lists over the clouds still evolving, rebuilt by loop_condition when a cloud
// has converged: act_cloud[a] is the a-th evolving cloud and act_pre[kind] the
// exclusive prefix of its work items (ACT_* in rd_engine.cuh), so kernels
// launched over fixed grids touch only active work.

struct ActiveList {
    const int32_t* pre;
    const int32_t* cloud;
    int nact;
    int total;
    bool single;
    __device__ ActiveList(const EngineView& v, int kind)
    {
        nact = v.ctr[CTR_NACT];
        pre = v.act_pre + (int64_t)kind * (v.n_clouds + 1);
        cloud = v.act_cloud;
        total = (v.single && kind == ACT_CHUNK) ? (nact ? v.one.n_chunks : 0) : pre[nact];
        single = v.single != 0;
    }
    // item t < total -> (cloud, item index inside that cloud)
    __device__ __forceinline__ void locate(int t, int& c, int& local) const
    {
        if (single) {
            c = 0;
            local = t;
            return;
        }
        int lo = 0, hi = nact - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (pre[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        c = cloud[lo];
        local = t - pre[lo];
    }
};


// ---------------------------------------------------------------------------
// choose: rd/cpu/brute_force/choose.hpp:37-70, one CTA per cloud.
// Blocks of BLOCK points are visited in order.  Phase 1 (all threads) drops
// every point that has a chosen point within r1 among those chosen by earlier
// blocks, looked up through a hashed grid of cell edge > r1 (the grid only
// prunes; the test itself is the exact FP32 one).  Phase 2 applies the greedy
// rule to the block's survivors (choose_survivors).  Chosen coordinates and
// hash chains are mirrored in shared memory for the first SCAP chosen points.
// ---------------------------------------------------------------------------
template <int DIM>
struct ChooseSmem {
    static constexpr int HBITS = 13;
    static constexpr int HB = 1 << HBITS;
    static constexpr int SCAP = (DIM <= 2) ? 6144 : 4096;
    static constexpr int BLOCK = 1024;
};
constexpr int CHOOSE_G = 128;             // survivors resolved together
constexpr int CHOOSE_GW = CHOOSE_G / 32;  // words of a conflict row

// Scratch of choose_survivors: the conflict rows of a group, its picks, and the
// warp counts of the compaction.
struct ChooseResolve {
    uint32_t adj[CHOOSE_G * CHOOSE_GW];
    int pick[CHOOSE_G];
    int npick;
    int wsum[32];
};

template <int DIM, class CS>
constexpr int choose_smem_bytes()
{
    return CS::HB * 4 + CS::SCAP * 4 + CS::SCAP * DIM * 4 + CS::BLOCK * DIM * 8;
}

// The sequential greedy rule over the block's survivors s_sp[0..tot) (in
// visiting order, none within r1 of a point chosen before the block), for the
// whole CTA: returns the new chosen count.  A survivor is chosen when no
// earlier chosen one lies within r1, and "within r1" among the survivors does
// not depend on what is chosen: the first CHOOSE_G survivors write that
// relation down as bit rows (all threads), one warp walks the group's alive
// bits -- take the lowest, clear its row -- and the rest of the survivors drop
// those within r1 of the group's picks and close up, in order, before the next
// group.  Bound by the walk, about 50 ns per chosen point, and by five barriers
// per group; a grid lookup by one warp per survivor, chosen or not, took
// 0.25-0.4 us (first 4,096 points of the 1M helix: 436 us before,
// 105 us now; 1,000 points of the 2D sine: 262 us before, 20 now).
template <int DIM, class CS>
__device__ int choose_survivors(int tot, int ns, const float rsq, float* s_sp, int32_t* s_scell,
                                int32_t* s_heads, int32_t* s_next, float* s_S, float* gS,
                                int32_t* gnext, const bool mirror, ChooseResolve& cr)
{
    constexpr int BLOCK = CS::BLOCK;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    while (tot > 0) {
        const int m = min(CHOOSE_G, tot);
        // conflict rows: a warp shares the word (its points j are broadcast
        // reads) and takes consecutive rows i
        for (int t = tid; t < CHOOSE_G * CHOOSE_GW; t += BLOCK) {
            const int i = t % CHOOSE_G, w = t / CHOOSE_G;
            uint32_t row = 0;
            if (i < m && w * 32 + 31 > i) {
                float p[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d) p[d] = s_sp[i * DIM + d];
                const int j1 = min(m - w * 32, 32);
                for (int b = 0; b < j1; ++b) {
                    const int j = w * 32 + b;
                    if (sqdist_exact<DIM>(s_sp + j * DIM, p) <= rsq) row |= 1u << b;
                }
                // later points only
                if (w * 32 <= i) row &= ~((2u << (i - w * 32)) - 1u);
            }
            cr.adj[i * CHOOSE_GW + w] = row;
        }
        __syncthreads();
        if (warp == 0) {
            uint32_t alive = 0;
            if (lane < CHOOSE_GW) {
                const int left = m - lane * 32;
                alive = left >= 32 ? 0xffffffffu : (left > 0 ? (1u << left) - 1u : 0u);
            }
            int k = 0;
            for (;;) {
                const unsigned any = __ballot_sync(FULL, alive != 0);
                if (!any) break;
                const int l = __ffs(any) - 1;
                const int i = l * 32 + __ffs(__shfl_sync(FULL, alive, l)) - 1;
                if (lane == 0) cr.pick[k] = i;
                ++k;
                if (lane == l) alive &= alive - 1;
                if (lane < CHOOSE_GW) alive &= ~cr.adj[i * CHOOSE_GW + lane];
            }
            if (lane == 0) cr.npick = k;
        }
        __syncthreads();
        const int k = cr.npick;
        for (int r = tid; r < k; r += BLOCK) {
            const int i = cr.pick[r], q = ns + r;
            const uint32_t b = cell_hash<DIM>(s_scell + i * DIM) & (uint32_t)(CS::HB - 1);
            const int head = atomicExch(&s_heads[b], q);   // any order inside a bucket
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const float x = s_sp[i * DIM + d];
                gS[(int64_t)q * DIM + d] = x;
                if (q < CS::SCAP) s_S[q * DIM + d] = x;
            }
            if (q < CS::SCAP) s_next[q] = head;
            if (mirror || q >= CS::SCAP) gnext[q] = head;
        }
        __syncthreads();
        // the rest: one survivor per thread (tot <= BLOCK)
        const int j = m + tid;
        bool surv = j < tot;
        float p[DIM];
        int cc[DIM];
        if (surv) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                p[d] = s_sp[j * DIM + d];
                cc[d] = s_scell[j * DIM + d];
            }
            for (int q = ns; q < ns + k && surv; ++q) {
                float s[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d)
                    s[d] = (q < CS::SCAP) ? s_S[q * DIM + d] : gS[(int64_t)q * DIM + d];
                surv = !(sqdist_exact<DIM>(p, s) <= rsq);
            }
        }
        const unsigned bal = __ballot_sync(FULL, surv);
        if (lane == 0) cr.wsum[warp] = __popc(bal);
        __syncthreads();
        int pos = __popc(bal & lanemask_lt()), left = 0;
#pragma unroll
        for (int w = 0; w < BLOCK / 32; ++w) {
            const int x = cr.wsum[w];
            pos += (w < warp) ? x : 0;
            left += x;
        }
        if (surv) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                s_sp[pos * DIM + d] = p[d];
                s_scell[pos * DIM + d] = cc[d];
            }
        }
        ns += k;
        tot = left;
        __syncthreads();
    }
    return ns;
}

template <int DIM, class CS>
__global__ void __launch_bounds__(CS::BLOCK) k_choose(EngineView v)
{
    constexpr int BLOCK = CS::BLOCK;
    constexpr int NB = Pow3<DIM>::v;
    __shared__ ChooseResolve s_cr;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int32_t* s_heads = reinterpret_cast<int32_t*>(smem_raw);          // HB
    int32_t* s_next = s_heads + CS::HB;                                // SCAP
    float* s_S = reinterpret_cast<float*>(s_next + CS::SCAP);          // SCAP*DIM
    float* s_sp = s_S + CS::SCAP * DIM;                                // BLOCK*DIM
    int32_t* s_scell = reinterpret_cast<int32_t*>(s_sp + BLOCK * DIM); // BLOCK*DIM
    __shared__ int s_wsum[BLOCK / 32];
    int ns = 0;   // the same in every thread

    const int c = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const CloudDesc cd = v.cl[c];
    const int n = cd.n_own;
    const float rsq = sqr_rn(cd.r1);
    const double inv = 1.0 / ((double)cd.r1 * (1.0 + 1.0 / 1024.0));
    const uint32_t hmask = CS::HB - 1;
    float* gS = v.S + cd.s_off * DIM;
    int32_t* gnext = v.next + cd.s_off;
    const float* P = v.P + cd.p_off * DIM;

    for (int h = tid; h < CS::HB; h += BLOCK) s_heads[h] = -1;
    __syncthreads();

    auto coord = [&](int q, int d) -> float {
        return (q < CS::SCAP) ? s_S[q * DIM + d] : gS[(int64_t)q * DIM + d];
    };
    auto nxt = [&](int q) -> int { return (q < CS::SCAP) ? s_next[q] : gnext[q]; };
    // any chosen point within r1 of p, over the given neighbour cells
    auto query = [&](const float* p, const int* cc, int o) -> bool {
        int nc[DIM];
        neighbour_cell<DIM>(cc, o, nc);
        int q = s_heads[cell_hash<DIM>(nc) & hmask];
        while (q >= 0) {
            float s[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) s[d] = coord(q, d);
            if (sqdist_exact<DIM>(p, s) <= rsq) return true;
            q = nxt(q);
        }
        return false;
    };

    for (int base = 0; base < n; base += BLOCK) {
        const int i = base + tid;
        const bool valid = i < n;
        float p[DIM];
        int cc[DIM];
        bool surv = false;
        if (valid) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                p[d] = P[(int64_t)i * DIM + d];
                cc[d] = cell_of(p[d], inv);
            }
            bool hit = false;
            for (int t = 0; t < NB && !hit; ++t) hit = query(p, cc, (t + NB / 2) % NB);
            surv = !hit;
        }
        // compact survivors in visiting order
        const unsigned bal = __ballot_sync(FULL, surv);
        if (lane == 0) s_wsum[warp] = __popc(bal);
        __syncthreads();
        int wbase = 0, tot = 0;
        for (int w = 0; w < BLOCK / 32; ++w) {
            const int x = s_wsum[w];
            wbase += (w < warp) ? x : 0;
            tot += x;
        }
        if (surv) {
            const int pos = wbase + __popc(bal & lanemask_lt());
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                s_sp[pos * DIM + d] = p[d];
                s_scell[pos * DIM + d] = cc[d];
            }
        }
        __syncthreads();
        ns = choose_survivors<DIM, CS>(tot, ns, rsq, s_sp, s_scell, s_heads, s_next, s_S, gS, gnext,
                                       false, s_cr);
    }
    if (tid == 0) {
        v.ns[c] = ns;
        v.phase[c] = (ns > 0) ? PH_EVOLVE : PH_DONE;
    }
}

// ---------------------------------------------------------------------------
// choose for one large cloud, in rounds over growing ranges [a, b) of its
// points (same semantics as k_choose).  k_choose_filter, spread over the whole
// GPU, drops every point of the range that has a point chosen in earlier rounds
// within r1 (hash grid read from global memory); a stable compaction lists the
// survivors in order; k_choose_resolve, one CTA, walks that list and applies
// the sequential greedy rule with a shared-memory mirror of the grid, then
// writes the grid back for the next round's filter.
// ---------------------------------------------------------------------------
template <int DIM>
__global__ void __launch_bounds__(256) k_choose_filter(EngineView v, int c, int a, int b,
                                                       uint8_t* __restrict__ surv)
{
    using CS = ChooseSmem<DIM>;
    constexpr int NB = Pow3<DIM>::v;
    const CloudDesc cd = v.cl[c];
    const float rsq = sqr_rn(cd.r1);
    const double inv = 1.0 / ((double)cd.r1 * (1.0 + 1.0 / 1024.0));
    const uint32_t hmask = CS::HB - 1;
    const int32_t* heads = v.hash;
    const float* gS = v.S + cd.s_off * DIM;
    const int32_t* gnext = v.next + cd.s_off;
    const float* P = v.P + cd.p_off * DIM;
    for (int i = a + blockIdx.x * blockDim.x + threadIdx.x; i < b; i += gridDim.x * blockDim.x) {
        float p[DIM];
        int cc[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            p[d] = P[(int64_t)i * DIM + d];
            cc[d] = cell_of(p[d], inv);
        }
        bool hit = false;
        for (int t = 0; t < NB && !hit; ++t) {
            int nc[DIM];
            neighbour_cell<DIM>(cc, (t + NB / 2) % NB, nc);
            for (int q = heads[cell_hash<DIM>(nc) & hmask]; q >= 0 && !hit; q = gnext[q]) {
                float s[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d) s[d] = gS[(int64_t)q * DIM + d];
                hit = sqdist_exact<DIM>(p, s) <= rsq;
            }
        }
        surv[i - a] = hit ? 0 : 1;
    }
}

// sel: the survivors of [a, b) in order, *nsel of them (nullptr in the first
// round, where every point of the range is a candidate).  The candidates are
// taken in blocks of BLOCK as k_choose takes its points: all threads load
// their candidates, compute their cells and drop those within r1 of a point
// chosen so far (earlier rounds and earlier blocks of this one); choose_survivors
// then applies the greedy rule to the block's survivors.
template <int DIM, class CS>
__global__ void __launch_bounds__(CS::BLOCK) k_choose_resolve(EngineView v, int c, int a, int b,
                                                          const int32_t* __restrict__ sel,
                                                          const int32_t* __restrict__ nsel,
                                                          int first)
{
    constexpr int BLOCK = CS::BLOCK;
    __shared__ ChooseResolve s_cr;
    constexpr int NB = Pow3<DIM>::v;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    int32_t* s_heads = reinterpret_cast<int32_t*>(smem_raw);          // HB
    int32_t* s_next = s_heads + CS::HB;                                // SCAP
    float* s_S = reinterpret_cast<float*>(s_next + CS::SCAP);          // SCAP*DIM
    float* s_sp = s_S + CS::SCAP * DIM;                                // BLOCK*DIM
    int32_t* s_scell = reinterpret_cast<int32_t*>(s_sp + BLOCK * DIM); // BLOCK*DIM
    __shared__ int s_wsum[BLOCK / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const CloudDesc cd = v.cl[c];
    const float rsq = sqr_rn(cd.r1);
    const double inv = 1.0 / ((double)cd.r1 * (1.0 + 1.0 / 1024.0));
    const uint32_t hmask = CS::HB - 1;
    float* gS = v.S + cd.s_off * DIM;
    int32_t* gnext = v.next + cd.s_off;
    const float* P = v.P + cd.p_off * DIM;
    const int ns0 = first ? 0 : v.ns[c];
    for (int h = tid; h < CS::HB; h += BLOCK) s_heads[h] = first ? -1 : v.hash[h];
    for (int q = tid; q < min(ns0, CS::SCAP); q += BLOCK) {
        s_next[q] = gnext[q];
#pragma unroll
        for (int d = 0; d < DIM; ++d) s_S[q * DIM + d] = gS[(int64_t)q * DIM + d];
    }
    int ns = ns0;   // the same in every thread
    __syncthreads();
    auto coord = [&](int q, int d) -> float {
        return (q < CS::SCAP) ? s_S[q * DIM + d] : gS[(int64_t)q * DIM + d];
    };
    auto nxt = [&](int q) -> int { return (q < CS::SCAP) ? s_next[q] : gnext[q]; };
    // any chosen point within r1 of p, over the given neighbour cells
    auto query = [&](const float* p, const int* cc, int o) -> bool {
        int nc[DIM];
        neighbour_cell<DIM>(cc, o, nc);
        int q = s_heads[cell_hash<DIM>(nc) & hmask];
        while (q >= 0) {
            float s[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) s[d] = coord(q, d);
            if (sqdist_exact<DIM>(p, s) <= rsq) return true;
            q = nxt(q);
        }
        return false;
    };
    const int cnt = sel ? *nsel : (b - a);
    for (int base = 0; base < cnt; base += BLOCK) {
        const int j = base + tid;
        float p[DIM];
        int cc[DIM];
        bool surv = false;
        if (j < cnt) {
            const int i = sel ? sel[j] : a + j;
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                p[d] = P[(int64_t)i * DIM + d];
                cc[d] = cell_of(p[d], inv);
            }
            bool hit = false;
            for (int t = 0; t < NB && !hit; ++t) hit = query(p, cc, (t + NB / 2) % NB);
            surv = !hit;
        }
        // compact the block's survivors in visiting order
        const unsigned bal = __ballot_sync(FULL, surv);
        if (lane == 0) s_wsum[warp] = __popc(bal);
        __syncthreads();
        int wbase = 0, tot = 0;
        for (int w = 0; w < BLOCK / 32; ++w) {
            const int x = s_wsum[w];
            wbase += (w < warp) ? x : 0;
            tot += x;
        }
        if (surv) {
            const int pos = wbase + __popc(bal & lanemask_lt());
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                s_sp[pos * DIM + d] = p[d];
                s_scell[pos * DIM + d] = cc[d];
            }
        }
        __syncthreads();
        ns = choose_survivors<DIM, CS>(tot, ns, rsq, s_sp, s_scell, s_heads, s_next, s_S, gS, gnext,
                                       true, s_cr);
    }
    for (int h = tid; h < CS::HB; h += BLOCK) v.hash[h] = s_heads[h];
    if (tid == 0) {
        v.ns[c] = ns;
        v.phase[c] = (ns > 0) ? PH_EVOLVE : PH_DONE;
    }
}

// ---------------------------------------------------------------------------
// assign: rd/cpu/brute_force/evolve.hpp:43-66 over one chunk of CHUNK cloud
// points per work item; writes the key of every point and the chunk's key
// histogram row.  This is the hot kernel.
// ---------------------------------------------------------------------------
template <int DIM>
__device__ __forceinline__ void load_chosen(const float* sS, int kk, float* s)
{
    constexpr int DP = PadDim<DIM>::v;
    if constexpr (DP == 4) {
        const float4 t = reinterpret_cast<const float4*>(sS)[kk];
        s[0] = t.x; s[1] = t.y; s[2] = t.z;
        if constexpr (DIM == 4) s[3] = t.w;
    } else if constexpr (DP == 2) {
        const float2 t = reinterpret_cast<const float2*>(sS)[kk];
        s[0] = t.x; s[1] = t.y;
    } else {
#pragma unroll
        for (int d = 0; d < DIM; ++d) s[d] = sS[kk * DP + d];
    }
}

constexpr int ASSIGN_TS = 1024;  // chosen points per shared-memory tile

template <int DIM, int BLOCK, int ITEMS>
__global__ void __launch_bounds__(BLOCK) k_assign(EngineView v)
{
    pdl_enter();
    constexpr int DP = PadDim<DIM>::v;
    constexpr int TS = ASSIGN_TS;
    __shared__ __align__(16) float sS[TS * DP];
    __shared__ int s_item;
    extern __shared__ int s_hist[];
    const int tid = threadIdx.x;

    const ActiveList al(v, ACT_CHUNK);
    for (;;) {
        if (tid == 0) s_item = atomicAdd(&v.ctr[CTR_WORK], 1);
        __syncthreads();
        const int item = s_item;
        __syncthreads();
        if (item >= al.total) break;
        int c, lc;
        al.locate(item, c, lc);
        const CloudDesc cd = v.cl[c];
        // chunks split the cloud evenly (at most BLOCK*ITEMS points each)
        const int start = (int)(((int64_t)lc * cd.n_all) / cd.n_chunks);
        const int n = (int)(((int64_t)(lc + 1) * cd.n_all) / cd.n_chunks);  // chunk end
        const int ns = v.ns[c];
        const float* P = v.P + cd.p_off * DIM;
        const float* gS = v.S + cd.s_off * DIM;

        // Two-level argmin.  The inner loop keeps only the running minimum
        // (one min per pair instead of compare + two selects) and records the
        // block of KB chosen points in which it last decreased; the exact
        // index is then the first point of that block at exactly the minimum.
        // Strict decrease per block and first match inside the block give the
        // reference's rule: lowest index among equal minima.
        constexpr int KB = 8;
        constexpr float FAR = 1e30f;  // padding: (FAR - p)^2 overflows to +inf
        static_assert(ITEMS % 2 == 0, "points are processed in pairs");
        float p[ITEMS][DIM];
        float2 np2[ITEMS / 2][DIM];  // negated coordinates of point pairs (2jj, 2jj+1)
        float best[ITEMS];
        int blk[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const int i = start + j * BLOCK + tid;
#pragma unroll
            for (int d = 0; d < DIM; ++d) p[j][d] = (i < n) ? P[(int64_t)i * DIM + d] : 0.0f;
            best[j] = FLT_MAX;
            blk[j] = -1;
        }
#pragma unroll
        for (int jj = 0; jj < ITEMS / 2; ++jj)
#pragma unroll
            for (int d = 0; d < DIM; ++d) np2[jj][d] = make_float2(-p[2 * jj][d], -p[2 * jj + 1][d]);
        for (int t0 = 0; t0 < ns; t0 += TS) {
            const int tl = min(TS, ns - t0);
            const int tlp = (tl + KB - 1) / KB * KB;
            __syncthreads();
            for (int e = tid; e < tlp; e += BLOCK) {
#pragma unroll
                for (int d = 0; d < DIM; ++d)
                    sS[e * DP + d] = (e < tl) ? gS[(int64_t)(t0 + e) * DIM + d] : FAR;
            }
            __syncthreads();
            for (int kb = 0; kb < tlp; kb += KB) {
                float old[ITEMS];
#pragma unroll
                for (int j = 0; j < ITEMS; ++j) old[j] = best[j];
#pragma unroll
                for (int u = 0; u < KB; ++u) {
                    float s[DIM];
                    load_chosen<DIM>(sS, kb + u, s);
#pragma unroll
                    for (int jj = 0; jj < ITEMS / 2; ++jj) {
                        const float2 q = sqdist2_exact<DIM>(s, np2[jj]);
                        best[2 * jj] = fminf(best[2 * jj], q.x);
                        best[2 * jj + 1] = fminf(best[2 * jj + 1], q.y);
                    }
                }
#pragma unroll
                for (int j = 0; j < ITEMS; ++j) blk[j] = (best[j] < old[j]) ? (t0 + kb) : blk[j];
            }
        }
        const float rsq = sqr_rn(cd.r1);
        int key[ITEMS];
#pragma unroll
        for (int j = 0; j < ITEMS; ++j) {
            const int i = start + j * BLOCK + tid;
            int idx = -1;
            if (i < n && best[j] <= rsq && blk[j] >= 0) {
                for (int u = 0; u < KB; ++u) {
                    const int k = blk[j] + u;
                    if (k >= ns) break;
                    float s[DIM];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) s[d] = gS[(int64_t)k * DIM + d];
                    if (sqdist_exact<DIM>(s, p[j]) == best[j]) { idx = k; break; }
                }
            }
            key[j] = idx;
            if (i < n) v.keys[cd.p_off + i] = key[j];
        }
        // chunk histogram row (row length ns_cap, first ns entries used)
        int32_t* row = v.hist + cd.hist_off + (int64_t)lc * cd.ns_cap;
        if (ns <= v.hist_smem) {
            for (int k = tid; k < ns; k += BLOCK) s_hist[k] = 0;
            __syncthreads();
#pragma unroll
            for (int j = 0; j < ITEMS; ++j)
                if (key[j] >= 0) atomicAdd(&s_hist[key[j]], 1);
            __syncthreads();
            for (int k = tid; k < ns; k += BLOCK) row[k] = s_hist[k];
        } else {
            for (int k = tid; k < ns; k += BLOCK) row[k] = 0;
            __syncthreads();
#pragma unroll
            for (int j = 0; j < ITEMS; ++j)
                if (key[j] >= 0) atomicAdd(&row[key[j]], 1);
        }
    }
}

// ---------------------------------------------------------------------------
// Culled assignment: the same keys as k_assign, over the spatial order (Ps,
// built once per run by launch_spatial_prep, DIM padded to PadDim) instead of
// the slot order, and only where a key can have changed.  A block is 32 x ITEMS
// consecutive points of that order, one warp each, with the bounding boxes of
// its two parts (rd_spatial.cu says where they part); "the box" below is their
// union and the gap to it the smaller of the two.
//
// Which chosen points a block looks at.  A chosen point s takes part in a
// block's argmin only when the squared gap between s and the box, g2, is at
// most thr = r1^2 (1 + 2^-10) (rounded up).  Exactness: the computed g2 exceeds
// the exact squared gap G by at most a relative 2^-20 (a few roundings of
// non-negative terms), and every computed distance from s to a point of the box
// is at least G (1 - 2^-20); so g2 > thr makes every such distance > r1^2.  A
// skipped chosen point can then neither be the nearest one within r1 nor tie
// with it, and the minimum over the remaining points, visited in index order
// with strict '<', is the reference's (rd/cpu/brute_force/evolve.hpp:54-66).
// The bound needs r1^2 in the normal range; any other r1 disables the skip.
// NaN gaps never skip.
//
// Which blocks are looked at.  An evaluation leaves the block's slack: the
// smallest margin of its points.  For a point with nearest chosen point at
// distance d1 <= r1 and the next kept one at d2 the margin is
// (min(d2, r1) - d1) / 2; for a point with none within r1 it is d1 - r1, at
// most 4e-4 r1; both less 1e-5 r1 for the roundings (distances carry a relative
// error below 2^-21).  k_merge_fold lists every chosen point it moves with its
// old and new place and the length of the move (rounded up).  Let D be the
// largest move, in this pass, of a chosen point within thr of the box before or
// after it.  The slack is lowered by D (rounded down), and while it stays
// positive no key of the block can have changed: the nearest chosen point, in
// range of the box all along, is at most d1 + sum D away.  Any other one was,
// when last out of range, more than r1 away, or it was kept and at least d2
// away, and came at most sum D closer since; with the margin above both stay
// behind the nearest one, and that one within r1.  A point with none within r1
// stays so: kept chosen points were d1 away, others at least r1 (1 + 4.8e-4).
// `full` clouds (first pass, after a decimation, after new chosen points)
// evaluate every block.  A block first tries the largest move of the whole
// cloud, one comparison, and scans the list of moves only when that does not do.
//
// Candidates.  A block keeps the list, in index order, of the chosen points
// within R = r1 + r1/4 of its box (with the same 2^-10 on R^2) as its last scan
// of the whole chosen set found them, while the moves D since then -- taken
// over the chosen points within R of the box, which covers those within r1 --
// add up to less than r1/4: any other chosen point is then still more than
// r1 (1 + 4.8e-4) away.  An evaluation reads that list, at most CAND_MAX
// entries, instead of every chosen point; a block with more candidates keeps
// none and scans.
//
// Only changed keys are written: to the points' slots, to the spatial copy
// (ksp), as -1/+1 in the histogram row of their slot-order chunk (which so
// always holds the current counts), and as an edit of both keys' member lists
// (push_edit); k_merge_fold then touches the keys with edits only.  A key with
// unchanged members keeps its sum, and its chosen point has answered the
// movement test for that sum already (it moved to the mean, or stayed within
// the threshold).
//
// 1M-point helix, 285 passes: the median pass changes 0.1% of the keys; the
// kernel that evaluated every block, with its keys and counts written anew,
// took 36 us per pass; this one 45 us in the first pass (candidate lists built),
// 25-40 us while every chosen point moves, 11-22 us after.  Bound by the few
// blocks whose candidates do not fit a list, then by instruction issue.
// ---------------------------------------------------------------------------
constexpr int AC_BLOCK = 256;             // threads of k_assign_cull
constexpr int AC_WARPS = AC_BLOCK / 32;

// squared gap between s and the box [lo, hi] (0 inside; NaN-free for NaN s)
template <int DIM>
__device__ __forceinline__ float box_gap2(const float* s, const float* lo, const float* hi)
{
    float g2 = 0.0f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const float gap = fmaxf(fmaxf(__fsub_rn(lo[d], s[d]), __fsub_rn(s[d], hi[d])), 0.0f);
        g2 = __fadd_rn(g2, __fmul_rn(gap, gap));
    }
    return g2;
}

// the same for the nearer of a block's two boxes, b[2][lo, hi] (an empty one is
// infinitely far; a NaN gap stays NaN, which never skips)
template <int DIM>
__device__ __forceinline__ float block_gap2(const float* s, const float (&b)[2][2 * DIM])
{
    const float g0 = box_gap2<DIM>(s, b[0], b[0] + DIM), g1 = box_gap2<DIM>(s, b[1], b[1] + DIM);
    return (g0 > g1) ? g1 : g0;
}

// One chosen point against the block's points: nearest and second nearest.
template <int DIM, int ITEMS>
__device__ __forceinline__ void assign_one(const float* sk, const int k, const float2 (&np2)[ITEMS / 2][DIM],
                                           float (&best)[ITEMS], float (&sec)[ITEMS], int (&key)[ITEMS])
{
#pragma unroll
    for (int jj = 0; jj < ITEMS / 2; ++jj) {
        const float2 dd = sqdist2_exact<DIM>(sk, np2[jj]);
        sec[2 * jj] = fminf(sec[2 * jj], fmaxf(best[2 * jj], dd.x));
        sec[2 * jj + 1] = fminf(sec[2 * jj + 1], fmaxf(best[2 * jj + 1], dd.y));
        if (dd.x < best[2 * jj]) { best[2 * jj] = dd.x; key[2 * jj] = k; }
        if (dd.y < best[2 * jj + 1]) { best[2 * jj + 1] = dd.y; key[2 * jj + 1] = k; }
    }
}

// moves of a single cloud staged in shared memory
constexpr int AC_MOVES = 512;
constexpr int EDIT_IN = (int)0x80000000;   // edit of a member list: this point joins (else it leaves)
constexpr int EDIT_MAX = 512;              // edits of one key that k_merge_fold takes

// rows of a key's region of the grouped lists with n members at the rebuild:
// room for its list to grow before the next rebuild (without lists every pass
// rebuilds)
__device__ __forceinline__ int list_cap(const EngineView& v, const int n)
{
    return v.lists ? list_room(n) : n;
}

// A pass regroups all points of a cloud by key: its chosen points are new or
// renumbered, or a key got more edits than it takes.
__device__ __forceinline__ bool rebuilds(const EngineView& v, const int c)
{
    return !v.lists || v.full[c] != 0 || v.reb[c] != 0;
}

// One edit of key k's member list.  The first one of the pass lists the key as
// work for k_merge_fold.
__device__ __forceinline__ void push_edit(const EngineView& v, const int c, const CloudDesc& cd,
                                          const int k, const int edit)
{
    const int64_t s = cd.key_off + k;
    const int at = atomicAdd(&v.ecnt[s], 1);
    if (at == 0) v.dlist[atomicAdd(&v.ctr[CTR_NDIRTY], 1)] = (int)s;
    const int2 reg = *reinterpret_cast<const int2*>(v.kinfo + s);   // base, capacity
    if (at < min(EDIT_MAX, reg.y)) v.edit[cd.reg_off + reg.x + at] = edit;
    else v.reb[c] = 1;
}

// resident CTAs the registers are held to: the evaluation waits on memory
// (points, keys, candidates, in three dependent steps), so warps in flight
// count; eight points per lane need the registers
template <int DIM, int ITEMS>
__global__ void __launch_bounds__(AC_BLOCK, ITEMS <= 4 ? 4 : 2) k_assign_cull(EngineView v)
{
    pdl_enter();
    static_assert(ITEMS % 2 == 0, "points are evaluated in pairs");
    constexpr int DP = PadDim<DIM>::v;
    constexpr int WPTS = 32 * ITEMS;
    const int lane = threadIdx.x & 31;
    __shared__ float s_mv[2 * DIM + 1][AC_MOVES];
    const ActiveList al(v, ACT_CHUNK);
    int n_staged = 0;   // the cloud's moves are in s_mv
    if (v.single) {
        const int m = v.mvn[0];
        if (m <= AC_MOVES && !v.full[0]) {
            for (int e = threadIdx.x; e < (2 * DIM + 1) * m; e += AC_BLOCK)
                s_mv[e / m][e % m] = v.mv[(int64_t)(e / m) * v.n_slots + e % m];
            n_staged = m;
        }
        __syncthreads();
    }
    const int wpc_log = 31 - __clz(v.chunk_pts / WPTS);   // blocks per chunk, a power of two
    const int total = al.total << wpc_log;
    const int nw = gridDim.x * AC_WARPS;
    // a warp takes blocks nw apart, one per lane: the lanes find their blocks'
    // clouds and make the one-comparison test at the same time
    for (int64_t base = blockIdx.x * AC_WARPS + (threadIdx.x >> 5); base < total; base += (int64_t)32 * nw) {
        const int64_t t = base + (int64_t)lane * nw;
        int my_c = 0, my_i = 0, my_full = 0;
        float my_slack = 0.0f;
        bool need = false;
        if (t < total) {
            int lc;
            al.locate((int)(t >> wpc_log), my_c, lc);
            my_i = (lc << wpc_log) + ((int)t & ((1 << wpc_log) - 1));
            const int my_n = v.single ? v.one.n_all : v.cl[my_c].n_all;
            if ((int64_t)my_i * WPTS < my_n) {
                const int64_t wb =
                    ((v.single ? v.one.chunk_begin : v.cl[my_c].chunk_begin) << wpc_log) + my_i;
                my_full = v.full[my_c];
                const float dmax = __int_as_float(v.dmax[my_c]);
                my_slack = v.bslack[wb];
                need = my_full || !(my_slack > dmax);
                if (!need && dmax > 0.0f) {
                    v.bslack[wb] = __fsub_rd(my_slack, dmax);
                    v.lslack[wb] = __fsub_rd(v.lslack[wb], dmax);
                }
            }
        }
        for (unsigned todo = __ballot_sync(FULL, need); todo; todo &= todo - 1) {
            const int src = __ffs(todo) - 1;
            const int c = __shfl_sync(FULL, my_c, src);
            const int bi = __shfl_sync(FULL, my_i, src);
            const int full = __shfl_sync(FULL, my_full, src);
            const CloudDesc cd = cloud_desc(v, c);
            const int ns = v.ns[c];
            const int64_t wb = (cd.chunk_begin << wpc_log) + bi;
            const float rsq = sqr_rn(cd.r1);
            const bool may_skip = rsq >= 1.0e-30f && rsq <= 1.0e30f;
            const float thr = __fmul_ru(rsq, 1.0009765625f);
            float box[2][2 * DIM];
#pragma unroll
            for (int e = 0; e < 2 * DIM; ++e) {
                box[0][e] = v.bbox[wb * 4 * DIM + e];
                box[1][e] = v.bbox[wb * 4 * DIM + 2 * DIM + e];
            }
            // this lane's points and their keys (positions past the cloud: slot < 0)
            const int pos0 = bi * WPTS + lane;
            const float* Ps = v.Ps + cd.p_off * DP;
            int32_t* ksp = v.ksp + cd.p_off;
            const int m = v.mvn[c];
            const float reach = __fadd_ru(cd.r1, 0.25f * cd.r1);
            const float thr_list = __fmul_ru(__fmul_ru(reach, reach), 1.0009765625f);
            float dl = __int_as_float(v.dmax[c]);
            // a list longer than half the chosen set costs about as much as the
            // evaluation it may save
            if (!full && 2 * m <= ns + 64) {
                unsigned dloc = 0;
                const bool staged = m == n_staged;
                const float* mv = staged ? &s_mv[0][0] : v.mv + cd.key_off;
                const int64_t pitch = staged ? AC_MOVES : v.n_slots;
                for (int j = lane; j < m; j += 32) {
                    float o[DIM], q[DIM];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) {
                        o[d] = mv[d * pitch + j];
                        q[d] = mv[(DIM + d) * pitch + j];
                    }
                    const bool out = may_skip && block_gap2<DIM>(o, box) > thr_list &&
                                     block_gap2<DIM>(q, box) > thr_list;
                    // lengths are not negative (or NaN): they order as their bits do
                    if (!out) dloc = max(dloc, __float_as_uint(mv[2 * DIM * pitch + j]));
                }
                dl = __uint_as_float(__reduce_max_sync(FULL, dloc));
                const float slack = __shfl_sync(FULL, my_slack, src);
                if (slack > dl) {
                    if (lane == 0 && dl > 0.0f) {
                        v.bslack[wb] = __fsub_rd(slack, dl);
                        v.lslack[wb] = __fsub_rd(v.lslack[wb], dl);
                    }
                    continue;
                }
            }
            const float list_left = full ? 0.0f : __fsub_rd(v.lslack[wb], dl);
            const int n_list = (list_left > 0.0f) ? v.blen[wb] : -1;
            int32_t* list = v.blist + wb * CAND_MAX;
            float2 np2[ITEMS / 2][DIM];
            int old[ITEMS];
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const int i = pos0 + j * 32;
                float p[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d) p[d] = 0.0f;
                old[j] = -1;
                if (i < cd.n_all) {
                    load_chosen<DIM>(Ps, i, p);
                    old[j] = ksp[i];
                }
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    if (j & 1) np2[j / 2][d].y = -p[d];
                    else np2[j / 2][d].x = -p[d];
                }
            }
            float best[ITEMS], sec[ITEMS];
            int key[ITEMS];
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                best[j] = FLT_MAX;
                sec[j] = FLT_MAX;
                key[j] = -1;
            }
            const float* gS = v.S + cd.s_off * DIM;
            // kept chosen points in index order, from their lanes' registers
            auto take = [&](unsigned kept, const float (&s)[DIM], const int k_of_lane) {
                while (kept) {
                    const int b = __ffs(kept) - 1;
                    kept &= kept - 1;
                    float sk[DIM];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) sk[d] = __shfl_sync(FULL, s[d], b);
                    assign_one<DIM, ITEMS>(sk, __shfl_sync(FULL, k_of_lane, b), np2, best, sec, key);
                }
            };
            float s[DIM];
            if (n_list >= 0) {
                for (int q0 = 0; q0 < n_list; q0 += 32) {
                    const bool in = q0 + lane < n_list;
                    const int k = in ? list[q0 + lane] : 0;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) s[d] = gS[(int64_t)k * DIM + d];
                    take(__ballot_sync(FULL, in && !(may_skip && block_gap2<DIM>(s, box) > thr)), s, k);
                }
                if (lane == 0) v.lslack[wb] = list_left;
            } else {
                float sn[DIM];
                int len = 0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) sn[d] = (lane < ns) ? gS[(int64_t)lane * DIM + d] : 0.0f;
                for (int q0 = 0; q0 < ns; q0 += 32) {
                    const int q = q0 + lane;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) {
                        s[d] = sn[d];
                        sn[d] = (q + 32 < ns) ? gS[(int64_t)(q + 32) * DIM + d] : 0.0f;
                    }
                    const float g2 = block_gap2<DIM>(s, box);
                    const bool near = q < ns && !(may_skip && g2 > thr_list);
                    const unsigned nb = __ballot_sync(FULL, near);
                    if (!nb) continue;
                    const int at = len + __popc(nb & lanemask_lt());
                    if (near && at < CAND_MAX) list[at] = q;
                    len += __popc(nb);
                    take(__ballot_sync(FULL, q < ns && !(may_skip && g2 > thr)), s, q);
                }
                if (lane == 0) {
                    v.blen[wb] = len;
                    v.lslack[wb] = (may_skip && len <= CAND_MAX) ? 0.25f * cd.r1 : 0.0f;
                }
            }
            const float r1 = cd.r1;
            float margin = FLT_MAX;
            int32_t* hist = v.hist + cd.hist_off;
#pragma unroll
            for (int j = 0; j < ITEMS; ++j) {
                const int i = pos0 + j * 32;
                if (i >= cd.n_all) continue;
                const bool in = best[j] <= rsq;
                const int k = in ? key[j] : -1;
                const float d1 = sqrtf(best[j]);
                const float mj = in ? 0.5f * (fminf(sqrtf(sec[j]), r1) - d1) : fminf(d1 - r1, 4.0e-4f * r1);
                margin = fminf(margin, mj);
                if (k != old[j]) {
                    const int slot = v.sorder[cd.p_off + i];
                    int32_t* row = hist + (int64_t)v.srow[cd.p_off + i] * cd.ns_cap;
                    v.keys[slot] = k;
                    ksp[i] = k;
                    if (old[j] >= 0) {
                        atomicAdd(&row[old[j]], -1);
                        if (!full) push_edit(v, c, cd, old[j], (int)(slot - cd.p_off));
                    }
                    if (k >= 0) {
                        atomicAdd(&row[k], 1);
                        if (!full) push_edit(v, c, cd, k, (int)(slot - cd.p_off) | EDIT_IN);
                    }
                }
            }
            // never negative, so that it orders as its bits do; 0: evaluate again
            margin = may_skip ? fmaxf(margin - 1.0e-5f * r1, 0.0f) : 0.0f;
            const unsigned mb = __reduce_min_sync(FULL, __float_as_uint(margin));
            if (lane == 0) v.bslack[wb] = __uint_as_float(mb);
        }
    }
}

// ---------------------------------------------------------------------------
// Chunk scan, for the clouds that regroup in this pass (rebuilds): for every
// chosen point k, the exclusive prefix over the cloud's chunks of the chunk x
// key histogram (hpre row lc: members in earlier chunks) and the member count
// cnt[k].  Work item = block of KBLK keys, one key per lane.
//   k_chunkscan_cta   clouds with many chunk rows or chosen points (scan_by_cta):
//                     one CTA per item; the CS_W warps take contiguous row ranges, sum
//                     them, exchange the warp totals, and rescan their rows
//                     writing the prefixes;
//   k_chunkscan_warp  the other clouds: one warp per item, a single pass.
// The key bases follow in the same kernel: the CTA (warp) that finishes the
// last key block of a cloud -- a per-cloud counter of finished blocks says
// which -- lays out the cloud's lists (each key's region starts after the
// regions of the keys before it) and lists every key as work for k_merge_fold.
// In most passes no cloud regroups: the threads of a CTA (lanes of a warp) look
// at its next items' clouds together, so that it is done after one look.
// ---------------------------------------------------------------------------
constexpr int CS_W = 16;   // warps of the CTA-wide scan
constexpr int CSW_W = 8;   // items (warps) per CTA of the warp-wide scan
constexpr int CS_LOADS = 16;  // histogram loads in flight per lane
constexpr int CS_REG = 32;    // rows per warp kept in registers between the two passes

// the moves of the last pass have been read: empty every active cloud's list
__device__ __forceinline__ void clear_moves(const EngineView& v, const int first, const int stride)
{
    const int nact = v.ctr[CTR_NACT];
    for (int a = first; a < nact; a += stride) {
        v.mvn[v.act_cloud[a]] = 0;
        v.dmax[v.act_cloud[a]] = 0;
    }
}

// key k (global slot s) of a rebuilt cloud: its region [at, at + cap)
__device__ __forceinline__ void place_key(const EngineView& v, const int64_t s, const int at, const int cap)
{
    v.base[s] = at;
    // a long list takes no edits: the first one regroups the cloud
    v.kinfo[s] = make_int4(at, cap < v.merge_cap ? cap : 0, v.cnt[s], 0);
    if (v.ecnt[s] == 0) v.dlist[atomicAdd(&v.ctr[CTR_NDIRTY], 1)] = (int)s;  // else push_edit did
}

// key bases of cloud c by the whole CTA (any multiple of 32 threads)
__device__ void key_bases_cta(const EngineView& v, const int c, int* s_w, int& s_carry)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const CloudDesc cd = v.cl[c];
    const int ns = v.ns[c];
    const int32_t* cnt = v.cnt + cd.key_off;
    __syncthreads();  // earlier readers of s_w / s_carry are done
    if (threadIdx.x == 0) s_carry = 0;
    for (int k0 = 0; k0 < ns; k0 += blockDim.x) {
        __syncthreads();
        const int k = k0 + threadIdx.x;
        const int x = (k < ns) ? list_cap(v, cnt[k]) : 0;
        int incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_w[warp] = incl;
        __syncthreads();
        int wpre = 0, tot = 0;
        for (int w = 0; w < nw; ++w) {
            wpre += (w < warp) ? s_w[w] : 0;
            tot += s_w[w];
        }
        const int carry = s_carry;
        if (k < ns) place_key(v, cd.key_off + k, carry + wpre + incl - x, x);
        __syncthreads();
        if (threadIdx.x == 0) s_carry = carry + tot;
    }
}

// the same by one warp
__device__ void key_bases_warp(const EngineView& v, const int c, const int lane)
{
    const CloudDesc cd = v.cl[c];
    const int ns = v.ns[c];
    const int32_t* cnt = v.cnt + cd.key_off;
    int carry = 0;
    for (int k0 = 0; k0 < ns; k0 += 32) {
        const int k = k0 + lane;
        const int x = (k < ns) ? list_cap(v, cnt[k]) : 0;
        int incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        if (k < ns) place_key(v, cd.key_off + k, carry + incl - x, x);
        carry += __shfl_sync(FULL, incl, 31);
    }
}

__global__ void __launch_bounds__(CS_W * 32) k_chunkscan_cta(EngineView v)
{
    pdl_enter();
    __shared__ int s_part[CS_W][32];
    __shared__ int s_w[CS_W];
    __shared__ int s_carry, s_last, s_n;
    __shared__ int2 s_item[CS_W * 32];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    clear_moves(v, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    const ActiveList al(v, ACT_KBLK);
    for (int64_t item0 = blockIdx.x; item0 < al.total; item0 += (int64_t)gridDim.x * blockDim.x) {
        // this thread's look: the CTA's threadIdx.x-th next item
        const int64_t mine = item0 + (int64_t)threadIdx.x * gridDim.x;
        int my_c = -1, my_kb = 0;
        if (mine < al.total) {
            al.locate((int)mine, my_c, my_kb);
            if (!rebuilds(v, my_c)) my_c = -1;
        }
        if (!__syncthreads_or(my_c >= 0)) continue;
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        if (my_c >= 0) {
            const int at = atomicAdd(&s_n, 1);
            s_item[at] = make_int2(my_c, my_kb);
        }
        __syncthreads();
        const int n_items = s_n;
        for (int q = 0; q < n_items; ++q) {
        const int c = s_item[q].x, kb = s_item[q].y;
        const CloudDesc cd = v.cl[c];
        const int ns = v.ns[c];
        const int k = kb * KBLK + lane;
        const bool ok = k < ns;
        const int rows = cd.n_chunks;
        const int rw0 = (warp * rows) / CS_W, rw1 = ((warp + 1) * rows) / CS_W;
        const int32_t* h = v.hist + cd.hist_off + k;
        int32_t* hp = v.hpre + cd.hist_off + k;
        // the first CS_REG rows of the warp's range stay in registers for the
        // rescan; longer ranges reload the rest
        int xr[CS_REG];
        int sum = 0;
#pragma unroll
        for (int u = 0; u < CS_REG; ++u)
            xr[u] = (ok && rw0 + u < rw1) ? h[(int64_t)(rw0 + u) * cd.ns_cap] : 0;
#pragma unroll
        for (int u = 0; u < CS_REG; ++u) sum += xr[u];
        for (int r0 = rw0 + CS_REG; r0 < rw1; r0 += CS_LOADS) {
            int x[CS_LOADS];
#pragma unroll
            for (int u = 0; u < CS_LOADS; ++u)
                x[u] = (ok && r0 + u < rw1) ? h[(int64_t)(r0 + u) * cd.ns_cap] : 0;
#pragma unroll
            for (int u = 0; u < CS_LOADS; ++u) sum += x[u];
        }
        s_part[warp][lane] = sum;
        __syncthreads();
        int run = 0, tot = 0;
#pragma unroll
        for (int w = 0; w < CS_W; ++w) {
            const int y = s_part[w][lane];
            run += (w < warp) ? y : 0;
            tot += y;
        }
#pragma unroll
        for (int u = 0; u < CS_REG; ++u) {
            if (ok && rw0 + u < rw1) hp[(int64_t)(rw0 + u) * cd.ns_cap] = run;
            run += xr[u];
        }
        for (int r0 = rw0 + CS_REG; r0 < rw1; r0 += CS_LOADS) {
            int x[CS_LOADS];
#pragma unroll
            for (int u = 0; u < CS_LOADS; ++u)
                x[u] = (ok && r0 + u < rw1) ? h[(int64_t)(r0 + u) * cd.ns_cap] : 0;
#pragma unroll
            for (int u = 0; u < CS_LOADS; ++u) {
                if (ok && r0 + u < rw1) hp[(int64_t)(r0 + u) * cd.ns_cap] = run;
                run += x[u];
            }
        }
        if (warp == 0 && ok) v.cnt[cd.key_off + k] = tot;
        // the last key block of the cloud: its key bases
        __threadfence();
        __syncthreads();  // also: s_part is reused by the next item
        if (threadIdx.x == 0)
            s_last = atomicAdd(&v.kbdone[c], 1) == (ns + KBLK - 1) / KBLK - 1;
        __syncthreads();
        if (s_last) {
            __threadfence();
            key_bases_cta(v, c, s_w, s_carry);
            if (threadIdx.x == 0) v.kbdone[c] = 0;
        }
        }
        __syncthreads();   // s_item and s_n are read no more
    }
}

__global__ void __launch_bounds__(CSW_W * 32) k_chunkscan_warp(EngineView v)
{
    pdl_enter();
    const int lane = threadIdx.x & 31;
    clear_moves(v, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
    const ActiveList al(v, ACT_KBLK_WARP);
    const int stride = gridDim.x * CSW_W;
    for (int64_t item0 = blockIdx.x * CSW_W + (threadIdx.x >> 5); item0 < al.total;
         item0 += (int64_t)32 * stride) {
        // this lane's look: the warp's lane-th next item
        const int64_t mine = item0 + (int64_t)lane * stride;
        int my_c = -1, my_kb = 0;
        if (mine < al.total) {
            al.locate((int)mine, my_c, my_kb);
            if (!rebuilds(v, my_c)) my_c = -1;
        }
        for (unsigned todo = __ballot_sync(FULL, my_c >= 0); todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        const int c = __shfl_sync(FULL, my_c, src), kb = __shfl_sync(FULL, my_kb, src);
        const CloudDesc cd = v.cl[c];
        const int ns = v.ns[c];
        const int k = kb * KBLK + lane;
        const bool ok = k < ns;
        const int rows = cd.n_chunks;
        const int32_t* h = v.hist + cd.hist_off + k;
        int32_t* hp = v.hpre + cd.hist_off + k;
        int run = 0;
        for (int r0 = 0; r0 < rows; r0 += CS_LOADS) {
            int x[CS_LOADS];
#pragma unroll
            for (int u = 0; u < CS_LOADS; ++u)
                x[u] = (ok && r0 + u < rows) ? h[(int64_t)(r0 + u) * cd.ns_cap] : 0;
#pragma unroll
            for (int u = 0; u < CS_LOADS; ++u) {
                if (ok && r0 + u < rows) hp[(int64_t)(r0 + u) * cd.ns_cap] = run;
                run += x[u];
            }
        }
        if (ok) v.cnt[cd.key_off + k] = run;
        // the last key block of the cloud: its key bases
        __threadfence();
        __syncwarp();
        int last = 0;
        if (lane == 0) last = atomicAdd(&v.kbdone[c], 1) == (ns + KBLK - 1) / KBLK - 1;
        if (__shfl_sync(FULL, last, 0)) {
            __threadfence();
            key_bases_warp(v, c, lane);
            if (lane == 0) v.kbdone[c] = 0;
        }
        }
    }
}

// ---------------------------------------------------------------------------
// stable scatter: one warp per chunk walks its points in index order and
// writes each assigned point's coordinates to the next free row of its key's
// segment of the grouped copy Pg, so every segment lists its members in
// cloud-point index order as one contiguous stream for the folds.  Keys of the chunk and the per-key start slots are
// staged in shared memory first; the ordered walk then touches shared memory
// only (match_any groups equal keys of 32 consecutive points, the group
// leader advances the key's cursor).
// ---------------------------------------------------------------------------
template <int DIM>
__device__ void scatter_chunk(const EngineView& v, int c, int lc, int* s_keys, int lane);

// row r of a grouped copy (PadDim<DIM> floats per row)
template <int DIM>
__device__ __forceinline__ void store_row(float* rows, int64_t r, const float (&q)[DIM])
{
    constexpr int DP = PadDim<DIM>::v;
    if constexpr (DP == 4) {
        reinterpret_cast<float4*>(rows)[r] =
            make_float4(q[0], DIM > 1 ? q[DIM > 1 ? 1 : 0] : 0.0f, DIM > 2 ? q[DIM > 2 ? 2 : 0] : 0.0f,
                        DIM > 3 ? q[DIM > 3 ? 3 : 0] : 0.0f);
    } else if constexpr (DP == 2) {
        reinterpret_cast<float2*>(rows)[r] = make_float2(q[0], q[1]);
    } else {
#pragma unroll
        for (int d = 0; d < DIM; ++d) rows[r * DP + d] = q[d];
    }
}


// One CTA per chunk for clouds with at most SCAT_HMAX chosen points.  The
// chunk is split into SCAT_W contiguous warp ranges; every warp counts its
// range's keys, an exclusive scan over the warps (per key) gives every warp
// its own start slots, and the warps then place their ranges at the same time,
// each in index order.  Ranges are in index order too, so the placement stays
// stable while the dependent placement chain is SCAT_W times shorter.  Larger
// chosen sets use scatter_chunk (one warp) in warp 0.
// Only the clouds that regroup in this pass are scattered; the threads of a CTA
// look at its next chunks' clouds together.
// groups of more clouds than this are gathered and compacted one thread per
// cloud (decimate_group)
constexpr int DEC_CLOUDS_SERIAL = 32;
constexpr int SCAT_W = 8;
constexpr int SCAT_HMAX = 1024;
constexpr int SCAT_KS = 8;   // chunk keys per thread loaded together (covers 2,048-point chunks)
constexpr int SCAT_SP = 8;   // placement steps whose coordinates are loaded together
static_assert(SCAT_HMAX % (SCAT_W * 32) == 0, "key bases: whole loads per thread");

template <int DIM>
__global__ void __launch_bounds__(SCAT_W * 32) k_scatter_cta(EngineView v)
{
    pdl_enter();
    constexpr int DP = PadDim<DIM>::v;
    extern __shared__ int s_dyn[];
    __shared__ int2 s_item[SCAT_W * 32];
    __shared__ int s_n;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const ActiveList al(v, ACT_CHUNK);
    for (int64_t item0 = blockIdx.x; item0 < al.total; item0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t mine = item0 + (int64_t)tid * gridDim.x;
        int my_c = -1, my_lc = 0;
        if (mine < al.total) {
            al.locate((int)mine, my_c, my_lc);
            if (!rebuilds(v, my_c)) my_c = -1;
        }
        if (tid == 0) s_n = 0;
        if (!__syncthreads_or(my_c >= 0)) continue;
        if (my_c >= 0) s_item[atomicAdd(&s_n, 1)] = make_int2(my_c, my_lc);
        __syncthreads();
        const int n_items = s_n;
        for (int q = 0; q < n_items; ++q) {
        __syncthreads();  // the previous chunk's readers are done
        const int c = s_item[q].x, lc = s_item[q].y;
        const CloudDesc cd = v.cl[c];
        const int ns = v.ns[c];
        if (ns > SCAT_HMAX) {
            if (warp == 0) scatter_chunk<DIM>(v, c, lc, s_dyn, lane);
            continue;
        }
        const int start = (int)(((int64_t)lc * cd.n_all) / cd.n_chunks);
        const int end = (int)(((int64_t)(lc + 1) * cd.n_all) / cd.n_chunks);
        const int len = end - start;
        int* s_keys = s_dyn;                 // chunk_max
        int* hw = s_dyn + v.chunk_max;       // SCAT_W x ns: counts, then start slots
        const int32_t* keys = v.keys + cd.p_off + start;
        const int32_t* row = v.hpre + cd.hist_off + (int64_t)lc * cd.ns_cap;
        const int32_t* bs = v.base + cd.key_off;
        const float* Pc = v.P + (cd.p_off + start) * DIM;
        float* Pg = v.Lr[0] + cd.reg_off * DP;
        int32_t* Ls = v.Ls[0] + cd.reg_off;
        const int r0 = (warp * len) / SCAT_W, r1 = ((warp + 1) * len) / SCAT_W;
        int kv[SCAT_KS];
#pragma unroll
        for (int u = 0; u < SCAT_KS; ++u) {
            const int e = u * SCAT_W * 32 + tid;
            kv[u] = (e < len) ? keys[e] : -1;
        }
        // Every global load of the chunk is issued up front -- its key bases
        // and histogram row, and the coordinates of this warp's first SCAT_SP
        // placement steps -- so the chunk waits for one memory round trip
        // instead of one per loop step.
        int bsv[SCAT_HMAX / (SCAT_W * 32)], rwv[SCAT_HMAX / (SCAT_W * 32)];
#pragma unroll
        for (int u = 0; u < SCAT_HMAX / (SCAT_W * 32); ++u) {
            const int k = u * SCAT_W * 32 + tid;
            bsv[u] = (k < ns) ? bs[k] : 0;
            rwv[u] = (k < ns) ? row[k] : 0;
        }
        float pc[SCAT_SP][DIM];
#pragma unroll
        for (int q = 0; q < SCAT_SP; ++q) {
            const int i = r0 + q * 32 + lane;
#pragma unroll
            for (int d = 0; d < DIM; ++d) pc[q][d] = (i < r1) ? Pc[(int64_t)i * DIM + d] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < SCAT_KS; ++u) {
            const int e = u * SCAT_W * 32 + tid;
            if (e < len) s_keys[e] = kv[u];
        }
        for (int e = SCAT_KS * SCAT_W * 32 + tid; e < len; e += SCAT_W * 32) s_keys[e] = keys[e];
        for (int e = tid; e < SCAT_W * ns; e += SCAT_W * 32) hw[e] = 0;
        __syncthreads();
        // per-warp key counts (order-free: shared-memory adds into the
        // warp's own row)
        for (int i = r0 + lane; i < r1; i += 32) {
            const int key = s_keys[i];
            if (key >= 0) atomicAdd(&hw[warp * ns + key], 1);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < SCAT_HMAX / (SCAT_W * 32); ++u) {
            const int k = u * SCAT_W * 32 + tid;
            if (k < ns) {
                int run = bsv[u] + rwv[u];
#pragma unroll
                for (int w = 0; w < SCAT_W; ++w) {
                    const int x = hw[w * ns + k];
                    hw[w * ns + k] = run;
                    run += x;
                }
            }
        }
        __syncthreads();
        int* cur = hw + warp * ns;
        for (int g0 = r0; g0 < r1; g0 += 32 * SCAT_SP) {
            if (g0 > r0) {  // ranges longer than SCAT_SP steps: the next steps' coordinates
#pragma unroll
                for (int q = 0; q < SCAT_SP; ++q) {
                    const int i = g0 + q * 32 + lane;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) pc[q][d] = (i < r1) ? Pc[(int64_t)i * DIM + d] : 0.0f;
                }
            }
#pragma unroll
            for (int q = 0; q < SCAT_SP; ++q) {
                const int i0 = g0 + q * 32;
                if (i0 >= r1) break;
                const int i = i0 + lane;
                const WarpRun r = warp_runs((i < r1) ? s_keys[i] : -1, lane);
                int b = 0;
                if (r.key >= 0 && lane == r.head) {
                    b = cur[r.key];
                    cur[r.key] = b + r.count;
                }
                b = __shfl_sync(FULL, b, r.head);
                float qv[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d) qv[d] = __shfl_sync(FULL, pc[q][d], r.src);
                if (r.key >= 0) {
                    store_row<DIM>(Pg, b + r.rank, qv);
                    if (v.lists) Ls[b + r.rank] = start + i0 + r.src;
                }
            }
        }
        }
        __syncthreads();  // s_item and s_n are read no more
    }
}

// dynamic shared memory of k_scatter_cta
inline int scatter_cta_smem_bytes(const EngineView& v)
{
    const int block_path = v.chunk_max + SCAT_W * SCAT_HMAX;
    const int warp_path = v.chunk_max + v.scat_smem;
    return 4 * (block_path > warp_path ? block_path : warp_path);
}

template <int DIM>
__device__ void scatter_chunk(const EngineView& v, int c, int lc, int* s_keys, int lane)
{
    constexpr int DP = PadDim<DIM>::v;
    const CloudDesc cd = v.cl[c];
    const int ns = v.ns[c];
    int32_t* row = v.hpre + cd.hist_off + (int64_t)lc * cd.ns_cap;
    const int32_t* bs = v.base + cd.key_off;
    const bool in_smem = ns <= v.scat_smem;
    // the row's prefixes are not needed after this chunk
    int32_t* ctr = in_smem ? (s_keys + v.chunk_max) : row;
    const int start = (int)(((int64_t)lc * cd.n_all) / cd.n_chunks);
    const int end = (int)(((int64_t)(lc + 1) * cd.n_all) / cd.n_chunks);
    const int len = end - start;
    const int32_t* keys = v.keys + cd.p_off + start;
    // stage the chunk's keys and the per-key start slots: eight independent
    // loads per lane in flight before the first shared-memory store, so the
    // staging costs a few load latencies instead of one per 32 elements
    for (int e0 = 0; e0 < len; e0 += 32 * 8) {
        int t[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + u * 32 + lane;
            t[u] = (e < len) ? keys[e] : -1;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = e0 + u * 32 + lane;
            if (e < len) s_keys[e] = t[u];
        }
    }
    for (int k0 = 0; k0 < ns; k0 += 32 * 4) {
        int a[4], r[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * 32 + lane;
            a[u] = (k < ns) ? bs[k] : 0;
            r[u] = (k < ns) ? row[k] : 0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + u * 32 + lane;
            if (k < ns) ctr[k] = a[u] + r[u];
        }
    }
    __syncwarp();
    const float* Pc = v.P + (cd.p_off + start) * DIM;
    float* Pg = v.Lr[0] + cd.reg_off * DP;
    int32_t* Ls = v.Ls[0] + cd.reg_off;
    for (int off = 0; off < len; off += 32) {
        const int i = off + lane;
        float pc[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) pc[d] = (i < len) ? Pc[(int64_t)i * DIM + d] : 0.0f;
        const WarpRun r = warp_runs((i < len) ? s_keys[i] : -1, lane);
        int b = 0;
        if (r.key >= 0 && lane == r.head) {
            b = ctr[r.key];
            ctr[r.key] = b + r.count;
        }
        b = __shfl_sync(FULL, b, r.head);
        float q[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) q[d] = __shfl_sync(FULL, pc[d], r.src);
        if (r.key >= 0) {
            store_row<DIM>(Pg, b + r.rank, q);
            if (v.lists) Ls[b + r.rank] = start + off + r.src;
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// ordered sums: lane d (< DIM) of a warp folds coordinate d of a key's members in
// index order with rounded adds, exactly as rd/cpu/brute_force/evolve.hpp:71-74
// accumulates, then applies the movement test of evolve.hpp:143-177.
// ---------------------------------------------------------------------------
constexpr int SUM_BP = 128;  // members staged per step of the ordered fold
// points (keys) per lane loaded together by the fused tile kernel's
// assignment (placement) loop
constexpr int TILE_PPL = 8;
// members from which the fused tile kernel folds a key with the whole CTA
// (warp-segmented exact evaluation, rd_segfold.cuh) instead of one warp's add
// chain
constexpr int FOLD_CTA_MIN = 4096;
// the same for the light tiles of the cluster kernel: the heavy tiles, whose
// keys need the CTA-wide folds, went to clusters; the others fold faster with
// every warp on its own keys
constexpr int FOLD_CTA_MIN_LIGHT = 1 << 30;

// Sequential FP32 fold, in list order, of the points P[perm[0..n)] (one warp;
// the sum of coordinate d is returned in lane d < DIM).
template <int DIM, int BP = SUM_BP>
__device__ float fold_members(const int32_t* __restrict__ perm, const int n,
                              const float* __restrict__ P, float* buf, int* sidx, const int lane)
{
    constexpr int R = BP * DIM / 32;    // floats per lane per step
    float nxt[R];
    // Two-stage pipeline: member indices of block b+2 and coordinates of
    // block b+1 are in flight while block b is folded.
    int pnx[BP / 32];
    auto load_perm = [&](int off) {
        const int m = min(BP, n - off);
#pragma unroll
        for (int u = 0; u < BP / 32; ++u) {
            const int j = u * 32 + lane;
            pnx[u] = (off < n && j < m) ? perm[off + j] : 0;
        }
    };
    auto load_coords = [&](int off) {  // indices of block `off` are in sidx
        const int m = min(BP, n - off);
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int e = u * 32 + lane;
            const int j = e / DIM, d = e - (e / DIM) * DIM;
            nxt[u] = (j < m) ? P[(int64_t)sidx[j] * DIM + d] : 0.0f;
        }
    };
    auto stage_perm = [&]() {
#pragma unroll
        for (int u = 0; u < BP / 32; ++u) sidx[u * 32 + lane] = pnx[u];
        __syncwarp();
    };
    load_perm(0);
    stage_perm();
    load_coords(0);
    load_perm(BP);
    float sum = 0.0f;
    for (int off = 0; off < n; off += BP) {
        const int m = min(BP, n - off);
        __syncwarp();  // every lane is done reading sidx of the previous stage
#pragma unroll
        for (int u = 0; u < R; ++u) buf[u * 32 + lane] = nxt[u];
        if (off + BP < n) {
            stage_perm();               // indices of block off+BP
            load_coords(off + BP);      // in flight during the fold
            load_perm(off + 2 * BP);    // in flight during the fold
        }
        __syncwarp();
        if (lane < DIM) {
            if (m == BP) {
#pragma unroll 32
                for (int j = 0; j < BP; ++j) sum = __fadd_rn(sum, buf[j * DIM + lane]);
            } else {
                for (int j = 0; j < m; ++j) sum = __fadd_rn(sum, buf[j * DIM + lane]);
            }
        }
        __syncwarp();
    }
    return sum;
}

// The shift of chosen point k of cloud c from its members' sum (lane d < DIM
// holds coordinate d): evolve.hpp:143-177, or the plain mean for the
// adjoint's forward step.  Called by one whole warp.
template <int DIM>
__device__ void apply_shift(const EngineView& v, int c, const CloudDesc& cd, int k, int n, float sum,
                            int lane)
{
    int moved = 0, changed = 0;
    float was = 0.0f, now = 0.0f;
    if (lane < DIM) {
        float* s = v.S + (cd.s_off + k) * DIM + lane;
        was = now = *s;
        if (v.flags & ENG_ALWAYS_MOVE) {
            now = __fdiv_rn(sum, (float)n);  // mean, no movement test
            changed = !(now == was);
            *s = now;
        } else {
            changed = moved = shift_coord(sum, n, now);
            if (moved) *s = now;
        }
    }
    if (__any_sync(FULL, moved) && lane == 0) v.cont[c] = 1;
    if (!v.lists || !__any_sync(FULL, changed)) return;
    // the move, for the blocks of points near it (k_assign_cull): old and new
    // place, and its length rounded up
    const float dd = fabsf(__fsub_rn(now, was));
    float len2 = 0.0f;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        const float x = __shfl_sync(FULL, dd, d);
        len2 = __fadd_ru(len2, __fmul_ru(x, x));
    }
    // (the difference was rounded to nearest: one part in 2^20 covers it; a
    // length that underflows counts as the smallest one that matters)
    const float len = fmaxf(__fmul_ru(__fsqrt_ru(len2), 1.000001f), 1.0e-30f);
    int at = 0;
    if (lane == 0) {
        at = atomicAdd(&v.mvn[c], 1);
        atomicMax(&v.dmax[c], (len2 == len2) ? __float_as_int(len) : 0x7fc00000);
    }
    at = __shfl_sync(FULL, at, 0);
    float* mv = v.mv + cd.key_off + at;
    if (lane < DIM) {
        mv[(int64_t)lane * v.n_slots] = was;
        mv[(int64_t)(DIM + lane) * v.n_slots] = now;
    }
    if (lane == 0) mv[(int64_t)(2 * DIM) * v.n_slots] = (len2 == len2) ? len : __int_as_float(0x7fc00000);
}

// Sequential FP32 fold, in order, of n contiguous rows of a grouped copy
// (PadDim<DIM> floats each); one warp, the sum of coordinate d returned in
// lane d < DIM.  A block of BP rows is loaded with coalesced vector loads into
// the warp's buffer (BP x PadDim floats) while the previous block is folded.
template <int DIM, int BP>
__device__ float fold_rows(const float* __restrict__ rows, const int n, float* buf, const int lane)
{
    constexpr int DP = PadDim<DIM>::v;
    constexpr int VW = (DP == 4) ? 4 : (DP == 2 ? 2 : 1);  // floats per vector load
    constexpr int R = BP * DP / (32 * VW);                 // vector loads per lane per block
    static_assert(BP * DP % (32 * VW) == 0, "block of whole vector loads");
    float nxt[R][VW];
    auto load = [&](int off) {
        const int lim = min(BP, n - off) * DP;  // valid floats of the block
        const float* src = rows + (int64_t)off * DP;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int e = (u * 32 + lane) * VW;
            if constexpr (VW == 4) {
                const float4 t = (e < lim) ? reinterpret_cast<const float4*>(src)[u * 32 + lane]
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
                nxt[u][0] = t.x; nxt[u][VW > 1 ? 1 : 0] = t.y;
                nxt[u][VW > 2 ? 2 : 0] = t.z; nxt[u][VW > 3 ? 3 : 0] = t.w;
            } else if constexpr (VW == 2) {
                const float2 t = (e < lim) ? reinterpret_cast<const float2*>(src)[u * 32 + lane]
                                           : make_float2(0.f, 0.f);
                nxt[u][0] = t.x; nxt[u][VW > 1 ? 1 : 0] = t.y;
            } else {
                nxt[u][0] = (e < lim) ? src[e] : 0.0f;
            }
        }
    };
    load(0);
    float sum = 0.0f;
    for (int off = 0; off < n; off += BP) {
        const int m = min(BP, n - off);
        __syncwarp();  // every lane is done reading the previous block
#pragma unroll
        for (int u = 0; u < R; ++u)
#pragma unroll
            for (int w = 0; w < VW; ++w) buf[(u * 32 + lane) * VW + w] = nxt[u][w];
        if (off + BP < n) load(off + BP);  // in flight during the fold
        __syncwarp();
        if (lane < DIM) {
            if (m == BP) {
#pragma unroll 32
                for (int j = 0; j < BP; ++j) sum = __fadd_rn(sum, buf[j * DP + lane]);
            } else {
                for (int j = 0; j < m; ++j) sum = __fadd_rn(sum, buf[j * DP + lane]);
            }
        }
    }
    __syncwarp();
    return sum;
}

// ---------------------------------------------------------------------------
// Member lists, ordered sum and shift: one CTA per listed key (dlist).
//
// Every key keeps its members' coordinates and positions in index order, in its
// region of the grouped lists, from pass to pass.  In a cloud that regroups
// (rebuilds) the scatter has just written the lists anew; otherwise the key's
// edits of this pass are merged in.  The edits are sorted by position in shared
// memory (each counts the smaller ones).  All warps but one take the old list in
// chunks of one row per thread, the next two chunks' loads in flight.  The position of
// each chunk's first row says which edits fall into the chunk; a row finds by
// binary search how many of them come before it, which gives its new place (or
// that it leaves), and takes along the points that join right before it; a
// chunk without edits moves as a whole.  New rows go to a ring in shared memory
// and to the other buffer; the last warp folds the ring behind them with the
// reference's chain of rounded adds (lane d: coordinate d;
// rd/cpu/brute_force/evolve.hpp:71-74) and applies the movement test
// (evolve.hpp:143-177).  A list that outgrows its region is folded all the
// same, and the cloud regroups in the next pass.
//
// Bound by the add chain of the longest listed key, about 2.3 ns per member;
// the merge of a chunk runs beside it and takes less.  Keys without edits cost
// nothing.  1M-point helix, after the assignment: scan, scatter and one-warp
// folds of every key took 70 us per pass; this kernel takes 20-40 us (790 keys of
// 1,266 members, most with edits), 12-20 us (few keys with edits), 45-50 us (116
// keys of 8,300 members, 20 us of it the add chain of the longest).
// ---------------------------------------------------------------------------
// CTA size: 256 threads for one cloud; 128 for several, whose pass has thousands
// of short lists, each a chain of loads and barriers: seven CTAs per SM instead
// of four (2,048 clouds: 635 -> 600 ms)
constexpr int MF_BLOCK = 256, MF_BLOCK_MANY = 128;
constexpr int MF_RING = 1024;               // two chunks and every edit fit
constexpr int MF_STAGES = 3;                // chunks of the old list in flight
constexpr int MF_CUTS = 256;                // chunks whose edits are looked up at once
constexpr int MF_CHAIN = 32;                // terms the chain takes at a time
static_assert(2 * (MF_BLOCK - 32) + EDIT_MAX + MF_CHAIN <= MF_RING && MF_RING % MF_CHAIN == 0,
              "ring of new rows");

template <int DIM, int BLOCK>
struct MergeSmem {
    static constexpr int PROD = BLOCK - 32;   // threads that merge, rows per chunk
    union {
        float ring[DIM][MF_RING + 4];   // per coordinate: the chain loads four terms at once
        SegFoldSmem<BLOCK / 32, DIM> seg;
    };
    alignas(16) float old[MF_STAGES][PROD * PadDim<DIM>::v];   // chunks of the old list
    int pos[MF_STAGES][PROD + 1];                     // their positions, after the row before's
    alignas(16) float joins[EDIT_MAX * PadDim<DIM>::v];   // coordinates of the joining edits
    int raw[EDIT_MAX];        // edits as listed
    int ed[EDIT_MAX];         // by position
    int ins[EDIT_MAX + 1];    // joining ones among the first i
    int cut[MF_CUTS + 1];     // edits before the first row of each chunk
};

// cloud c after a pass: the next one evaluates and regroups what this one left
__device__ __forceinline__ void next_pass(const EngineView& v, const int c)
{
    v.full[c] = v.lists ? 0 : 1;
    v.reb[c] = v.rebnext[c];
    v.rebnext[c] = 0;
}

// the per-cloud control step after a pass (k_control), over clouds first,
// first + stride, ... of the active list
__device__ int control_clouds(const EngineView& v, const int first, const int stride);
__device__ void loop_condition(const EngineView& v, cudaGraphConditionalHandle h, int use_handle,
                               int count_iter);

// the end of an iteration that leaves `a` clouds unfinished (one thread):
// counters for the next one, and the loop condition
__device__ __forceinline__ void next_iteration(const EngineView& v, int a, cudaGraphConditionalHandle h,
                                               const int use_handle, const int count_iter)
{
    v.ctr[CTR_WORK] = 0;
    v.ctr[CTR_NREADY] = 0;
    v.ctr[CTR_NDIRTY] = 0;
    v.ctr[CTR_TILE_HEAVY] = 0;
    const int it = v.ctr[CTR_ITERS] + (count_iter ? 1 : 0);
    v.ctr[CTR_ITERS] = it;
    if (it >= v.max_iters && a > 0) {
        v.ctr[CTR_ERR] |= ERRB_EVOLVE_CAP;
        v.ctr[CTR_NACT] = 0;   // nor do the graph round's passes after this one
        a = 0;
    }
    v.ctr[CTR_ACTIVE] = a;
    if (use_handle) cudaGraphSetConditional(h, a > 0 ? 1u : 0u);
}

template <int DIM>
__device__ __forceinline__ void load_row(const float* rows, const int64_t r, float (&q)[DIM])
{
    constexpr int DP = PadDim<DIM>::v;
    if constexpr (DP == 4) {
        const float4 t = reinterpret_cast<const float4*>(rows)[r];
        q[0] = t.x;
        if constexpr (DIM > 1) q[1] = t.y;
        if constexpr (DIM > 2) q[2] = t.z;
        if constexpr (DIM > 3) q[3] = t.w;
    } else if constexpr (DP == 2) {
        const float2 t = reinterpret_cast<const float2*>(rows)[r];
        q[0] = t.x;
        q[1] = t.y;
    } else {
        q[0] = rows[r];
    }
}

// edits at positions below x, which are at least lo and at most hi
__device__ __forceinline__ int edits_below(const int* ed, int lo, int hi, const int x)
{
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if ((ed[mid] & ~EDIT_IN) < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

__device__ __forceinline__ void lds_f32x4(const uint32_t a, float* x)
{
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(x[0]), "=f"(x[1]), "=f"(x[2]), "=f"(x[3]) : "r"(a));
}

// copies BYTES (4, 8 or 16) of global memory to shared memory, asynchronously
template <int BYTES>
__device__ __forceinline__ void copy_async(void* to, const void* from)
{
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(to);
    if constexpr (BYTES == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(from) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(a), "l"(from), "n"(BYTES) : "memory");
}

// sum + term 0 + term 1 + ... (`n` groups of MF_CHAIN terms in the ring from
// address a on, its end at `end`; in order, each add rounded): half a group is
// loaded, four terms at a time, while the half before it is added, so that a
// term costs its add (4 cycles) and not the load's latency.  A function of its
// own: inlined into the merge, its registers were spilled and every add waited
// for its load.
__device__ __noinline__ float chain_add(uint32_t a, const int n, const uint32_t end, float sum)
{
    constexpr int B = MF_CHAIN / 2;
    float x[B], y[B];
#pragma unroll
    for (int u = 0; u < B; u += 4) lds_f32x4(a + u * 4, x + u);
    for (int g = 0; g < n; ++g) {
#pragma unroll
        for (int u = 0; u < B; u += 4) lds_f32x4(a + (B + u) * 4, y + u);
#pragma unroll
        for (int u = 0; u < B; ++u) sum = __fadd_rn(sum, x[u]);
        a += MF_CHAIN * 4;
        if (a >= end) a -= MF_RING * 4;
        // (the group after the last one is read and not used)
#pragma unroll
        for (int u = 0; u < B; u += 4) lds_f32x4(a + u * 4, x + u);
#pragma unroll
        for (int u = 0; u < B; ++u) sum = __fadd_rn(sum, y[u]);
    }
    return sum;
}

// the last m < MF_CHAIN terms
__device__ __noinline__ float chain_tail(const uint32_t a, const int m, float sum)
{
    float x[MF_CHAIN];
#pragma unroll
    for (int u = 0; u < MF_CHAIN; u += 4) lds_f32x4(a + u * 4, x + u);
#pragma unroll
    for (int u = 0; u < MF_CHAIN; ++u)
        if (u < m) sum = __fadd_rn(sum, x[u]);
    return sum;
}

// apart, so that its registers do not weigh on the merge
template <int DIM, int W, bool LONG>
__device__ __noinline__ void fold_long_list(const float* rows, const int n, SegFoldSmem<W, DIM>& sm)
{
    fold_members_seg_src<W, DIM>(RowSrc<DIM>{rows}, n, sm);
}

template <int DIM, int BLOCK, bool LONG>
__device__ void merge_fold_key(const EngineView& v, const int slot, const bool seg_ok,
                               MergeSmem<DIM, BLOCK>& sm)
{
    constexpr int MF_PROD = BLOCK - 32, MF_ROWS = MF_PROD;
    constexpr int DP = PadDim<DIM>::v;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = v.single ? 0 : v.slot_cloud[slot];
    const int4 info = v.kinfo[slot];
    const int edits = v.ecnt[slot];
    const CloudDesc cd = cloud_desc(v, c);
    const int k = (int)(slot - cd.key_off);
    const bool fresh = rebuilds(v, c);
    const int64_t at = cd.reg_off + info.x;
    const int cap = info.y;
    const int n_old = info.z;
    const int par = info.w;                    // (0 when fresh)
    const int ne = fresh ? 0 : edits;          // at most EDIT_MAX, or the cloud rebuilds
    const float* src = v.Lr[par] + at * DP;
    __syncthreads();  // the previous key's scratch, and its state, are read no more
    for (int i = tid; i < ne; i += BLOCK) sm.raw[i] = v.edit[at + i];
    __syncthreads();
    for (int i = tid; i < ne; i += BLOCK) {
        const int e = sm.raw[i], x = e & ~EDIT_IN;
        int r = 0;
        float p[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) p[d] = v.P[(cd.p_off + x) * DIM + d];
        for (int j = 0; j < ne; ++j) r += (sm.raw[j] & ~EDIT_IN) < x;   // positions differ
        sm.ed[r] = e;
        store_row<DIM>(sm.joins, r, p);
    }
    __syncthreads();
    if (warp == 0) {
        int carry = 0;
        for (int i0 = 0; i0 < ne; i0 += 32) {
            const bool in = i0 + lane < ne && sm.ed[i0 + lane] < 0;
            const unsigned bal = __ballot_sync(FULL, in);
            if (i0 + lane < ne) sm.ins[i0 + lane] = carry + __popc(bal & lanemask_lt());
            carry += __popc(bal);
        }
        if (lane == 0) sm.ins[ne] = carry;
    }
    __syncthreads();
    const int n_new = n_old + 2 * sm.ins[ne] - ne;
    const bool seg = seg_ok && ne == 0 && n_old >= (LONG ? SUM_BIG_MIN : SUM_BIG_MIN_SLOW);
    const int steps = seg ? 0 : (max(n_old, 1) + MF_ROWS - 1) / MF_ROWS;
    float sum = 0.0f;
    const int32_t* pos = v.lists ? v.Ls[par] + at : nullptr;
    // edits before chunk s's first row (those before the list's first row go to chunk 0)
    auto find_cuts = [&](const int s0) {
        for (int i = tid; i <= MF_CUTS; i += BLOCK) {
            const int s = s0 + i;
            sm.cut[i] = (s == 0 || ne == 0) ? 0
                        : (s < steps) ? edits_below(sm.ed, 0, ne, pos[s * MF_ROWS]) : ne;
        }
    };
    // new rows before chunk s (of the current window of chunks)
    auto rows_before = [&](const int s, const int s0) {
        if (s >= steps) return n_new;
        const int e = sm.cut[s - s0];
        return s * MF_ROWS - e + 2 * sm.ins[e];
    };
    int r = 0;   // rows folded (warp 0)
    for (int s0 = 0; s0 == 0 || s0 < steps; s0 += MF_CUTS) {
        find_cuts(s0);
        __syncthreads();
        const int s1 = min(steps, s0 + MF_CUTS);
        if (warp == 0) {
            // the chain follows the merge one chunk behind
            for (int s = s0; s <= s1; ++s) {
                if (s > s0) {
                    // whole groups; the rest waits for the next chunk
                    const int end = rows_before(s, s0), n = (end - r) / MF_CHAIN;
                    if (lane < DIM) {
                        const uint32_t ring = (uint32_t)__cvta_generic_to_shared(sm.ring[lane]);
                        if (n > 0) sum = chain_add(ring + (r & (MF_RING - 1)) * 4, n, ring + MF_RING * 4, sum);
                        if (s == steps)
                            sum = chain_tail(ring + ((r + n * MF_CHAIN) & (MF_RING - 1)) * 4,
                                             end - r - n * MF_CHAIN, sum);
                    }
                    r += n * MF_CHAIN;
                }
                __syncthreads();
            }
        } else {
            float* dst = v.Lr[par ^ 1] + at * DP;
            int32_t* dpos = (v.lists ? v.Ls[par ^ 1] + at : nullptr);
            const int pt = tid - 32;
            auto load = [&](const int s) {
                const int j = s * MF_ROWS + pt, b = s % MF_STAGES;
                if (j < n_old) {
                    copy_async<DP * 4>(sm.old[b] + pt * DP, src + (int64_t)j * DP);
                    if (ne > 0) {
                        copy_async<4>(&sm.pos[b][pt + 1], pos + j);
                        if (pt == 0 && j > 0) copy_async<4>(&sm.pos[b][0], pos + j - 1);
                    }
                }
                if (pt == 0 && s == 0) sm.pos[b][0] = -1;
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            auto put = [&](const int r, const float (&p)[DIM], const int i) {
#pragma unroll
                for (int d = 0; d < DIM; ++d) sm.ring[d][r & (MF_RING - 1)] = p[d];
                if (r < cap) {
                    store_row<DIM>(dst, r, p);
                    dpos[r] = i;
                }
            };
            // joining edit e, right before old row j (or at the end)
            auto join = [&](const int e, const int j) {
                float p[DIM];
                load_row<DIM>(sm.joins, e, p);
                put(j - e + 2 * sm.ins[e], p, sm.ed[e] & ~EDIT_IN);
            };
            load(s0);
            load(s0 + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            named_bar_sync(1, MF_PROD);   // chunk s0 is here
            for (int s = s0; s <= s1; ++s) {
                if (s < s1) {
                    load(s + 2);
                    const int e0 = sm.cut[s - s0], e1 = sm.cut[s - s0 + 1];
                    const int last = min(n_old, (s + 1) * MF_ROWS) - 1;
                    const int j = s * MF_ROWS + pt, b3 = s % MF_STAGES;
                    if (j <= last) {
                        float q[DIM];
                        load_row<DIM>(sm.old[b3], pt, q);
                        if (ne == 0) {
#pragma unroll
                            for (int d = 0; d < DIM; ++d) sm.ring[d][j & (MF_RING - 1)] = q[d];
                        } else {
                            const int x = sm.pos[b3][pt + 1];
                            if (e0 == e1) {
                                put(j + 2 * sm.ins[e0] - e0, q, x);
                            } else {
                                const int xp = sm.pos[b3][pt];
                                const int b = edits_below(sm.ed, e0, e1, x);   // before this row
                                for (int e = b - 1; e >= e0 && (sm.ed[e] & ~EDIT_IN) > xp; --e) join(e, j);
                                const bool leaves = b < e1 && (sm.ed[b] & ~EDIT_IN) == x;
                                if (!leaves) put(j - b + 2 * sm.ins[b], q, x);
                                if (j == last)   // and those before the next chunk's first row
                                    for (int e = b + (leaves ? 1 : 0); e < e1; ++e) join(e, j + 1);
                            }
                        }
                    }
                    if (n_old == 0)
                        for (int e = pt; e < ne; e += MF_PROD) join(e, 0);
                    asm volatile("cp.async.wait_group 1;" ::: "memory");   // chunk s + 1 is here
                }
                __syncthreads();
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        if (s1 == steps) break;
        __syncthreads();   // cut is looked up anew
    }
    if (seg) {
        __syncthreads();  // the ring is read no more
        fold_long_list<DIM, BLOCK / 32, LONG>(src, n_old, sm.seg);
        if (warp == 0 && lane < DIM) sum = sm.seg.out[lane];
    }
    if (warp == 0) {
        if (lane == 0) {
            v.ecnt[slot] = 0;
            v.cnt[slot] = n_new;
            v.kinfo[slot] = make_int4(info.x, cap, n_new, (ne > 0) ? par ^ 1 : par);
            if (ne > 0 && n_new > cap) v.rebnext[c] = 1;
        }
        if (n_new > 0) apply_shift<DIM>(v, c, cd, k, n_new, sum, lane);
    }
}

// control: what the last CTA to finish does.  MF_CONTROL: the control step of
// k_control (the moved flags of every fold are then complete) and, when that
// leaves no group to decimate, the loop condition, so that k_decimate has
// nothing to wait for.  MF_STEP (passes whose number the caller sets, over the
// same clouds): make ready for the next pass.
enum : int { MF_CONTROL = 1, MF_STEP = 2 };

template <int DIM, int BLOCK, bool LONG>
__global__ void __launch_bounds__(BLOCK, LONG ? 1 : BLOCK == MF_BLOCK ? 4 : 7)
    k_merge_fold(EngineView v, cudaGraphConditionalHandle h, int control, int use_handle)
{
    pdl_enter();
    __shared__ __align__(16) MergeSmem<DIM, BLOCK> sm;
    __shared__ int s_last;
    const int nd = v.ctr[CTR_NDIRTY];
    for (int t = blockIdx.x; t < nd; t += gridDim.x)
        merge_fold_key<DIM, BLOCK, LONG>(v, v.dlist[t], nd <= (int)gridDim.x, sm);
    // every thread's writes (chosen points, moved flags) before the count
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&v.ctr[CTR_SUM_DONE], 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (control == MF_STEP) {
        const int nact = v.ctr[CTR_NACT];
        for (int a = threadIdx.x; a < nact; a += blockDim.x) next_pass(v, v.act_cloud[a]);
        if (threadIdx.x == 0) {
            v.ctr[CTR_SUM_DONE] = 0;
            v.ctr[CTR_NDIRTY] = 0;
            v.ctr[CTR_WORK] = 0;
        }
        return;
    }
    if (v.ctr[CTR_NACT] == 0) {   // a pass after the last one
        if (threadIdx.x == 0) {
            v.ctr[CTR_SUM_DONE] = 0;
            v.ctr[CTR_COND_DONE] = 1;
        }
        return;
    }
    const int conv = __syncthreads_or(control_clouds(v, threadIdx.x, blockDim.x));
    if (!conv) {
        // every cloud goes on: the work lists stay as they are
        if (threadIdx.x == 0) {
            v.ctr[CTR_SUM_DONE] = 0;
            v.ctr[CTR_COND_DONE] = 1;
            next_iteration(v, v.ctr[CTR_ACTIVE], h, use_handle, 1);
        }
        return;
    }
    __threadfence();
    __syncthreads();
    const bool idle = *reinterpret_cast<volatile int32_t*>(&v.ctr[CTR_NREADY]) == 0;
    if (threadIdx.x == 0) {
        v.ctr[CTR_SUM_DONE] = 0;
        v.ctr[CTR_COND_DONE] = idle ? 1 : 0;
    }
    if (idle) loop_condition(v, h, use_handle, 1);
}

// ---------------------------------------------------------------------------
// Fused per-tile evolve (tiled runs): one CTA evolves one tile to convergence
// without leaving the kernel, so tiles proceed independently instead of in
// lockstep passes.  Every pass is the same exact computation as the pass
// pipeline (assign with the two-level argmin, stable grouping, index-order
// fold, movement test), done inside the CTA:
//   * warp w owns the contiguous point range [w n/W, (w+1) n/W); its per-key
//     counts go to hist[w][key];
//   * a key's members are laid out warp range by warp range, each range in
//     index order (match_any ranks inside 32-point steps), i.e. in index order;
//   * warp w folds keys w, w+W, ... (fold_members) and applies the shift.
// Shared memory: chosen points (TILE_NS_MAX, padded to float4 for DIM 3),
// W x (ns+1) counters, key bases.
// ---------------------------------------------------------------------------
// Assignment of the points [r0, r1w) of a tile by one warp (steps of 32 x
// TILE_PPL points, loads first): keys[i] = nearest chosen point within r1
// (first index of the minimum), and the warp's members per key in whist.
// With at most TILE_KB chosen points the counts are kept per key in
// warp-uniform registers (one ballot per key and step) and stored at the end;
// otherwise one shared-memory add per distinct key of a step.
constexpr int TILE_KB = 8;

template <int DIM>
__device__ __forceinline__ void tile_assign_range(const float* __restrict__ P, const int r0,
                                                  const int r1w, const float* sS, const int ns,
                                                  const int nsp, const float rsq,
                                                  int32_t* __restrict__ keys, int* whist,
                                                  const int lane)
{
    constexpr int KB = TILE_KB;
    int kc[KB];
#pragma unroll
    for (int k = 0; k < KB; ++k) kc[k] = 0;
    for (int i0 = r0; i0 < r1w; i0 += 32 * TILE_PPL) {
        float p[TILE_PPL][DIM];
#pragma unroll
        for (int h = 0; h < TILE_PPL; ++h) {
            const int i = i0 + h * 32 + lane;
#pragma unroll
            for (int d = 0; d < DIM; ++d) p[h][d] = (i < r1w) ? P[(int64_t)i * DIM + d] : 0.0f;
        }
        if (ns <= KB) {
            // first index of the minimum, directly: each chosen point is read
            // once for the step's TILE_PPL points
            float best[TILE_PPL];
            int bk[TILE_PPL];
#pragma unroll
            for (int h = 0; h < TILE_PPL; ++h) {
                best[h] = FLT_MAX;
                bk[h] = -1;
            }
            for (int k = 0; k < ns; ++k) {
                float s[DIM];
                load_chosen<DIM>(sS, k, s);
#pragma unroll
                for (int h = 0; h < TILE_PPL; ++h) {
                    const float dd = sqdist_exact<DIM>(s, p[h]);
                    if (dd < best[h]) { best[h] = dd; bk[h] = k; }
                }
            }
#pragma unroll
            for (int h = 0; h < TILE_PPL; ++h) {
                const int i = i0 + h * 32 + lane;
                const int key = (i < r1w && best[h] <= rsq) ? bk[h] : -1;
                if (i < r1w) keys[i] = key;
#pragma unroll
                for (int k = 0; k < KB; ++k)
                    if (k < ns) kc[k] += __popc(__ballot_sync(FULL, key == k));
            }
            continue;
        }
#pragma unroll
        for (int h = 0; h < TILE_PPL; ++h) {
            const int i = i0 + h * 32 + lane;
            int key = -1;
            if (i < r1w) {
                float best = FLT_MAX;
                int blk = -1;
                for (int kb = 0; kb < nsp; kb += KB) {
                    const float old = best;
#pragma unroll
                    for (int u = 0; u < KB; ++u) {
                        float s[DIM];
                        load_chosen<DIM>(sS, kb + u, s);
                        best = fminf(best, sqdist_exact<DIM>(s, p[h]));
                    }
                    blk = (best < old) ? kb : blk;
                }
                if (best <= rsq && blk >= 0) {
                    for (int u = 0; u < KB && blk + u < ns; ++u) {
                        float s[DIM];
                        load_chosen<DIM>(sS, blk + u, s);
                        if (sqdist_exact<DIM>(s, p[h]) == best) { key = blk + u; break; }
                    }
                }
                keys[i] = key;
            }
            // a tile's warp step holds few distinct keys: the match
            // instruction is cheap there (warp_runs suits many keys)
            const unsigned mm = __match_any_sync(FULL, key);
            if (key >= 0 && lane == __ffs(mm) - 1) atomicAdd(&whist[key], __popc(mm));
        }
    }
    if (ns <= KB && lane == 0)
#pragma unroll
        for (int k = 0; k < KB; ++k)
            if (k < ns) whist[k] += kc[k];
}

// Stable placement of the warp's points [r0, r1w): the coordinates of the
// members of key k go, in index order, to rows cur[k], cur[k] + 1, ... of the
// grouped copy Pg (cur advanced).
template <int DIM>
__device__ __forceinline__ void tile_place_range(const float* __restrict__ P,
                                                 const int32_t* __restrict__ keys, const int r0,
                                                 const int r1w, int* cur, const int ns,
                                                 float* __restrict__ Pg, const int lane)
{
    constexpr int KB = TILE_KB;
    int base[KB];
    if (ns <= KB) {
#pragma unroll
        for (int k = 0; k < KB; ++k) base[k] = (k < ns) ? cur[k] : 0;
    }
    for (int i0 = r0; i0 < r1w; i0 += 32 * TILE_PPL) {
        int kq[TILE_PPL];
        float pq[TILE_PPL][DIM];
#pragma unroll
        for (int h = 0; h < TILE_PPL; ++h) {
            const int i = i0 + h * 32 + lane;
            kq[h] = (i < r1w) ? keys[i] : -1;
#pragma unroll
            for (int d = 0; d < DIM; ++d) pq[h][d] = (i < r1w) ? P[(int64_t)i * DIM + d] : 0.0f;
        }
#pragma unroll
        for (int h = 0; h < TILE_PPL; ++h) {
            const int key = kq[h];
            if (ns <= KB) {
#pragma unroll
                for (int k = 0; k < KB; ++k) {
                    if (k < ns) {
                        const unsigned m = __ballot_sync(FULL, key == k);
                        if (key == k) store_row<DIM>(Pg, base[k] + __popc(m & lanemask_lt()), pq[h]);
                        base[k] += __popc(m);
                    }
                }
            } else {
                const unsigned m = __match_any_sync(FULL, key);
                const int leader = __ffs(m) - 1;
                int b = 0;
                if (key >= 0 && lane == leader) {
                    b = cur[key];
                    cur[key] = b + __popc(m);
                }
                b = __shfl_sync(FULL, b, leader);
                if (key >= 0) store_row<DIM>(Pg, b + __popc(m & lanemask_lt()), pq[h]);
            }
        }
    }
}

template <int DIM, int BLOCK>
struct TileCtaSmem {
    float buf[BLOCK / 32][SUM_BP * PadDim<DIM>::v];   // fold_rows blocks
    int moved;
    SegFoldSmem<BLOCK / 32, DIM> seg;
};

// One CTA evolves tile c to convergence (see above); dyn is the dynamic
// shared memory laid out as tile_evolve_smem_bytes describes.  hand_over()
// (thread 0, after every pass): leave the tile as this pass left it to somebody
// else; then true is returned.
template <int DIM, int BLOCK, class HandOver>
__device__ bool tile_evolve_one(const EngineView& v, const int c, const int fold_cta_min,
                                unsigned char* dyn, TileCtaSmem<DIM, BLOCK>& ts,
                                HandOver&& hand_over)
{
    constexpr int W = BLOCK / 32;
    constexpr int DP = PadDim<DIM>::v;
    constexpr int KB = 8;
    constexpr float FAR = 1e30f;
    float* sS = reinterpret_cast<float*>(dyn);                              // TILE_NS_MAX*DP
    int* hist = reinterpret_cast<int*>(sS + TILE_NS_MAX * DP);             // W*(TILE_NS_MAX+1)
    int* kbase = hist + W * (TILE_NS_MAX + 1);                              // TILE_NS_MAX+1
    auto& s_buf = ts.buf;
    int& s_moved = ts.moved;
    auto& s_seg = ts.seg;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    {
        const CloudDesc cd = v.cl[c];
        const int n = cd.n_all;
        const int ns = v.ns[c];
        const float* P = v.P + cd.p_off * DIM;
        float* gS = v.S + cd.s_off * DIM;
        int32_t* keys = v.keys + cd.p_off;
        float* Pg = v.Pg + cd.p_off * DP;
        const float rsq = sqr_rn(cd.r1);
        const int nsp = (ns + KB - 1) / KB * KB;
        __syncthreads();
        for (int e = tid; e < nsp; e += BLOCK)
#pragma unroll
            for (int d = 0; d < DIM; ++d) sS[e * DP + d] = (e < ns) ? gS[(int64_t)e * DIM + d] : FAR;
        const int r0 = (int)(((int64_t)warp * n) / W), r1w = (int)(((int64_t)(warp + 1) * n) / W);
        int pass = 0;
        bool handed = false;
        for (;;) {
            // 1. assignment of the warp's range + per-warp key counts
            //    (counts added once per distinct key of a warp step)
            for (int k = lane; k <= ns; k += 32) hist[warp * (TILE_NS_MAX + 1) + k] = 0;
            __syncthreads();
            int* whist = hist + warp * (TILE_NS_MAX + 1);
            tile_assign_range<DIM>(P, r0, r1w, sS, ns, nsp, rsq, keys, whist, lane);
            __syncthreads();
            // 2. key bases and per-warp starts (thread per key)
            for (int k = tid; k < ns; k += BLOCK) {
                int tot = 0;
                for (int w = 0; w < W; ++w) tot += hist[w * (TILE_NS_MAX + 1) + k];
                kbase[k + 1] = tot;  // counts for the scan below
            }
            if (tid == 0) { kbase[0] = 0; s_moved = 0; }
            __syncthreads();
            if (warp == 0) {  // inclusive scan of counts -> kbase[k] = first slot of key k
                int carry = 0;
                for (int k0 = 0; k0 < ns; k0 += 32) {
                    const int k = k0 + lane;
                    const int x = (k < ns) ? kbase[k + 1] : 0;
                    int incl = x;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(FULL, incl, o);
                        if (lane >= o) incl += y;
                    }
                    if (k < ns) kbase[k + 1] = carry + incl;
                    carry += __shfl_sync(FULL, incl, 31);
                }
            }
            __syncthreads();
            for (int k = tid; k < ns; k += BLOCK) {
                int run = kbase[k];
                for (int w = 0; w < W; ++w) {
                    const int x = hist[w * (TILE_NS_MAX + 1) + k];
                    hist[w * (TILE_NS_MAX + 1) + k] = run;
                    run += x;
                }
            }
            __syncthreads();
            // 3. stable placement, warp range by warp range (keys of
            //    TILE_PPL warp steps loaded ahead of the dependent placement
            //    chain)
            tile_place_range<DIM>(P, keys, r0, r1w, hist + warp * (TILE_NS_MAX + 1), ns, Pg, lane);
            __syncthreads();
            // 4a. very large keys, one at a time, folded by the whole CTA
            for (int k = 0; k < ns; ++k) {
                const int cnt = kbase[k + 1] - kbase[k];
                if (cnt < fold_cta_min) continue;
                fold_members_seg_src<W, DIM>(RowSrc<DIM>{Pg + (int64_t)kbase[k] * DP}, cnt, s_seg);
                if (tid < DIM) {
                    float cval = sS[k * DP + tid];
                    if (shift_coord(s_seg.out[tid], cnt, cval)) {
                        sS[k * DP + tid] = cval;
                        s_moved = 1;
                    }
                }
                __syncthreads();
            }
            // 4b. index-order fold and movement test, warp w takes keys w, w+W, ...
            for (int k = warp; k < ns; k += W) {
                const int cnt = kbase[k + 1] - kbase[k];
                if (cnt == 0 || cnt >= fold_cta_min) continue;
                const float sum = fold_rows<DIM, SUM_BP>(Pg + (int64_t)kbase[k] * DP, cnt, s_buf[warp], lane);
                int moved = 0;
                if (lane < DIM) {
                    float cval = sS[k * DP + lane];
                    moved = shift_coord(sum, cnt, cval);
                    if (moved) sS[k * DP + lane] = cval;
                }
                if (__any_sync(FULL, moved) && lane == 0) s_moved = 1;
            }
            __syncthreads();
            ++pass;
            if (tid == 0) {
                v.pairs[c] += (unsigned long long)n * (unsigned long long)ns;
            }
            if (!s_moved) break;
            if (pass >= v.max_passes) {
                if (tid == 0) v.err[c] |= ERRB_EVOLVE_CAP;
                break;
            }
            handed = __syncthreads_or(tid == 0 ? hand_over() : 0);
            if (handed) break;
        }
        // results back and control (as k_control does after the last pass)
        for (int e = tid; e < ns; e += BLOCK)
#pragma unroll
            for (int d = 0; d < DIM; ++d) gS[(int64_t)e * DIM + d] = sS[e * DP + d];
        if (tid == 0) {
            v.passes[c] += pass;
            v.total_passes[c] += pass;
            v.cont[c] = 0;
            if (!handed) {
                v.phase[c] = PH_CONVERGED;
                const GroupDesc gd = v.gr[cd.group];
                if (atomicAdd(&v.group_conv[cd.group], 1) + 1 == gd.n_clouds)
                    v.ready[atomicAdd(&v.ctr[CTR_NREADY], 1)] = cd.group;
            }
        }
        return handed;
    }
}

template <int DIM, int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_tile_evolve(EngineView v)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TileCtaSmem<DIM, BLOCK> ts;
    const int nact = v.ctr[CTR_NACT];
    for (int a = blockIdx.x; a < nact; a += gridDim.x)
        tile_evolve_one<DIM, BLOCK>(v, v.act_cloud[a], FOLD_CTA_MIN, smem_raw, ts, [] { return 0; });
}

__host__ __device__ constexpr int tile_evolve_smem_bytes(int dim)
{
    const int dp = (dim == 3) ? 4 : dim;
    const int w = 8;
    return TILE_NS_MAX * dp * 4 + w * (TILE_NS_MAX + 1) * 4 + (TILE_NS_MAX + 1) * 4;
}

}  // namespace
}  // namespace rdb
#include "rd_tile_cluster.cuh"
namespace rdb {
namespace {

// ---------------------------------------------------------------------------
// control: one thread per cloud after each pass.
// ---------------------------------------------------------------------------
// (returns whether one of this thread's clouds converged)
__device__ int control_clouds(const EngineView& v, const int first, const int stride)
{
    int any = 0;
    const int nact = v.ctr[CTR_NACT];
    for (int a = first; a < nact; a += stride) {
        const int c = v.act_cloud[a];
        const CloudDesc cd = cloud_desc(v, c);
        v.pairs[c] += (unsigned long long)cd.n_all * (unsigned long long)v.ns[c];
        v.passes[c] += 1;
        v.total_passes[c] += 1;
        bool conv = false;
        if (v.cont[c] == 0) {
            conv = true;
        } else if (v.passes[c] >= v.max_passes) {
            v.err[c] |= ERRB_EVOLVE_CAP;
            conv = true;
        }
        v.cont[c] = 0;
        next_pass(v, c);
        any |= conv;
        if (conv && (v.flags & ENG_EVOLVE_ONLY)) {
            v.phase[c] = PH_DONE;
        } else if (conv) {
            v.phase[c] = PH_CONVERGED;
            // the last member of a group to converge queues the group
            const GroupDesc gd = v.gr[cd.group];
            if (atomicAdd(&v.group_conv[cd.group], 1) + 1 == gd.n_clouds)
                v.ready[atomicAdd(&v.ctr[CTR_NREADY], 1)] = cd.group;
        }
    }
    return any;
}

__global__ void k_control(EngineView v)
{
    pdl_enter();
    control_clouds(v, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// ---------------------------------------------------------------------------
// decimate: one CTA per group, rd/cpu/brute_force/decimate.hpp:41-81 (brute
// force) or :85-127 (decimateNoCopy, tiled), on the group's chosen points in
// cloud order.  Neighbour counts within r2 and 2*r2 (self included) come from a
// hashed grid of cell edge > 2*r2; the in-order scan is kept exact by updating
// the counts of a removed point's neighbours at the moment of its removal, and
// a warp ballot skips runs of points that cannot be removed.
// ---------------------------------------------------------------------------
template <int DIM, int BLOCK>
__device__ void decimate_group(const EngineView& v, const int g)
{
    const GroupDesc gd = v.gr[g];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ int s_off[33];
    __syncthreads();

    const CloudDesc c0 = v.cl[gd.cloud_begin];
    float* X = v.dx + gd.s_scratch * DIM;
    int32_t* cell = v.dcell + gd.s_scratch * DIM;
    int32_t* alive = v.dalive + gd.s_scratch;
    int32_t* c1 = v.dc1 + gd.s_scratch;
    int32_t* c2 = v.dc2 + gd.s_scratch;
    int32_t* items = v.ditems + gd.s_scratch;
    const int hbits = v.dec_hbits[g];
    const uint32_t hmask = (1u << hbits) - 1;
    int32_t* bstart = v.dbstart + v.dec_hoff[g];

    // Groups of many clouds (tiled runs) are walked one thread per cloud: the
    // clouds' offsets in the group's list come from a block-wide scan of their
    // chosen counts, or from the GPU-wide preparation (dcpre) when it ran.
    const int big = v.dbig[1] == g ? v.dbig[0] : 0;   // 1: lists are ready, 3: rounds are done too
    const int prepared = (big == 1 || big == 3) ? big : 0;
    const bool per_thread = gd.n_clouds > DEC_CLOUDS_SERIAL;
    // f(ci, c, ns, off) for every cloud of the group, one thread each; returns
    // the group's total (the same in every thread)
    auto for_clouds = [&](auto&& f) -> int {
        __shared__ int s_w[BLOCK / 32];
        __shared__ int s_carry;
        if (tid == 0) s_carry = 0;
        __syncthreads();
        for (int c0 = 0; c0 < gd.n_clouds; c0 += BLOCK) {
            const int ci = c0 + tid;
            const int c = gd.cloud_begin + ci;
            const int x = (ci < gd.n_clouds) ? v.ns[c] : 0;
            int incl = x;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) s_w[warp] = incl;
            __syncthreads();
            int pre = 0, tot = 0;
            for (int w = 0; w < BLOCK / 32; ++w) {
                pre += (w < warp) ? s_w[w] : 0;
                tot += s_w[w];
            }
            const int carry = s_carry;
            if (ci < gd.n_clouds) f(ci, c, x, prepared ? v.dcpre[ci] : carry + pre + incl - x);
            __syncthreads();
            if (tid == 0) s_carry = carry + tot;
            __syncthreads();
        }
        return s_carry;
    };
    // gather the group's chosen points (cloud order) into X, unless the
    // GPU-wide preparation kernels already did (large group)
    int total = 0;
    if (prepared) {
        total = v.dbig[2];
    } else if (per_thread) {
        total = for_clouds([&](int, int c, int ns, int off) {
            const int64_t so = v.cl[c].s_off;
            for (int e = 0; e < ns * DIM; ++e) X[(int64_t)off * DIM + e] = v.S[so * DIM + e];
        });
        __syncthreads();
    } else {
        for (int i = 0; i < gd.n_clouds; ++i) {
            const int c = gd.cloud_begin + i;
            const CloudDesc cd = v.cl[c];
            const int ns = v.ns[c];
            for (int e = tid; e < ns * DIM; e += BLOCK) X[(int64_t)total * DIM + e] = v.S[cd.s_off * DIM + e];
            total += ns;
        }
    }
    extern __shared__ __align__(16) unsigned char dec_smem[];
    // small sets over bit matrices, in shared memory where they fit behind the
    // counts, else in the room of the neighbour lists
    const int64_t mat = dec_bits_matrix(total);
    const bool bits_smem = dec_matrix_bytes(total) <= v.dec_dyn;
    bool bits = !prepared && total <= DEC_BITS_MAX && dec_bits_fixed(total) <= v.dec_dyn &&
                (bits_smem || mat <= (int64_t)4 * v.dec_nb_pp * gd.s_cap);
    __syncthreads();   // X is complete
    // Matrices in global memory cost the square of the points whatever lies near them,
    // the lists' walks (thread per point, 3^DIM cells each) grow with the neighbours.
    // 2D, 1,500 / 3,000 / 4,096 points, us, lists / matrices: 12 neighbours within 2 r2
    // 335 / 617, 546 / 1,642, 814 / 2,550; 48: 564 / 545, 1,189 / 1,507, 1,817 / 2,392;
    // 160: 1,044 / 498, 2,716 / 1,413, 4,079 / 2,280.  3D, 24: 780 / 830, 1,672 / 1,999,
    // 3,835 / 3,180; 96: 1,628 / 642, 4,104 / 1,874, 7,377 / 3,044.
    if (bits && !bits_smem)
        bits = dec_near_samples<DIM, BLOCK>([&](int i, int d) { return X[(int64_t)i * DIM + d]; }, total,
                                            c0.r2) > DEC_SAMPLES * (DIM <= 2 ? 48 : 24);
    if (bits) {
        uint32_t* m = bits_smem ? reinterpret_cast<uint32_t*>(dec_smem + (dec_bits_fixed(total) + 15) / 16 * 16)
                                : reinterpret_cast<uint32_t*>(v.dnb + (int64_t)v.dec_nb_pp * gd.s_scratch);
        decimate_bits<DIM, BLOCK>(X, total, c0.r2, gd.nocopy, alive, m, dec_smem, &v.err[gd.cloud_begin],
                                  v.ctr + CTR_DEC_PASSES);
    } else
    decimate_scan_lists<DIM, BLOCK>(X, total, c0.r2, gd.nocopy, cell, alive, c1, c2, items, bstart,
                                    hmask, v.dnb_off + gd.s_scratch + g,
                                    v.dnb + (int64_t)v.dec_nb_pp * gd.s_scratch,
                                    (int64_t)v.dec_nb_pp * gd.s_cap, dec_smem, v.dec_smem_max,
                                    &v.err[gd.cloud_begin], prepared, v.ctr + CTR_DEC_PASSES,
                                    prepared == 3 ? v.dbig[3] : 0);
    // compaction back into each cloud, in order
    int running = 0, total_after = 0;
    if (per_thread) {
        __shared__ int s_after;
        if (tid == 0) s_after = 0;
        __syncthreads();
        int mine = 0;
        for_clouds([&](int, int c, int ns, int off) {
            const int64_t so = v.cl[c].s_off;
            int kept = 0;
            for (int k = 0; k < ns; ++k) {
                if (!alive[off + k]) continue;
#pragma unroll
                for (int d = 0; d < DIM; ++d) v.S[(so + kept) * DIM + d] = X[(int64_t)(off + k) * DIM + d];
                ++kept;
            }
            v.ns[c] = kept;
            mine += kept;
        });
        if (mine) atomicAdd(&s_after, mine);
        __syncthreads();
        total_after = s_after;
    }
    for (int ci = 0; !per_thread && ci < gd.n_clouds; ++ci) {
        const int c = gd.cloud_begin + ci;
        const CloudDesc cd = v.cl[c];
        const int ns = v.ns[c];
        int kept = 0;
        for (int k0 = 0; k0 < ns; k0 += BLOCK) {
            const int k = k0 + tid;
            const bool a = (k < ns) && alive[running + k];
            const unsigned bal = __ballot_sync(FULL, a);
            if (lane == 0) s_off[warp] = __popc(bal);
            __syncthreads();
            int pre = 0, tot = 0;
            for (int w = 0; w < BLOCK / 32; ++w) {
                pre += (w < warp) ? s_off[w] : 0;
                tot += s_off[w];
            }
            if (a) {
                const int pos = kept + pre + __popc(bal & lanemask_lt());
#pragma unroll
                for (int d = 0; d < DIM; ++d)
                    v.S[(cd.s_off + pos) * DIM + d] = X[(int64_t)(running + k) * DIM + d];
            }
            kept += tot;
            __syncthreads();
        }
        running += ns;
        total_after += kept;
        if (tid == 0) v.ns[c] = kept;
    }
    __syncthreads();
    // outer-loop control: stop when decimation removed nothing
    const bool stable = (total_after == total);
    for (int i = tid; i < gd.n_clouds; i += BLOCK) {
        const int c = gd.cloud_begin + i;
        v.outer[c] += 1;
        v.passes[c] = 0;
        v.full[c] = 1;   // the chosen points have new indices
        if (stable) {
            v.phase[c] = PH_DONE;
        } else if (v.outer[c] >= v.max_outer) {
            v.err[c] |= ERRB_OUTER_CAP;
            v.phase[c] = PH_DONE;
        } else {
            v.phase[c] = PH_EVOLVE;
        }
    }
    if (tid == 0) {
        v.group_conv[g] = 0;
        if (prepared) v.dbig[0] = 0;
    }
    __syncthreads();
}

// ---------------------------------------------------------------------------
// GPU-wide preparation of a large decimation (tiled runs, whose one group may
// hold thousands of tiles, and rd_decimate).  When exactly one group is ready and it
// holds more than DEC_BIG_MIN points, these kernels build its gathered points, hash
// buckets, neighbour counts and neighbour lists across all SMs, and k_dec_rounds
// resolves its passes.  dbig = {state, group, total}: state 1 =
// prepared, 2 = lists overflowed (k_decimate rebuilds on its own), 3 = prepared
// and its rounds done (k_dec_rounds), 0 = idle.
// ---------------------------------------------------------------------------
// About the largest set whose bit matrices one CTA keeps in shared memory (205-250
// us for 790 points); from there on the kernels below take 200-350 us up to 4,097
// points and 40 neighbours, one CTA 500-3,200.
constexpr int DEC_BIG_MIN = 704;

template <int DIM>
__global__ void __launch_bounds__(1024) k_decbig_setup(EngineView v)
{
    __shared__ int s_w[32];
    __shared__ int s_carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) { v.dbig[0] = 0; s_carry = 0; }
    if (v.ctr[CTR_NREADY] != 1) return;
    const int g = v.ready[0];
    const GroupDesc gd = v.gr[g];
    __syncthreads();
    // exclusive prefix of the members' chosen counts -> dcpre
    for (int i0 = 0; i0 < gd.n_clouds; i0 += 1024) {
        const int i = i0 + tid;
        const int x = (i < gd.n_clouds) ? v.ns[gd.cloud_begin + i] : 0;
        int incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_w[warp] = incl;
        __syncthreads();
        int pre = 0, tot = 0;
        for (int w = 0; w < 32; ++w) {
            pre += (w < warp) ? s_w[w] : 0;
            tot += s_w[w];
        }
        const int carry = s_carry;
        if (i < gd.n_clouds) v.dcpre[i] = carry + pre + incl - x;
        __syncthreads();
        if (tid == 0) s_carry = carry + tot;
        __syncthreads();
    }
    const int total = s_carry;
    if (total <= DEC_BIG_MIN) return;
    // a quarter of the set around every point: lists as long as that take longer than
    // the bit matrices of one CTA (all within 2 r2, 1,000 / 4,000 points: 965 / 3,649
    // us, matrices 273 / 2,148; 40% of 790 in 3D 375 and 231; 4% of 4,096 349 and 2,280)
    if (total <= DEC_BITS_MAX) {
        auto coord = [&](int i, int d) {
            int lo = 0, hi = gd.n_clouds - 1;   // last member with dcpre <= i
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (v.dcpre[mid] <= i) lo = mid;
                else hi = mid - 1;
            }
            const CloudDesc& cd = v.cl[gd.cloud_begin + lo];
            return v.S[(cd.s_off + i - v.dcpre[lo]) * DIM + d];
        };
        if (dec_near_samples<DIM, 1024>(coord, total, v.cl[gd.cloud_begin].r2) > DEC_SAMPLES / 4 * total)
            return;
    }
    const int hbits = v.dec_hbits[g];
    int32_t* bstart = v.dbstart + v.dec_hoff[g];
    for (int h = tid; h <= (1 << hbits); h += 1024) bstart[h] = 0;
    if (tid == 0) {
        v.dcpre[gd.n_clouds] = total;
        v.dbig[1] = g;
        v.dbig[2] = total;
        v.dbig[0] = 1;
    }
}

template <int DIM>
__global__ void __launch_bounds__(256) k_decbig_gather(EngineView v)
{
    if (v.dbig[0] != 1) return;
    const int g = v.dbig[1], total = v.dbig[2];
    const GroupDesc gd = v.gr[g];
    const CloudDesc c0 = v.cl[gd.cloud_begin];
    const double inv = 1.0 / (2.0 * (double)c0.r2 * (1.0 + 1.0 / 1024.0));
    const uint32_t hmask = (1u << v.dec_hbits[g]) - 1;
    float* X = v.dx + gd.s_scratch * DIM;
    int32_t* cell = v.dcell + gd.s_scratch * DIM;
    int32_t* bstart = v.dbstart + v.dec_hoff[g];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        int lo = 0, hi = gd.n_clouds - 1;  // last member with dcpre <= t
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (v.dcpre[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        const CloudDesc cd = v.cl[gd.cloud_begin + lo];
        const int local = t - v.dcpre[lo];
        int cc[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            const float x = v.S[(cd.s_off + local) * DIM + d];
            X[(int64_t)t * DIM + d] = x;
            cc[d] = cell_of(x, inv);
            cell[(int64_t)t * DIM + d] = cc[d];
        }
        atomicAdd(&bstart[(cell_hash<DIM>(cc) & hmask) + 1], 1);
    }
}

// exclusive prefix over the big group's buckets (bstart[b] -> start of bucket b)
__global__ void __launch_bounds__(1024) k_decbig_scan_buckets(EngineView v)
{
    if (v.dbig[0] != 1) return;
    __shared__ int s_w[32];
    __shared__ int s_carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = v.dbig[1];
    const int n = (1 << v.dec_hbits[g]) + 1;
    int32_t* bstart = v.dbstart + v.dec_hoff[g];
    if (tid == 0) s_carry = 0;
    __syncthreads();
    for (int i0 = 0; i0 < n; i0 += 1024) {
        const int i = i0 + tid;
        const int x = (i < n) ? bstart[i] : 0;
        int incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_w[warp] = incl;
        __syncthreads();
        int pre = 0, tot = 0;
        for (int w = 0; w < 32; ++w) {
            pre += (w < warp) ? s_w[w] : 0;
            tot += s_w[w];
        }
        const int carry = s_carry;
        if (i < n) bstart[i] = carry + pre + incl;  // inclusive of the shifted counts
        __syncthreads();
        if (tid == 0) s_carry = carry + tot;
        __syncthreads();
    }
}

template <int DIM>
__global__ void __launch_bounds__(256) k_decbig_fill(EngineView v)
{
    if (v.dbig[0] != 1) return;
    const int g = v.dbig[1], total = v.dbig[2];
    const GroupDesc gd = v.gr[g];
    const uint32_t hmask = (1u << v.dec_hbits[g]) - 1;
    const int32_t* cell = v.dcell + gd.s_scratch * DIM;
    int32_t* items = v.ditems + gd.s_scratch;
    int32_t* bstart = v.dbstart + v.dec_hoff[g];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        int cc[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) cc[d] = cell[(int64_t)t * DIM + d];
        items[atomicAdd(&bstart[cell_hash<DIM>(cc) & hmask], 1)] = t;
    }
}

template <int DIM>
__global__ void __launch_bounds__(256) k_decbig_count(EngineView v)
{
    if (v.dbig[0] != 1) return;
    const int g = v.dbig[1], total = v.dbig[2];
    const GroupDesc gd = v.gr[g];
    const CloudDesc c0 = v.cl[gd.cloud_begin];
    const float rsq = sqr_rn(c0.r2);
    const float rsq4 = __fmul_rn(4.0f, rsq);
    const uint32_t hmask = (1u << v.dec_hbits[g]) - 1;
    const float* X = v.dx + gd.s_scratch * DIM;
    const int32_t* cell = v.dcell + gd.s_scratch * DIM;
    const int32_t* items = v.ditems + gd.s_scratch;
    const int32_t* bstart = v.dbstart + v.dec_hoff[g];
    int32_t* c1 = v.dc1 + gd.s_scratch;
    int32_t* c2 = v.dc2 + gd.s_scratch;
    int32_t* nb_off = v.dnb_off + gd.s_scratch + g;
    // a warp per point, a neighbour cell per lane: the cells' chains of dependent
    // loads (bounds, member, its cell and coordinates) run side by side (10,000
    // points, 40 neighbours: 238 -> 59 us, the lists 290 -> 65)
    const int lane = threadIdx.x & 31;
    for (int t = blockIdx.x * 8 + (threadIdx.x >> 5); t < total; t += gridDim.x * 8) {
        int n1 = 0, n2 = 0;
        dec_for_neighbours<DIM>(t, X, cell, items, bstart, hmask, rsq, rsq4,
                                [&](int, bool w1) { ++n2; n1 += w1; }, lane, 32);
        n1 = __reduce_add_sync(FULL, n1);
        n2 = __reduce_add_sync(FULL, n2);
        if (lane == 0) {
            c1[t] = n1 + 1;
            c2[t] = n2 + 1;
            nb_off[t] = n2;
        }
    }
}

// exclusive prefix of the list lengths; flags overflow of the list capacity
__global__ void __launch_bounds__(1024) k_decbig_scan_lists(EngineView v)
{
    if (v.dbig[0] != 1) return;
    __shared__ int s_w[32];
    __shared__ int64_t s_carry;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = v.dbig[1], total = v.dbig[2];
    const GroupDesc gd = v.gr[g];
    int32_t* nb_off = v.dnb_off + gd.s_scratch + g;
    if (tid == 0) s_carry = 0;
    __syncthreads();
    for (int i0 = 0; i0 < total; i0 += 1024) {
        const int i = i0 + tid;
        const int x = (i < total) ? list_len(nb_off[i]) : 0;
        int incl = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) s_w[warp] = incl;
        __syncthreads();
        int64_t pre = 0, tot = 0;
        for (int w = 0; w < 32; ++w) {
            pre += (w < warp) ? s_w[w] : 0;
            tot += s_w[w];
        }
        const int64_t carry = s_carry;
        if (i < total) nb_off[i] = (int)(carry + pre + incl - x);
        __syncthreads();
        if (tid == 0) s_carry = carry + tot;
        __syncthreads();
    }
    if (tid == 0) {
        nb_off[total] = (int)s_carry;
        if (!lists_fit(s_carry, (int64_t)v.dec_nb_pp * gd.s_cap)) v.dbig[0] = 2;
    }
}

template <int DIM>
__global__ void __launch_bounds__(256) k_decbig_lists(EngineView v)
{
    if (v.dbig[0] != 1) return;
    const int g = v.dbig[1], total = v.dbig[2];
    const GroupDesc gd = v.gr[g];
    const CloudDesc c0 = v.cl[gd.cloud_begin];
    const float rsq = sqr_rn(c0.r2);
    const float rsq4 = __fmul_rn(4.0f, rsq);
    const uint32_t hmask = (1u << v.dec_hbits[g]) - 1;
    const float* X = v.dx + gd.s_scratch * DIM;
    const int32_t* cell = v.dcell + gd.s_scratch * DIM;
    const int32_t* items = v.ditems + gd.s_scratch;
    const int32_t* bstart = v.dbstart + v.dec_hoff[g];
    const int32_t* nb_off = v.dnb_off + gd.s_scratch + g;
    int32_t* nb = v.dnb + (int64_t)v.dec_nb_pp * gd.s_scratch;
    // as k_decbig_count; the order inside a list does not matter
    __shared__ int s_at[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t = blockIdx.x * 8 + warp; t < total; t += gridDim.x * 8) {
        __syncwarp();
        if (lane == 0) s_at[warp] = nb_off[t];
        __syncwarp();
        dec_for_neighbours<DIM>(
            t, X, cell, items, bstart, hmask, rsq, rsq4,
            [&](int q, bool w1) { nb[atomicAdd(&s_at[warp], 1)] = w1 ? (q | (int)0x80000000) : q; },
            lane, 32);
    }
}

// The passes of the prepared decimation in parallel rounds, as
// decimate_round_passes (rd_grid.cuh) resolves them, by a cluster of DR_CTAS
// CTAs of 1,024 threads: a point is some thread's own, its state is published in
// global memory and copied into every CTA's shared memory between rounds, so
// that a neighbour's state is a shared-memory read.  One CTA alone waited for a
// chain of list loads, 20 points per thread: 10,000 points with about 40
// neighbours each 13.8 ms before (with its buckets and lists), 0.27 ms here and
// 0.24 in the other kernels now.
// Leaves dbig[0] = 3 and dbig[3] = alive count, or -1 - count where the
// minimum-count rule may act (k_decimate goes on with the sequential scan);
// larger sets than its shared memory holds are left to k_decimate.
constexpr int DR_CTAS = 8, DR_BLOCK = 1024;
constexpr int DR_MAX = 32 * 1024;
constexpr int DR_PTS = DR_MAX / (DR_CTAS * DR_BLOCK);

__global__ void __cluster_dims__(DR_CTAS, 1, 1) __launch_bounds__(DR_BLOCK) k_dec_rounds(EngineView v)
{
    __shared__ __align__(16) unsigned char st[DR_MAX];   // 0 dead, 1 alive, 2 kept, 3 removed
    __shared__ int s_left[2], s_removed;
    const int total = v.dbig[2];
    if (v.dbig[0] != 1 || total > DR_MAX) return;        // the same in every CTA
    namespace cgx = cooperative_groups;
    cgx::cluster_group cl = cgx::this_cluster();
    const int rank = (int)cl.block_rank(), tid = threadIdx.x;
    const int g = v.dbig[1];
    const GroupDesc gd = v.gr[g];
    int32_t* alive = v.dalive + gd.s_scratch;
    unsigned* pub = reinterpret_cast<unsigned*>(alive);  // one byte per point until the end
    unsigned char* pub8 = reinterpret_cast<unsigned char*>(alive);
    int32_t* c1 = v.dc1 + gd.s_scratch;
    int32_t* c2 = v.dc2 + gd.s_scratch;
    const int32_t* nb_off = v.dnb_off + gd.s_scratch + g;
    const int32_t* nb = v.dnb + (int64_t)v.dec_nb_pp * gd.s_scratch;
    int32_t* err = &v.err[gd.cloud_begin];
    const int words = (total + 3) / 4;
    // this thread's points, their lists and counts
    int lo[DR_PTS], hi[DR_PTS], n1[DR_PTS], n2[DR_PTS];
#pragma unroll
    for (int u = 0; u < DR_PTS; ++u) {
        const int i = (u * DR_CTAS + rank) * DR_BLOCK + tid;
        lo[u] = (i < total) ? nb_off[i] : 0;
        hi[u] = (i < total) ? nb_off[i + 1] : 0;
        n1[u] = (i < total) ? c1[i] : 0;
        n2[u] = (i < total) ? c2[i] : 0;
        if (i < total) pub8[i] = 1;
    }
    for (int i = tid; i < DR_MAX; i += DR_BLOCK) st[i] = i < total ? 1 : 0;
    // bytes past the last point of its word stay what they are: never read
    cl.sync();
    int cnt = total, guard = 0, flip = 0;
    bool fallback = false;
    while (cnt > 3) {
        if (++guard > total + 2) {
            if (rank == 0 && tid == 0) atomicOr(err, ERRB_DEC_CAP);
            break;
        }
        for (int round = 0;; ++round, flip ^= 1) {
            int left = 0;
#pragma unroll
            for (int u = 0; u < DR_PTS; ++u) {
                const int i = (u * DR_CTAS + rank) * DR_BLOCK + tid;
                if (i >= total || st[i] != 1) continue;
                int rem1 = 0, und1 = 0, rem2 = 0, und2 = 0;
#pragma unroll 8
                for (int t = lo[u]; t < hi[u]; ++t) {
                    const int e = nb[t];
                    const int q = e & 0x7fffffff;
                    const int sq = (q < i) ? st[q] : 0;
                    const int w1 = (e < 0) ? 1 : 0;
                    rem2 += (sq == 3);
                    rem1 += (sq == 3) & w1;
                    und2 += (sq == 1);
                    und1 += (sq == 1) & w1;
                }
                const int a = n1[u] - rem1, b = n2[u] - rem2;
                if (a - und1 >= 4 || b < 3) pub8[i] = 3;
                else if (a < 4 && b - und2 >= 3) pub8[i] = 2;
                else left = 1;
            }
            left = __syncthreads_or(left);
            if (tid == 0) s_left[flip] = left;
            cl.sync();   // decisions and flags of every CTA
            left = 0;
            for (int q = 0; q < DR_CTAS; ++q) left |= *cl.map_shared_rank(&s_left[flip], q);
            for (int w = tid; w < words; w += DR_BLOCK)
                reinterpret_cast<unsigned*>(st)[w] = __ldcg(pub + w);
            if (rank == 0 && tid == 0) atomicAdd(&v.ctr[CTR_DEC_ROUNDS], 1);
            __syncthreads();
            if (!left) break;
            if (round > total) {   // cannot happen: every round decides a point
                if (rank == 0 && tid == 0) atomicOr(err, ERRB_DEC_CAP);
                break;
            }
        }
        flip ^= 1;
        if (tid == 0) s_removed = 0;
        if (rank == 0 && tid == 0) atomicAdd(&v.ctr[CTR_DEC_PASSES], 1);
        __syncthreads();
        int mine = 0;
        for (int i = tid; i < total; i += DR_BLOCK) mine += (st[i] == 3);
        if (mine) atomicAdd(&s_removed, mine);
        __syncthreads();
        const int removed = s_removed;   // the same in every CTA
        const bool apply = removed > 0 && cnt - removed >= 3;
        for (int i = tid; i < total; i += DR_BLOCK)
            st[i] = (st[i] == 3) ? (apply ? 0 : 1) : (st[i] == 2 ? 1 : st[i]);
        cl.sync();       // every CTA has copied the last round
#pragma unroll
        for (int u = 0; u < DR_PTS; ++u) {
            const int i = (u * DR_CTAS + rank) * DR_BLOCK + tid;
            if (i < total) pub8[i] = st[i];
        }
        cl.sync();       // the new states are published (the next round copies all of them)
        if (removed == 0) break;            // a pass that changed nothing ends the loop
        if (!apply) {                       // the minimum-count rule may act
            fallback = true;
            break;
        }
        cnt -= removed;
        // exact counts of the alive points for the next pass
#pragma unroll
        for (int u = 0; u < DR_PTS; ++u) {
            const int i = (u * DR_CTAS + rank) * DR_BLOCK + tid;
            if (i >= total || st[i] != 1) continue;
            int a = 1, b = 1;
#pragma unroll 8
            for (int t = lo[u]; t < hi[u]; ++t) {
                const int e = nb[t];
                const int on = st[e & 0x7fffffff] == 1;
                b += on;
                a += on & (e < 0 ? 1 : 0);
            }
            n1[u] = a;
            n2[u] = b;
        }
    }
    cl.sync();   // the published bytes are read no more
#pragma unroll
    for (int u = 0; u < DR_PTS; ++u) {
        const int i = (u * DR_CTAS + rank) * DR_BLOCK + tid;
        if (i >= total) continue;
        alive[i] = st[i] != 0;
        c1[i] = n1[u];
        c2[i] = n2[u];
    }
    if (rank == 0 && tid == 0) {
        v.dbig[3] = fallback ? -1 - cnt : cnt;
        v.dbig[0] = 3;
    }
}

template <int DIM>
cudaError_t launch_decbig(const EngineView& v, cudaStream_t st)
{
    const int grid = v.n_sms * 8;
    k_decbig_setup<DIM><<<1, 1024, 0, st>>>(v);
    k_decbig_gather<DIM><<<grid, 256, 0, st>>>(v);
    k_decbig_scan_buckets<<<1, 1024, 0, st>>>(v);
    k_decbig_fill<DIM><<<grid, 256, 0, st>>>(v);
    k_decbig_count<DIM><<<grid, 256, 0, st>>>(v);
    k_decbig_scan_lists<<<1, 1024, 0, st>>>(v);
    k_decbig_lists<DIM><<<grid, 256, 0, st>>>(v);
    k_dec_rounds<<<DR_CTAS, DR_BLOCK, 0, st>>>(v);
    return cudaGetLastError();
}

__device__ void loop_condition(const EngineView& v, cudaGraphConditionalHandle h, int use_handle,
                               int count_iter);

// one CTA per group queued by the control step in this iteration; with_cond:
// the last CTA to finish then runs the loop-condition step (the phases and
// chosen counts of every group are final by then)
template <int DIM, int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_decimate(EngineView v, cudaGraphConditionalHandle h,
                                                    int with_cond, int use_handle)
{
    pdl_enter();
    __shared__ int s_last;
    const int nready = v.ctr[CTR_NREADY];
    if (v.ctr[CTR_COND_DONE]) return;   // nothing ready: k_merge_fold ended the iteration
    for (int r = blockIdx.x; r < nready; r += gridDim.x) decimate_group<DIM, BLOCK>(v, v.ready[r]);
    if (!with_cond) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&v.ctr[CTR_DEC_DONE], 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) v.ctr[CTR_DEC_DONE] = 0;
    loop_condition(v, h, use_handle, 1);
}

// ---------------------------------------------------------------------------
// loop condition: any unfinished cloud?  Sets the graph WHILE handle (graph
// mode) and/or leaves the count in ctr[CTR_ACTIVE] for the host (plain mode).
// Run by one whole CTA (any size up to 1024 threads).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(1024) k_loopcond(EngineView v, cudaGraphConditionalHandle h,
                                                   int use_handle, int count_iter)
{
    loop_condition(v, h, use_handle, count_iter);
}

__device__ void loop_condition(const EngineView& v, cudaGraphConditionalHandle h, int use_handle,
                               int count_iter)
{
    __shared__ int s_act;
    __shared__ int s_w[32][ACT_KINDS + 1];
    __shared__ int s_carry[ACT_KINDS + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        s_act = 0;
        for (int q = 0; q <= ACT_KINDS; ++q) s_carry[q] = 0;
    }
    __syncthreads();
    int act = 0;
    for (int c = tid; c < v.n_clouds; c += blockDim.x) act += (v.phase[c] != PH_DONE);
    if (act) atomicAdd(&s_act, act);
    // work lists of the next iteration: evolving clouds, prefixes of their
    // chunks and chosen-point blocks
    const int nc = v.n_clouds;
    for (int c0 = 0; c0 < nc; c0 += blockDim.x) {
        const int c = c0 + tid;
        const bool ev = (c < nc) && v.phase[c] == PH_EVOLVE;
        int x[ACT_KINDS + 1];
        x[0] = ev ? 1 : 0;
        const int rows = ev ? v.cl[c].n_chunks : 0;
        const int nkb = ev ? (v.ns[c] + KBLK - 1) / KBLK : 0;
        x[1 + ACT_CHUNK] = rows;
        const bool by_cta = ev && scan_by_cta(rows, v.cl[c].ns_cap);
        x[1 + ACT_KBLK] = by_cta ? nkb : 0;
        x[1 + ACT_KBLK_WARP] = by_cta ? 0 : nkb;
        int incl[ACT_KINDS + 1];
#pragma unroll
        for (int q = 0; q <= ACT_KINDS; ++q) {
            incl[q] = x[q];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(FULL, incl[q], o);
                if (lane >= o) incl[q] += y;
            }
            if (lane == 31) s_w[warp][q] = incl[q];
        }
        __syncthreads();
        int excl[ACT_KINDS + 1], tot[ACT_KINDS + 1];
#pragma unroll
        for (int q = 0; q <= ACT_KINDS; ++q) {
            int pre = 0, t = 0;
            for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
                pre += (w < warp) ? s_w[w][q] : 0;
                t += s_w[w][q];
            }
            excl[q] = s_carry[q] + pre + incl[q] - x[q];
            tot[q] = t;
        }
        if (ev) {
            v.act_cloud[excl[0]] = c;
#pragma unroll
            for (int q = 0; q < ACT_KINDS; ++q) v.act_pre[q * (nc + 1) + excl[0]] = excl[1 + q];
        }
        __syncthreads();
        if (tid == 0) {
#pragma unroll
            for (int q = 0; q <= ACT_KINDS; ++q) s_carry[q] += tot[q];
        }
        __syncthreads();
    }
    if (tid == 0) {
        const int nact = s_carry[0];
        for (int q = 0; q < ACT_KINDS; ++q) v.act_pre[q * (nc + 1) + nact] = s_carry[1 + q];
        v.ctr[CTR_NACT] = nact;
        next_iteration(v, s_act, h, use_handle, count_iter);
    }
}

// chosen counts are given in v.ns: evolving phase for non-empty clouds, or
// (queue_decimation) converged phase with every group queued for decimation
__global__ void k_set_given(EngineView v, int queue_decimation)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < v.n_clouds) {
        if (queue_decimation) v.phase[c] = PH_CONVERGED;
        else v.phase[c] = (v.ns[c] > 0) ? PH_EVOLVE : PH_DONE;
    }
    if (queue_decimation && c < v.n_groups) {
        v.ready[c] = c;
        v.group_conv[c] = v.gr[c].n_clouds;
    }
    if (c == 0) v.ctr[CTR_NREADY] = queue_decimation ? v.n_groups : 0;
}

__global__ void k_reset(EngineView v)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < CTR_COUNT && blockIdx.x == 0) v.ctr[c] = 0;
    if (c == 0) v.dbig[0] = 0;
    if (c < v.n_groups) v.group_conv[c] = 0;
    if (c >= v.n_clouds) return;
    v.kbdone[c] = 0;
    v.full[c] = 1;
    v.reb[c] = 0;
    v.rebnext[c] = 0;
    v.mvn[c] = 0;
    v.dmax[c] = 0;
    v.cont[c] = 0;
    v.passes[c] = 0;
    v.total_passes[c] = 0;
    v.outer[c] = 0;
    v.err[c] = 0;
    v.pairs[c] = 0;
}

// The dynamic shared memory a kernel may take is a property of the function, not of a
// launch, and another thread's run sets it between this one's call and its launch: it is
// always set to the most any run takes.  (Set to what the own run takes, a run of
// larger sets beside one of smaller ones failed to launch or to capture.)
template <int DIM, int BLOCK, int ITEMS>
cudaError_t set_assign_attrs()
{
    return cudaFuncSetAttribute(k_assign<DIM, BLOCK, ITEMS>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * HIST_SMEM_MAX);
}
template <int DIM>
cudaError_t set_decimate_attrs()
{
    return cudaFuncSetAttribute(k_decimate<DIM, 512>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                DEC_SMEM_MOST);
}
template <int DIM>
cudaError_t set_scatter_attrs()
{
    return cudaFuncSetAttribute(k_scatter_cta<DIM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                4 * (CHUNK_PTS_MAX + std::max(SCAT_W * SCAT_HMAX, SCAT_SMEM_MAX)));
}

// launch with programmatic stream serialisation (pdl != 0): the kernel may
// start while the previous kernel on the stream drains; it waits in
// pdl_enter(). Single-cloud passes (small, latency-bound grids) gain from it
// (33.7 -> 33.5 ms per 1M-point helix solve); batches of thousands of clouds
// lose 1% with it, so they launch plainly.
template <typename... KArgs, typename... Args>
static cudaError_t launch_pdl(int pdl, void (*kernel)(KArgs...), int grid, int block, size_t smem,
                              cudaStream_t st, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// persistent grid of k_assign_cull: every resident CTA, at most one warp per block
template <int DIM, int ITEMS>
cudaError_t launch_assign_cull(const EngineView& v, int pdl, cudaStream_t st)
{
    static std::atomic<int> per_sm{0};
    int b = per_sm.load(std::memory_order_relaxed);
    if (b == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_assign_cull<DIM, ITEMS>, AC_BLOCK, 0) !=
                cudaSuccess || b < 1)
            b = 1;
        per_sm.store(b, std::memory_order_relaxed);
    }
    const int wpc = v.chunk_pts / (32 * ITEMS);
    if (wpc < 1 || (wpc & (wpc - 1))) return cudaErrorInvalidValue;  // the kernel's block numbers need 2^k
    const int64_t ctas = ((int64_t)v.n_chunks * wpc + AC_WARPS - 1) / AC_WARPS;
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>(ctas, (int64_t)v.n_sms * b));
    return launch_pdl(pdl, k_assign_cull<DIM, ITEMS>, g, AC_BLOCK, 0, st, v);
}

// grid of k_merge_fold: every resident CTA, at most one per chosen point
template <int DIM, int BLOCK, bool LONG>
int merge_grid(const EngineView& v)
{
    static std::atomic<int> per_sm{0};
    int b = per_sm.load(std::memory_order_relaxed);
    if (b == 0) {
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_merge_fold<DIM, BLOCK, LONG>, BLOCK, 0) !=
                cudaSuccess || b < 1)
            b = 1;
        per_sm.store(b, std::memory_order_relaxed);
    }
    return (int)std::max<int64_t>(1, std::min<int64_t>(v.n_slots, (int64_t)v.n_sms * b));
}

template <int DIM>
cudaError_t prepare_pass_dim(const EngineView& v, const TuneParams& tp)
{
    cudaError_t e = cudaErrorInvalidValue;
#define RD_PREP_CASE(B, I) \
    if (tp.block == B && tp.items == I) e = set_assign_attrs<DIM, B, I>();
    RD_PREP_CASE(128, 8) RD_PREP_CASE(128, 4) RD_PREP_CASE(256, 4) RD_PREP_CASE(256, 8)
    RD_PREP_CASE(128, 16)
#undef RD_PREP_CASE
    if (e != cudaSuccess) return e;
    if (dec_smem_bytes(v) > DEC_SMEM_MOST || v.chunk_max > CHUNK_PTS_MAX) return cudaErrorInvalidValue;
    e = set_decimate_attrs<DIM>();
    if (e != cudaSuccess) return e;
    return set_scatter_attrs<DIM>();
}

// the kernels of an evolve pass; control: see k_merge_fold
template <int DIM>
cudaError_t launch_evolve_kernels(const EngineView& v, const TuneParams& tp, int assign_grid,
                                  const LoopCond& lc, int control, cudaStream_t st,
                                  cudaEvent_t a0 = nullptr, cudaEvent_t a1 = nullptr,
                                  int assign_pdl = 0)
{
    const int hist_bytes = v.hist_smem * 4;
    const int sms = v.n_sms;
    if (a0) cudaEventRecord(a0, st);
    if (v.cull) {
        cudaError_t e;
        if (!v.lists) {
            // assigned and counted anew (the counts' rows hold the last pass's prefixes)
            e = cudaMemsetAsync(v.hist, 0, 4 * (size_t)v.hist_ints, st);
            if (e == cudaSuccess) e = cudaMemsetAsync(v.keys, 0xff, 4 * (size_t)v.n_points, st);
            if (e == cudaSuccess) e = cudaMemsetAsync(v.ksp, 0xff, 4 * (size_t)v.n_points, st);
            if (e != cudaSuccess) return e;
            assign_pdl = 0;   // follows no kernel
        }
        if (tp.cull_items == 2) e = launch_assign_cull<DIM, 2>(v, assign_pdl, st);
        else if (tp.cull_items == 8) e = launch_assign_cull<DIM, 8>(v, assign_pdl, st);
        else e = launch_assign_cull<DIM, 4>(v, assign_pdl, st);
        if (e != cudaSuccess) return e;
    } else {
#define RD_ASSIGN_CASE(B, I)                                                                  \
    if (tp.block == B && tp.items == I) {                                                     \
        k_assign<DIM, B, I><<<assign_grid, B, hist_bytes, st>>>(v);                           \
    } else
    RD_ASSIGN_CASE(128, 8)
    RD_ASSIGN_CASE(128, 4)
    RD_ASSIGN_CASE(256, 4)
    RD_ASSIGN_CASE(256, 8)
    RD_ASSIGN_CASE(128, 16)
    { return cudaErrorInvalidValue; }
#undef RD_ASSIGN_CASE
    }
    if (a1) cudaEventRecord(a1, st);
    // fixed grids; every kernel walks only the current work lists
    // every kernel after the assignment is a programmatic dependent of the one
    // before it (pdl_enter) when a single cloud evolves
    const int pdl = v.n_clouds == 1;
    cudaError_t e = cudaSuccess;
    if (v.n_kblk > 0)
        e = launch_pdl(pdl, k_chunkscan_cta, std::min(v.n_kblk, sms * 4), CS_W * 32, 0, st, v);
    if (e == cudaSuccess && v.n_kblk_warp > 0)
        e = launch_pdl(pdl, k_chunkscan_warp, std::min((v.n_kblk_warp + CSW_W - 1) / CSW_W, sms * 8),
                       CSW_W * 32, 0, st, v);
    if (e == cudaSuccess && v.n_chunks > 0)
        e = launch_pdl(pdl, k_scatter_cta<DIM>, std::min(v.n_chunks, sms * 8), SCAT_W * 32,
                       scatter_cta_smem_bytes(v), st, v);
    if (e != cudaSuccess) return e;
    if (v.n_slots > 0) {
        auto merge = [&](auto block, auto lng) {
            constexpr int B = decltype(block)::value;
            constexpr bool LONG = decltype(lng)::value;
            return launch_pdl(pdl, k_merge_fold<DIM, B, LONG>, merge_grid<DIM, B, LONG>(v), B, 0, st, v,
                              lc.h, control, lc.use_handle);
        };
        using Many = std::integral_constant<int, MF_BLOCK_MANY>;
        using One = std::integral_constant<int, MF_BLOCK>;
        if (v.long_lists) e = merge(One{}, std::true_type{});
        else if (v.n_clouds == 1) e = merge(One{}, std::false_type{});
        else e = merge(Many{}, std::false_type{});
    } else {
        e = launch_pdl(pdl, k_control, std::min((v.n_clouds + 255) / 256, sms), 256, 0, st, v);
    }
    return e;
}

template <int DIM>
cudaError_t launch_pass_dim(const EngineView& v, const TuneParams& tp, int assign_grid,
                            const LoopCond& lc, cudaStream_t st, cudaEvent_t a0, cudaEvent_t a1,
                            bool follows_pass)
{
    const int pdl = v.n_clouds == 1;
    const cudaError_t e = launch_evolve_kernels<DIM>(v, tp, assign_grid, lc, MF_CONTROL, st, a0, a1,
                                                     pdl && follows_pass);
    if (e != cudaSuccess) return e;
    return launch_pdl(pdl, k_decimate<DIM, 512>, std::min(v.n_groups, v.n_sms * 2), 512,
                      dec_smem_bytes(v), st, v, lc.h, 1, lc.use_handle);
}

template <int DIM>
cudaError_t launch_choose_dim(const EngineView& v, cudaStream_t st)
{
    using CS = ChooseSmem<DIM>;
    constexpr int bytes = choose_smem_bytes<DIM, CS>();
    cudaError_t e =
        cudaFuncSetAttribute(k_choose<DIM, CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    k_choose<DIM, CS><<<v.n_clouds, CS::BLOCK, bytes, st>>>(v);
    return cudaGetLastError();
}

// rounds over [0, n): 4096 points first, then four times as many each; needs
// v.hash (HB ints) and surv (n bytes).  The points a round leaves to the one-CTA
// resolve are those no earlier round covers, few after the first rounds, so
// the number of rounds (a filter, a compaction and a resolve each, 50-80 us) is
// what counts: growing four-fold instead of two-fold takes five instead of
// eight on 1M points.
template <int DIM>
cudaError_t launch_choose_rounds_dim(const EngineView& v, int c, int n, uint8_t* surv,
                                     int32_t* sel, void* tmp, size_t tmp_bytes, cudaStream_t st)
{
    using CS = ChooseSmem<DIM>;
    constexpr int B = CS::BLOCK;
    constexpr int bytes = choose_smem_bytes<DIM, CS>();
    cudaError_t e = cudaFuncSetAttribute(k_choose_resolve<DIM, CS>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    int a = 0, size = 4096, first = 1;
    int32_t* nsel = sel + n;
    while (a < n) {
        const int b = (int)std::min<int64_t>((int64_t)n, (int64_t)a + size);
        if (first) {
            k_choose_resolve<DIM, CS><<<1, B, bytes, st>>>(v, c, a, b, nullptr, nullptr, first);
        } else {
            const int grid = std::max(1, std::min((b - a + 255) / 256, 148 * 16));
            k_choose_filter<DIM><<<grid, 256, 0, st>>>(v, c, a, b, surv);
            size_t tb = tmp_bytes;
            e = cub::DeviceSelect::Flagged(tmp, tb, cub::CountingInputIterator<int32_t>(a), surv, sel,
                                           nsel, b - a, st);
            if (e != cudaSuccess) return e;
            k_choose_resolve<DIM, CS><<<1, B, bytes, st>>>(v, c, a, b, sel, nsel, first);
        }
        a = b;
        size = (int)std::min<int64_t>((int64_t)size * 4, 1 << 30);
        first = 0;
    }
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_choose_rounds(int dim, const EngineView& v, int c, int n, uint8_t* surv,
                                 int32_t* sel, void* tmp, size_t tmp_bytes, cudaStream_t st)
{
    return with_dim(dim, [&](auto D) {
        return launch_choose_rounds_dim<decltype(D)::value>(v, c, n, surv, sel, tmp, tmp_bytes, st);
    });
}

int choose_hash_buckets() { return ChooseSmem<2>::HB; }

size_t choose_select_scratch_bytes(int64_t n)
{
    size_t tb = 0;
    cub::DeviceSelect::Flagged(nullptr, tb, cub::CountingInputIterator<int32_t>(0), (const uint8_t*)nullptr,
                               (int32_t*)nullptr, (int32_t*)nullptr, (int)std::max<int64_t>(n, 1));
    return tb + 256;
}

cudaError_t launch_choose(int dim, const EngineView& v, cudaStream_t st)
{
    return with_dim(dim, [&](auto D) { return launch_choose_dim<decltype(D)::value>(v, st); });
}

cudaError_t prepare_pass(int dim, const EngineView& v, const TuneParams& tp)
{
    return with_dim(dim, [&](auto D) { return prepare_pass_dim<decltype(D)::value>(v, tp); });
}

cudaError_t launch_pass(int dim, const EngineView& v, const TuneParams& tp, int assign_grid,
                        const LoopCond& lc, cudaStream_t st, cudaEvent_t a0, cudaEvent_t a1,
                        bool follows_pass)
{
    return with_dim(dim, [&](auto D) {
        return launch_pass_dim<decltype(D)::value>(v, tp, assign_grid, lc, st, a0, a1, follows_pass);
    });
}

cudaError_t launch_loopcond(const EngineView& v, cudaGraphConditionalHandle h, int use_handle,
                            cudaStream_t st, int count_iter)
{
    k_loopcond<<<1, 1024, 0, st>>>(v, h, use_handle, count_iter);
    return cudaGetLastError();
}

static std::atomic<int> g_tile_cl_on{1}, g_tile_cl_min{0}, g_tile_seg_min{0};
TileClusterParams tile_cluster_params()
{
    return TileClusterParams{g_tile_cl_on.load() != 0, g_tile_cl_min.load(), g_tile_seg_min.load()};
}
void set_tile_cluster_params(const TileClusterParams& p)
{
    g_tile_cl_on.store(p.enabled ? 1 : 0);
    g_tile_cl_min.store(p.min_points);
    g_tile_seg_min.store(p.seg_min);
}

// launch configuration of the cluster tile kernel: one CTA per resident slot
// (TCL-CTA clusters), dynamic shared memory as tile_cluster_smem_bytes
template <int DIM>
static void tile_cl_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int grid)
{
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(256, 1, 1);
    cfg.dynamicSmemBytes = tile_cluster_smem_bytes(DIM);
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = TCL;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

template <int DIM>
static cudaError_t tile_cl_prepare(int* cl_grid)
{
    cudaError_t e = cudaFuncSetAttribute(k_tile_evolve_cl<DIM, 256>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         tile_cluster_smem_bytes(DIM));
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    tile_cl_config<DIM>(cfg, at, TCL);
    int ncl = 0;
    e = cudaOccupancyMaxActiveClusters(&ncl, k_tile_evolve_cl<DIM, 256>, &cfg);
    if (e != cudaSuccess) return e;
    *cl_grid = (ncl > 0) ? ncl * TCL : 0;
    return cudaSuccess;
}

cudaError_t prepare_tile_pass(int dim, const EngineView& v, int* cl_grid)
{
    *cl_grid = 0;
    return with_dim(dim, [&](auto D) {
        constexpr int DIM = decltype(D)::value;
        cudaError_t e = cudaFuncSetAttribute(k_tile_evolve<DIM, 256>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             tile_evolve_smem_bytes(DIM));
        if (e != cudaSuccess) return e;
        if (v.tile_clusters) {
            e = tile_cl_prepare<DIM>(cl_grid);
            if (e != cudaSuccess) return e;
        }
        return set_decimate_attrs<DIM>();
    });
}

cudaError_t launch_tile_pass(int dim, const EngineView& v, const LoopCond& lc, cudaStream_t st,
                             cudaEvent_t a0, cudaEvent_t a1)
{
    const int smem = tile_evolve_smem_bytes(dim);
    const int grid = std::max(1, std::min(v.n_clouds, v.n_sms * 3));
    const int dgrid = std::max(1, std::min(v.n_groups, v.n_sms * 2));
    return with_dim(dim, [&](auto D) {
        constexpr int DIM = decltype(D)::value;
        if (a0) cudaEventRecord(a0, st);
        if (v.tile_cl_grid > 0) {
            cudaLaunchConfig_t cfg;
            cudaLaunchAttribute at[1];
            tile_cl_config<DIM>(cfg, at, v.tile_cl_grid);
            cfg.stream = st;
            const cudaError_t e = cudaLaunchKernelEx(&cfg, k_tile_evolve_cl<DIM, 256>, v);
            if (e != cudaSuccess) return e;
        } else {
            k_tile_evolve<DIM, 256><<<grid, 256, smem, st>>>(v);
        }
        if (a1) cudaEventRecord(a1, st);
        launch_decbig<DIM>(v, st);
        k_decimate<DIM, 512><<<dgrid, 512, dec_smem_bytes(v), st>>>(v, lc.h, 1, lc.use_handle);
        return cudaGetLastError();
    });
}

template <int DIM>
__global__ void __launch_bounds__(32) k_ordered_sum(const float* P, const int32_t* idx, int n,
                                                   float* out, int method)
{
    __shared__ float s_buf[SUM_BP * DIM];
    __shared__ int s_idx[SUM_BP];
    const int lane = threadIdx.x;
    const float r = (method == 1) ? fold_members_par<DIM>(idx, n, P, lane)
                                  : fold_members<DIM>(idx, n, P, s_buf, s_idx, lane);
    if (lane < DIM) out[lane] = r;
}

template <int DIM>
__global__ void __launch_bounds__(256) k_ordered_sum_cta(const float* P, const int32_t* idx, int n,
                                                         float* out)
{
    __shared__ FoldCtaSmem<8, DIM> sm;
    fold_members_cta<8, DIM>(idx, n, P, sm);
    if (threadIdx.x < DIM) out[threadIdx.x] = sm.s[threadIdx.x];
}

template <int DIM, int BLOCK>
__global__ void __launch_bounds__(BLOCK) k_ordered_sum_seg(const float* P, const int32_t* idx, int n,
                                                           float* out)
{
    __shared__ SegFoldSmem<BLOCK / 32, DIM> sm;
    fold_members_seg<BLOCK / 32, DIM>(idx, n, P, sm);
    if (threadIdx.x < DIM) out[threadIdx.x] = sm.out[threadIdx.x];
}

cudaError_t launch_ordered_sum(int dim, const float* P, const int32_t* idx, int n, float* out,
                               int method, cudaStream_t st)
{
    return with_dim(dim, [&](auto D) {
        constexpr int DIM = decltype(D)::value;
        if (method == 3) k_ordered_sum_seg<DIM, 256><<<1, 256, 0, st>>>(P, idx, n, out);
        else if (method == 4) k_ordered_sum_seg<DIM, 1024><<<1, 1024, 0, st>>>(P, idx, n, out);
        else if (method == 2) k_ordered_sum_cta<DIM><<<1, 256, 0, st>>>(P, idx, n, out);
        else k_ordered_sum<DIM><<<1, 32, 0, st>>>(P, idx, n, out, method);
        return cudaGetLastError();
    });
}

cudaError_t launch_set_given(const EngineView& v, int queue_decimation, cudaStream_t st)
{
    const int n = v.n_clouds > v.n_groups ? v.n_clouds : v.n_groups;
    k_set_given<<<(n + 255) / 256, 256, 0, st>>>(v, queue_decimation);
    return cudaGetLastError();
}

int dec_smem_points()
{
    static const int n = [] {
        int m = 1;
        while (m < DEC_BITS_MAX && dec_matrix_bytes(m + 1) <= DEC_BITS_SMEM) ++m;
        return m;
    }();
    return n;
}

int dec_dyn_bytes(int points)
{
    // the largest group's matrices where they fit; otherwise its counts, and room
    // for the matrices of groups of up to about 700 points
    const int b = std::min(points, DEC_BITS_MAX);
    const int64_t all = dec_matrix_bytes(b);
    const int bits = all <= DEC_BITS_SMEM ? (int)all : std::max(dec_bits_fixed(b), 128 * 1024);
    return std::max(dec_list_bytes(points), bits);
}

cudaError_t launch_decimate(int dim, const EngineView& view, int64_t points, cudaStream_t st)
{
    EngineView v = view;
    // the one group's size is known: its matrices fit shared memory, or (more than
    // DEC_BITS_MAX points) it has none
    const bool big = v.n_groups == 1 && v.dec_dyn < dec_matrix_bytes((int)std::min<int64_t>(points, DEC_BITS_MAX));
    if (big && points > DEC_BITS_MAX) v.dec_dyn = dec_list_bytes(v.dec_smem_max);
    const int grid = std::max(1, std::min(v.n_groups, v.n_sms * 2));
    const int smem = dec_smem_bytes(v);
    cudaError_t e = cudaSuccess;
    e = with_dim(dim, [&](auto D) {
        constexpr int DIM = decltype(D)::value;
        cudaError_t r = set_decimate_attrs<DIM>();
        // one large group: its buckets, lists and rounds over more of the GPU
        if (r == cudaSuccess && big) r = launch_decbig<DIM>(v, st);
        if (r == cudaSuccess) k_decimate<DIM, 512><<<grid, 512, smem, st>>>(v, 0, 0, 0);
        return r;
    });
    if (e != cudaSuccess) return e;
    return cudaGetLastError();
}

cudaError_t launch_evolve_step(int dim, const EngineView& v, const TuneParams& tp, int assign_grid,
                               cudaStream_t st)
{
    return with_dim(dim, [&](auto D) {
        return launch_evolve_kernels<decltype(D)::value>(v, tp, assign_grid, LoopCond(), MF_STEP, st);
    });
}

cudaError_t launch_reset(const EngineView& v, cudaStream_t st)
{
    int n = v.n_clouds > CTR_COUNT ? v.n_clouds : CTR_COUNT;
    n = n > v.n_groups ? n : v.n_groups;
    k_reset<<<(n + 255) / 256, 256, 0, st>>>(v);
    return cudaGetLastError();
}

bool tune_supported(int dim, const TuneParams& tp)
{
    (void)dim;
    const bool cull_ok = tp.cull_items == 2 || tp.cull_items == 4 || tp.cull_items == 8;
    return cull_ok && ((tp.block == 128 && (tp.items == 4 || tp.items == 8 || tp.items == 16)) ||
                       (tp.block == 256 && (tp.items == 4 || tp.items == 8)));
}

int long_list_avg() { return LONG_AVG; }
int merge_cap(bool long_lists) { return long_lists ? MERGE_CAP_LONG : MERGE_CAP; }

int assign_smem_bytes(int dim, const TuneParams& tp, int hist_ints)
{
    (void)tp;
    const int dp = (dim == 3) ? 4 : dim;
    return ASSIGN_TS * dp * 4 + 16 + hist_ints * 4;
}

template <int DIM, int B, int I>
static int occ_of(int dyn)
{
    int nb = 0;
    if (set_assign_attrs<DIM, B, I>() != cudaSuccess) return 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_assign<DIM, B, I>, B, dyn);
    return nb;
}

int max_assign_blocks_per_sm(int dim, const TuneParams& tp, int hist_ints)
{
    const int dyn = hist_ints * 4;
#define RD_OCC(D, B, I) \
    if (dim == D && tp.block == B && tp.items == I) return occ_of<D, B, I>(dyn);
    RD_OCC(1, 128, 8) RD_OCC(1, 128, 4) RD_OCC(1, 256, 4) RD_OCC(1, 256, 8) RD_OCC(1, 128, 16)
    RD_OCC(2, 128, 8) RD_OCC(2, 128, 4) RD_OCC(2, 256, 4) RD_OCC(2, 256, 8) RD_OCC(2, 128, 16)
    RD_OCC(3, 128, 8) RD_OCC(3, 128, 4) RD_OCC(3, 256, 4) RD_OCC(3, 256, 8) RD_OCC(3, 128, 16)
    RD_OCC(4, 128, 8) RD_OCC(4, 128, 4) RD_OCC(4, 256, 4) RD_OCC(4, 256, 8) RD_OCC(4, 128, 16)
#undef RD_OCC
    return 0;
}

}  // namespace rdb
