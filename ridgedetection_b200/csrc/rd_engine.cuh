// rd_engine.cuh -- the device-side batch engine shared by every entry point.
//
// One engine run solves a batch of independent "clouds" (see CloudDesc) that
// share the point dimension DIM:
//   choose      one CTA per cloud, greedy r1-separated subset in input order
//               over a hashed uniform grid (exact test, grid only prunes);
//   evolve      passes over all clouds still evolving: assignment, of the blocks of
//               points whose keys can have changed, then the member lists of the keys
//               with changes (merge of the pass's edits, or chunk scan and stable
//               scatter of a cloud that regroups), their ordered sums and shifts, and
//               control; the per-chosen coordinate sums are formed in cloud-point
//               index order, exactly as the reference's serial loop forms them;
//   decimate    one CTA per group with the reference's in-order semantics;
//   loop        a device flag says whether any cloud is unfinished; it drives a
//               CUDA-graph WHILE node (graph mode) or is read by the host (plain).
#pragma once

#include "rd_internal.cuh"
#include "rd_listroom.hpp"
#include "rd_tile_rule.hpp"

#include <cstddef>
#include <cstdint>
#include <string>
#include <vector>

namespace rdb {

enum : int {
    ENG_EVOLVE_ONLY = 1,   // converged clouds finish without decimation
    ENG_ALWAYS_MOVE = 2,   // adjoint forward: every non-empty cluster moves to its mean
};

// neighbour-list capacity of the decimation, per chosen point: at least
// DEC_NB_MIN_PER_POINT, more (up to all points of the largest group) while the whole
// list buffer stays within DEC_NB_BUDGET entries (lists that do not fit fall back to
// walking the hash buckets)
constexpr int DEC_NB_MIN_PER_POINT = 32;
constexpr int DEC_NB_MAX_PER_POINT = 4096;
constexpr int64_t DEC_NB_BUDGET = int64_t(1) << 28;
// points whose int16 counts live in the decimation's shared memory (a count
// never exceeds the number of points, so int16 holds it)
constexpr int DEC_SMEM_MAX_POINTS = 32752;
// fused per-tile evolve: chosen points per tile it can hold
constexpr int TILE_NS_MAX = 1024;

// kinds of work list over the evolving clouds (rebuilt by loop_condition when a cloud
// converges): assignment chunks; blocks of KBLK chosen points of the clouds scanned by
// CTAs (scan_by_cta) and of the others (one warp per block)
enum : int { ACT_CHUNK = 0, ACT_KBLK = 1, ACT_KBLK_WARP = 2, ACT_KINDS = 3 };
// Clouds whose histogram a CTA scans per block of chosen points: those of many chunk
// rows, and those of many chosen points, where the last block lays out every key's
// region, 32 keys after 32 in one warp (one pass over 30,000 points with 29,849 chosen
// ones 3.6 ms, by CTAs 2.8).
constexpr int SCAN_ROWS_WARP = 64, SCAN_KEYS_WARP = 2048;
__host__ __device__ inline bool scan_by_cta(const int n_chunks, const int ns_cap)
{
    return n_chunks > SCAN_ROWS_WARP || ns_cap > SCAN_KEYS_WARP;
}

enum : int {
    CTR_WORK = 0,      // assignment work ticket
    CTR_ACTIVE = 1,    // unfinished clouds after the last control step
    CTR_ITERS = 2,     // loop iterations run
    CTR_ERR = 3,       // OR of global error bits
    CTR_NACT = 4,      // evolving clouds in the current work lists
    CTR_NREADY = 5,    // groups ready for decimation in this iteration
    CTR_NDIRTY = 6,    // keys listed for folding in the current pass
    CTR_TILE_HEAVY = 7,// heavy-tile ticket of the cluster tile kernel
    CTR_SUM_DONE = 8,  // CTAs of k_merge_fold finished (the last one runs the control step)
    CTR_DEC_DONE = 9,  // CTAs of k_decimate finished (the last one sets the loop condition)
    CTR_DEC_PASSES = 10,  // decimation passes resolved in parallel rounds (this run)
    CTR_DEC_ROUNDS = 11,  // rounds they took
    CTR_COND_DONE = 12,   // k_merge_fold ended this iteration (no group was ready)
    CTR_HANDED = 13,      // light tiles handed over to a cluster (this run)
    CTR_COUNT = 14,
};

struct EngineView {
    const CloudDesc* cl;
    const GroupDesc* gr;
    const int32_t* chunk_cloud;  // chunk -> cloud
    const int32_t* slot_cloud;   // chosen slot -> cloud
    float* P;                    // packed evolve points, ROW_MAJOR
    float* S;                    // chosen points, ROW_MAJOR, capacity n_own per cloud
    int32_t* keys;               // per point slot: assigned chosen index or -1
    float* Pg;                   // per point slot: the points' coordinates grouped by key in
                                 // index order, PadDim floats each (tiled kernels)
    // lockstep passes: each key's members in index order, in its region
    // [base, base + kcap) of its cloud's part (reg_off) of two buffers; the
    // current list is in buffer par
    float* Lr[2];                // coordinates, PadDim floats per row
    int32_t* Ls[2];              // the points' positions in their cloud (with lists)
    int4* kinfo;                 // per chosen slot: base, kcap, members, par
    int32_t* edit;               // per row: edits of this pass, at the key's region
    int32_t* ecnt;               // per chosen slot: edits of this pass
    int32_t* dlist;              // chosen slots to fold in this pass
    int32_t* reb;                // per cloud: regroup all points in this pass
    int32_t* rebnext;            // per cloud: and in the next one
    int32_t* hist;               // per cloud: n_chunks x ns_cap key histogram
    int32_t* hpre;               // the same shape: its exclusive prefix over the chunks (hist itself
                                 // in runs without lists, which count anew in every pass)
    int32_t* cnt;                // per chosen slot: members in the last pass
    int32_t* base;               // per chosen slot: first row of its region
    int32_t* kbdone;             // per cloud: key blocks of the chunk scan finished in this pass
    int32_t* hash;               // choose hash heads
    int32_t* next;               // per chosen slot: choose hash chain
    int32_t* ns;                 // per cloud: current chosen count
    int32_t* phase;              // per cloud: PH_*
    int32_t* cont;               // per cloud: a coordinate moved in this pass
    int32_t* passes;             // per cloud: passes of the current evolve run
    int32_t* total_passes;       // per cloud: all passes
    int32_t* outer;              // per cloud: evolve/decimate rounds
    int32_t* err;                // per cloud: ERRB_* bits
    unsigned long long* pairs;   // per cloud: sum over passes of n_all * ns
    int32_t* ctr;                // CTR_* counters
    int32_t* act_cloud;          // evolving clouds, in cloud order (n_clouds)
    int32_t* act_pre;            // ACT_KINDS x (n_clouds+1) exclusive prefixes of their work items
    int32_t* group_conv;         // per group: members converged in this round
    int32_t* ready;              // groups ready for decimation (n_groups)
    // decimation scratch, per group (offsets in GroupDesc / dec_hoff)
    float* dx;                   // coordinates of the group's chosen points
    int32_t* dcell;              // their grid cells
    int32_t* dalive;
    int32_t* dc1;                // alive neighbours within r2 (self included)
    int32_t* dc2;                // alive neighbours within 2*r2 (self included)
    int32_t* dbstart;            // bucket starts (HB+1 per group)
    int32_t* ditems;             // bucket members
    int32_t* dnb_off;            // per group: neighbour-list offsets (total+1)
    int32_t* dnb;                // per group: neighbour lists, dec_nb_pp per scratch slot
    int32_t* dbig;               // GPU-wide prepared decimation: {state, group, total, left}
    int32_t* dcpre;              // its members' chosen-count prefix (n_clouds+1)
    int32_t dec_smem_max;        // points whose counts fit the decimation's shared memory
    int32_t dec_nb_pp;           // neighbour-list entries per scratch slot
    int32_t dec_dyn;             // bytes of the decimation's dynamic shared memory
    const int64_t* dec_hoff;     // per group: start of its bucket arrays
    const int32_t* dec_hbits;    // per group: log2 buckets
    int32_t n_clouds;
    int32_t n_groups;
    int32_t n_chunks;
    int32_t n_slots;
    int32_t n_kblk;              // blocks of KBLK chosen slots, clouds scanned by CTAs
    int32_t n_kblk_warp;         // the same over the other clouds
    int32_t chunk_pts;           // max points per assignment chunk (BLOCK*ITEMS)
    int32_t chunk_max;           // largest chunk actually used (scatter staging)
    int32_t hist_smem;           // ints of dynamic smem for the assign histogram
    int32_t scat_smem;           // ints of dynamic smem per scatter warp
    int32_t max_passes;
    int32_t max_outer;
    int32_t max_iters;
    int32_t n_sms;
    int32_t flags;               // ENG_* run-mode bits
    int32_t single;              // a run of one cloud: cl[0] is also here
    CloudDesc one;
    // exact chunk-box culling of the assignment (see k_assign_cull)
    const float* Ps;             // evolve points in spatial order inside each cloud
    const int32_t* sorder;       // spatial position -> packed point slot
    const int32_t* srow;         // spatial position -> its slot's chunk in the cloud (histogram row)
    int32_t* ksp;                // spatial position -> its point's key (as keys holds it by slot)
    const float* bbox;           // per block of 32 x cull_items spatial positions: two boxes (lo, hi)
    float* bslack;               // per block: moves that leave its keys as they are (see k_assign_cull)
    float* lslack;               // per block: moves that leave its candidate list complete
    int32_t* blen;               // per block: entries of its candidate list
    int32_t* blist;              // per block: the list (CAND_MAX entries)
    int32_t* full;               // per cloud: the next pass evaluates every block and every key
    int32_t* mvn;                // per cloud: chosen points moved in the last pass
    int32_t* dmax;               // per cloud: bits of the longest of those moves
    float* mv;                   // 2*DIM+1 arrays of n_slots: each cloud's moves at its key_off
                                 // (old place, new place, length rounded up)
    int32_t cull;                // passes assign with k_assign_cull
    int32_t lists;               // and keep member lists, candidates and slacks from pass to pass
                                 // (else every pass evaluates and regroups every point)
    int64_t hist_ints;           // entries of hist
    int64_t n_points;
    int32_t long_lists;          // few chosen points: k_merge_fold's variant for long lists
    int32_t merge_cap;           // a key with a region this large regroups its cloud when edited
    // fused tiled runs: tiles by decreasing evolve points, the first n_heavy
    // evolved by whole thread-block clusters (rd_tile_cluster.cuh)
    const int32_t* tile_order;
    int32_t n_heavy;
    int32_t tile_clusters;       // the cluster kernel runs
    int32_t tile_hand;           // and hands over light tiles
    int32_t tile_cl_grid;        // CTAs of the cluster tile kernel (0 = one-CTA kernel)
    int32_t tile_seg_min;        // members of a key the cluster folds in segments
};

// dynamic shared memory of the decimation kernel's list path: two int16 counts
// and an alive byte per point, then a candidate bit per point; the bit-matrix
// path lays it out as rd_decbits.cuh describes
inline int dec_list_bytes(int points) { return ((points * 5 + 15) / 16) * 16 + 4 * ((points + 31) / 32) + 16; }
constexpr int DEC_BITS_MAX = 4096;           // points decimated over bit matrices
constexpr int DEC_BITS_SMEM = 200 * 1024;    // shared memory for them
// most dynamic shared memory of the decimation: the matrices, or the counts and flags
// of DEC_SMEM_MAX_POINTS points (dec_list_bytes)
constexpr int DEC_SMEM_MOST = DEC_BITS_SMEM;
static_assert(DEC_SMEM_MAX_POINTS * 5 + 16 + DEC_SMEM_MAX_POINTS / 8 + 32 <= DEC_SMEM_MOST, "decimation smem");
constexpr int DEC_SAMPLES = 32;              // points sampled for the choice between them and lists
inline int dec_smem_bytes(const EngineView& v) { return v.dec_dyn; }
// bytes for groups of up to `points` points
int dec_dyn_bytes(int points);
// largest set whose bit matrices that includes
int dec_smem_points();

// points of an assignment chunk (block x items), and the most ints of shared memory for
// a chunk's key histogram and a scatter warp's key starts
constexpr int CHUNK_PTS_MAX = 2048, HIST_SMEM_MAX = 24 * 1024, SCAT_SMEM_MAX = 4 * 1024;

// launch configuration picked by the tuner per (dim, cloud size, r1) bucket
struct TuneParams {
    int block;          // assign CTA size (all-pairs kernel); with items, the chunk size
    int items;          // points per assign thread
    int cull_items = 4; // culled kernel: points per lane (a warp's box holds 32 x this)
};

// host-side launchers (rd_kernels.cu); all enqueue on `st`
cudaError_t launch_choose(int dim, const EngineView& v, cudaStream_t st);
// the settings of the cluster path of fused tiled runs (process-wide, read when a
// run starts; rd_tile_rule.hpp)
TileClusterParams tile_cluster_params();
void set_tile_cluster_params(const TileClusterParams& p);
// choose of one large cloud c (n own points) in GPU-wide rounds; v.hash must
// hold choose_hash_buckets() ints and surv n bytes
cudaError_t launch_choose_rounds(int dim, const EngineView& v, int c, int n, uint8_t* surv,
                                 int32_t* sel, void* tmp, size_t tmp_bytes, cudaStream_t st);
// scratch of the survivor compaction of launch_choose_rounds for n points;
// sel holds n + 1 ints (the list, then its length)
size_t choose_select_scratch_bytes(int64_t n);
int choose_hash_buckets();
cudaError_t prepare_pass(int dim, const EngineView& v, const TuneParams& tp);
// How an iteration ends: the last CTA of its decimation kernel rebuilds the
// work lists and sets the loop condition (k_loopcond's step), leaving the
// count of unfinished clouds in ctr[CTR_ACTIVE] and, with use_handle, setting
// the graph WHILE handle.
struct LoopCond {
    cudaGraphConditionalHandle h = 0;
    int use_handle = 0;
};
// One iteration: evolve pass, control, decimation, loop condition.  a0/a1
// (optional) are recorded on `st` right before and after the assign kernel.
// follows_pass: the kernel before on `st` is the last one of such an iteration.
cudaError_t launch_pass(int dim, const EngineView& v, const TuneParams& tp, int assign_grid,
                        const LoopCond& lc, cudaStream_t st, cudaEvent_t a0 = nullptr,
                        cudaEvent_t a1 = nullptr, bool follows_pass = false);
// Sets the loop condition and rebuilds the work lists of the next iteration
// as a kernel of its own (count_iter = 0 for the initial build before the
// first iteration).
cudaError_t launch_loopcond(const EngineView& v, cudaGraphConditionalHandle h, int use_handle,
                            cudaStream_t st, int count_iter = 1);
cudaError_t launch_reset(const EngineView& v, cudaStream_t st);
// phases from the chosen counts already in v.ns (evolve or decimate from a given set)
cudaError_t launch_set_given(const EngineView& v, int queue_decimation, cudaStream_t st);
// fused per-tile evolve (every active cloud to convergence, one CTA each) +
// decimation of the groups that became ready; needs every ns <= TILE_NS_MAX
cudaError_t prepare_tile_pass(int dim, const EngineView& v, int* cl_grid);
// a0/a1 (optional) are recorded right before and after the tile-evolve kernel;
// the iteration ends with the loop condition as in launch_pass
cudaError_t launch_tile_pass(int dim, const EngineView& v, const LoopCond& lc, cudaStream_t st,
                             cudaEvent_t a0 = nullptr, cudaEvent_t a1 = nullptr);
// points: of the largest group
cudaError_t launch_decimate(int dim, const EngineView& v, int64_t points, cudaStream_t st);
// quality metrics (rd_quality.cu)
cudaError_t launch_min_dist(int dim, const float* A, int na, const float* B, int nb, float* out,
                            cudaStream_t st);
cudaError_t launch_axis_dist(int dim, const float* T, int n, float* out, cudaStream_t st);
cudaError_t launch_max2(const float* a, int na, const float* b, int nb, float* out, cudaStream_t st);
cudaError_t launch_dist_stats(float* d, int n, float* sorted, int32_t* iota, void* temp,
                              size_t temp_bytes, float* out, cudaStream_t st);
size_t dist_stats_temp_bytes(int n);
// chains of a ridge (rd_order.cu): alive ns bytes, deq 2*ns+1 ints of scratch;
// order ns ints, chain_start ns+1 ints, n_chains one int (all device)
cudaError_t launch_order_chains(int dim, const float* S, int ns, float rsq, unsigned char* alive,
                                int32_t* deq, int32_t* order, int32_t* chain_start,
                                int32_t* n_chains, cudaStream_t st);
// out[d] = ordered FP32 sum of P[idx[i]*dim + d] (method 0 chain, 1 parallel exact)
cudaError_t launch_ordered_sum(int dim, const float* P, const int32_t* idx, int n, float* out,
                               int method, cudaStream_t st);
// Spatial order of every cloud's points for the culled assignment: cells of
// edge r1/4, Morton order of the cells (cloud first), slot order inside a
// cell; Ps/sorder receive the reordered points and their slots.  Needs
// contiguous clouds in cloud order and n_points < 2^31; scratch of
// spatial_prep_scratch_bytes(n).
size_t spatial_prep_scratch_bytes(int64_t n_points);
// Also writes the boxes of the blocks of 32 x items positions and clears keys
// and ksp.
cudaError_t launch_spatial_prep(int dim, const EngineView& v, int items, int64_t n_points,
                                void* scratch, size_t scratch_bytes, float* Ps, int32_t* sorder,
                                float* bbox, cudaStream_t st);
// the kernels of one evolve pass without control and decimation (adjoint
// forward), again and again over the work lists of one launch_loopcond
cudaError_t launch_evolve_step(int dim, const EngineView& v, const TuneParams& tp, int assign_grid,
                               cudaStream_t st);
// points per chosen point from which a run takes the variant for long lists
int long_list_avg();
int merge_cap(bool long_lists);   // EngineView::merge_cap
int assign_smem_bytes(int dim, const TuneParams& tp, int hist_ints);
int max_assign_blocks_per_sm(int dim, const TuneParams& tp, int hist_ints);
bool tune_supported(int dim, const TuneParams& tp);

}  // namespace rdb
