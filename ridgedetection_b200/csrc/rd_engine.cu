// rd_engine.cu -- host side of the batch engine (see rd_engine_host.hpp).
#include "rd_engine_host.hpp"

#include <algorithm>
#include <cmath>
#include <tuple>
#include <atomic>
#include <cstring>
#include <map>
#include <mutex>

namespace rdb {

// ---------------------------------------------------------------------------
// tuning table
// ---------------------------------------------------------------------------
namespace {
std::mutex g_tune_mu;
// (dim, size bucket, r1 bucket) -> shape; r1 bucket TUNE_ANY_R1 = any radius
std::map<std::tuple<int, int, int>, TuneParams> g_tune;
}  // namespace

int tune_bucket(int64_t n)
{
    int b = 0;
    while (b < 62 && (int64_t(1) << (b + 1)) <= std::max<int64_t>(n, 1)) ++b;
    return b;
}

int tune_r1_bucket(float r1)
{
    if (!(r1 > 0.0f) || !(r1 < INFINITY)) return TUNE_ANY_R1;
    const double b = std::floor(2.0 * std::log2((double)r1));   // half octaves
    return (int)std::max(-256.0, std::min(256.0, b));
}

TuneParams tune_lookup(int dim, int64_t n, float r1)
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    const int nb = tune_bucket(n), rb = tune_r1_bucket(r1);
    auto it = g_tune.find({dim, nb, rb});
    if (it != g_tune.end()) return it->second;
    it = g_tune.find({dim, nb, TUNE_ANY_R1});
    if (it != g_tune.end()) return it->second;
    // the nearest radius bucket tuned for this dimension and size
    const TuneParams* best = nullptr;
    int bd = 1 << 30;
    for (const auto& kv : g_tune) {
        if (std::get<0>(kv.first) != dim || std::get<1>(kv.first) != nb) continue;
        const int d = std::abs(std::get<2>(kv.first) - rb);
        if (d < bd) { bd = d; best = &kv.second; }
    }
    return best ? *best : TuneParams{128, 8, 4};
}

bool tune_find_exact(int dim, int64_t n, float r1, TuneParams* out)
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto it = g_tune.find({dim, tune_bucket(n), tune_r1_bucket(r1)});
    if (it == g_tune.end()) return false;
    *out = it->second;
    return true;
}

void tune_store(int dim, int64_t n, float r1, const TuneParams& tp)
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune[{dim, tune_bucket(n), tune_r1_bucket(r1)}] = tp;
}

void tune_clear()
{
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune.clear();
}

const std::vector<TuneParams>& tune_candidates(bool culled)
{
    static const std::vector<TuneParams> all_pairs = {
        {128, 4, 4}, {128, 8, 4}, {128, 16, 4}, {256, 4, 4}, {256, 8, 4}};
    static const std::vector<TuneParams> cull = [] {
        std::vector<TuneParams> c;
        for (const TuneParams& s : all_pairs)
            for (int ci : {2, 4, 8}) c.push_back(TuneParams{s.block, s.items, ci});
        return c;
    }();
    return culled ? cull : all_pairs;
}


static std::atomic<int> g_assign_cull{1};
void set_assign_cull(bool on) { g_assign_cull.store(on ? 1 : 0); }
bool assign_cull_enabled() { return g_assign_cull.load() != 0; }

namespace {
thread_local DevArena* t_arena = nullptr;
std::atomic<uint64_t> g_arena_gen{1};
constexpr size_t ARENA_ALIGN = 256;
}  // namespace

DevArena* current_arena() { return t_arena; }

ArenaScope::ArenaScope(DevArena* a) : prev(t_arena)
{
    a->gen = g_arena_gen.fetch_add(1);
    t_arena = a;
}

ArenaScope::~ArenaScope() { t_arena = prev; }

cudaError_t DevBuf::ensure(size_t want)
{
    if (want == 0) want = 16;
    if (DevArena* a = t_arena) {
        if (borrowed && gen == a->gen && want <= bytes) return cudaSuccess;
        release();
        const size_t off = (a->used + ARENA_ALIGN - 1) / ARENA_ALIGN * ARENA_ALIGN;
        if (!a->measuring() && (off > a->cap || want > a->cap - off)) {
            a->exhausted = true;
            return cudaErrorMemoryAllocation;
        }
        // a measuring arena hands out distinct, aligned placeholders
        p = a->measuring() ? reinterpret_cast<void*>(uintptr_t(ARENA_ALIGN) + off) : a->base + off;
        a->used = off + want;
        bytes = want;
        borrowed = true;
        gen = a->gen;
        return cudaSuccess;
    }
    if (want <= bytes && (!borrowed || in_slab)) return cudaSuccess;
    release();
    cudaError_t e = cudaMalloc(&p, want);
    if (e != cudaSuccess) {
        p = nullptr;
        bytes = 0;
        return e;
    }
    bytes = want;
    return cudaSuccess;
}

void DevBuf::release()
{
    if (p && !borrowed) cudaFree(p);
    p = nullptr;
    bytes = 0;
    borrowed = in_slab = false;
}

cudaError_t ensure_together(DevBuf& slab, const std::vector<SlabItem>& items)
{
    cudaError_t e = cudaSuccess;
    if (t_arena) {
        for (const SlabItem& it : items)
            if ((e = it.buf->ensure(it.bytes)) != cudaSuccess) return e;
        return cudaSuccess;
    }
    bool fits = true;
    for (const SlabItem& it : items) {
        const bool own = it.buf->p && !it.buf->borrowed;
        if (it.bytes > SLAB_ITEM_MAX || (own && it.buf->bytes >= it.bytes)) {
            if (it.buf->in_slab) it.buf->release();
            if ((e = it.buf->ensure(it.bytes)) != cudaSuccess) return e;
        } else {
            if (own) it.buf->release();
            fits = fits && it.buf->in_slab && it.buf->bytes >= std::max<size_t>(it.bytes, 1);
        }
    }
    if (fits) return cudaSuccess;
    // the second try is for exactly what is asked
    const bool first = slab.p == nullptr;
    for (int exact = first ? 1 : 0; exact < 2; ++exact) {
        std::vector<size_t> off(items.size()), len(items.size());
        size_t total = 0;
        for (size_t i = 0; i < items.size(); ++i) {
            const SlabItem& it = items[i];
            if (it.buf->p && !it.buf->borrowed) continue;   // has its own
            len[i] = std::max<size_t>(it.bytes, 16);
            if (!exact) {
                const size_t had = it.buf->in_slab ? it.buf->bytes : 0;
                len[i] = std::max(had, len[i] > had ? len[i] + len[i] / 8 : len[i]);
            }
            total = (total + ARENA_ALIGN - 1) / ARENA_ALIGN * ARENA_ALIGN;
            off[i] = total;
            total += len[i];
        }
        slab.release();
        if (exact)
            for (const SlabItem& it : items)
                if (it.buf->borrowed) it.buf->release();
        if ((e = slab.ensure(total)) != cudaSuccess) {
            if (!exact) (void)cudaGetLastError();
            continue;
        }
        for (size_t i = 0; i < items.size(); ++i) {
            if (!len[i]) continue;
            DevBuf& b = *items[i].buf;
            b.release();
            b.p = static_cast<char*>(slab.p) + off[i];
            b.bytes = len[i];
            b.borrowed = b.in_slab = true;
        }
        return cudaSuccess;
    }
    return e;
}

Engine::Engine() {}

Engine::~Engine()
{
    if (exec_) cudaGraphExecDestroy(exec_);
    if (graph_) cudaGraphDestroy(graph_);
    if (cap_stream_) cudaStreamDestroy(cap_stream_);
}

int Engine::fail(const char* what, cudaError_t e)
{
    last_error = std::string(what) + ": " + cudaGetErrorString(e);
    return 2;  // RD_ERR_CUDA
}

#define RD_CK(call)                                   \
    do {                                              \
        cudaError_t e_ = (call);                      \
        if (e_ != cudaSuccess) return fail(#call, e_); \
    } while (0)

template <class T>
static cudaError_t upload(DevBuf& b, const std::vector<T>& h, cudaStream_t st)
{
    cudaError_t e = b.ensure(sizeof(T) * (h.size() + 1));
    if (e != cudaSuccess || h.empty()) return e;
    if (DevArena* a = current_arena(); a && a->measuring()) return cudaSuccess;
    return cudaMemcpyAsync(b.p, h.data(), sizeof(T) * h.size(), cudaMemcpyHostToDevice, st);
}

// n zero bytes (nothing to do while only sizes are planned)
static cudaError_t upload_zero(DevBuf& b, size_t n, cudaStream_t st)
{
    if (DevArena* a = current_arena(); a && a->measuring()) return cudaSuccess;
    return cudaMemsetAsync(b.p, 0, n, st);
}

int Engine::setup(int dim, const std::vector<CloudDesc>& clouds,
                  const std::vector<GroupDesc>& groups, int64_t total_points)
{
    if (!dim_supported(dim)) {
        last_error = "dim must be 1 to 4";
        return 6;  // RD_ERR_UNSUPPORTED
    }
    if (!tune_locked) {
        int64_t nmax = 1;
        float r1 = 0.0f;
        for (const CloudDesc& cd : clouds)
            if (cd.n_all >= nmax) {
                nmax = std::max<int64_t>(nmax, cd.n_all);
                r1 = cd.r1;
            }
        tune = tune_lookup(dim, nmax, r1);
    }
    if (!tune_supported(dim, tune)) {
        last_error = "unsupported tuning parameters";
        return 1;
    }
    dim_ = dim;
    total_points_ = total_points;
    h_cl_ = clouds;
    h_gr_ = groups;
    chunk_pts_ = tune.block * tune.items;
    int dev = 0;
    RD_CK(cudaGetDevice(&dev));
    RD_CK(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev));
    // Chunks split every cloud evenly into at most chunk_pts_ points each.  A
    // cloud big enough to fill the GPU on its own gets a multiple of the SM
    // count, so that the single wave of assignment CTAs is balanced.
    int64_t chunk = 0, s_off = 0;
    chunk_max_ = 0;
    h_chunk_cloud_.clear();
    for (size_t c = 0; c < h_cl_.size(); ++c) {
        CloudDesc& cd = h_cl_[c];
        cd.s_off = s_off;
        s_off += cd.n_own;
        cd.chunk_begin = chunk;
        int64_t nch = (cd.n_all + chunk_pts_ - 1) / chunk_pts_;
        if (h_cl_.size() == 1 && nch >= 2 * sms_) nch = (nch + sms_ - 1) / sms_ * sms_;
        cd.n_chunks = (int32_t)nch;
        if (nch > 0)
            chunk_max_ = std::max<int>(chunk_max_, (int)((cd.n_all + nch - 1) / nch));
        for (int k = 0; k < cd.n_chunks; ++k) h_chunk_cloud_.push_back((int32_t)c);
        chunk += cd.n_chunks;
    }
    n_chunks_ = (int32_t)chunk;
    const size_t nc = h_cl_.size();
    // the spatial order sorts by (cloud, cell): clouds must tile [0, total)
    // in cloud order
    spatial_ok_ = total_points < (int64_t(1) << 31) - 1;
    int64_t next_off = 0;
    for (const CloudDesc& cd : h_cl_) {
        spatial_ok_ = spatial_ok_ && cd.p_off == next_off;
        next_off += cd.n_all;
    }
    spatial_ok_ = spatial_ok_ && next_off == total_points;
    const size_t per = 4 * (nc + 1), per_group = 4 * (h_gr_.size() + 1);
    RD_CK(ensure_together(slab_setup_, {
        {&bRes_, res_bytes(nc)}, {&bPhase_, per}, {&bCont_, per}, {&bPasses_, per}, {&bOuter_, per},
        {&bKbDone_, per}, {&bFull_, per}, {&bReb_, per}, {&bRebNext_, per}, {&bMvn_, per},
        {&bDmax_, per}, {&bActCloud_, per}, {&bActPre_, ACT_KINDS * per}, {&bGroupConv_, per_group},
        {&bReady_, per_group}, {&bDbig_, 4 * 4}, {&bDcpre_, per},
        {&bCl_, sizeof(CloudDesc) * (nc + 1)}, {&bGr_, sizeof(GroupDesc) * (h_gr_.size() + 1)},
        {&bTileOrder_, per}, {&bChunkCloud_, 4 * (h_chunk_cloud_.size() + 1)},
        {&bP_, sizeof(float) * (size_t)(total_points * dim + 4)},
        {&bS_, sizeof(float) * (size_t)(s_off * dim + 4)},
        {&bNext_, sizeof(int32_t) * (size_t)(s_off + 1)},
        {&bKeys_, sizeof(int32_t) * (size_t)(total_points + 1)},
    }));
    return 0;
}

EngineView Engine::view() const
{
    EngineView v;
    std::memset(&v, 0, sizeof(v));
    v.cl = bCl_.as<CloudDesc>();
    v.gr = bGr_.as<GroupDesc>();
    v.chunk_cloud = bChunkCloud_.as<int32_t>();
    v.slot_cloud = bSlotCloud_.as<int32_t>();
    v.P = bP_.as<float>();
    v.S = bS_.as<float>();
    v.keys = bKeys_.as<int32_t>();
    v.Pg = bPg_.as<float>();
    v.hist = bHist_.as<int32_t>();
    v.hpre = lists_ ? bHpre_.as<int32_t>() : bHist_.as<int32_t>();
    v.cnt = bCnt_.as<int32_t>();
    v.base = bBase_.as<int32_t>();
    for (int b = 0; b < 2; ++b) {
        // otherwise the points are regrouped in every pass
        v.Lr[b] = lists_ ? bLr_[b].as<float>() : bPg_.as<float>();
        v.Ls[b] = lists_ ? bLs_[b].as<int32_t>() : nullptr;
    }
    v.kinfo = bKinfo_.as<int4>();
    v.edit = bEdit_.as<int32_t>();
    v.ecnt = bEcnt_.as<int32_t>();
    v.dlist = bDlist_.as<int32_t>();
    v.reb = bReb_.as<int32_t>();
    v.rebnext = bRebNext_.as<int32_t>();
    v.kbdone = bKbDone_.as<int32_t>();
    v.next = bNext_.as<int32_t>();
    v.hash = bHash_.as<int32_t>();
    // what collect() reads back, in one piece (res_bytes)
    const size_t nr = h_cl_.size() + 1;
    v.pairs = bRes_.as<unsigned long long>();
    v.ns = reinterpret_cast<int32_t*>(v.pairs + nr);
    v.total_passes = v.ns + nr;
    v.err = v.total_passes + nr;
    v.ctr = v.err + nr;
    v.phase = bPhase_.as<int32_t>();
    v.cont = bCont_.as<int32_t>();
    v.passes = bPasses_.as<int32_t>();
    v.outer = bOuter_.as<int32_t>();
    v.act_cloud = bActCloud_.as<int32_t>();
    v.act_pre = bActPre_.as<int32_t>();
    v.group_conv = bGroupConv_.as<int32_t>();
    v.ready = bReady_.as<int32_t>();
    v.dx = bDx_.as<float>();
    v.dcell = bDcell_.as<int32_t>();
    v.dalive = bDalive_.as<int32_t>();
    v.dc1 = bDc1_.as<int32_t>();
    v.dc2 = bDc2_.as<int32_t>();
    v.dbstart = bDbstart_.as<int32_t>();
    v.ditems = bDitems_.as<int32_t>();
    v.dnb_off = bDnbOff_.as<int32_t>();
    v.dnb = bDnb_.as<int32_t>();
    v.dbig = bDbig_.as<int32_t>();
    v.dcpre = bDcpre_.as<int32_t>();
    v.dec_smem_max = dec_smem_max_;
    v.dec_dyn = dec_dyn_;
    v.dec_nb_pp = dec_nb_pp_;
    v.dec_hoff = bDecHoff_.as<int64_t>();
    v.dec_hbits = bDecHbits_.as<int32_t>();
    v.n_clouds = (int32_t)h_cl_.size();
    v.n_groups = (int32_t)h_gr_.size();
    v.n_chunks = n_chunks_;
    v.n_slots = n_slots_;
    v.n_kblk = n_kblk_;
    v.n_kblk_warp = n_kblk_warp_;
    v.chunk_pts = chunk_pts_;
    v.chunk_max = chunk_max_;
    v.hist_smem = hist_smem_;
    v.scat_smem = scat_smem_;
    v.max_passes = max_passes;
    v.max_outer = max_outer;
    v.max_iters = max_iters;
    v.Ps = bPs_.as<float>();
    v.sorder = bSorder_.as<int32_t>();
    v.srow = bSorder_.as<int32_t>() + total_points_;  // second half of the same buffer
    v.ksp = bKsp_.as<int32_t>();
    v.bbox = bBox_.as<float>();
    v.bslack = bSlack_.as<float>();
    v.lslack = bLslack_.as<float>();
    v.blen = bBlen_.as<int32_t>();
    v.blist = bBlist_.as<int32_t>();
    v.full = bFull_.as<int32_t>();
    v.mvn = bMvn_.as<int32_t>();
    v.dmax = bDmax_.as<int32_t>();
    v.mv = bMv_.as<float>();
    v.cull = cull_ ? 1 : 0;
    v.lists = lists_ ? 1 : 0;
    v.hist_ints = hist_ints_;
    v.n_points = total_points_;
    v.long_lists = n_slots_ > 0 && total_points_ / n_slots_ >= long_list_avg() ? 1 : 0;
    v.merge_cap = merge_cap(v.long_lists != 0);
    v.tile_order = bTileOrder_.as<int32_t>();
    v.n_heavy = n_heavy_;
    v.tile_clusters = tile_clusters_ ? 1 : 0;
    v.tile_hand = tile_hand_ ? 1 : 0;
    v.tile_cl_grid = tile_cl_grid_;
    v.tile_seg_min = tile_seg_min_;
    v.n_sms = sms_;
    v.flags = flags_;
    v.single = h_cl_.size() == 1 ? 1 : 0;
    if (v.single) v.one = h_cl_[0];
    return v;
}

static int ceil_log2(int64_t x)
{
    int b = 0;
    while ((int64_t(1) << b) < x) ++b;
    return b;
}

// The chosen points a run of one cloud is laid out for: a few more than it has, and as
// many as the last one where that does, so that the clouds of a handle share their
// buffers and their graph.  Capturing and instantiating it anew takes about 0.4 ms
// (1,000 points, another cloud each time: 1.31 ms with exact counts, 0.92 with room).
int Engine::chosen_room(int ns)
{
    const CloudDesc& cd = h_cl_[0];
    int step = 64;
    while (8 * step <= ns) step *= 2;
    int64_t room = (int64_t)(ns + step - 1) / step * step;
    // the histogram has a row of them for every chunk
    if (4 * room * cd.n_chunks > int64_t(64) << 20 || current_arena()) return ns;
    if (room_points_ == cd.n_all && room_ >= ns && room_ <= 2 * room) return room_;
    room_points_ = cd.n_all;
    return room_ = (int)room;
}

int Engine::finish_setup_after_choose(cudaStream_t st, bool ns_given, bool exact)
{
    const size_t nc = h_cl_.size();
    h_ns_.resize(nc);
    if (DevArena* a = current_arena(); (a && a->measuring()) || ns_given) {
        // size planning: the counts the caller will give; or has given
        for (size_t c = 0; c < nc; ++c) h_ns_[c] = c < given_ns.size() ? given_ns[c] : h_cl_[c].n_own;
    } else {
        RD_CK(cudaMemcpyAsync(h_ns_.data(), view().ns, 4 * nc, cudaMemcpyDeviceToHost, st));
        RD_CK(cudaStreamSynchronize(st));
    }
    int64_t hist = 0, key = 0, kblk = 0, kblk_warp = 0;
    int max_ns = 0;
    h_slot_cloud_.clear();
    for (size_t c = 0; c < nc; ++c) {
        CloudDesc& cd = h_cl_[c];
        cd.ns_cap = nc == 1 && !exact ? chosen_room(h_ns_[c]) : h_ns_[c];
        max_ns = std::max(max_ns, cd.ns_cap);
        cd.hist_off = hist;
        hist += (int64_t)cd.n_chunks * cd.ns_cap;
        cd.key_off = key;
        key += cd.ns_cap;
        (scan_by_cta(cd.n_chunks, cd.ns_cap) ? kblk : kblk_warp) += (cd.ns_cap + KBLK - 1) / KBLK;
        for (int k = 0; k < cd.ns_cap; ++k) h_slot_cloud_.push_back((int32_t)c);
    }
    n_slots_ = (int32_t)key;
    hist_ints_ = hist;
    lay_out_lists(cull_possible());
    n_kblk_ = (int32_t)kblk;
    n_kblk_warp_ = (int32_t)kblk_warp;
    // group decimation scratch
    h_dec_hoff_.resize(h_gr_.size());
    h_dec_hbits_.resize(h_gr_.size());
    int64_t sscr = 0, hoff = 0, max_tot = 0;
    for (size_t g = 0; g < h_gr_.size(); ++g) {
        GroupDesc& gd = h_gr_[g];
        int64_t tot = 0;
        for (int i = 0; i < gd.n_clouds; ++i) tot += h_cl_[gd.cloud_begin + i].ns_cap;
        gd.s_scratch = sscr;
        gd.s_cap = (int32_t)tot;
        sscr += tot;
        max_tot = std::max(max_tot, tot);
        const int hb = std::min(20, std::max(6, ceil_log2(std::max<int64_t>(tot, 1))));
        h_dec_hbits_[g] = hb;
        h_dec_hoff_[g] = hoff;
        hoff += (int64_t(1) << hb) + 1;
    }
    // shared-memory budgets (ints)
    hist_smem_ = std::min(max_ns, HIST_SMEM_MAX);
    scat_smem_ = std::min(max_ns, SCAT_SMEM_MAX);
    dec_nb_pp_ = (int)std::max<int64_t>(
        DEC_NB_MIN_PER_POINT,
        std::min({(int64_t)DEC_NB_MAX_PER_POINT, DEC_NB_BUDGET / std::max<int64_t>(sscr, 1), max_tot}));
    const size_t slots = (size_t)key + 1, scr = (size_t)sscr + 1;
    RD_CK(ensure_together(slab_chosen_, {
        {&bSlotCloud_, 4 * (h_slot_cloud_.size() + 1)},
        {&bDecHoff_, 8 * (h_dec_hoff_.size() + 1)}, {&bDecHbits_, 4 * (h_dec_hbits_.size() + 1)},
        {&bHist_, 4 * (size_t)(hist + 1)},
        {&bCnt_, 4 * slots}, {&bBase_, 4 * slots}, {&bKinfo_, sizeof(int4) * slots},
        {&bEcnt_, 4 * slots}, {&bDlist_, 4 * slots},
        {&bDx_, 4 * scr * dim_}, {&bDcell_, 4 * scr * dim_}, {&bDalive_, 4 * scr},
        {&bDc1_, 4 * scr}, {&bDc2_, 4 * scr}, {&bDitems_, 4 * scr},
        {&bDbstart_, 4 * (size_t)(hoff + 1)},
        {&bDnbOff_, 4 * (size_t)(sscr + h_gr_.size() + 1)},
        {&bDnb_, 4 * (size_t)((int64_t)dec_nb_pp_ * sscr + 1)},
    }));
    RD_CK(upload(bCl_, h_cl_, st));
    RD_CK(upload(bGr_, h_gr_, st));
    RD_CK(upload(bSlotCloud_, h_slot_cloud_, st));
    RD_CK(upload(bDecHoff_, h_dec_hoff_, st));
    RD_CK(upload(bDecHbits_, h_dec_hbits_, st));
    RD_CK(upload_zero(bEcnt_, 4 * (size_t)(key + 1), st));
    dec_smem_max_ = (int)std::min<int64_t>(max_tot, DEC_SMEM_MAX_POINTS);
    // where a room beyond the count would leave the sets whose matrices fit, the largest
    // of those
    dec_dyn_ = dec_dyn_bytes(h_gr_.size() == 1 && nc == 1 && h_ns_[0] <= dec_smem_points()
                                 ? std::min(dec_smem_max_, dec_smem_points()) : dec_smem_max_);
    // persistent assignment grid: every resident CTA slot, at most one per chunk
    int dev = 0, sms = 0;
    RD_CK(cudaGetDevice(&dev));
    RD_CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const int per_sm = std::max(1, max_assign_blocks_per_sm(dim_, tune, hist_smem_));
    assign_grid_ = std::max(1, std::min(n_chunks_, sms * per_sm));
    return 0;
}

int Engine::build_graph(cudaStream_t st)
{
    (void)st;
    const EngineView v = view();
    std::vector<unsigned char> key(sizeof(v) + sizeof(TuneParams) + 2 * sizeof(int));
    const int fz = fused_ ? 1 : 0;
    std::memcpy(key.data(), &v, sizeof(v));
    std::memcpy(key.data() + sizeof(v), &tune, sizeof(TuneParams));
    std::memcpy(key.data() + sizeof(v) + sizeof(TuneParams), &assign_grid_, sizeof(int));
    std::memcpy(key.data() + sizeof(v) + sizeof(TuneParams) + sizeof(int), &fz, sizeof(int));
    if (exec_ && key == graph_key_) return 0;
    if (exec_) { cudaGraphExecDestroy(exec_); exec_ = nullptr; }
    if (graph_) { cudaGraphDestroy(graph_); graph_ = nullptr; }
    if (!cap_stream_) RD_CK(cudaStreamCreateWithFlags(&cap_stream_, cudaStreamNonBlocking));
    RD_CK(cudaGraphCreate(&graph_, 0));
    cudaGraphConditionalHandle h;
    RD_CK(cudaGraphConditionalHandleCreate(&h, graph_, 1, cudaGraphCondAssignDefault));
    alignas(cudaGraphNodeParams) unsigned char cp_raw[sizeof(cudaGraphNodeParams)];
    std::memset(cp_raw, 0, sizeof(cp_raw));
    cudaGraphNodeParams& cp = *reinterpret_cast<cudaGraphNodeParams*>(cp_raw);
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = h;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    cudaGraphNode_t node;
    RD_CK(cudaGraphAddNode(&node, graph_, nullptr, 0, &cp));
    cudaGraph_t body = cp.conditional.phGraph_out[0];
    RD_CK(cudaStreamBeginCaptureToGraph(cap_stream_, body, nullptr, nullptr, 0,
                                        cudaStreamCaptureModeThreadLocal));
    LoopCond lc;
    lc.h = h;
    lc.use_handle = 1;
    // One cloud: several passes per round of the WHILE node.  Inside a round a
    // pass's kernels follow the last one's as programmatic dependents; a new round
    // costs about as much as the pass's kernels do for a small cloud.  Passes
    // after the last one find empty work lists.  Solves, 1 / 4 passes a round, ms:
    // 1,000-point sine 0.97 / 0.90, 20,000 2.59 / 2.39, 77,777-point helix 7.25 / 6.66,
    // 1M helix 20.2 / 19.5; 8 a round: 0.91, 2.35, 6.58, 19.4.
    const int passes = (!fused_ && h_cl_.size() == 1 && n_slots_ > 0) ? 4 : 1;
    cudaError_t e1 = cudaSuccess;
    for (int p = 0; p < passes && e1 == cudaSuccess; ++p)
        e1 = fused_ ? launch_tile_pass(dim_, v, lc, cap_stream_)
                    : launch_pass(dim_, v, tune, assign_grid_, lc, cap_stream_, nullptr, nullptr, p > 0);
    cudaGraph_t out = nullptr;
    cudaError_t e3 = cudaStreamEndCapture(cap_stream_, &out);
    if (e1 != cudaSuccess || e3 != cudaSuccess) {
        graph_ = nullptr;   // half captured: left to the process, not destroyed
        return fail(e1 != cudaSuccess ? "capture pass" : "end capture", e1 != cudaSuccess ? e1 : e3);
    }
    RD_CK(cudaGraphInstantiate(&exec_, graph_, 0));
    graph_key_ = key;
    return 0;
}

// buffers of the choose of one large cloud
cudaError_t Engine::ensure_choose()
{
    const int64_t n = h_cl_[0].n_own;
    return ensure_together(slab_choose_, {{&bHash_, 4 * (size_t)choose_hash_buckets()},
                                          {&bSurv_, (size_t)n + 16},
                                          {&bSel_, 4 * (size_t)(n + 2)},
                                          {&bSelTmp_, choose_select_scratch_bytes(n)}});
}

int Engine::run(cudaStream_t st, bool use_graph, int mode)
{
    if (h_cl_.empty()) return 0;
    stats_ = RunStats();
    read_switches();
    flags_ = (mode == RUN_EVOLVE_ONLY) ? ENG_EVOLVE_ONLY : 0;
    RD_CK(upload(bCl_, h_cl_, st));
    RD_CK(upload(bGr_, h_gr_, st));
    RD_CK(upload(bChunkCloud_, h_chunk_cloud_, st));
    build_tile_order();
    RD_CK(upload(bTileOrder_, h_tile_order_, st));
    if (mode == RUN_EVOLVE_ONLY || mode == RUN_DECIMATE_ONLY) {
        // chosen sets supplied by the caller (given_ns, points already in S)
        if (given_ns.size() != h_cl_.size()) {
            last_error = "given chosen counts do not match the clouds";
            return 1;
        }
        for (size_t c = 0; c < h_cl_.size(); ++c)
            if (given_ns[c] < 0 || given_ns[c] > h_cl_[c].n_own) {
                last_error = "given chosen count exceeds the cloud's capacity";
                return 1;
            }
        EngineView v0 = view();
        RD_CK(launch_reset(v0, st));
        RD_CK(cudaMemcpyAsync(v0.ns, given_ns.data(), 4 * given_ns.size(),
                              cudaMemcpyHostToDevice, st));
        if (int rc = finish_setup_after_choose(st, true, mode == RUN_DECIMATE_ONLY)) return rc;
        const EngineView v1 = view();
        RD_CK(launch_set_given(v1, mode == RUN_DECIMATE_ONLY ? 1 : 0, st));
        if (mode == RUN_DECIMATE_ONLY) {
            int64_t points = 0;
            for (const GroupDesc& gd : h_gr_) points = std::max<int64_t>(points, gd.s_cap);
            RD_CK(launch_decimate(dim_, v1, points, st));
            return collect(st);
        }
    } else {
        // one large cloud: GPU-wide choose rounds; otherwise one CTA per cloud
        const bool rounds = h_cl_.size() == 1 && h_cl_[0].n_own >= (1 << 16);
        if (rounds) {
            RD_CK(ensure_choose());
        }
        EngineView v0 = view();
        RD_CK(launch_reset(v0, st));
        if (rounds)
            RD_CK(launch_choose_rounds(dim_, v0, 0, h_cl_[0].n_own, bSurv_.as<uint8_t>(),
                                       bSel_.as<int32_t>(), bSelTmp_.p, bSelTmp_.bytes, st));
        else
            RD_CK(launch_choose(dim_, v0, st));
        if (mode == RUN_CHOOSE_ONLY) {
            h_ns_.resize(h_cl_.size());
            RD_CK(cudaMemcpyAsync(h_ns_.data(), v0.ns, 4 * h_ns_.size(), cudaMemcpyDeviceToHost,
                                  st));
            RD_CK(cudaStreamSynchronize(st));
            return 0;
        }
        if (int rc = finish_setup_after_choose(st)) return rc;
    }
    // Tiled runs (one group of many clouds, every chosen set small enough)
    // evolve each tile to convergence inside one kernel; everything else runs
    // lockstep passes over all evolving clouds.
    int max_ns = 0;
    for (const CloudDesc& cd : h_cl_) max_ns = std::max(max_ns, cd.ns_cap);
    fused_ = fuse_tiles && h_gr_.size() == 1 && h_cl_.size() > 1 && max_ns <= TILE_NS_MAX &&
             flags_ == 0;
    cull_ = cull_possible() && !fused_;
    if (int rc = start_passes(st)) return rc;
    tile_cl_grid_ = 0;
    if (fused_) RD_CK(prepare_tile_pass(dim_, view(), &tile_cl_grid_));
    const EngineView v = view();
    RD_CK(prepare_pass(dim_, v, tune));
    // work lists of the first iteration
    RD_CK(launch_loopcond(v, cudaGraphConditionalHandle(), 0, st, 0));
    if (use_graph) {
        if (int rc = build_graph(st)) return rc;
        RD_CK(cudaGraphLaunch(exec_, st));
    } else {
        cudaEvent_t a0 = nullptr, a1 = nullptr;
        if (profile_assign || profile_pass) {
            RD_CK(cudaEventCreate(&a0));
            RD_CK(cudaEventCreate(&a1));
        }
        stats_.assign_ms = 0;
        stats_.assign_launches = 0;
        for (;;) {
            // profile_pass: the events bracket the whole iteration instead of
            // the assignment kernel
            cudaEvent_t k0 = profile_pass ? nullptr : a0, k1 = profile_pass ? nullptr : a1;
            if (profile_pass) RD_CK(cudaEventRecord(a0, st));
            const LoopCond lc;  // no handle: the count is read below
            if (fused_) RD_CK(launch_tile_pass(dim_, v, lc, st, k0, k1));
            else RD_CK(launch_pass(dim_, v, tune, assign_grid_, lc, st, k0, k1));
            if (profile_pass) RD_CK(cudaEventRecord(a1, st));
            int32_t act = 0;
            RD_CK(cudaMemcpyAsync(&act, v.ctr + CTR_ACTIVE, 4, cudaMemcpyDeviceToHost, st));
            RD_CK(cudaStreamSynchronize(st));
            if (a0) {
                float ms = 0;
                RD_CK(cudaEventElapsedTime(&ms, a0, a1));
                stats_.assign_ms += ms;
                stats_.assign_launches += 1;
            }
            if (act == 0) break;
        }
        if (a0) cudaEventDestroy(a0);
        if (a1) cudaEventDestroy(a1);
    }
    return collect(st);
}

// Where each cloud's grouped lists start.  With lists (keep), every key has a region
// with room to grow; otherwise a cloud's lists take its points' places.
void Engine::lay_out_lists(bool keep)
{
    lists_ = keep;
    for (const CloudDesc& cd : h_cl_) lists_ = lists_ && lists_possible(cd.n_all, cd.ns_cap);
    list_rows_ = 0;
    for (CloudDesc& cd : h_cl_) {
        cd.reg_off = list_rows_;
        list_rows_ += list_rows(cd.n_all, cd.ns_cap);
    }
    // A caller's scratch stays within LIST_WS_MAX of what it is without lists.
    if (current_arena() && list_bytes() > LIST_WS_MAX) lists_ = false;
    if (!lists_)
        for (CloudDesc& cd : h_cl_) cd.reg_off = cd.p_off;
}

int64_t Engine::list_bytes() const
{
    return list_rows_ * (2 * (pad_dim(dim_) * 4 + 4) + 4) + 4 * hist_ints_ +
           (int64_t)(2 * dim_ + 1) * 4 * n_slots_;
}

// buffers and state of the lockstep passes (cull_ is set)
int Engine::start_passes(cudaStream_t st)
{
    if (!cull_) lists_ = false;
    if (int rc = ensure_pass_buffers(st)) return rc;
    if (!cull_) return 0;
    const EngineView vs = view();
    RD_CK(launch_spatial_prep(dim_, vs, tune.cull_items, total_points_, bSpatialTmp_.p,
                              spatial_prep_scratch_bytes(total_points_), bPs_.as<float>(),
                              bSorder_.as<int32_t>(), bBox_.as<float>(), st));
    // no point has a key yet: with lists the assignment keeps the counts by its
    // changes
    RD_CK(cudaMemsetAsync(bHist_.p, 0, 4 * (size_t)(hist_ints_ + 1), st));
    return 0;
}

// Another thread may flip the switch at any time, and both the layout of the
// grouped lists (finish_setup_after_choose) and the choice of kernels and buffers
// follow from it: every run reads it once.
void Engine::read_switches()
{
    cull_on_ = cull_assign && assign_cull_enabled();
}

// whether the lockstep passes of this batch assign with culling
bool Engine::cull_possible() const
{
    return cull_on_ && spatial_ok_ && total_points_ > 0;
}

// blocks of points of the culled assignment
int64_t Engine::cull_blocks() const { return (int64_t)n_chunks_ * (chunk_pts_ / (32 * tune.cull_items)); }

// Buffers of the lockstep passes (sizes known after choose).  The kept lists take 25
// to 55 bytes a point and a second histogram more than regrouping in every pass does;
// where the device has no room for them the run goes without.
int Engine::ensure_pass_buffers(cudaStream_t st)
{
    const size_t n = (size_t)total_points_;
    const size_t blocks = (size_t)cull_blocks();
    if (cull_)
        RD_CK(ensure_together(slab_pass_, {
            {&bPs_, sizeof(float) * (n * pad_dim(dim_) + 4)},
            {&bSorder_, sizeof(int32_t) * (2 * n + 1)},
            {&bSpatialTmp_, spatial_prep_scratch_bytes(total_points_)},
            {&bBox_, sizeof(float) * (4 * dim_ * blocks + 1)},
            {&bSlack_, sizeof(float) * (blocks + 1)},
            {&bLslack_, sizeof(float) * (blocks + 1)},
            {&bBlen_, sizeof(int32_t) * (blocks + 1)},
            {&bKsp_, sizeof(int32_t) * (n + 1)},
            {&bBlist_, sizeof(int32_t) * (CAND_MAX * blocks + 1)},
        }));
    if (lists_) {
        const cudaError_t e = ensure_list_buffers();
        if (e == cudaErrorMemoryAllocation && !current_arena()) {
            (void)cudaGetLastError();
            for (DevBuf* b : {&bLr_[0], &bLr_[1], &bLs_[0], &bLs_[1], &bEdit_, &bHpre_, &bMv_, &slab_list_})
                b->release();
            lay_out_lists(false);
            RD_CK(upload(bCl_, h_cl_, st));
        } else if (e != cudaSuccess) {
            return fail("buffers of the member lists", e);
        }
    }
    if (!lists_) RD_CK(bPg_.ensure(sizeof(float) * (n * pad_dim(dim_) + 4)));
    return 0;
}

cudaError_t Engine::ensure_list_buffers()
{
    const size_t rows = (size_t)list_rows_;
    return ensure_together(slab_list_, {
        {&bHpre_, 4 * (size_t)(hist_ints_ + 1)},
        {&bLr_[0], sizeof(float) * (rows * pad_dim(dim_) + 4)},
        {&bLr_[1], sizeof(float) * (rows * pad_dim(dim_) + 4)},
        {&bLs_[0], sizeof(int32_t) * (rows + 1)},
        {&bLs_[1], sizeof(int32_t) * (rows + 1)},
        {&bEdit_, sizeof(int32_t) * (rows + 1)},
        {&bMv_, sizeof(float) * ((size_t)(2 * dim_ + 1) * n_slots_ + 1)},
    });
}

// Tiles (clouds) by decreasing evolve points; the heavy ones (evolved by a
// whole cluster in fused tiled runs) first.
void Engine::build_tile_order()
{
    const size_t nc = h_cl_.size();
    h_tile_order_.resize(nc);
    for (size_t c = 0; c < nc; ++c) h_tile_order_[c] = (int32_t)c;
    std::stable_sort(h_tile_order_.begin(), h_tile_order_.end(),
                     [&](int32_t a, int32_t b) { return h_cl_[a].n_all > h_cl_[b].n_all; });
    const TileRule rule = tile_rule(tile_cluster_params(), total_points_, sms_,
                                    nc > 1 ? h_cl_[h_tile_order_[0]].n_all : 0);
    tile_seg_min_ = rule.seg_min;
    tile_clusters_ = rule.clusters && nc > 1;
    tile_hand_ = rule.hand_over && nc > 1;
    n_heavy_ = 0;
    if (tile_clusters_)
        while (n_heavy_ < (int)nc && h_cl_[h_tile_order_[n_heavy_]].n_all >= rule.heavy) ++n_heavy_;
}

int Engine::plan_workspace(int mode)
{
    DevArena* a = current_arena();
    if (!a || !a->measuring()) {
        last_error = "workspace planning needs a measuring arena";
        return 1;
    }
    read_switches();
    // the buffers run() takes, in its order, for a single-cloud device step
    RD_CK(upload(bCl_, h_cl_, nullptr));
    RD_CK(upload(bGr_, h_gr_, nullptr));
    RD_CK(upload(bChunkCloud_, h_chunk_cloud_, nullptr));
    build_tile_order();
    RD_CK(upload(bTileOrder_, h_tile_order_, nullptr));
    if (mode == RUN_EVOLVE_ONLY || mode == RUN_DECIMATE_ONLY) {
        if (int rc = finish_setup_after_choose(nullptr, false, mode == RUN_DECIMATE_ONLY)) return rc;
        if (mode == RUN_EVOLVE_ONLY) {
            cull_ = cull_possible();
            if (int rc = ensure_pass_buffers(nullptr)) return rc;
        }
        return 0;
    }
    if (mode == RUN_CHOOSE_ONLY) {
        if (h_cl_.size() == 1 && h_cl_[0].n_own >= (1 << 16)) {
            RD_CK(ensure_choose());
        }
        return 0;
    }
    last_error = "workspace planning covers the choose, evolve and decimate steps only";
    return 1;
}

int Engine::adjoint_setup(cudaStream_t st)
{
    if (h_cl_.size() != 1 || given_ns.size() != 1) {
        last_error = "adjoint: one cloud with a given chosen set";
        return 1;
    }
    if (given_ns[0] < 1 || given_ns[0] > h_cl_[0].n_own) {
        last_error = "adjoint: chosen count out of range";
        return 1;
    }
    stats_ = RunStats();
    flags_ = ENG_ALWAYS_MOVE;
    fused_ = false;
    read_switches();
    cull_ = cull_possible();
    RD_CK(upload(bCl_, h_cl_, st));
    RD_CK(upload(bGr_, h_gr_, st));
    EngineView v0 = view();
    RD_CK(launch_reset(v0, st));
    RD_CK(cudaMemcpyAsync(v0.ns, given_ns.data(), 4, cudaMemcpyHostToDevice, st));
    RD_CK(upload(bChunkCloud_, h_chunk_cloud_, st));
    if (int rc = finish_setup_after_choose(st, true)) return rc;
    if (int rc = start_passes(st)) return rc;
    const EngineView v = view();
    RD_CK(launch_set_given(v, 0, st));
    RD_CK(prepare_pass(dim_, v, tune));
    RD_CK(launch_loopcond(v, cudaGraphConditionalHandle(), 0, st, 0));  // work lists and tickets
    return 0;
}

int Engine::adjoint_step(cudaStream_t st)
{
    const EngineView v = view();
    RD_CK(launch_evolve_step(dim_, v, tune, assign_grid_, st));
    return 0;
}

int Engine::adjoint_restart(cudaStream_t st)
{
    // any value but 0: the next pass evaluates and regroups everything
    RD_CK(cudaMemsetAsync(bFull_.p, 1, sizeof(int32_t), st));
    return 0;
}

int Engine::collect(cudaStream_t st)
{
    const size_t nc = h_cl_.size();
    // pairs, chosen counts, passes, errors and counters in one copy (five copies of
    // pageable memory cost about 15 us each)
    h_res_.resize((res_bytes(nc) + 7) / 8);
    RD_CK(cudaMemcpyAsync(h_res_.data(), bRes_.p, res_bytes(nc), cudaMemcpyDeviceToHost, st));
    RD_CK(cudaStreamSynchronize(st));
    const uint64_t* pr = h_res_.data();
    const int32_t* ns = reinterpret_cast<const int32_t*>(pr + nc + 1);
    const int32_t *tp = ns + nc + 1, *er = tp + nc + 1, *ctr = er + nc + 1;
    h_ns_.assign(ns, ns + nc);
    h_err_.assign(er, er + nc);
    stats_.loop_iters = ctr[CTR_ITERS];
    stats_.err_bits = ctr[CTR_ERR];
    stats_.handed_tiles = ctr[CTR_HANDED];
    stats_.dec_passes = ctr[CTR_DEC_PASSES];
    stats_.dec_rounds = ctr[CTR_DEC_ROUNDS];
    for (size_t c = 0; c < nc; ++c) {
        stats_.total_passes += tp[c];
        stats_.max_passes = std::max<int64_t>(stats_.max_passes, tp[c]);
        stats_.pairs += (double)pr[c];
        stats_.point_passes += (double)h_cl_[c].n_all * (double)tp[c];
        stats_.err_bits |= h_err_[c];
    }
    if (stats_.err_bits & (ERRB_EVOLVE_CAP | ERRB_OUTER_CAP | ERRB_DEC_CAP)) {
        last_error = "iteration limit reached before convergence";
        return 4;  // RD_ERR_NOT_CONVERGED
    }
    if (stats_.err_bits & ERRB_CAPACITY) {
        last_error = "device capacity exceeded";
        return 3;
    }
    return 0;
}

}  // namespace rdb
