// fused.cu -- host side of the one-launch refinement (fused_kernels.cuh): when
// it applies, its working memory, the launch, and the one-shot call of a small
// host graph.
#include <algorithm>
#include <chrono>
#include <cstring>
#include <new>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/rbsc.h"
#include "common.cuh"
#include "fused_kernels.cuh"
#include "deep_kernels.cuh"
#include "list_kernels.cuh"
#include "check_kernels.cuh"
#include "scan.cuh"
#include "internal.h"

using namespace rbsc;

namespace {

// Graphs that fit one block's shared memory (fused_fits_block) run there, the
// next larger ones on one cluster of 8 blocks, larger ones on the whole chip (us a refinement, cluster / chip: 3,000 nodes and 12,000 arcs
// 70 / 71, 8,000 and 32,000 76-97 / 72-84, 16,000 and 64,000 115-135 / 80-87).
constexpr uint32_t kClusterNodes = 8192;
constexpr uint64_t kClusterArcs = 1u << 15;
constexpr unsigned kClusterBlocks = 8;
// A host graph of at most this many bytes goes through one pinned staging
// buffer and one copy.
constexpr size_t kStageBytes = 256u << 10;
constexpr uint32_t kStageNodes = 16384;

bool default_knobs(const rbsc_opts& o)
{
    return o.relabel == RBSC_RELABEL_HASH && o.use_graph && o.persist_log2 == 0 && o.grid_per_sm == 0 && o.sig_kernel == 0 &&
           o.persist_bps == 0 && o.persist_sig == 0;
}

bool one_cluster(uint32_t n, uint64_t m) { return n <= kClusterNodes && m <= kClusterArcs; }

rbsc_status launch(rbsc_ctx* ctx, FusedArgs& a, const FusedLayout& l, bool block, cudaStream_t s)
{
    const bool cluster = one_cluster(a.n, a.m);
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = kFuThreads;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    if (block) {
        const void* k = a.wt ? (const void*)k_refine_block<true> : (const void*)k_refine_block<false>;
        EK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFuBlockSmem));
        cfg.gridDim = 1;
        cfg.dynamicSmemBytes = fused_block_smem(a, l);
        ++rbsc::launch_counter();
        EK(a.wt ? cudaLaunchKernelEx(&cfg, k_refine_block<true>, a, l) : cudaLaunchKernelEx(&cfg, k_refine_block<false>, a, l));
        return RBSC_OK;
    }
    if (cluster) {
        cfg.gridDim = kClusterBlocks;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = kClusterBlocks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
    } else {
        // one block per SM (1024 threads of 64 registers)
        cfg.gridDim = (unsigned)ctx->sm_count;
        at.id = cudaLaunchAttributeCooperative;
        at.val.cooperative = 1;
        EK(cudaMemsetAsync(a.w, 0, sizeof(FusedWords), s));
    }
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    ++rbsc::launch_counter();
    if (cluster) EK(a.wt ? cudaLaunchKernelEx(&cfg, k_refine_fused<kFuCluster, true>, a) : cudaLaunchKernelEx(&cfg, k_refine_fused<kFuCluster, false>, a));
    else EK(a.wt ? cudaLaunchKernelEx(&cfg, k_refine_fused<kFuGrid, true>, a) : cudaLaunchKernelEx(&cfg, k_refine_fused<kFuGrid, false>, a));
    return RBSC_OK;
}

// The rows are a CSR's.
bool rows_side_by_side(const FusedArgs& a) { return a.off_end == static_cast<const char*>(a.off) + (a.off64 ? 8 : 4); }

rbsc_status ensure_pinned(rbsc_ctx* ctx)
{
    if (!ctx->h_fused) EKS(host_alloc(ctx, &ctx->h_fused, sizeof(FusedResult)));
    return RBSC_OK;
}

void common_args(const rbsc_ctx* ctx, FusedArgs& a)
{
    a.res = static_cast<FusedResult*>(ctx->h_fused);  // page-locked, written by the kernel
    a.verify = ctx->opts.verify ? 1 : 0;
    a.seed = ctx->opts.seed;
    a.max_rounds = ctx->opts.max_rounds ? ctx->opts.max_rounds : a.n + 1u;
    a.hash_bits = ctx->opts.test_hash_bits < 0 ? 64u : (uint32_t)ctx->opts.test_hash_bits;
}

// When to look for a deep refinement: once the passes so far have cost about
// as much as the change to the work list does (us; a pass takes about 6 + 1 per
// 100,000 arcs and per 33,000 nodes, the change 150 + 1 per 20,000 arcs and per
// 3,000 nodes).
uint32_t deep_round(uint32_t n, uint64_t m)
{
    const double pass = 6.0 + (double)m / 100e3 + n / 33e3, change = 150.0 + (double)m / 20e3 + n / 3e3;
    return (uint32_t)std::max(6.0, change / pass);
}

// The passes after a launch that ended with kFuDeep, on a work list: the
// classes of its last two passes are in a.col.  Leaves the launch that
// confirms (or goes on, as it does when there is no memory for the list) in `a`.
rbsc_status deep_tail(rbsc_ctx* ctx, FusedArgs& a, cudaStream_t s)
{
    FusedResult& r = *static_cast<FusedResult*>(ctx->h_fused);
    const uint32_t n = a.n, passes = r.rounds - a.round0;
    uint32_t* col = a.col[passes & 1u];
    const uint32_t* old = a.col[(passes & 1u) ^ 1u];
    // a new id is a new class, and there are at most n classes; room for the
    // ids of one more pass keeps k_inc_passes' own bound from ever ending it
    const size_t slots = (size_t)1 << a.log2tab, ids = slots + n + kIncCap;
    Scratch sc(ctx);
    // zeroed together: class sizes, in-degrees, T stamps, largest parts, counters
    const size_t z_size = 0, z_deg = z_size + 4 * ids, z_flag = z_deg + 4 * (size_t)n, z_ctr = z_flag + 4 * (size_t)n,
                 z_best = (z_ctr + sizeof(IncCounters) + 255) & ~(size_t)255, z_bytes = z_best + 8 * slots;
    unsigned char* z = nullptr;
    unsigned long long *sig = nullptr, *S = nullptr;
    uint32_t *cursor = nullptr, *tsrc = nullptr, *colm = nullptr, *tlist = nullptr;
    uint64_t* twt = nullptr;
    unsigned char* tmp = nullptr;
    const auto room = [&]() {
        return sc.get(&z, z_bytes) == RBSC_OK && sc.get(&S, ids) == RBSC_OK && sc.get(&sig, n) == RBSC_OK && sc.get(&cursor, n) == RBSC_OK &&
               sc.get(&colm, n) == RBSC_OK && sc.get(&tlist, kIncCap) == RBSC_OK && sc.get(&tsrc, a.m) == RBSC_OK &&
               (!a.wt || sc.get(&twt, a.m) == RBSC_OK) && sc.get(&tmp, scan_temp_bytes<uint32_t>((uint64_t)n + 1) + 1024) == RBSC_OK;
    };
    a.start = col;
    a.validate = 0;
    if (!room()) {  // full passes to the end
        a.round0 = r.rounds;
        a.deep_round = 0;
        return RBSC_OK;
    }
    uint32_t* size = reinterpret_cast<uint32_t*>(z + z_size);
    uint32_t* deg = reinterpret_cast<uint32_t*>(z + z_deg);
    IncCounters* ctr = reinterpret_cast<IncCounters*>(z + z_ctr);
    unsigned long long* best = reinterpret_cast<unsigned long long*>(z + z_best);
    EK(cudaMemsetAsync(z, 0, z_bytes, s));
    EK(cudaMemsetAsync(S, 0xff, 8 * ids, s));
    const unsigned grid = (unsigned)ctx->sm_count * 8;
    const uint64_t salt = pass_salt1(a.seed, 0x40000000u + r.rounds);
    rbsc::launch_counter() += 5;
    k_inc_degrees<<<grid, 256, 0, s>>>(a, col, size, deg);
    EK((exclusive_scan<uint32_t, uint32_t>(deg, cursor, n, (uint32_t*)nullptr, tmp, s)));
    if (a.wt) k_inc_transpose<true><<<grid, 256, 0, s>>>(a, col, old, size, cursor, tsrc, twt, best);
    else k_inc_transpose<false><<<grid, 256, 0, s>>>(a, col, old, size, cursor, tsrc, twt, best);
    k_inc_mark<<<grid, 256, 0, s>>>(n, col, old, best, colm);
    if (a.wt) k_inc_sums<true><<<grid, 256, 0, s>>>(a, colm, size, salt, sig, S, tlist, ctr);
    else k_inc_sums<false><<<grid, 256, 0, s>>>(a, colm, size, salt, sig, S, tlist, ctr);
    IncArgs t{};
    t.col = col;
    t.sig = sig;
    t.S = S;
    t.size = size;
    t.tend = cursor;
    t.tsrc = tsrc;
    t.twt = twt;
    t.tflag = reinterpret_cast<uint32_t*>(z + z_flag);
    t.tlist = tlist;
    t.ctr = ctr;
    t.res = &r;
    t.salt = salt;
    t.first_id = (uint32_t)slots;
    t.end_id = (uint32_t)ids;
    t.round = r.rounds;
    t.blocks = r.blocks;
    t.max_rounds = a.max_rounds;
    const void* k = a.wt ? (const void*)k_inc_passes<true> : (const void*)k_inc_passes<false>;
    EK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(IncSmem)));
    if (a.wt) k_inc_passes<true><<<1, 1024, sizeof(IncSmem), s>>>(t);
    else k_inc_passes<false><<<1, 1024, sizeof(IncSmem), s>>>(t);
    EK(cudaGetLastError());
    IncCounters h{};
    EK(cudaMemcpyAsync(&h, ctr, sizeof h, cudaMemcpyDeviceToHost, s));
    EK(cudaStreamSynchronize(s));
    if (h.over) return rbsc_fail(ctx, RBSC_ERR_NOT_CONVERGED, "no fixpoint after %u passes", h.rounds);
    // the pass that found nothing to change is run again in full, to confirm it
    a.round0 = h.done ? h.rounds - 1u : h.rounds;
    a.deep_round = h.done ? 0u : 2u * h.rounds;
    return RBSC_OK;
}

// One launch, waited for.
rbsc_status launch_and_wait(rbsc_ctx* ctx, FusedArgs& a, const FusedLayout& l, bool block, cudaStream_t s)
{
    std::unique_lock<std::mutex> lock;
    if (!block && !one_cluster(a.n, a.m)) lock = coop_lock(ctx->device);
    EKS(launch(ctx, a, l, block, s));
    EK(cudaEventRecord(ctx->ev[1], s));
    EK(cudaStreamSynchronize(s));
    return RBSC_OK;
}

// Table slots of a batch of rows in check_rows (12 bytes each).
constexpr uint64_t kCheckSlots = 1u << 23;

// The rows that a launch's check left undecided (check_kernels.cuh), in batches
// whose tables fit kCheckSlots, or one row; col: the final colours, nlist: the
// check's list length on the device.  *equal: all of them are as their class's
// smallest member is.  False too when the tables cannot be had or the rows are
// read too often (one long member beside many short rows of the same sums):
// the launch-per-phase check, which sorts each row once, decides then.
rbsc_status check_rows(rbsc_ctx* ctx, const FusedArgs& a, const uint32_t* col, const uint32_t* nlist, cudaStream_t s, bool* equal)
{
    *equal = false;
    uint32_t n = 0, count = 0;
    EK(cudaMemcpyAsync(&n, nlist, 4, cudaMemcpyDeviceToHost, s));
    EK(cudaStreamSynchronize(s));
    Scratch sc(ctx);
    uint32_t *words = nullptr, *keys = nullptr;  // words: rows, differences
    unsigned long long* vals = nullptr;
    CheckRow* rows = nullptr;
    if (sc.get(&words, 2) != RBSC_OK || sc.get(&rows, n) != RBSC_OK) return RBSC_OK;
    EK(cudaMemsetAsync(words, 0, 8, s));
    const unsigned grid = (unsigned)ctx->sm_count * 8;
    ++rbsc::launch_counter();
    k_check_rows<<<grid, 256, 0, s>>>(a, n, col, rows, words);
    EK(cudaGetLastError());
    EK(cudaMemcpyAsync(&count, words, 4, cudaMemcpyDeviceToHost, s));
    EK(cudaStreamSynchronize(s));
    std::vector<CheckRow> h;
    try {
        h.resize(count);
    } catch (const std::bad_alloc&) {
        return RBSC_OK;
    }
    EK(cudaMemcpyAsync(h.data(), rows, sizeof(CheckRow) * count, cudaMemcpyDeviceToHost, s));
    EK(cudaStreamSynchronize(s));
    uint64_t arcs = 0, most = 0;
    for (CheckRow& x : h) {
        arcs += (uint64_t)x.du + x.dr;
        // equal rows of unit weights have the member's colours; others may have
        // colours whose weights add up to 0
        const uint64_t colours = std::min<uint64_t>(a.wt ? (uint64_t)x.du + x.dr : x.dr, a.n);
        uint64_t slots = 1024;
        while (slots < 2 * colours) slots <<= 1;
        x.mask = (uint32_t)(slots - 1);
        most = std::max(most, slots);
    }
    if (arcs > 8 * a.m) return RBSC_OK;
    const uint64_t cap = std::max(most, std::min<uint64_t>(kCheckSlots, 2 * a.m));
    if (sc.get(&keys, cap) != RBSC_OK || sc.get(&vals, cap) != RBSC_OK) return RBSC_OK;
    for (size_t i = 0; i < h.size();) {
        uint64_t used = 0, pieces = 0;
        size_t e = i;
        for (; e < h.size(); ++e) {
            CheckRow& x = h[e];
            if (used + x.mask + 1 > cap) break;
            x.base = used;
            x.first = (uint32_t)pieces;
            used += (uint64_t)x.mask + 1;
            pieces += ((uint64_t)x.du + kCkChunk - 1) / kCkChunk + ((uint64_t)x.dr + kCkChunk - 1) / kCkChunk;
        }
        EK(cudaMemcpyAsync(rows + i, h.data() + i, sizeof(CheckRow) * (e - i), cudaMemcpyHostToDevice, s));
        EK(cudaMemsetAsync(keys, 0xff, 4 * used, s));
        EK(cudaMemsetAsync(vals, 0, 8 * used, s));
        rbsc::launch_counter() += 2;
        if (a.wt) k_check_count<true><<<grid, 256, 0, s>>>(a, col, rows + i, (uint32_t)(e - i), (uint32_t)pieces, keys, vals, words + 1);
        else k_check_count<false><<<grid, 256, 0, s>>>(a, col, rows + i, (uint32_t)(e - i), (uint32_t)pieces, keys, vals, words + 1);
        k_check_zero<<<grid, 256, 0, s>>>(used, vals, words + 1);
        EK(cudaGetLastError());
        i = e;
    }
    uint32_t bad = 0;
    EK(cudaMemcpyAsync(&bad, words + 1, 4, cudaMemcpyDeviceToHost, s));
    EK(cudaEventRecord(ctx->ev[1], s));
    EK(cudaStreamSynchronize(s));
    *equal = bad == 0;
    return RBSC_OK;
}

// The launch, and where it stops early the work-list passes and a launch that
// confirms them, and the rows that its check left; waits for the stream.  ev[0]
// and ev[1] enclose it.
rbsc_status run(rbsc_ctx* ctx, FusedArgs& a, const FusedLayout& l, cudaStream_t s)
{
    FusedResult& r = *static_cast<FusedResult*>(ctx->h_fused);
    // one block keeps its classes in shared memory: nothing to continue from
    // (and a pass there costs less than one on the work list)
    const bool block = rows_side_by_side(a) && fused_fits_block(a, l);
    a.deep_round = block ? 0u : deep_round(a.n, a.m);
    EK(cudaEventRecord(ctx->ev[0], s));
    EKS(launch_and_wait(ctx, a, l, block, s));
    const uint32_t initial = r.initial_blocks;
    const uint64_t t0 = r.t[0], t1 = r.t[1];
    while (r.status == kFuDeep) {
        EKS(deep_tail(ctx, a, s));
        EKS(launch_and_wait(ctx, a, l, false, s));
        r.initial_blocks = initial;
        r.t[0] = t0;
        r.t[1] = t1;
    }
    if (r.status == kFuUndecided && !r.failed) {
        bool equal = false;
        EKS(check_rows(ctx, a, a.col[(r.rounds - a.round0 + r.repairs) & 1u], &a.w->nlist[r.repairs & 1u], s, &equal));
        if (equal) r.status = kFuOk;
    }
    return RBSC_OK;
}

// Status and statistics of a finished launch.  *handled false: the exact
// check is not decided, or found a difference that the launch could not split
// off; the caller refines the graph launch by launch.
rbsc_status outcome(rbsc_ctx* ctx, rbsc_stats* stats, float ms, bool* handled)
{
    const FusedResult& r = *static_cast<const FusedResult*>(ctx->h_fused);
    *handled = r.status != kFuUndecided;
    switch (r.status) {
        case kFuBadOffsets:
            return rbsc_fail(ctx, RBSC_ERR_INVALID, "offsets are not a valid CSR (must start at 0, be non-decreasing and end at M)");
        case kFuBadHead: return rbsc_fail(ctx, RBSC_ERR_INVALID, "an arc head is >= N");
        case kFuNotConverged: return rbsc_fail(ctx, RBSC_ERR_NOT_CONVERGED, "no fixpoint after %u passes", r.rounds);
        case kFuBarrier: return rbsc_fail(ctx, RBSC_ERR_DEVICE, "fused refinement: a grid barrier timed out");
        default: break;
    }
    if (stats && *handled) {
        stats->rounds = r.rounds;
        stats->blocks = r.blocks;
        stats->done = 1;
        stats->verified = ctx->opts.verify ? 1u : 0u;
        stats->repairs = r.repairs;
        stats->initial_blocks = r.initial_blocks;
        stats->device_ms = ms;
        stats->init_ms = (double)(r.t[1] - r.t[0]) * 1e-6;
        stats->loop_ms = (double)(r.t[2] - r.t[1]) * 1e-6;
        stats->verify_ms = (double)(r.t[3] - r.t[2]) * 1e-6;
        for (uint32_t i = 0; i < 64 && i <= r.rounds; ++i) stats->round_blocks[i] = r.round_blocks[i];
    }
    return RBSC_OK;
}

}  // namespace

// Below 2^22 arcs one launch always wins (sparse resident graphs apart: see
// refine_resident).  Above, the first pass by tiles with list_kernels.cuh after
// it catches up, first where it has more to offer (rival: hot heads, or heads
// whose copy overlaps the first pass).  us a refinement, one launch / after the
// first signatures / launch by launch, from one class: R-MAT-20 with 8 M arcs 385
// / 287 / 571, with 16 M 430 / 343 / 595, R-MAT-21 with 32 M 840 / 545 / 799,
// Erdos-Renyi with 16 M 211 / 261 / 558, a lift with 8.4 M 336 / 391 / 675: the line
// at 24 M lies between, since a graph's skew is not known before it is prepared.
// Weighted (whose rows the launch-per-phase check sorts), one launch / launch by
// launch: R-MAT-20 with 16 M 627 / 1001, R-MAT-21 1114 / 1435, from degree colours
// 467 / 789 and 863 / 1081, R-MAT-22 with 65 M 1560 / 1657: the line at 2^25, and
// the rival that resident ones with colours have from 2^22, are older than these.
constexpr uint64_t kSmallArcs = 1ull << 22, kLargeArcs = 3ull << 23, kLargeWeighted = 1ull << 25;

std::unique_lock<std::mutex> coop_lock(int device)
{
    static std::mutex mu[64];
    return std::unique_lock<std::mutex>(mu[(unsigned)device % 64u]);
}

bool fused_wanted(const rbsc_ctx* ctx, uint32_t n, uint64_t m, bool weighted, bool rival)
{
    if (!default_knobs(ctx->opts) || n == 0 || n > kIncMaxNodes) return false;
    if (m >= kSmallArcs && (rival || m >= (weighted ? kLargeWeighted : kLargeArcs))) return false;
    // a server's contexts (whose no_persist keeps k_refine_persistent out) take
    // it too: cooperative launches wait for one another (coop_lock)
    return ctx->shared_gpu || !ctx->opts.no_persist;
}

static rbsc_status ensure_work(rbsc_ctx* ctx, rbsc_graph* g, size_t bytes)
{
    if (g->fused_bytes >= bytes) return RBSC_OK;
    dev_free(ctx, g->d_fused);
    g->fused_bytes = 0;
    EKS(dev_alloc(ctx, &g->d_fused, bytes));
    g->fused_bytes = bytes;
    return RBSC_OK;
}

// From here on launch by launch; makes room for that path's arc sets.
static void launch_gave_up(rbsc_ctx* ctx, rbsc_graph* g)
{
    g->launch_off = true;
    dev_free(ctx, g->d_fused);
    g->fused_bytes = 0;
}

// The working arrays of k_refine_rows behind its counters.  Its second table and
// the classes' smallest members lie in d_tab8 and d_srank, which the initial pass
// is done with (sized by all nodes, so no smaller): the launch needs no more than
// the arc sets and check keys of the launch-per-phase path, which a server counts.
static FusedLayout list_layout(const rbsc_ctx* ctx, const rbsc_graph* g, size_t* seg = nullptr, uint32_t* seg_len = nullptr)
{
    FusedLayout l{};
    size_t at = fused_al(sizeof(ListWords));
    auto take = [&](size_t bytes) {
        const size_t r = at;
        at += fused_al(bytes);
        return r;
    };
    l.log2tab = 10;
    while ((1ull << l.log2tab) < 2ull * g->K) ++l.log2tab;
    l.long_cap = (uint32_t)std::min<uint64_t>(g->K, g->m / (kFuGroupRow + 1)) + 1u;
    l.chunk_cap = (uint32_t)(g->m / kFuChunk) + l.long_cap;
    l.tab[0] = take(8ull << l.log2tab);
    l.tab[2] = take(8ull << l.log2tab);
    l.list = take(4ull * g->K);
    l.lrow = take(4ull * l.long_cap);
    l.lfirst = take(4ull * l.long_cap);
    l.lsum = take(8ull * l.long_cap);
    l.ldone = take(4ull * l.long_cap);
    l.lchunk = take(4ull * l.chunk_cap);
    const uint64_t warps = (uint64_t)ctx->sm_count * (kFuThreads / 32), len = (g->K + 32 * warps - 1) / (32 * warps) * 32;
    const size_t sg = take(12ull * warps * len);
    if (seg) *seg = sg;
    if (seg_len) *seg_len = (uint32_t)len;
    l.bytes = at;
    return l;
}

// Graphs that fused_wanted leaves over, from 2^22 arcs: see the figures in
// list_kernels.cuh.  Below, the launch-per-phase path is only taken with options
// that this one does not know.
bool list_wanted(const rbsc_ctx* ctx, const rbsc_graph* g)
{
    return default_knobs(ctx->opts) && (ctx->shared_gpu || !ctx->opts.no_persist) && ctx->opts.test_hash_bits == 0 && !g->weighted &&
           !g->host_arcs && !g->launch_off && g->K > 0 && g->m >= kSmallArcs && g->m < (1ull << 32) && g->n < kListMaxNodes &&
           g->K <= (1u << 28);
}

bool list_reserve(rbsc_ctx* ctx, rbsc_graph* g) { return ensure_work(ctx, g, list_layout(ctx, g).bytes) == RBSC_OK; }

rbsc_status list_clear(rbsc_ctx* ctx, rbsc_graph* g, cudaStream_t s)
{
    const FusedLayout l = list_layout(ctx, g);
    unsigned char* b = static_cast<unsigned char*>(g->d_fused);
    EK(cudaMemsetAsync(b, 0, sizeof(ListWords), s));
    EK(cudaMemsetAsync(g->d_tab8, 0, 8ull << l.log2tab, s));
    EK(cudaMemsetAsync(b + l.tab[2], 0, 8ull << l.log2tab, s));
    return RBSC_OK;
}

rbsc_status list_arcless(rbsc_ctx* ctx, rbsc_graph* g, uint32_t* d_out)
{
    ++rbsc::launch_counter();
    k_list_arcless<<<(unsigned)ctx->sm_count * 8, 256, 0, ctx->stream>>>(g->n, g->d_bare, g->d_initlab, g->d_grep, d_out,
                                                                        &static_cast<ListWords*>(g->d_fused)->arcless);
    EK(cudaGetLastError());
    return RBSC_OK;
}

rbsc_status list_refine(rbsc_ctx* ctx, rbsc_graph* g, const uint32_t* d_init, uint32_t* d_out, uint32_t initial_blocks, rbsc_stats* stats,
                        bool* handled)
{
    *handled = false;
    cudaStream_t s = ctx->stream;
    ListArgs x{};
    size_t seg = 0;
    const FusedLayout l = list_layout(ctx, g, &seg, &x.seg_len);
    EKS(ensure_pinned(ctx));
    fused_bind(x.f, l, static_cast<unsigned char*>(g->d_fused));
    x.f.n = g->n;
    x.f.m = g->m;
    fused_csr(x.f, g->d_off, true);
    x.f.idx = g->d_idx;
    x.f.init = d_init;
    x.f.out = d_out;
    common_args(ctx, x.f);
    x.K = g->K;
    x.rows = g->d_rows;
    x.seg = reinterpret_cast<uint2*>(static_cast<unsigned char*>(g->d_fused) + seg);
    x.alone = reinterpret_cast<uint32_t*>(x.seg + (size_t)ctx->sm_count * (kFuThreads / 32) * x.seg_len);
    x.sig = g->d_sig;
    x.f.tab[1] = g->d_tab8;
    x.f.minm = g->d_srank;
    // a node without arcs keeps the words that the initial pass left in both
    x.f.col[0] = g->d_initlab;
    x.f.col[1] = g->d_col[0];
    x.w = reinterpret_cast<ListWords*>(g->d_fused);
    x.err = &g->d_st->error;
    x.initial = initial_blocks;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = (unsigned)ctx->sm_count;
    cfg.blockDim = kFuThreads;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    FusedResult& r = *static_cast<FusedResult*>(ctx->h_fused);
    // other contexts' cooperative launches need not wait for this graph's copies
    if (ctx->shared_gpu || g->oneshot) EK(cudaEventSynchronize(ctx->ev_sig[1]));
    {
        const std::unique_lock<std::mutex> lock = coop_lock(ctx->device);
        ++rbsc::launch_counter();
        EK(cudaLaunchKernelEx(&cfg, k_refine_rows, x));
        EK(cudaEventRecord(ctx->ev[1], s));
        EK(cudaStreamSynchronize(s));
    }
    if (r.status == kFuBadHead) {
        // what the first pass found wrong: the caller reports the state's error bits
        return RBSC_OK;
    }
    if (r.status == kFuUndecided && !r.failed) {
        bool equal = false;
        EKS(check_rows(ctx, x.f, x.f.col[r.rounds & 1u], &x.w->f.nlist[0], s, &equal));
        if (equal) r.status = kFuOk;
    }
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    EKS(outcome(ctx, stats, ms, handled));
    if (!*handled) launch_gave_up(ctx, g);
    return RBSC_OK;
}

rbsc_status fused_refine(rbsc_ctx* ctx, rbsc_graph* g, const uint32_t* d_init, uint32_t* d_out, rbsc_stats* stats, bool* handled)
{
    *handled = false;
    cudaStream_t s = ctx->stream;
    const uint64_t lc0 = rbsc::launch_counter();
    const FusedLayout l = fused_layout(g->n, g->m);
    // (the launch-per-phase path may have its buffers already)
    if (ensure_work(ctx, g, l.bytes) != RBSC_OK) return RBSC_OK;
    // labels may be asked for over the initial colours, which the check reads;
    // and a call that runs out of rounds leaves the caller's array alone
    uint32_t* const asked = d_out;
    if (!d_out || ctx->opts.max_rounds || labels_over_init(d_init, d_out, g->n)) {
        if (!g->d_out) EKS(dev_alloc(ctx, (void**)&g->d_out, 4 * (size_t)g->n));
        d_out = g->d_out;
    }
    EKS(ensure_pinned(ctx));
    FusedArgs a{};
    fused_bind(a, l, static_cast<unsigned char*>(g->d_fused));
    a.n = g->n;
    a.m = g->m;
    fused_csr(a, g->d_off, true);
    a.idx = g->d_idx;
    a.wt = g->weighted ? g->d_wt : nullptr;
    a.init = d_init;
    a.out = d_out;
    a.validate = g->prepared ? 0 : 1;
    common_args(ctx, a);
    EKS(run(ctx, a, l, s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    if (!g->prepared) cudaEventElapsedTime(&g->up_ms, ctx->ev[2], ctx->ev[3]);
    EKS(outcome(ctx, stats, ms, handled));
    if (!*handled) launch_gave_up(ctx, g);
    if (*handled && asked && asked != d_out) {
        EK(cudaMemcpyAsync(asked, d_out, 4 * (size_t)g->n, cudaMemcpyDeviceToDevice, s));
        EK(cudaStreamSynchronize(s));
    }
    if (stats && *handled) stats->kernel_launches = rbsc::launch_counter() - lc0;
    return RBSC_OK;
}

rbsc_status fused_refine_rows(rbsc_ctx* ctx, const FusedRows& r, const uint32_t* d_init, uint32_t* d_out, rbsc_stats* stats, bool* handled)
{
    *handled = false;
    cudaStream_t s = ctx->stream;
    const FusedLayout l = fused_layout(r.n, r.m);
    Scratch sc(ctx);
    unsigned char* d = nullptr;
    EKS(sc.get(&d, l.bytes));
    EKS(ensure_pinned(ctx));
    FusedArgs a{};
    fused_bind(a, l, d);
    a.n = r.n;
    a.m = r.m;
    a.off = r.begin;
    a.off_end = r.end;
    a.idx = r.idx;
    a.wt = r.wt;
    a.init = d_init;
    a.out = d_out;
    common_args(ctx, a);
    EKS(run(ctx, a, l, s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    if (stats) std::memset(stats, 0, sizeof *stats);
    return outcome(ctx, stats, ms, handled);
}

// A small host graph, labels back in host memory: the arrays are gathered in a
// pinned buffer, go to the device in one copy, and the kernel writes the
// labels and counts into pinned memory.
rbsc_status fused_oneshot(rbsc_ctx* ctx, const rbsc_csr* c, const uint32_t* init, uint32_t* out, rbsc_stats* stats, bool* handled,
                          bool* gave_up)
{
    *handled = *gave_up = false;
    const uint64_t lc0 = rbsc::launch_counter();
    if (c->m > kStageBytes / 4 || c->n > kStageNodes) return RBSC_OK;  // before the sizes below are added up
    const uint32_t n = c->n;
    auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
    const size_t b_off = (size_t)c->offset_bytes * ((size_t)n + 1), b_idx = 4 * (size_t)c->m, b_wt = c->weights ? 8 * (size_t)c->m : 0,
                 b_init = init ? 4 * (size_t)n : 0;
    const size_t in = al(b_off) + al(b_idx) + al(b_wt) + al(b_init);
    if (!fused_wanted(ctx, n, c->m, c->weights != nullptr, false) || in > kStageBytes) return RBSC_OK;
    const auto t0 = std::chrono::steady_clock::now();
    EK(cudaSetDevice(ctx->device));
    cudaStream_t s = ctx->stream;
    EKS(ensure_pinned(ctx));
    if (!ctx->h_stage) EKS(host_alloc(ctx, &ctx->h_stage, kStageBytes + 4 * (size_t)kStageNodes));
    unsigned char* h = static_cast<unsigned char*>(ctx->h_stage);
    uint32_t* h_out = reinterpret_cast<uint32_t*>(h + kStageBytes);
    const size_t o_idx = al(b_off), o_wt = o_idx + al(b_idx), o_init = o_wt + al(b_wt);
    std::memcpy(h, c->offsets, b_off);
    if (b_idx) std::memcpy(h + o_idx, c->indices, b_idx);
    if (b_wt) std::memcpy(h + o_wt, c->weights, b_wt);
    if (b_init) std::memcpy(h + o_init, init, b_init);
    const FusedLayout l = fused_layout(n, c->m);
    FusedArgs a{};
    a.n = n;
    a.m = c->m;
    auto bind_input = [&](unsigned char* p) {
        fused_csr(a, p, c->offset_bytes == 8);
        a.idx = reinterpret_cast<const uint32_t*>(p + o_idx);
        a.wt = b_wt ? reinterpret_cast<const uint64_t*>(p + o_wt) : nullptr;
        a.init = b_init ? reinterpret_cast<const uint32_t*>(p + o_init) : nullptr;
    };
    bind_input(h);
    const bool block = fused_fits_block(a, l);
    Scratch sc(ctx);
    EK(cudaEventRecord(ctx->ev[2], s));
    if (!block) {  // one block brings the arrays in itself, straight from the pinned buffer
        unsigned char* d = nullptr;
        EKS(sc.get(&d, l.bytes + in));
        fused_bind(a, l, d);
        bind_input(d + l.bytes);
        EK(cudaMemcpyAsync(d + l.bytes, h, in, cudaMemcpyHostToDevice, s));
    }
    EK(cudaEventRecord(ctx->ev[3], s));
    a.out = h_out;
    a.validate = 1;
    common_args(ctx, a);
    EKS(run(ctx, a, l, s));
    float ms = 0.f, up = 0.f;
    cudaEventElapsedTime(&up, ctx->ev[2], ctx->ev[3]);
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    if (stats) std::memset(stats, 0, sizeof *stats);
    EKS(outcome(ctx, stats, ms, handled));
    *gave_up = !*handled;
    if (!*handled) return RBSC_OK;
    if (out) std::memcpy(out, h_out, 4 * (size_t)n);
    if (stats) {
        stats->kernel_launches = rbsc::launch_counter() - lc0;
        stats->h2d_ms = up;
        stats->h2d_bytes = b_off + b_idx + b_wt + b_init;
        stats->d2h_bytes = out ? 4ull * n : 0;
        stats->time_s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    }
    return RBSC_OK;
}
