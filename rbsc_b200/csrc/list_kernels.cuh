// list_kernels.cuh -- the passes of a large refinement after its first
// signature pass, in one launch.
//
// A large graph's first pass is worth its own kernel (hot heads, narrow ranks,
// heads that arrive while it runs); what follows it touches far fewer arcs and
// was spent in a dozen launches per pass: an insert that wrote slots for a
// relabel to look up, node lists and arc sets rebuilt, a tail kernel, a check
// that classified every node into lists.  k_refine_rows takes the first pass's
// signatures and finishes the refinement as fused_kernels.cuh does: a pass's
// colour is the slot its key takes, one barrier per pass, three tables in turn,
// nodes alone in their class marked when the next pass finds nobody joined.
// Only rows with arcs are visited, each read where it lies in the graph's own
// arrays (no arc set is rebuilt).  A node without arcs (9.4 of R-MAT-24's 16.8 M)
// belongs to the class of its initial colour for good: its colour words are
// those that the initial pass left, so col[] are the initial pass's own arrays
// and a row's word carries kSlotBit to differ from them.
//
// Each warp owns the rows of every nw-th group of 32 (the low ids of an R-MAT
// graph are hubs; this deals them out) and keeps those still in play in a list
// of its own: no atomics, and a late pass walks 1.7 M rows instead of 7.4 M.  A
// pass first drops the rows that nobody joined, four loads in flight per lane
// (their words are written to both arrays, the second time a pass later, when
// nobody reads it); the rest is folded and inserted in groups of 32 that a
// block's warps take as they become free.  The tables' windows follow
// the rows in play (twice their number).  Rows too long for a warp are queued as
// a pass meets them and shared out after a barrier.
//
// Bound by the random 32-byte sectors of the gathers and inserts: the passes
// move about 3.5 TB/s of them.  R-MAT-24 from degree colours (263 M arcs), B200:
// the kernel takes 1.28 ms (passes 190 / 425 / 250 / 135 / 107 us, labels and
// check 166), a refinement 2.33 ms; launch by launch 3.15.  From degree colours,
// one launch after the signatures / launch per phase, us: a lift of 4.2 M arcs
// 338 / 519, of 8.4 M 472 / 743, Erdos-Renyi of 5 M 236 / 477, of 16 M 528 / 875;
// R-MAT-21 from one class 589 / 820.  Walking all rows in every pass, without the
// warps' lists: 2.84 ms on R-MAT-24; lists that kept a row one pass longer: 2.62;
// each warp folding its own list only, without dealing a block's groups out (35 %
// of the warps' time went into waiting at barriers): 2.43.
//
// Unit weights.  Rows with more colours than the check's table holds, or more
// arcs than a block may count, are left to check_kernels.cuh.  When a node fails the check (a hash collision), the
// refinement is done again launch by launch.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "common.cuh"
#include "fused_kernels.cuh"

namespace rbsc {

constexpr uint32_t kSlotBit = 1u << 30;       // colour word: a slot; without it, the initial label of a node without arcs
constexpr uint32_t kListMaxNodes = 1u << 30;
constexpr uint32_t kQueued = 0xffffffffu;  // slot word: the row went through the queue, its slot is in the colour array

struct ListWords {
    FusedWords f;
    uint32_t nlong[2], nchunk[2];  // of the running pass (by its parity)
    uint32_t active[3];            // rows that took part in pass p, in turn
    uint32_t arcless;              // classes of nodes without arcs
};

struct ListArgs {
    FusedArgs f;               // (weights, start, fail and lists by node are not used)
    uint32_t K;
    const uint32_t* rows;      // nodes with arcs
    uint2* seg;                // each warp's rows in play (node, slot or kQueued), seg_len places per warp
    uint32_t* alone;           // those found alone in the last pass
    uint32_t seg_len;
    const Sig* sig;            // the first pass's signatures
    ListWords* w;
    const uint32_t* err;       // RoundState.error: a bad head met by the first pass
    uint32_t initial;          // initial classes
};

// Labels of the nodes without arcs (final) and the number of their classes.
// `bare` has a bit per such node: with the offsets read here and in
// k_group_reps instead, 16 bytes a node, R-MAT-24 took 2446 us against 2426.
static __global__ void __launch_bounds__(256) k_list_arcless(uint32_t n, const uint32_t* __restrict__ bare,
                                                             const uint32_t* __restrict__ initlab, const uint32_t* __restrict__ grep,
                                                             uint32_t* __restrict__ out, uint32_t* __restrict__ count)
{
    __shared__ BlockReserveSmem<256> sm;
    constexpr int U = 4;  // nodes per thread and step: their loads overlap
    const uint32_t stride = gridDim.x * 256;
    uint32_t made = 0;
    for (uint32_t base = blockIdx.x * 256 + threadIdx.x; base < n; base += U * stride) {
        uint32_t r[U];
        bool none[U];
#pragma unroll
        for (int j = 0; j < U; ++j) {
            const uint64_t u = (uint64_t)base + (uint64_t)j * stride;
            none[j] = u < n && (bare[u >> 5] >> (u & 31u) & 1u);
        }
#pragma unroll
        for (int j = 0; j < U; ++j) r[j] = none[j] ? initlab[base + j * stride] : 0u;
#pragma unroll
        for (int j = 0; j < U; ++j) r[j] = none[j] ? grep[r[j]] : 0u;
#pragma unroll
        for (int j = 0; j < U; ++j)
            if (none[j]) {
                out[base + j * stride] = r[j];
                made += r[j] == base + j * stride ? 1u : 0u;
            }
    }
    block_count<256>(made, count, sm);
}

static __global__ void __launch_bounds__(kFuThreads, 1) k_refine_rows(const __grid_constant__ ListArgs x)
{
    constexpr int MODE = kFuGrid;
    __shared__ FuCache s_cache;
    __shared__ __align__(16) unsigned long long s_buf[kFuThreads / 32 * 128];
    __shared__ uint32_t s_sum, s_act, s_flag, s_word[2];
    __shared__ uint32_t s_delta[kFuThreads];
    __shared__ uint32_t s_cnt[kFuThreads / 32], s_next;
    const FusedArgs& a = x.f;
    const int lane = threadIdx.x & 31;
    const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nw = gridDim.x * (kFuThreads / 32);
    const uint32_t gt = blockIdx.x * kFuThreads + threadIdx.x, nt = gridDim.x * kFuThreads;
    const uint32_t* __restrict__ idx = a.idx;
    const uint32_t K = x.K;
    uint2* const seg = x.seg + (size_t)gw * x.seg_len;
    uint32_t* const alone = x.alone + (size_t)gw * x.seg_len;
    uint32_t cnt = 0, nalone = 0, gone = 0;  // rows in them; rows that left for good
    FusedWords* const w = &x.w->f;
    FuSync sync;
    const bool first = gt == 0;
    uint64_t t0 = 0, t2 = 0;
    if (first) t0 = fu_timer();
    if (threadIdx.x == 0) {
        s_sum = s_act = 0u;
        s_word[0] = s_word[1] = 0u;
    }
    uint32_t round = 0, prev = x.initial;
    auto finish = [&](int status) {
        if (!first) return;
        a.res->rounds = round;
        a.res->blocks = prev;
        a.res->initial_blocks = x.initial;
        a.res->repairs = 0;
        a.res->status = status;
        a.res->t[0] = a.res->t[1] = t0;
        a.res->t[2] = t2;
        a.res->t[3] = fu_timer();
    };
    if (*x.err) {  // (written by earlier launches only)
        finish(kFuBadHead);
        return;
    }
    auto window = [&](uint32_t count) {
        uint32_t l = 10;
        while (l < a.log2tab && (1ull << l) < 2ull * count) ++l;
        return l;
    };
    auto clear = [&](unsigned long long* t, uint32_t lg) {
        ulonglong2* q = reinterpret_cast<ulonglong2*>(t);
        for (uint32_t i = gt; i < 1u << (lg - 1); i += nt) q[i] = make_ulonglong2(0ull, 0ull);
    };
    // The block's lists as one sequence of groups of 32 rows, dealt out as warps
    // become free: group t is group t / 32 of warp t % 32's list.
    constexpr uint32_t kWarps = kFuThreads / 32;
    auto share = [&]() -> uint32_t {
        if (lane == 0) s_cnt[threadIdx.x >> 5] = cnt;
        if (threadIdx.x == 0) s_next = 0u;
        __syncthreads();
        return (__reduce_max_sync(0xffffffffu, s_cnt[lane]) + 31u) / 32u * kWarps;
    };
    auto take = [&]() -> uint32_t {
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(&s_next, 1u);
        return __shfl_sync(0xffffffffu, t, 0);
    };
    uint2* const segs = x.seg + (size_t)blockIdx.x * x.seg_len;
    const size_t seg_warp = (size_t)gridDim.x * x.seg_len;  // from one warp's list to the block's next
    auto totals = [&](uint32_t made, uint32_t act) {
        made = __reduce_add_sync(0xffffffffu, made);
        act = __reduce_add_sync(0xffffffffu, act);
        if (lane == 0 && made) atomicAdd(&s_sum, made);
        if (lane == 0 && act) atomicAdd(&s_act, act);
        __syncthreads();
    };
    uint32_t p = 0, lg = window(K);
    if (first) a.res->round_blocks[0] = prev;
    if (!fu_barrier<MODE>(w, sync, 0u, nullptr, s_word)) {
        finish(kFuBarrier);
        return;
    }
    const uint32_t arcless = fu_cg<MODE>(&x.w->arcless);

    int status = kFuOk;
    for (;;) {
        // pass: col[p & 1] -> the other array, classes in tab[(p + 1) % 3]
        const uint32_t* __restrict__ co = a.col[p & 1u];
        uint32_t* __restrict__ cn = a.col[(p & 1u) ^ 1u];
        const unsigned long long* __restrict__ tp = a.tab[p % 3u];
        unsigned long long* tc = a.tab[(p + 1u) % 3u];
        const uint32_t par = p & 1u;
        fu_cache_clear(s_cache);
        if (threadIdx.x == 0) s_sum = s_act = 0u;
        __syncthreads();
        if (p) clear(a.tab[(p + 2u) % 3u], lg);  // (the next window is no larger; the first two were cleared before the launch)
        if (first) {
            x.w->nlong[par ^ 1u] = x.w->nchunk[par ^ 1u] = 0u;
            x.w->active[(p + 1u) % 3u] = 0u;  // (its readers passed the last barrier)
        }
        const uint64_t salt = pass_salt1(a.seed, round);
        const bool few = (uint64_t)prev * 1024ull < K;
        uint32_t made = 0;
        if (p == 0) {
            // the first pass's signatures are there: its classes
            // (a step ahead: the label and signature of the next row, the node after)
            const uint32_t step = nw * 32u;
            uint32_t k = gw * 32u + lane;
            uint32_t u = k < K ? __ldg(x.rows + k) : 0u, nu = k + step < K ? __ldg(x.rows + k + step) : 0u;
            uint32_t lab = k < K ? fu_cg<MODE>(co + u) : 0u;
            uint64_t s1 = k < K ? __ldcs(&x.sig[u].s1) : 0ull;
            for (uint32_t base = gw * 32u; base < K; base += step, k += step) {
                const bool act = k < K;
                const uint64_t fp = act ? fu_fingerprint(lab, s1, a.seed) : 0ull;
                const uint32_t v = u;
                u = nu;
                if (k + step < K) {
                    lab = fu_cg<MODE>(co + u);
                    s1 = __ldcs(&x.sig[u].s1);
                }
                nu = k + 2u * step < K ? __ldg(x.rows + k + 2u * step) : 0u;
                const uint32_t s = fu_insert_warp<MODE>(act, few, tc, lg, fp, s_cache, made);
                if (act) {
                    cn[v] = kSlotBit | s;
                    seg[cnt + lane] = make_uint2(v, s);
                }
                cnt += min(K - base, 32u);
            }
        } else {
            // rows found alone in the last pass: in both arrays now, and out
            for (uint32_t i = lane; i < nalone; i += 32u) {
                const uint32_t u = alone[i];
                cn[u] = kSingleton | u;
            }
            gone += nalone;
            __syncwarp();
            // nobody joined a row's slot: alone for good
            uint32_t kept = 0, mk = 0;
            for (uint32_t i = 0; i < cnt; i += 128u) {
                uint2 q[4];
                uint32_t e[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t at = i + 32u * k + lane;
                    q[k] = at < cnt ? seg[at] : make_uint2(0u, 0u);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (q[k].y == kQueued) q[k].y = fu_cg<MODE>(co + q[k].x) & ~kSlotBit;
#pragma unroll
                for (int k = 0; k < 4; ++k) e[k] = i + 32u * k + lane < cnt ? (uint32_t)fu_cg<MODE>(tp + q[k].y) & 1u : 2u;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const unsigned stay = __ballot_sync(0xffffffffu, e[k] == 1u), leave = __ballot_sync(0xffffffffu, e[k] == 0u);
                    const unsigned below = (1u << lane) - 1u;
                    if (e[k] == 1u) seg[kept + __popc(stay & below)] = q[k];
                    if (e[k] == 0u) {
                        const uint32_t u = q[k].x;
                        cn[u] = kSingleton | u;
                        a.out[u] = u;
                        alone[mk + __popc(leave & below)] = u;
                    }
                    kept += __popc(stay);
                    mk += __popc(leave);
                }
            }
            cnt = kept;
            nalone = mk;
            const uint32_t groups = share();
            for (uint32_t t = take(); t < groups; t = take()) {
                const uint32_t i = t / kWarps * 32u, rest = s_cnt[t % kWarps];
                if (i >= rest) continue;
                uint2* const row = segs + (t % kWarps) * seg_warp + i + lane;
                bool act = i + lane < rest;
                const uint2 q = act ? *row : make_uint2(0u, 0u);
                const uint32_t u = q.x, c = q.y;
                uint64_t b = 0;
                uint32_t d = 0;
                if (act) {
                    b = fu_off<MODE>(a, u);
                    d = (uint32_t)(fu_end<MODE>(a, u) - b);
                }
                const uint32_t da = act ? d : 0u;
                const bool queue = fu_shared_row(da, __reduce_add_sync(0xffffffffu, da));
                const unsigned qm = __ballot_sync(0xffffffffu, queue);
                if (qm) {
                    const uint32_t nc = queue ? (d + kFuChunk - 1) / kFuChunk : 0u;
                    uint32_t end = nc;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const uint32_t y = __shfl_up_sync(0xffffffffu, end, o);
                        if (lane >= o) end += y;
                    }
                    uint32_t j0 = 0, f0 = 0;
                    if (lane == 31) {
                        j0 = atomicAdd(&x.w->nlong[par], (uint32_t)__popc(qm));
                        f0 = atomicAdd(&x.w->nchunk[par], end);
                    }
                    const uint32_t j = __shfl_sync(0xffffffffu, j0, 31) + __popc(qm & ((1u << lane) - 1u));
                    const uint32_t f = __shfl_sync(0xffffffffu, f0, 31) + end - nc;
                    if (queue) {
                        act = false;
                        row->y = kQueued;
                        if (j < a.long_cap) {
                            a.lrow[j] = u;
                            a.lfirst[j] = f;
                            a.lsum[j] = 0ull;
                            a.ldone[j] = 0u;
                            for (uint32_t i = 0; i < nc && f + i < a.chunk_cap; ++i) a.lchunk[f + i] = j;
                        }
                    }
                }
                const uint64_t s1 = fu_row_sums<MODE, false>(act, b, d, idx, nullptr, co, salt, s_delta + (threadIdx.x & ~31u),
                                                             reinterpret_cast<ulonglong2*>(s_buf + (threadIdx.x >> 5) * 128));
                const uint64_t fp = act ? fu_fingerprint(c, s1, a.seed) : 0ull;
                const uint32_t s = fu_insert_warp<MODE>(act, few, tc, lg, fp, s_cache, made);
                if (act) {
                    cn[u] = kSlotBit | s;
                    row->y = s;
                }
            }
        }
        __syncwarp();
        totals(made + (lane == 0 ? gone + nalone : 0u), lane == 0 ? cnt : 0u);
        if (threadIdx.x == 0 && s_act) atomicAdd(&x.w->active[p % 3u], s_act);
        uint32_t count = 0;
        if (!fu_barrier<MODE>(w, sync, s_sum, &count, s_word)) {
            finish(kFuBarrier);
            return;
        }
        const uint32_t nchunk = min(fu_cg<MODE>(&x.w->nchunk[par]), a.chunk_cap);
        if (p > 0 && nchunk) {
            made = 0;
            for (uint32_t ch = gw; ch < nchunk; ch += nw) {
                const uint32_t j = a.lchunk[ch], u = a.lrow[j], f = a.lfirst[j];
                const uint32_t c = fu_cg<MODE>(co + u) & ~kSlotBit;
                const uint64_t b = fu_off<MODE>(a, u), e = fu_end<MODE>(a, u);
                const uint64_t s = b + (uint64_t)(ch - f) * kFuChunk, t = min(e, s + kFuChunk);
                uint64_t sum = 0;
#pragma unroll 8
                for (uint64_t i = s + lane; i < t; i += 32) sum += fu_term(fu_cg<MODE>(co + fu_ro<MODE>(idx + i)), salt);
                sum = fu_warp_sum(sum, 32);
                if (lane == 0) {
                    const uint32_t nc = (uint32_t)((e - b + kFuChunk - 1) / kFuChunk);
                    bool last = nc == 1u;
                    if (!last) {
                        atomicAdd(&a.lsum[j], (unsigned long long)sum);
                        __threadfence();
                        last = atomicAdd(&a.ldone[j], 1u) + 1u == nc;
                        if (last) {
                            __threadfence();
                            sum = atomicExch(&a.lsum[j], 0ull);
                        }
                    }
                    if (last) {
                        bool claimed;
                        cn[u] = kSlotBit | fu_insert<MODE>(tc, lg, fu_fingerprint(c, sum, a.seed), false, s_cache, claimed);
                        made += claimed ? 1u : 0u;
                    }
                }
            }
            __syncthreads();
            if (threadIdx.x == 0) s_sum = 0u;
            __syncthreads();
            totals(made, 0u);
            uint32_t more = 0;
            if (!fu_barrier<MODE>(w, sync, s_sum, &more, s_word)) {
                finish(kFuBarrier);
                return;
            }
            count += more;
        }
        count += arcless;
        const uint32_t in_play = fu_cg<MODE>(&x.w->active[p % 3u]);
        ++p;
        ++round;
        const bool done = count == prev;
        prev = count;
        if (first && round < (uint32_t)kRoundLog) a.res->round_blocks[round] = count;
        if (done) break;
        if (round >= a.max_rounds) {
            status = kFuNotConverged;
            break;
        }
        lg = min(lg, window(in_play));
    }
    if (status != kFuOk) {
        finish(status);
        return;
    }
    if (first) t2 = fu_timer();
    // labels and the exact check, as in fused_body
    const uint32_t* __restrict__ col = a.col[p & 1u];
    {
        uint4* q = reinterpret_cast<uint4*>(a.minm);
        for (uint32_t i = gt; i < 1u << (lg - 2); i += nt) q[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    }
    if (!fu_barrier<MODE>(w, sync, 0u, nullptr, s_word)) {
        finish(kFuBarrier);
        return;
    }
    for (uint32_t i = lane; i < cnt; i += 128u) {
        uint2 q[4];
        uint32_t r[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            q[k] = i + 32u * k < cnt ? seg[i + 32u * k] : make_uint2(0u, 0u);
            if (q[k].y == kQueued) q[k].y = fu_cg<MODE>(col + q[k].x) & ~kSlotBit;
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) r[k] = i + 32u * k < cnt ? fu_cg<MODE>(a.minm + q[k].y) : 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (r[k] > q[k].x) atomicMin(a.minm + q[k].y, q[k].x);
    }
    if (!fu_barrier<MODE>(w, sync, 0u, nullptr, s_word)) {
        finish(kFuBarrier);
        return;
    }
    uint32_t nbad = 0;
    const uint32_t groups = share();
    for (uint32_t t = take(); t < groups; t = take()) {
        const uint32_t i = t / kWarps * 32u, rest = s_cnt[t % kWarps];
        if (i >= rest) continue;
        const bool valid = i + lane < rest;
        const uint2 q = valid ? segs[(t % kWarps) * seg_warp + i + lane] : make_uint2(0u, 0u);
        const uint32_t u = q.x;
        const uint32_t r = valid ? fu_cg<MODE>(a.minm + (q.y != kQueued ? q.y : fu_cg<MODE>(col + u) & ~kSlotBit)) : 0u;
        if (valid) a.out[u] = r;
        const bool chk = a.verify && valid && r != u;
        if (!__any_sync(0xffffffffu, chk)) continue;
        uint64_t bu = 0, br = 0;
        uint32_t du = 0, dr = 0, iu = 0, ir = 0;
        if (chk) {
            bu = fu_off<MODE>(a, u);
            br = fu_off<MODE>(a, r);
            du = (uint32_t)(fu_end<MODE>(a, u) - bu);
            dr = (uint32_t)(fu_end<MODE>(a, r) - br);
            if (a.init) {
                iu = __ldg(a.init + u);
                ir = __ldg(a.init + r);
            }
        }
        bool bad = chk && (iu != ir || du != dr);
        const uint32_t mx = chk && !bad ? du : 0u;
        fu_check_rows<MODE, false, 8>(__ballot_sync(0xffffffffu, mx > 0 && mx <= 8), lane, idx, nullptr, col, bu, du, br, dr, bad);
        fu_check_rows<MODE, false, 16>(__ballot_sync(0xffffffffu, mx > 8 && mx <= 16), lane, idx, nullptr, col, bu, du, br, dr, bad);
        fu_check_rows<MODE, false, 32>(__ballot_sync(0xffffffffu, mx > 16 && mx <= 32), lane, idx, nullptr, col, bu, du, br, dr, bad);
        fu_check_long<MODE, 2>(__ballot_sync(0xffffffffu, mx > 32 && mx <= 64), lane, idx, col, bu, br, du, bad);
        fu_check_long<MODE, 4>(__ballot_sync(0xffffffffu, mx > 64 && mx <= 128), lane, idx, col, bu, br, du, bad);
        const unsigned ml = __ballot_sync(0xffffffffu, mx > 128);
        if (ml) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(&w->nlist[0], (uint32_t)__popc(ml));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (mx > 128) a.list[at + __popc(ml & ((1u << lane) - 1u))] = u;
        }
        nbad += bad ? 1u : 0u;
    }
    __syncthreads();
    if (threadIdx.x == 0) s_sum = 0u;
    __syncthreads();
    totals(nbad, 0u);
    uint32_t nfail = 0;
    if (!fu_barrier<MODE>(w, sync, s_sum, &nfail, s_word)) {
        finish(kFuBarrier);
        return;
    }
    const uint32_t nlist = fu_cg<MODE>(&w->nlist[0]);
    if (nlist && nfail == 0u) {
        unsigned long long* const val = s_buf;
        uint32_t* const key = reinterpret_cast<uint32_t*>(s_buf + kFuCheckSlots);
        nbad = 0;
        uint64_t spent = 0;
        const uint64_t most = kFuCheckArcs + 4 * (a.m / gridDim.x);
        for (uint32_t i = blockIdx.x; i < nlist; i += gridDim.x) {
            const uint32_t u = a.list[i] & ~kSingleton, r = fu_cg<MODE>(a.minm + (fu_cg<MODE>(col + u) & ~kSlotBit));
            spent += fu_end<MODE>(a, u) - fu_off<MODE>(a, u) + (fu_end<MODE>(a, r) - fu_off<MODE>(a, r));
            if (spent > most) {
                if (threadIdx.x == 0) {
                    atomicOr(&w->overflow, 1u);
                    a.list[i] = u | kSingleton;
                }
                continue;
            }
            for (uint32_t k = threadIdx.x; k < kFuCheckSlots; k += kFuThreads) {
                key[k] = 0xffffffffu;
                val[k] = 0ull;
            }
            if (threadIdx.x == 0) s_flag = 0u;
            __syncthreads();
            bool ok = true;
            for (int side = 0; side < 2 && ok; ++side) {
                const uint32_t v = side ? u : r;
                const uint64_t e = fu_end<MODE>(a, v);
                for (uint64_t q = fu_off<MODE>(a, v) + threadIdx.x; q < e && ok; q += kFuThreads)
                    ok = fu_count(key, val, kFuCheckSlots - 1u, kFuProbes, fu_cg<MODE>(col + fu_ro<MODE>(idx + q)), side ? ~0ull : 1ull);
            }
            if (!ok) atomicOr(&s_flag, 2u);
            __syncthreads();
            bool diff = false;
            for (uint32_t k = threadIdx.x; k < kFuCheckSlots; k += kFuThreads) diff |= val[k] != 0ull;
            if (diff) atomicOr(&s_flag, 1u);
            __syncthreads();
            if (threadIdx.x == 0) {
                if (s_flag & 2u) {
                    atomicOr(&w->overflow, 1u);
                    a.list[i] = u | kSingleton;
                } else {
                    nbad += s_flag;
                }
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) s_sum = 0u;
        __syncthreads();
        totals(nbad, 0u);
        if (!fu_barrier<MODE>(w, sync, s_sum, &nfail, s_word)) {
            finish(kFuBarrier);
            return;
        }
    }
    if (first) a.res->failed = nfail;
    finish(nfail || fu_cg<MODE>(&w->overflow) ? kFuUndecided : kFuOk);
}

}  // namespace rbsc
