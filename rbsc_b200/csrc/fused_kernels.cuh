// fused_kernels.cuh -- a whole refinement in one launch, for graphs whose
// passes are short (below 2^22 arcs, and on to 24 or 32 M arcs where nothing else
// is faster: fused_wanted).
//
// The launch-per-phase path spends such a graph's time on launches, host
// synchronisations and phase boundaries, not on work: the 131,072-node lift
// took 0.42 ms for four passes whose bytes take a few microseconds (0.10 ms
// here; a 1,000-arc one-shot call 0.44 -> 0.09 ms, R-MAT-18 with 3.9 M arcs
// 0.36 -> 0.18 ms, 5,000 nodes without allocation 0.18 -> 0.04 ms).  Here one
// launch checks the graph (on request), classes the initial colours, runs the
// passes to the fixpoint, checks the fixpoint exactly, repairs it if the check
// fails and writes the canonical labels.
//
// One barrier per pass.  A pass's new colour of a node is the *slot* its key
// (old colour, signature) takes in the pass's table, which the thread that
// inserts the key knows at once; no second phase has to look the class up,
// and no smallest member is kept until the end.  Colours ping-pong between
// two arrays (a pass reads the old ones while it writes the new ones), and
// three tables take turns: the pass inserts into one, reads the previous one
// (was a second node in my class? no: the node is alone for good and leaves
// the passes as kSingleton | node) and zeroes the third for the next pass.
// Any injective renaming of the colours gives the same partition, so blocks,
// rounds and the final labels are those of the launch-per-phase path.
//
// A table entry is one 64-bit word: a 63-bit fingerprint of the key and the
// joined bit (exact keys in the initial and repair passes).  Keys that share a
// fingerprint would merge two classes; the exact check finds that.
//
// Rows: nodes are dealt to warps 32 at a time, interleaved over the SMs.  The
// warp lays the arcs of its unfinished rows end to end and takes 128 of them
// per step, four per lane (the heads of neighbouring rows lie side by side in
// memory, so a step touches few lines, and no lane waits for a longer row);
// a running prefix sum is read off at the row starts, and a row's sum is the
// difference of two of them.  (One arc per lane and step took four times the
// shuffles: the 131,072-node lift 101 us against 96, a lift of 170 rounds 1102
// against 1045.)  Rows of more than kFuChunk arcs, and
// rows of more than kFuGroupRow arcs in a group of more than kFuGroupArcs (the
// low node ids of an R-MAT graph are all hubs), are cut into chunks that all
// warps share (the warp that completes a row's last chunk inserts it).
// R-MAT-14 (228,000 arcs), first pass with only rows above 512 arcs shared:
// 90 us, one warp holding most of the arcs.
//
// MODE: a cooperative grid with a counter barrier whose waits are bounded
// (kFuGrid); one cluster, whose blocks are resident together by construction
// (kFuCluster: hardware barrier, block totals exchanged through the blocks'
// shared memory); or one block with the graph and all working arrays in shared
// memory (kFuBlock): a pass of a 1,000-arc graph is then a microsecond of work
// instead of nine dependent trips to L2.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>
#include "common.cuh"
#include "refine_kernels.cuh"
#include "verify_kernels.cuh"

namespace rbsc {

constexpr int kFuThreads = 1024;
constexpr uint32_t kFuChunk = 256;
constexpr uint32_t kFuGroupArcs = 1024;  // a warp's 32 rows together: beyond this its rows of more than
constexpr uint32_t kFuGroupRow = 64;     // kFuGroupRow arcs are shared out too
constexpr uint32_t kFuCache = 512;         // per block: slots of classes it met that have two members
// Shared memory is kept small on purpose: what it leaves is L1, whose lines
// hold the gathers in flight (with 200 KB of check tables a pass of the
// 131,072-node lift took 16.5 us, with 48 KB 13 us).
constexpr uint32_t kFuCheckSlots = 2048;    // per block: colours of one long row (exact check)
constexpr uint32_t kFuWarpSlots = kFuCheckSlots / (kFuThreads / 32);
constexpr uint32_t kFuWarpRow = kFuWarpSlots - 8;  // rows up to this length are tried by one warp
constexpr uint32_t kFuWideSlots = 32768;    // per block, in global memory: any row of a graph of at most 16384 nodes

// Arcs that a block counts in its table of the check, beside 4 / blocks of the
// graph's: the others wait for it at a bounded barrier, so the rows beyond are
// left undecided.  A block counts an arc in 1.7 ns (two rows of 3 M arcs: 10 ms,
// shared by all warps 0.6), so these take 2 ms, and the share of a graph of 2^32
// arcs 0.2 s.
constexpr uint64_t kFuCheckArcs = 1ull << 20;
constexpr uint32_t kFuProbes = 256;  // of the shared table: one that takes longer is as good as full

// outcome of a launch (FusedResult.status)
// kFuUndecided: labels are written, but the exact check left rows to check_kernels.cuh (marked with
// kSingleton in the list) or, with `failed`, found a node that differs and could not split it off
constexpr int kFuOk = 0, kFuBadOffsets = 1, kFuBadHead = 2, kFuNotConverged = 3, kFuUndecided = 4, kFuBarrier = 5,
              kFuDeep = 6;  // stopped after deep_round passes or more: the last ones changed little (deep_kernels.cuh)

// Counters of one launch, zero at its start (zeroed by the launcher, or by
// block 0 of a cluster).
struct FusedWords {
    unsigned long long bar[2];  // barrier words (fu_barrier)
    uint32_t pad[28];
    uint32_t bad;          // 1 = offsets, 2 = a head
    uint32_t overflow;     // a row had more colours than the check's table, or too many arcs: marked in the list
    uint32_t nlong, nchunk;
    uint32_t nlist[2];     // long rows of the running check (by repair parity)
};

struct FusedResult {
    uint32_t rounds, blocks, initial_blocks, repairs;
    int32_t status;
    uint32_t failed;       // kFuUndecided: another node failed the check
    uint64_t t[4];         // globaltimer: start, initial colours done, fixpoint, end
    uint32_t round_blocks[kRoundLog];
};

struct FusedArgs {
    uint32_t n;
    uint64_t m;
    const void* off;       // where each row starts; rows may lie anywhere in idx
    const void* off_end;   // where it ends (CSR offsets: off + 1 entry)
    const uint32_t* idx;
    const uint64_t* wt;
    const uint32_t* init;
    const uint32_t* start; // classes to start from instead of init's (a continued refinement), or null
    uint32_t* out;
    uint32_t* col[2];
    unsigned long long* tab[3];
    uint32_t log2tab;
    uint32_t* minm;        // per slot of the final table: smallest member
    uint32_t* list;        // nodes whose check needs a shared table
    uint8_t* fail;
    unsigned char* wide;   // kFuWideSlots counters per block for rows with more colours than the
                           // shared table holds; null: such a row is left undecided (kFuUndecided)
    uint32_t* lrow;        // long rows: node, first chunk, running sum, chunks done
    uint32_t* lfirst;
    unsigned long long* lsum;
    uint32_t* ldone;
    uint32_t* lchunk;      // chunk -> long row
    uint32_t long_cap, chunk_cap;
    FusedWords* w;
    FusedResult* res;              // or:
    rbsc_noalloc_result* na_res;
    uint64_t seed;
    uint32_t max_rounds;
    uint32_t hash_bits;
    uint32_t round0;       // passes already run
    uint32_t deep_round;   // from this pass on stop (kFuDeep) when passes make few new classes; 0: never
    uint8_t off64, validate, verify;
};

// "few": at most kFuDeepNew, and no sharp drop for kFuDeepSteady passes: the last
// passes of a random graph make 200, 60, 15, 3, 1 and are soon over, a chain goes
// on making the same number.  (With the first alone, Erdos-Renyi of 2^20 nodes and
// 0.7 arcs per node took 1,509 us instead of 772, for the one pass saved.)  After
// twice deep_round's passes the first is enough: the numbers may go up and down.
constexpr uint32_t kFuDeepNew = 256, kFuDeepSteady = 3;

constexpr int kFuGrid = 0, kFuCluster = 1, kFuBlock = 2;

// Loads of arrays that the launch itself writes (at L2) and of its inputs; in
// kFuBlock both lie in shared memory.
template <int MODE, typename T> __device__ __forceinline__ T fu_cg(const T* p)
{
    if constexpr (MODE == kFuBlock) return *(const volatile T*)p;
    else return __ldcg(p);
}
template <int MODE, typename T> __device__ __forceinline__ T fu_ro(const T* p)
{
    if constexpr (MODE == kFuBlock) return *p;
    else return __ldg(p);
}
template <int MODE> __device__ __forceinline__ uint64_t fu_ld(const void* p, bool wide, uint32_t u)
{
    return wide ? fu_ro<MODE>(reinterpret_cast<const unsigned long long*>(p) + u)
                : (uint64_t)fu_ro<MODE>(reinterpret_cast<const uint32_t*>(p) + u);
}
template <int MODE = kFuGrid> __device__ __forceinline__ uint64_t fu_off(const FusedArgs& a, uint32_t u) { return fu_ld<MODE>(a.off, a.off64, u); }
template <int MODE = kFuGrid> __device__ __forceinline__ uint64_t fu_end(const FusedArgs& a, uint32_t u) { return fu_ld<MODE>(a.off_end, a.off64, u); }

// Whether a row of d arcs in a group of `group` arcs goes in chunks.
__device__ __forceinline__ bool fu_shared_row(uint32_t d, uint32_t group)
{
    return d > kFuChunk || (group > kFuGroupArcs && d > kFuGroupRow);
}

__device__ __forceinline__ uint64_t fu_timer()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// The per-arc term on the whole colour word (a bijection of it, salted).
__device__ __forceinline__ uint64_t fu_term(uint32_t c, uint64_t salt)
{
    uint64_t y = (uint64_t)(c ^ (uint32_t)salt) * 0x9e3779b97f4a7c15ull;
    y ^= y >> 32;
    y *= 0xd6e8feb86659fd93ull;
    y ^= y >> 32;
    return y + (salt >> 32);
}

// The table fingerprint of (colour, signature): bit 0 clear, never 0.
__device__ __forceinline__ uint64_t fu_fingerprint(uint32_t c, uint64_t s1, uint64_t seed)
{
    const uint64_t f = fmix64(s1 ^ (((uint64_t)c + 1ull) * kGolden ^ seed)) & ~1ull;
    return f ? f : 2ull;
}

__device__ __forceinline__ uint64_t fu_warp_sum(uint64_t v, int width)
{
    for (int d = width >> 1; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}

struct FuCache {
    unsigned long long key[kFuCache];
    uint32_t slot[kFuCache];
};

__device__ __forceinline__ void fu_cache_clear(FuCache& c)
{
    for (uint32_t i = threadIdx.x; i < kFuCache; i += kFuThreads) {
        c.key[i] = 0ull;
        c.slot[i] = 0xffffffffu;
    }
}

// Slot of fingerprint fp (bit 0 clear, not 0) for one node, or for several
// (multi); claimed: this call opened the class.  A class already met by the block with two members answers from
// shared memory: the few big classes of an early pass would otherwise be one
// L2 address for the whole grid.  A cache word is written once per pass, by
// the thread whose compare-and-swap took it.
template <int MODE>
__device__ __forceinline__ uint32_t fu_insert(unsigned long long* __restrict__ tab, uint32_t log2tab, uint64_t fp, bool multi, FuCache& cache,
                                              bool& claimed)
{
    const uint64_t h = fp * kGolden;
    const uint32_t ci = (uint32_t)(h >> 20) & (kFuCache - 1u);
    const uint64_t ck = MODE == kFuBlock ? 1ull : *(volatile unsigned long long*)&cache.key[ci];
    claimed = false;
    if (ck == fp) {
        const uint32_t s = *(volatile uint32_t*)&cache.slot[ci];
        if (s != 0xffffffffu) return s;
    }
    const uint32_t mask = (1u << log2tab) - 1u;
    uint32_t s = (uint32_t)(h >> (64 - log2tab));
    // at most half of the entries are taken, so an empty one ends the probe;
    // the bound only keeps a broken table from looping
    for (uint32_t probe = 0; probe <= mask; ++probe, s = (s + 1u) & mask) {
        unsigned long long e = fu_cg<MODE>(tab + s);
        if (e == 0ull) {
            e = atomicCAS(tab + s, 0ull, (unsigned long long)fp | (multi ? 1ull : 0ull));
            if (e == 0ull) {
                claimed = true;
                return s;
            }
        }
        if ((e & ~1ull) == fp) {
            if (!(e & 1ull)) atomicOr(tab + s, 1ull);
            if (ck == 0ull && atomicCAS(&cache.key[ci], 0ull, (unsigned long long)fp) == 0ull)
                *(volatile uint32_t*)&cache.slot[ci] = s;
            return s;
        }
    }
    return 0u;
}

// The lanes with `need` insert their keys; `few`: the classes are few beside
// the nodes, so lanes with equal keys send one of them (32 compare-and-swaps
// of a warp on one address would be served one after another).
template <int MODE>
__device__ __forceinline__ uint32_t fu_insert_warp(bool need, bool few, unsigned long long* __restrict__ tab, uint32_t log2tab,
                                                   uint64_t fp, FuCache& cache, uint32_t& made)
{
    const unsigned m = __ballot_sync(0xffffffffu, need);
    uint32_t s = 0;
    if (need) {
        bool claimed = false;
        if (few) {
            const unsigned peers = __match_any_sync(m, (unsigned long long)fp);
            const int leader = __ffs(peers) - 1;
            if ((int)(threadIdx.x & 31) == leader) s = fu_insert<MODE>(tab, log2tab, fp, (peers & (peers - 1u)) != 0u, cache, claimed);
            s = __shfl_sync(peers, s, leader);
        } else {
            s = fu_insert<MODE>(tab, log2tab, fp, false, cache, claimed);
        }
        made += claimed ? 1u : 0u;
    }
    return s;
}

// Barrier over the whole grid that also adds up `val` over the blocks (thread
// 0's values): *total = the sum.  A word counts arrivals in its low half and
// the values in its high half, both over all barriers so far, so one atomic
// and one polled load do both.  Two words take turns: a block that is already
// at the next barrier adds to the other one, so what this barrier reads is the
// same for every block.  False: a wait ran out.
struct FuSync {
    uint32_t epoch = 0;           // barriers so far
    uint32_t seen0 = 0, seen1 = 0;  // the words' high halves after their last barriers
};

template <int MODE>
__device__ __forceinline__ bool fu_barrier(FusedWords* w, FuSync& y, uint32_t val, uint32_t* total, uint32_t* s_word)
{
    const uint32_t par = y.epoch & 1u;
    const unsigned target = ((y.epoch >> 1) + 1u) * gridDim.x;  // arrivals at this word
    ++y.epoch;
    if constexpr (MODE == kFuBlock) {
        __syncthreads();
        if (total) *total = val;  // every thread of the block has its total
        return true;
    }
    if constexpr (MODE == kFuCluster) {
        // thread i hands the block's value to block i: the sums need no trip to L2
        uint32_t* const part = s_word + 2 + 8 * par;
        if (threadIdx.x < gridDim.x) {
            uint32_t mine = (uint32_t)__cvta_generic_to_shared(part + blockIdx.x), there;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(mine), "r"(threadIdx.x));
            asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(there), "r"(val) : "memory");
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (total) {
            uint32_t all = 0;
            for (uint32_t i = 0; i < gridDim.x; ++i) all += *(volatile uint32_t*)(part + i);
            *total = all;
        }
        return true;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long* const word = &w->bar[par];
        const unsigned long long add = ((unsigned long long)val << 32) | 1ull;
        __threadfence();
        unsigned long long v = atomicAdd(word, add) + add;
        uint32_t it = 0;
        while ((uint32_t)v < target) {
            if (++it > (1u << 22)) {  // about two seconds
                s_word[1] = 1u;
                break;
            }
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word) : "memory");
        }
        s_word[0] = (uint32_t)(v >> 32);
        __threadfence();
    }
    __syncthreads();
    const uint32_t all = *(volatile uint32_t*)&s_word[0];
    if (total) *total = all - (par ? y.seen1 : y.seen0);
    if (par) y.seen1 = all;
    else y.seen0 = all;
    return *(volatile uint32_t*)&s_word[1] == 0u;
}

// Group g (of 32 / G) of a warp takes the g-th set bit of `m` as its source
// lane (-1: none); the bits taken are cleared.
template <int G>
__device__ __forceinline__ int fu_take(unsigned& m, int lane)
{
    int src = -1;
#pragma unroll
    for (int q = 0; q < 32 / G; ++q) {
        const int b = m ? __ffs(m) - 1 : -1;
        if (m) m &= m - 1u;
        if (lane / G == q) src = b;
    }
    return src;
}

// The arc sums of a warp's 32 rows (lane: row [b, b + d) where act; see the top
// of the file).  delta: 32 words, pre: 128 sums of shared memory of the warp.
template <int MODE, bool WEIGHTED>
__device__ __forceinline__ uint64_t fu_row_sums(bool act, uint64_t b, uint32_t d, const uint32_t* __restrict__ idx,
                                                const uint64_t* __restrict__ wt, const uint32_t* __restrict__ co, uint64_t salt,
                                                uint32_t* delta, ulonglong2* pre)
{
    const int lane = threadIdx.x & 31;
    const unsigned rows = __ballot_sync(0xffffffffu, act && d > 0);
    const uint32_t dd = act ? d : 0u;
    uint32_t end = dd;  // inclusive prefix: where the row ends in the warp's sequence
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += x;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, end, 31), start = end - dd;
    if (dd) delta[__popc(rows & ((1u << lane) - 1u))] = (uint32_t)b - start;
    __syncwarp();
    uint64_t run = 0, at_start = 0;
    uint32_t before = 0;  // rows that start before the step
    // a step: 128 arcs, four consecutive ones per lane
    for (uint32_t j0 = 0; j0 < total; j0 += 128) {
        // bit i of heads[w]: a row starts at position j0 + 32 w + i
        uint32_t heads[4], rank = before;
        const uint32_t rel = start - j0;
#pragma unroll
        for (int w = 0; w < 4; ++w)
            heads[w] = __reduce_or_sync(0xffffffffu, dd && rel - 32u * w < 32u ? 1u << (rel & 31u) : 0u);
        uint32_t mine = heads[0];
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            if (w < lane >> 3) {
                rank += __popc(heads[w]);
                mine = heads[w + 1 < 4 ? w + 1 : 3];
            }
            before += __popc(heads[w]);
        }
        // (a lane's positions past the end read nothing and add nothing)
        const uint32_t left = total - min(total, j0 + 4u * lane);
        uint32_t cc[4];
        uint64_t t[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t r = rank + __popc(mine & (0xffffffffu >> (31 - ((lane & 7) * 4 + q))));
            cc[q] = q < left ? delta[r - 1u] + j0 + 4u * lane + q : 0u;
        }
        if (WEIGHTED) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                t[q] = q < left ? fu_ro<MODE>(reinterpret_cast<const unsigned long long*>(wt) + cc[q]) : 0ull;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) cc[q] = q < left ? fu_ro<MODE>(idx + cc[q]) : 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) cc[q] = q < left ? fu_cg<MODE>(co + cc[q]) : 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (WEIGHTED) t[q] *= fu_term(cc[q], salt);
            else t[q] = q < left ? fu_term(cc[q], salt) : 0ull;
        }
        const uint64_t sum = t[0] + t[1] + t[2] + t[3];
        uint64_t in = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint64_t y = __shfl_up_sync(0xffffffffu, in, o);
            if (lane >= o) in += y;
        }
        // the sums before each position, for the rows that start there
        const uint64_t ex = run + in - sum;
        pre[2 * lane] = make_ulonglong2(ex, ex + t[0]);
        pre[2 * lane + 1] = make_ulonglong2(ex + t[0] + t[1], ex + t[0] + t[1] + t[2]);
        run += __shfl_sync(0xffffffffu, in, 31);
        __syncwarp();
        if (dd && rel < 128u) at_start = reinterpret_cast<const unsigned long long*>(pre)[rel];
        __syncwarp();
    }
    // a row ends where the next one starts
    const unsigned above = lane == 31 ? 0u : rows & (0xffffffffu << (lane + 1));
    const uint64_t next = __shfl_sync(0xffffffffu, at_start, above ? __ffs(above) - 1 : 0);
    __syncwarp();
    return dd ? (above ? next : run) - at_start : 0ull;
}

// Exact comparison of two rows of at most G arcs by groups of G lanes: lane gl
// of a group holds arc gl of both rows (colour 0xffffffff and weight 0 past a
// row's end).  Unit weights: both rows sorted in registers.  Weighted: every
// lane adds up its colour's weight over both rows; a difference that is not 0
// (mod 2^64) is one.
template <bool WEIGHTED, int G>
__device__ __forceinline__ bool fu_lane_differs(uint32_t a, uint32_t b, uint64_t wa, uint64_t wb)
{
    if (!WEIGHTED) return group_sort<G>(a) != group_sort<G>(b);
    uint64_t da = 0, db = 0;
#pragma unroll
    for (int j = 0; j < G; ++j) {
        const uint32_t ca = __shfl_sync(0xffffffffu, a, j, G), cb = __shfl_sync(0xffffffffu, b, j, G);
        const uint64_t va = __shfl_sync(0xffffffffu, wa, j, G), vb = __shfl_sync(0xffffffffu, wb, j, G);
        if (ca == a) da += va;
        if (cb == a) da -= vb;
        if (ca == b) db += va;
        if (cb == b) db -= vb;
    }
    return (a != 0xffffffffu && da != 0) || (b != 0xffffffffu && db != 0);
}

// The rows (bu, du) and (br, dr) of the lanes in `m`, G lanes each; sets the
// owner lane's `bad`.
template <int MODE, bool WEIGHTED, int G>
__device__ __forceinline__ void fu_check_rows(unsigned m, int lane, const uint32_t* __restrict__ idx, const uint64_t* __restrict__ wt,
                                              const uint32_t* __restrict__ col, uint64_t bu, uint32_t du, uint64_t br, uint32_t dr,
                                              bool& bad)
{
    const int gl = lane & (G - 1);
    while (m) {
        const unsigned m0 = m;
        const int src = fu_take<G>(m, lane);
        const int s = src < 0 ? 0 : src;
        const uint64_t xbu = __shfl_sync(0xffffffffu, bu, s), xbr = __shfl_sync(0xffffffffu, br, s);
        const uint32_t xdu = __shfl_sync(0xffffffffu, du, s), xdr = __shfl_sync(0xffffffffu, dr, s);
        uint32_t a = 0xffffffffu, b = 0xffffffffu;
        uint64_t wa = 0, wb = 0;
        if (src >= 0) {
            if ((uint32_t)gl < xdu) {
                a = fu_cg<MODE>(col + fu_ro<MODE>(idx + xbu + gl));
                if (WEIGHTED) wa = fu_ro<MODE>(reinterpret_cast<const unsigned long long*>(wt) + xbu + gl);
            }
            if ((uint32_t)gl < xdr) {
                b = fu_cg<MODE>(col + fu_ro<MODE>(idx + xbr + gl));
                if (WEIGHTED) wb = fu_ro<MODE>(reinterpret_cast<const unsigned long long*>(wt) + xbr + gl);
            }
        }
        const unsigned diff = __ballot_sync(0xffffffffu, fu_lane_differs<WEIGHTED, G>(a, b, wa, wb));
        // which of this step's groups is the lane's own row in?
        unsigned left = m0;
#pragma unroll
        for (int q = 0; q < 32 / G; ++q) {
            if (!left) break;
            const int b0 = __ffs(left) - 1;
            left &= left - 1u;
            const unsigned gm = G == 32 ? 0xffffffffu : (((1u << (G & 31)) - 1u) << (q * G));
            if (lane == b0 && (diff & gm)) bad = true;
        }
    }
}

// Ascending bitonic sort of 32 * K values, K per lane (value i of the
// sequence: register i / 32 of lane i % 32).
template <int K> __device__ __forceinline__ void fu_sort(uint32_t (&v)[K])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32 * K; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
#pragma unroll
                for (int q = 0; q < K; ++q)
                    if (!(q & (j / 32))) {
                        const bool up = ((q * 32) & k) == 0;
                        const uint32_t x = v[q], y = v[q | (j / 32)];
                        v[q] = up ? min(x, y) : max(x, y);
                        v[q | (j / 32)] = up ? max(x, y) : min(x, y);
                    }
            } else {
#pragma unroll
                for (int q = 0; q < K; ++q) {
                    const uint32_t o = __shfl_xor_sync(0xffffffffu, v[q], j);
                    const bool up = ((q * 32 + lane) & k) == 0;
                    v[q] = ((lane & j) == 0) == up ? min(v[q], o) : max(v[q], o);
                }
            }
        }
}

// The rows of the lanes in `m` (unit weights, equal lengths of at most 32 * K
// arcs), one after another by the whole warp.
template <int MODE, int K>
__device__ __forceinline__ void fu_check_long(unsigned m, int lane, const uint32_t* __restrict__ idx, const uint32_t* __restrict__ col,
                                              uint64_t bu, uint64_t br, uint32_t d, bool& bad)
{
    while (m) {
        const int s = __ffs(m) - 1;
        m &= m - 1u;
        const uint64_t xbu = __shfl_sync(0xffffffffu, bu, s), xbr = __shfl_sync(0xffffffffu, br, s);
        const uint32_t xd = __shfl_sync(0xffffffffu, d, s);
        uint32_t a[K], b[K];
#pragma unroll
        for (int q = 0; q < K; ++q) {
            const uint32_t i = 32u * q + lane;
            a[q] = i < xd ? fu_cg<MODE>(col + fu_ro<MODE>(idx + xbu + i)) : 0xffffffffu;
            b[q] = i < xd ? fu_cg<MODE>(col + fu_ro<MODE>(idx + xbr + i)) : 0xffffffffu;
        }
        fu_sort<K>(a);
        fu_sort<K>(b);
        bool diff = false;
#pragma unroll
        for (int q = 0; q < K; ++q) diff |= a[q] != b[q];
        if (__any_sync(0xffffffffu, diff) && lane == s) bad = true;
    }
}

// Adds sign * weight to colour c in an open-addressed table; false when it
// finds no place in so many probes.
__device__ __forceinline__ bool fu_count(uint32_t* key, unsigned long long* val, uint32_t mask, uint32_t probes, uint32_t c, uint64_t w)
{
    uint32_t h = (c * 0x9e3779b1u) >> 7 & mask;
    for (uint32_t p = 0; p < probes; ++p, h = (h + 1u) & mask) {
        const uint32_t k = atomicCAS(&key[h], 0xffffffffu, c);
        if (k == 0xffffffffu || k == c) {
            atomicAdd(&val[h], (unsigned long long)w);
            return true;
        }
    }
    return false;
}

template <int MODE, bool WEIGHTED>
__device__ __forceinline__ void fused_body(const FusedArgs& a)
{
    __shared__ FuCache s_cache;
    // the passes' prefix sums (128 per warp); the check's table of one long row
    __shared__ __align__(16) unsigned long long s_buf[kFuThreads / 32 * 128];
    static_assert(sizeof s_buf >= kFuCheckSlots * 12, "values, then keys");
    unsigned long long* const s_val = s_buf;
    uint32_t* const s_key = reinterpret_cast<uint32_t*>(s_buf + kFuCheckSlots);
    __shared__ uint32_t s_sum, s_flag, s_next, s_word[2 + 16];
    __shared__ uint32_t s_delta[kFuThreads];  // per warp: its rows' (first arc - position) by rank
    const uint32_t n = a.n;
    const int lane = threadIdx.x & 31;
    // warps dealt over the blocks: neighbouring node groups on different SMs
    const uint32_t gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    const uint32_t nw = gridDim.x * (kFuThreads / 32);
    const uint32_t gt = blockIdx.x * kFuThreads + threadIdx.x;
    const uint32_t nt = gridDim.x * kFuThreads;
    const uint32_t* __restrict__ idx = a.idx;
    const uint64_t* __restrict__ wt = a.wt;
    FusedWords* const w = a.w;
    FuSync sync;
    const bool first = gt == 0;
    uint64_t t0 = 0, t1 = 0, t2 = 0;
    if (first) t0 = fu_timer();
    if (threadIdx.x == 0) {
        s_sum = 0u;
        s_word[0] = s_word[1] = 0u;
    }
    fu_cache_clear(s_cache);
    if constexpr (MODE != kFuGrid) {
        if (first) {
            w->bad = w->overflow = 0u;
            w->nlong = w->nchunk = 0u;
            w->nlist[0] = w->nlist[1] = 0u;
        }
        if constexpr (MODE == kFuBlock) __syncthreads();
        else asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    }

    auto finish = [&](int status, uint32_t rounds, uint32_t blocks, uint32_t initial, uint32_t repairs) {
        if (!first) return;
        if (a.res) {
            a.res->rounds = rounds;
            a.res->blocks = blocks;
            a.res->initial_blocks = initial;
            a.res->repairs = repairs;
            a.res->status = status;
            a.res->t[0] = t0;
            a.res->t[1] = t1;
            a.res->t[2] = t2;
            a.res->t[3] = fu_timer();
        }
        if (a.na_res) {
            a.na_res->blocks = blocks;
            a.na_res->rounds = rounds;
            a.na_res->repairs = repairs;
            a.na_res->status = status == kFuOk                                        ? RBSC_OK
                               : status == kFuBadOffsets || status == kFuBadHead ? RBSC_ERR_INVALID
                               : status == kFuNotConverged                            ? RBSC_ERR_NOT_CONVERGED
                                                                                      : RBSC_ERR_DEVICE;
        }
    };

    if (n == 0) {
        finish(kFuOk, 0u, 0u, 0u, 0u);
        return;
    }

    // clear the tables, check the graph, list the long rows
    const uint32_t tabn = 1u << a.log2tab;
    auto clear_tab = [&](unsigned long long* t) {
        ulonglong2* q = reinterpret_cast<ulonglong2*>(t);
        for (uint32_t i = gt; i < tabn / 2; i += nt) q[i] = make_ulonglong2(0ull, 0ull);
    };
    auto clear_min = [&]() {
        uint4* q = reinterpret_cast<uint4*>(a.minm);
        for (uint32_t i = gt; i < tabn / 4; i += nt) q[i] = make_uint4(~0u, ~0u, ~0u, ~0u);
    };
    clear_tab(a.tab[0]);
    clear_tab(a.tab[1]);
    clear_min();
    const uint32_t* __restrict__ const ini = a.start ? a.start : a.init;
    uint32_t bad_in = 0;
    for (uint32_t base = gw * 32u; base < n; base += nw * 32u) {
        const uint32_t u = base + lane;
        uint64_t b = 0, e = 0;
        bool bad = false;
        if (u < n) {
            b = fu_off<MODE>(a, u);
            e = fu_end<MODE>(a, u);
            bad = a.validate && (b > e || e > a.m || (u == 0 && b != 0) || (u == n - 1 && e != a.m));
            if (!ini) a.col[0][u] = 0u;
        }
        // (with a bad row anywhere nothing below is used)
        const uint32_t d = bad ? 0u : (uint32_t)(e - b);
        if (fu_shared_row(d, __reduce_add_sync(0xffffffffu, d))) {
            const uint32_t nc = (d + kFuChunk - 1) / kFuChunk;
            const uint32_t j = atomicAdd(&w->nlong, 1u), f = atomicAdd(&w->nchunk, nc);
            if (j < a.long_cap) {
                a.lrow[j] = u;
                a.lfirst[j] = f;
                a.lsum[j] = 0ull;
                a.ldone[j] = 0u;
                for (uint32_t i = 0; i < nc && f + i < a.chunk_cap; ++i) a.lchunk[f + i] = j;
            }
        }
        bad_in |= bad ? 1u : 0u;
    }
    if (a.validate)
        for (uint64_t k = gt; k < a.m; k += nt)
            if (fu_ro<MODE>(idx + k) >= n) bad_in |= 2u;
    if (bad_in) atomicOr(&w->bad, bad_in);
    if (!fu_barrier<MODE>(w, sync, 0u, nullptr, s_word)) {
        finish(kFuBarrier, 0u, 0u, 0u, 0u);
        return;
    }
    {
        const uint32_t bad = fu_cg<MODE>(&w->bad);
        if (bad) {  // nothing is written, nothing read through the graph
            finish((bad & 1u) ? kFuBadOffsets : kFuBadHead, 0u, 0u, 0u, 0u);
            return;
        }
    }
    const uint32_t nchunk = min(fu_cg<MODE>(&w->nchunk), a.chunk_cap);

    uint32_t p = 0;  // current colours: col[p & 1], classes: tab[p % 3]
    uint32_t made = 0;
    auto block_total = [&](uint32_t v) -> uint32_t {
        v = __reduce_add_sync(0xffffffffu, v);
        if (lane == 0 && v) atomicAdd(&s_sum, v);
        __syncthreads();
        return *(volatile uint32_t*)&s_sum;
    };
    uint32_t prev = 1;
    bool has_classes = ini != nullptr;
    if (ini) {
        for (uint32_t base = gw * 32u; base < n; base += nw * 32u) {
            const uint32_t u = base + lane;
            const bool valid = u < n;
            const uint64_t fp = valid ? ((uint64_t)fu_cg<MODE>(ini + u) + 1ull) << 1 : 0ull;
            const uint32_t s = fu_insert_warp<MODE>(valid, true, a.tab[0], a.log2tab, fp, s_cache, made);
            if (valid) a.col[0][u] = s;
        }
        const uint32_t tot = block_total(made);
        if (!fu_barrier<MODE>(w, sync, tot, &prev, s_word)) {
            finish(kFuBarrier, 0u, 0u, 0u, 0u);
            return;
        }
    }
    const uint32_t initial = prev;
    if (first) {
        t1 = fu_timer();
        if (a.res && !a.start) a.res->round_blocks[0] = prev;
    }

    // The next group of a block's warp: groups are dealt out as warps become free
    // (the first ones are fixed), since rows differ in length.  Every nw-th group
    // for each warp instead: weighted R-MAT-20 695 us against 640, R-MAT-20 480
    // against 459, a lift of 8.4 M arcs 375 against 352.
    auto next_group = [&](uint32_t base) -> uint32_t {
        if constexpr (MODE != kFuGrid) return base + nw * 32u;
        uint32_t t = 0;
        if (lane == 0) t = atomicAdd(&s_next, 1u);
        t = __shfl_sync(0xffffffffu, t, 0) + kFuThreads / 32;
        return (t * gridDim.x + blockIdx.x) * 32u;
    };
    // one pass from col[p & 1] to the other array; REPAIR: the key is (colour,
    // failed) instead of (colour, signature).  Returns false on a timeout.
    uint32_t round = a.round0, repairs = 0, count = 0;
    uint32_t trend = 0;  // classes that the last pass made (kIncMaxNodes at most); from bit 24: passes since a sharp drop
    auto pass = [&](bool repair) -> bool {
        const uint32_t* __restrict__ co = a.col[p & 1u];
        uint32_t* __restrict__ cn = a.col[(p & 1u) ^ 1u];
        const unsigned long long* __restrict__ tp = a.tab[p % 3u];
        unsigned long long* tc = a.tab[(p + 1u) % 3u];
        fu_cache_clear(s_cache);
        if (threadIdx.x == 0) s_sum = s_next = 0u;
        __syncthreads();
        clear_tab(a.tab[(p + 2u) % 3u]);
        if (repair) clear_min();
        const uint64_t salt = pass_salt1(a.seed, round);
        const bool uniform = !has_classes && !WEIGHTED;  // one class: a row's sum is its length times one term
        const bool few = (uint64_t)prev * 1024ull < n;
        const uint64_t t_one = fu_term(0u, salt);
        const uint64_t hmask = a.hash_bits == 0 ? ~0ull : a.hash_bits >= 64 ? 0ull : (1ull << a.hash_bits) - 1ull;
        made = 0;
        auto fingerprint = [&](uint32_t c, uint64_t s1) { return fu_fingerprint(c, s1 & hmask, a.seed); };
        for (uint32_t base = gw * 32u; base < n; base = next_group(base)) {
            const uint32_t u = base + lane;
            const bool valid = u < n;
            uint32_t c = valid ? fu_cg<MODE>(co + u) : kSingleton;
            bool act = !(c & kSingleton);
            unsigned long long e = 1ull;
            uint64_t b = 0;
            uint32_t d = 0;
            if (valid && !repair) {
                b = fu_off<MODE>(a, u);
                d = (uint32_t)(fu_end<MODE>(a, u) - b);
            }
            if (act) {
                if (has_classes) e = fu_cg<MODE>(tp + c);
                else e = n > 1u ? 1ull : 0ull;
                if (!(e & 1ull)) {  // nobody joined: alone for good
                    act = false;
                    c = kSingleton | u;
                }
            }
            if (valid && !act) {
                cn[u] = c;
                ++made;
            }
            uint64_t fp = 0;
            if (repair) {
                if (act) fp = ((((uint64_t)c << 1) | (a.fail[u] ? 1ull : 0ull)) + 1ull) << 1;
            } else {
                uint64_t s1 = 0;
                if (uniform) {
                    s1 = t_one * d;
                } else {
                    if (fu_shared_row(d, __reduce_add_sync(0xffffffffu, d))) act = false;  // in chunks, below
                    s1 = fu_row_sums<MODE, WEIGHTED>(act, b, d, idx, wt, co, salt, s_delta + (threadIdx.x & ~31u),
                                                     reinterpret_cast<ulonglong2*>(s_buf + (threadIdx.x >> 5) * 128));
                }
                if (act) fp = fingerprint(c, s1);
            }
            const uint32_t s = fu_insert_warp<MODE>(act, few, tc, a.log2tab, fp, s_cache, made);
            if (act) cn[u] = s;
        }
        if (!repair && !uniform)
            for (uint32_t ch = nw - 1u - gw; ch < nchunk; ch += nw) {
                const uint32_t j = a.lchunk[ch], u = a.lrow[j], f = a.lfirst[j];
                const uint32_t c = fu_cg<MODE>(co + u);
                if ((c & kSingleton) || (has_classes && !(fu_cg<MODE>(tp + c) & 1ull)) || n == 1u) continue;
                const uint64_t b = fu_off<MODE>(a, u), e = fu_end<MODE>(a, u);
                const uint64_t s = b + (uint64_t)(ch - f) * kFuChunk, t = min(e, s + kFuChunk);
                uint64_t sum = 0;
#pragma unroll 8
                for (uint64_t i = s + lane; i < t; i += 32) {
                    const uint64_t x = fu_term(fu_cg<MODE>(co + fu_ro<MODE>(idx + i)), salt);
                    sum += WEIGHTED ? x * fu_ro<MODE>(reinterpret_cast<const unsigned long long*>(wt) + i) : x;
                }
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
                            a.ldone[j] = 0u;
                        }
                    }
                    if (last) {
                        bool claimed;
                        cn[u] = fu_insert<MODE>(tc, a.log2tab, fingerprint(c, sum), false, s_cache, claimed);
                        made += claimed ? 1u : 0u;
                    }
                }
            }
        const uint32_t tot = block_total(made);
        if (!fu_barrier<MODE>(w, sync, tot, &count, s_word)) return false;
        ++p;
        has_classes = true;
        return true;
    };

    int status = kFuOk;
    for (;;) {
        // hashed passes to the fixpoint
        for (;;) {
            if (!pass(false)) {
                finish(kFuBarrier, round, prev, initial, repairs);
                return;
            }
            ++round;
            const bool done = count == prev;
            const uint32_t fresh = count - prev;
            trend = fresh | (fresh <= kFuDeepNew && fresh * 4u >= (trend & 0xffffffu) * 3u ? (trend & 0xff000000u) + 0x1000000u : 0u);
            prev = count;
            if (first && a.res && round < (uint32_t)kRoundLog) a.res->round_blocks[round] = count;
            if (done) break;
            if (round >= a.max_rounds) {
                status = kFuNotConverged;
                break;
            }
            if (a.deep_round && round >= a.deep_round && (trend & 0xffffffu) <= kFuDeepNew && repairs == 0u &&
                (trend >> 24 >= kFuDeepSteady || round >= 2u * a.deep_round)) {
                if (first) t2 = fu_timer();
                finish(kFuDeep, round, prev, initial, repairs);
                return;
            }
        }
        if (first) t2 = fu_timer();
        // the smallest member of every class
        const uint32_t* __restrict__ col = a.col[p & 1u];
        const uint32_t par = repairs & 1u;
        if (first) w->nlist[par ^ 1u] = 0u;
        if (threadIdx.x == 0) s_next = 0u;  // (the barrier below)
        for (uint32_t u = gt; u < n; u += nt) {
            const uint32_t c = fu_cg<MODE>(col + u);
            if (!(c & kSingleton) && fu_cg<MODE>(a.minm + c) > u) atomicMin(a.minm + c, u);
        }
        if (!fu_barrier<MODE>(w, sync, 0u, nullptr, s_word)) {
            finish(kFuBarrier, round, prev, initial, repairs);
            return;
        }
        // labels, and the exact check of every node against that member
        const bool check = a.verify && status == kFuOk;
        uint32_t nbad = 0;
        for (uint32_t base = gw * 32u; base < n; base = next_group(base)) {
            const uint32_t u = base + lane;
            const bool valid = u < n;
            const uint32_t c = valid ? fu_cg<MODE>(col + u) : kSingleton;
            const uint32_t r = (c & kSingleton) ? u : fu_cg<MODE>(a.minm + c);
            if (valid) a.out[u] = r;
            if (!check) continue;
            const bool chk = valid && r != u;
            uint64_t bu = 0, br = 0;
            uint32_t du = 0, dr = 0, iu = 0, ir = 0;
            if (chk) {
                bu = fu_off<MODE>(a, u);
                br = fu_off<MODE>(a, r);
                du = (uint32_t)(fu_end<MODE>(a, u) - bu);
                dr = (uint32_t)(fu_end<MODE>(a, r) - br);
                if (a.init) {
                    iu = fu_ro<MODE>(a.init + u);
                    ir = fu_ro<MODE>(a.init + r);
                }
            }
            bool bad = chk && (iu != ir || (!WEIGHTED && du != dr));
            const uint32_t mx = chk && !bad ? max(du, dr) : 0u;
            fu_check_rows<MODE, WEIGHTED, 8>(__ballot_sync(0xffffffffu, mx > 0 && mx <= 8), lane, idx, wt, col, bu, du, br, dr, bad);
            fu_check_rows<MODE, WEIGHTED, 16>(__ballot_sync(0xffffffffu, mx > 8 && mx <= 16), lane, idx, wt, col, bu, du, br, dr, bad);
            fu_check_rows<MODE, WEIGHTED, 32>(__ballot_sync(0xffffffffu, mx > 16 && mx <= 32), lane, idx, wt, col, bu, du, br, dr, bad);
            uint32_t reg = 32;  // longest row compared in registers
            if (!WEIGHTED) {
                fu_check_long<MODE, 2>(__ballot_sync(0xffffffffu, mx > 32 && mx <= 64), lane, idx, col, bu, br, du, bad);
                fu_check_long<MODE, 4>(__ballot_sync(0xffffffffu, mx > 64 && mx <= 128), lane, idx, col, bu, br, du, bad);
                reg = 128;
            }
            const unsigned ml = __ballot_sync(0xffffffffu, mx > reg);
            if (ml) {
                uint32_t at = 0;
                if (lane == 0) at = atomicAdd(&w->nlist[par], (uint32_t)__popc(ml));
                at = __shfl_sync(0xffffffffu, at, 0);
                if (mx > reg) a.list[at + __popc(ml & ((1u << lane) - 1u))] = u;
            }
            if (valid && !(c & kSingleton)) a.fail[u] = bad ? 1 : 0;
            nbad += bad ? 1u : 0u;
        }
        if (!check) {
            finish(status, round, prev, initial, repairs);
            return;
        }
        if (threadIdx.x == 0) s_sum = 0u;
        __syncthreads();
        uint32_t tot = block_total(nbad), nfail = 0, more = 0;
        if (!fu_barrier<MODE>(w, sync, tot, &nfail, s_word)) {
            finish(kFuBarrier, round, prev, initial, repairs);
            return;
        }
        const uint32_t nlist = fu_cg<MODE>(&w->nlist[par]);
        if (nlist) {
            // longer rows: colours counted in a table, + for the member's row
            // and - for the node's; all must end at 0.  A warp tries the short
            // ones (weighted) in its part of the block's table and leaves them
            // to the block when they do not fit.
            nbad = 0;
            auto add_arc = [&](uint32_t* key, unsigned long long* val, uint32_t mask, uint32_t probes, uint64_t i, bool minus) -> bool {
                const uint64_t v = WEIGHTED ? fu_ro<MODE>(reinterpret_cast<const unsigned long long*>(wt) + i) : 1ull;
                return fu_count(key, val, mask, probes, fu_cg<MODE>(col + fu_ro<MODE>(idx + i)), minus ? 0ull - v : v);
            };
            auto longest = [&](uint32_t u, uint32_t r) {
                return max((uint32_t)(fu_end<MODE>(a, u) - fu_off<MODE>(a, u)), (uint32_t)(fu_end<MODE>(a, r) - fu_off<MODE>(a, r)));
            };
            if (WEIGHTED) {
                const uint32_t wi = threadIdx.x >> 5;
                uint32_t* key = s_key + wi * kFuWarpSlots;
                unsigned long long* val = s_val + wi * kFuWarpSlots;
                for (uint32_t i = gw; i < nlist; i += nw) {
                    const uint32_t u = a.list[i], r = fu_cg<MODE>(a.minm + fu_cg<MODE>(col + u));
                    if (longest(u, r) > kFuWarpRow) continue;
                    for (uint32_t k = lane; k < kFuWarpSlots; k += 32) {
                        key[k] = 0xffffffffu;
                        val[k] = 0ull;
                    }
                    __syncwarp();
                    bool ok = true;
                    for (int side = 0; side < 2; ++side) {
                        const uint64_t b = fu_off<MODE>(a, side ? u : r), e = fu_end<MODE>(a, side ? u : r);
                        for (uint64_t k = b + lane; k < e; k += 32) ok &= add_arc(key, val, kFuWarpSlots - 1u, kFuWarpSlots, k, side);
                    }
                    __syncwarp();
                    bool diff = false;
                    for (uint32_t k = lane; k < kFuWarpSlots; k += 32) diff |= val[k] != 0ull;
                    ok = __all_sync(0xffffffffu, ok);
                    diff = __any_sync(0xffffffffu, diff);
                    if (lane == 0) {
                        if (!ok) a.fail[u] = 2;  // undecided
                        else if (diff) {
                            a.fail[u] = 1;
                            ++nbad;
                        }
                    }
                    __syncwarp();
                }
                // the undecided marks are read by other blocks
                if (!fu_barrier<MODE>(w, sync, 0u, nullptr, s_word)) {
                    finish(kFuBarrier, round, prev, initial, repairs);
                    return;
                }
            }
            uint64_t spent = 0;
            const uint64_t most = kFuCheckArcs + 4 * (a.m / gridDim.x);
            for (uint32_t i = blockIdx.x; i < nlist; i += gridDim.x) {
                // (thread 0 may be marking it already)
                const uint32_t u = a.list[i] & ~kSingleton, r = fu_cg<MODE>(a.minm + fu_cg<MODE>(col + u));
                if (WEIGHTED && longest(u, r) <= kFuWarpRow && fu_cg<MODE>(a.fail + u) != 2) continue;
                if (MODE != kFuBlock && !a.wide) {
                    spent += fu_end<MODE>(a, u) - fu_off<MODE>(a, u) + (fu_end<MODE>(a, r) - fu_off<MODE>(a, r));
                    if (spent > most) {
                        if (threadIdx.x == 0) {
                            atomicOr(&w->overflow, 1u);
                            a.list[i] = u | kSingleton;
                        }
                        continue;
                    }
                }
                uint32_t* key = s_key;
                unsigned long long* val = s_val;
                // (a graph in shared memory has fewer nodes than the table half its slots)
                uint32_t slots = kFuCheckSlots, probes = MODE == kFuBlock ? kFuCheckSlots : kFuProbes;
                for (;;) {
                    for (uint32_t k = threadIdx.x; k < slots; k += kFuThreads) {
                        key[k] = 0xffffffffu;
                        val[k] = 0ull;
                    }
                    if (threadIdx.x == 0) s_flag = 0u;
                    __syncthreads();
                    bool ok = true;  // (false: the table is full, and what it holds is of no use)
                    for (int side = 0; side < 2 && ok; ++side) {
                        const uint64_t b = fu_off<MODE>(a, side ? u : r), e = fu_end<MODE>(a, side ? u : r);
                        for (uint64_t k = b + threadIdx.x; k < e && ok; k += kFuThreads) ok = add_arc(key, val, slots - 1u, probes, k, side);
                    }
                    if (!ok) atomicOr(&s_flag, 2u);
                    __syncthreads();
                    bool diff = false;
                    for (uint32_t k = threadIdx.x; k < slots; k += kFuThreads) diff |= val[k] != 0ull;
                    if (diff) atomicOr(&s_flag, 1u);
                    __syncthreads();
                    const uint32_t f = *(volatile uint32_t*)&s_flag;
                    __syncthreads();
                    if ((f & 2u) && key == s_key && a.wide) {
                        // more colours than the shared table holds: once more in global memory
                        val = reinterpret_cast<unsigned long long*>(a.wide + (size_t)blockIdx.x * kFuWideSlots * 12);
                        key = reinterpret_cast<uint32_t*>(val + kFuWideSlots);
                        slots = probes = kFuWideSlots;
                        continue;
                    }
                    if (threadIdx.x == 0) {
                        if (f & 2u) {
                            atomicOr(&w->overflow, 1u);
                            a.list[i] = u | kSingleton;
                        } else {
                            a.fail[u] = (f & 1u) ? 1 : 0;
                            nbad += f & 1u;
                        }
                    }
                    break;
                }
            }
            if (threadIdx.x == 0) s_sum = 0u;
            __syncthreads();
            tot = block_total(nbad);
            if (!fu_barrier<MODE>(w, sync, tot, &more, s_word)) {
                finish(kFuBarrier, round, prev, initial, repairs);
                return;
            }
            if (fu_cg<MODE>(&w->overflow)) {
                if (first && a.res) a.res->failed = nfail + more;
                finish(kFuUndecided, round, prev, initial, repairs);
                return;
            }
        }
        if (nfail + more == 0u) {
            finish(kFuOk, round, prev, initial, repairs);
            return;
        }
        // split the failed nodes off and refine on
        ++repairs;
        if (!pass(true)) {
            finish(kFuBarrier, round, prev, initial, repairs);
            return;
        }
        prev = count;
        if (round >= a.max_rounds) {
            // no pass left: the labels of the partition as it stands, unchecked
            status = kFuNotConverged;
            const uint32_t* __restrict__ cc = a.col[p & 1u];
            for (uint32_t u = gt; u < n; u += nt) {
                const uint32_t c = fu_cg<MODE>(cc + u);
                if (!(c & kSingleton) && fu_cg<MODE>(a.minm + c) > u) atomicMin(a.minm + c, u);
            }
            if (!fu_barrier<MODE>(w, sync, 0u, nullptr, s_word)) {
                finish(kFuBarrier, round, prev, initial, repairs);
                return;
            }
            for (uint32_t u = gt; u < n; u += nt) {
                const uint32_t c = fu_cg<MODE>(cc + u);
                a.out[u] = (c & kSingleton) ? u : fu_cg<MODE>(a.minm + c);
            }
            finish(status, round, prev, initial, repairs);
            return;
        }
    }
}

template <int MODE, bool WEIGHTED>
static __global__ void __launch_bounds__(kFuThreads, 1) k_refine_fused(const __grid_constant__ FusedArgs a)
{
    static_assert(MODE != kFuBlock, "k_refine_block");
    fused_body<MODE, WEIGHTED>(a);
}

struct FusedLayout;
inline __host__ __device__ size_t fused_al(size_t b) { return (b + 255) & ~(size_t)255; }

// Working memory of a fused refinement: offsets of its arrays in one block.
struct FusedLayout {
    size_t col[2], tab[3], minm, list, fail, lrow, lfirst, lsum, ldone, lchunk, words, bytes;
    uint32_t log2tab, long_cap, chunk_cap;
};

inline FusedLayout fused_layout(uint32_t n, uint64_t m)
{
    FusedLayout l{};
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t r = at;
        at += fused_al(bytes);
        return r;
    };
    l.log2tab = 10;
    while ((1ull << l.log2tab) < 2ull * n) ++l.log2tab;
    l.long_cap = (uint32_t)std::min<uint64_t>(n, m / (kFuGroupRow + 1)) + 1u;  // rows that go in chunks
    l.chunk_cap = (uint32_t)(m / kFuChunk) + l.long_cap;                         // at most one partial chunk each
    l.words = take(sizeof(FusedWords));
    for (int i = 0; i < 2; ++i) l.col[i] = take(4ull * n);
    for (int i = 0; i < 3; ++i) l.tab[i] = take(8ull << l.log2tab);
    l.minm = take(4ull << l.log2tab);
    l.list = take(4ull * n);
    l.fail = take(n);
    l.lrow = take(4ull * l.long_cap);
    l.lfirst = take(4ull * l.long_cap);
    l.lsum = take(8ull * l.long_cap);
    l.ldone = take(4ull * l.long_cap);
    l.lchunk = take(4ull * l.chunk_cap);
    l.bytes = at;
    return l;
}

// The rows of a CSR with offsets of 4 or 8 bytes.
inline void fused_csr(FusedArgs& a, const void* off, bool off64)
{
    a.off = off;
    a.off_end = static_cast<const char*>(off) + (off64 ? 8 : 4);
    a.off64 = off64 ? 1 : 0;
}

__host__ __device__ inline void fused_bind(FusedArgs& a, const FusedLayout& l, unsigned char* base)
{
    a.w = reinterpret_cast<FusedWords*>(base + l.words);
    for (int i = 0; i < 2; ++i) a.col[i] = reinterpret_cast<uint32_t*>(base + l.col[i]);
    for (int i = 0; i < 3; ++i) a.tab[i] = reinterpret_cast<unsigned long long*>(base + l.tab[i]);
    a.log2tab = l.log2tab;
    a.minm = reinterpret_cast<uint32_t*>(base + l.minm);
    a.list = reinterpret_cast<uint32_t*>(base + l.list);
    a.fail = base + l.fail;
    a.lrow = reinterpret_cast<uint32_t*>(base + l.lrow);
    a.lfirst = reinterpret_cast<uint32_t*>(base + l.lfirst);
    a.lsum = reinterpret_cast<unsigned long long*>(base + l.lsum);
    a.ldone = reinterpret_cast<uint32_t*>(base + l.ldone);
    a.lchunk = reinterpret_cast<uint32_t*>(base + l.lchunk);
    a.long_cap = l.long_cap;
    a.chunk_cap = l.chunk_cap;
}

// kFuBlock: the graph's arrays are copied to shared memory (from device or
// page-locked host memory), behind the working arrays.
constexpr uint32_t kFuBlockNodes = 1024;
constexpr uint64_t kFuBlockArcs = 8192;
constexpr size_t kFuBlockSmem = 184u << 10;  // beside 43 KB of static shared memory

inline size_t fused_block_smem(const FusedArgs& a, const FusedLayout& l)
{
    return l.bytes + fused_al((size_t)(a.off64 ? 8 : 4) * ((size_t)a.n + 1)) + fused_al(4 * (size_t)a.m) +
           (a.wt ? fused_al(8 * (size_t)a.m) : 0) + (a.init ? fused_al(4 * (size_t)a.n) : 0);
}

// A CSR small enough for one block (offsets side by side, as fused_csr sets them).
inline bool fused_fits_block(const FusedArgs& a, const FusedLayout& l)
{
    return a.n <= kFuBlockNodes && a.m <= kFuBlockArcs && fused_block_smem(a, l) <= kFuBlockSmem;
}

template <bool WEIGHTED>
static __global__ void __launch_bounds__(kFuThreads, 1) k_refine_block(const __grid_constant__ FusedArgs in, const __grid_constant__ FusedLayout l)
{
    extern __shared__ __align__(256) unsigned char s_work[];
    __shared__ FusedArgs s_args;
    const size_t ob = in.off64 ? 8 : 4;
    unsigned char* const off = s_work + l.bytes;
    unsigned char* const idx = off + fused_al(ob * ((size_t)in.n + 1));
    unsigned char* const wt = idx + fused_al(4 * (size_t)in.m);
    unsigned char* const init = wt + (WEIGHTED ? fused_al(8 * (size_t)in.m) : 0);
    auto bring = [&](unsigned char* dst, const void* src, size_t bytes) {
        for (size_t i = threadIdx.x; i < bytes / 4; i += kFuThreads)
            reinterpret_cast<uint32_t*>(dst)[i] = reinterpret_cast<const uint32_t*>(src)[i];
    };
    bring(off, in.off, ob * ((size_t)in.n + 1));
    bring(idx, in.idx, 4 * (size_t)in.m);
    if (WEIGHTED) bring(wt, in.wt, 8 * (size_t)in.m);
    if (in.init) bring(init, in.init, 4 * (size_t)in.n);
    if (threadIdx.x == 0) {
        s_args = in;
        fused_bind(s_args, l, s_work);
        s_args.off = off;
        s_args.off_end = off + ob;
        s_args.idx = reinterpret_cast<const uint32_t*>(idx);
        s_args.wt = reinterpret_cast<const uint64_t*>(wt);
        if (in.init) s_args.init = reinterpret_cast<const uint32_t*>(init);
    }
    __syncthreads();
    fused_body<kFuBlock, WEIGHTED>(s_args);
}

}  // namespace rbsc
