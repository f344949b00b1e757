// deep_kernels.cuh -- the long tail of a deep refinement, driven by changes.
//
// A graph with long chains needs hundreds of passes in which only a few nodes
// change class, yet a full pass reads every active arc (170 passes over a
// 325,000-node lift beside a chain of 170 nodes: 38 us each).  Once the passes
// are known to be many (fused.cu), the rest runs on a work list:
//
//   sig[u]   the sum of u's arc terms under one salt, kept up to date: when v
//            moves from class a to class b, every predecessor u of v gets
//            w * (H(b) - H(a)) (predecessors from a transpose of the arcs
//            between nodes that can still change)
//   T        the nodes whose sum changed in the last pass
//   S[c]     the sum shared by the members of class c that are not in T
//
// A pass groups the members of T whose sum differs from S[class] by (class,
// sum).  A class that keeps a member outside keeps its id; of a class whose
// members all moved, the largest group keeps it; the other groups are new
// classes.  Ids are not used again: a class of s nodes that sheds one node a
// pass, by a change of all others, uses s - 2 of them.  That is the partition
// a full pass gives: members outside T see the same multiset of classes as
// before, and a node in T sees a class id that no node outside T sees.  No new
// class: the fixpoint (the same pass that a full pass would find unchanged).
//
// One block of 1024 threads runs the passes with its lists and tables in
// shared memory: about five dependent L2 accesses a pass, 4 us, no grid barrier
// (that lift: 6.3 -> 1.13 ms, of which 0.65 the 161 passes here, 0.12 the
// transpose and sums, 0.29 the 9 full passes before, 0.12 the confirmation).
// A pass with more than kIncCap changed sums ends it (done = 0) and the
// full passes go on.  The result is confirmed by one full pass and the exact
// check, as any other.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "common.cuh"
#include "fused_kernels.cuh"

namespace rbsc {

constexpr uint32_t kIncCap = 2048;      // changed sums of a pass
constexpr uint32_t kIncSlots = 4096;    // per table, at most half taken
constexpr uint32_t kIncMark = 1u << 30; // colour word of k_inc_mark: the node changed class in the last full pass
constexpr uint32_t kIncMaxNodes = 1u << 22;  // class ids (slots below 2^23, then at most 2^22 new ones) stay below kIncMark
constexpr uint64_t kIncNoSum = ~0ull;   // S of a class with no member outside T

struct IncCounters {
    uint32_t tcount;   // nodes in T
    uint32_t done;
    uint32_t rounds;   // passes run, including earlier ones
    uint32_t blocks;
    uint32_t over;     // max_rounds reached
};

// Class sizes; the in-degrees of nodes that can change, over sources that can.
static __global__ void k_inc_degrees(FusedArgs a, const uint32_t* __restrict__ col, uint32_t* __restrict__ size,
                                     uint32_t* __restrict__ indeg)
{
    const uint32_t gl = threadIdx.x & 7u, g = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, ng = (gridDim.x * blockDim.x) >> 3;
    for (uint32_t u = g; u < a.n; u += ng) {
        const uint32_t c = col[u];
        if (c & kSingleton) continue;
        if (gl == 0) atomicAdd(&size[c], 1u);
        const uint64_t e = fu_end(a, u);
        for (uint64_t i = fu_off(a, u) + gl; i < e; i += 8) {
            const uint32_t v = a.idx[i];
            if (!(col[v] & kSingleton)) atomicAdd(&indeg[v], 1u);
        }
    }
}

// The transpose (cursor: row starts on entry, row ends on exit), and for each
// class of the previous pass its largest part: best = size << 32 | class.
template <bool WEIGHTED>
static __global__ void k_inc_transpose(FusedArgs a, const uint32_t* __restrict__ col, const uint32_t* __restrict__ old,
                                       const uint32_t* __restrict__ size, uint32_t* __restrict__ cursor, uint32_t* __restrict__ tsrc,
                                       uint64_t* __restrict__ twt, unsigned long long* __restrict__ best)
{
    const uint32_t gl = threadIdx.x & 7u, g = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, ng = (gridDim.x * blockDim.x) >> 3;
    for (uint32_t u = g; u < a.n; u += ng) {
        const uint32_t c = col[u];
        if (c & kSingleton) continue;
        if (gl == 0) {
            const unsigned long long v = ((unsigned long long)size[c] << 32) | c;
            if (__ldcg(&best[old[u]]) < v) atomicMax(&best[old[u]], v);
        }
        const uint64_t e = fu_end(a, u);
        for (uint64_t i = fu_off(a, u) + gl; i < e; i += 8) {
            const uint32_t v = a.idx[i];
            if (col[v] & kSingleton) continue;
            const uint32_t p = atomicAdd(&cursor[v], 1u);
            tsrc[p] = u;
            if (WEIGHTED) twt[p] = a.wt[i];
        }
    }
}

// colm = colour word, marked when the node is not in its old class's largest part.
static __global__ void k_inc_mark(uint32_t n, const uint32_t* __restrict__ col, const uint32_t* __restrict__ old,
                                  const unsigned long long* __restrict__ best, uint32_t* __restrict__ colm)
{
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
        const uint32_t c = col[u];
        colm[u] = !(c & kSingleton) && (uint32_t)best[old[u]] != c ? c | kIncMark : c;
    }
}

// The sums under the tail's salt; T = the nodes with a marked successor, S from the others.
template <bool WEIGHTED>
static __global__ void k_inc_sums(FusedArgs a, const uint32_t* __restrict__ colm, const uint32_t* __restrict__ size, uint64_t salt,
                                  unsigned long long* __restrict__ sig, unsigned long long* __restrict__ S,
                                  uint32_t* __restrict__ tlist, IncCounters* __restrict__ ctr)
{
    const uint32_t gl = threadIdx.x & 7u, g = (blockIdx.x * blockDim.x + threadIdx.x) >> 3, ng = (gridDim.x * blockDim.x) >> 3;
    for (uint32_t u0 = g & ~3u; u0 < a.n; u0 += ng) {  // the four groups of a warp run together
        const uint32_t u = u0 + (g & 3u);
        const uint32_t c = u < a.n ? colm[u] & ~kIncMark : kSingleton;
        const bool act = !(c & kSingleton);
        uint64_t s = 0;
        uint32_t touched = 0;
        if (act) {
            const uint64_t e = fu_end(a, u);
            for (uint64_t i = fu_off(a, u) + gl; i < e; i += 8) {
                const uint32_t w = colm[a.idx[i]];
                touched |= w & kIncMark;
                const uint64_t t = fu_term(w & ~kIncMark, salt);
                s += WEIGHTED ? t * a.wt[i] : t;
            }
        }
#pragma unroll
        for (int d = 4; d > 0; d >>= 1) {
            s += __shfl_xor_sync(0xffffffffu, s, d);
            touched |= __shfl_xor_sync(0xffffffffu, touched, d);
        }
        if (act && gl == 0) {
            sig[u] = s;
            if (touched) {
                const uint32_t p = atomicAdd(&ctr->tcount, 1u);
                if (p < kIncCap) tlist[p] = u;
            } else {
                S[c] = s;  // the same value from every such member
            }
        }
    }
}

struct IncArgs {
    uint32_t* col;               // class ids, kSingleton | node for a class of one
    unsigned long long* sig;
    unsigned long long* S;       // per class id (end_id words)
    uint32_t* size;
    const uint32_t* tend;        // transpose: row ends (a row starts where the one before ends)
    const uint32_t* tsrc;
    const uint64_t* twt;
    uint32_t* tflag;             // pass that last put the node into T (zero at the start)
    const uint32_t* tlist;
    IncCounters* ctr;
    FusedResult* res;
    uint64_t salt;
    uint32_t first_id, end_id;   // ids from the one on are free, up to the other
    uint32_t round, blocks, max_rounds;
};

struct IncSmem {
    unsigned long long ts[kIncCap];     // sum of each changed node
    unsigned long long kkey[kIncSlots]; // groups: fingerprint of (class, sum)
    unsigned long long cbest[kIncSlots];// classes: largest group (count << 32 | group)
    uint32_t tu[2][kIncCap];            // T of this pass and the next
    uint32_t tk[kIncCap];               // group (kIncSlots: unchanged)
    uint32_t tb[kIncCap], te[kIncCap];  // transpose row
    uint32_t wl[kIncCap];               // positions of the nodes that change class
    uint32_t kcnt[kIncSlots], kid[kIncSlots], kcls[kIncSlots];
    uint32_t ckey[kIncSlots], cch[kIncSlots], csize[kIncSlots];
    uint32_t nt, nnext, nw, nnew, nid;
};

template <bool WEIGHTED>
static __global__ void __launch_bounds__(1024, 1) k_inc_passes(IncArgs a)
{
    extern __shared__ __align__(16) unsigned char s_raw[];
    IncSmem& s = *reinterpret_cast<IncSmem*>(s_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    uint32_t round = a.round, blocks = a.blocks, cur = 0, stamp = 0, done = 0, over = 0;
    uint32_t nt = a.ctr->tcount;
    // the tables' first 2^lg slots are used, at least twice the nodes of T
    auto log2_slots = [](uint32_t t) { return t <= 32u ? 6u : 33u - (uint32_t)__clz(t - 1u); };
    uint32_t lg = 12;
    auto clear = [&]() {
        for (uint32_t i = tid; i < (1u << lg); i += 1024) {
            s.kkey[i] = 0ull;
            s.kcnt[i] = 0u;
            s.ckey[i] = 0xffffffffu;
            s.cch[i] = 0u;
            s.cbest[i] = 0ull;
        }
    };
    clear();
    if (nt <= kIncCap)
        for (uint32_t i = tid; i < nt; i += 1024) s.tu[0][i] = a.tlist[i];
    if (tid == 0) s.nid = a.first_id;
    __syncthreads();
    while (nt <= kIncCap) {
        if (round >= a.max_rounds) {
            over = 1;
            break;
        }
        if (nt > a.end_id - s.nid) break;  // a pass takes at most an id per node of T
        ++stamp;
        lg = log2_slots(nt);
        const uint32_t slots = 1u << lg, mask = slots - 1u;
        if (tid == 0) s.nnext = s.nw = s.nnew = 0u;
        // group the changed nodes by (class, sum); count them per class
        for (uint32_t i = tid; i < nt; i += 1024) {
            const uint32_t u = s.tu[cur][i];
            const uint32_t c = __ldcg(a.col + u);
            const uint64_t x = __ldcg(a.sig + u);
            s.tb[i] = u ? __ldg(a.tend + u - 1) : 0u;
            s.te[i] = __ldg(a.tend + u);
            uint32_t k = kIncSlots;
            if (!(c & kSingleton)) {
                const uint32_t n_c = __ldcg(a.size + c);
                if (x != __ldcg(a.S + c)) {
                    uint32_t h = (c * 0x9e3779b1u) >> (32 - lg);
                    for (;; h = (h + 1u) & mask) {  // at most half of the slots are taken
                        const uint32_t o = atomicCAS(&s.ckey[h], 0xffffffffu, c);
                        if (o == 0xffffffffu || o == c) break;
                    }
                    if (atomicAdd(&s.cch[h], 1u) == 0u) s.csize[h] = n_c;
                    uint64_t f = fmix64(x ^ (((uint64_t)c + 1ull) * kGolden));
                    f = f ? f : 1ull;
                    k = (uint32_t)(f >> (64 - lg));
                    for (;; k = (k + 1u) & mask) {
                        const unsigned long long o = atomicCAS(&s.kkey[k], 0ull, (unsigned long long)f);
                        if (o == 0ull || o == f) break;
                    }
                    if (atomicAdd(&s.kcnt[k], 1u) == 0u) s.kcls[k] = h;
                    s.ts[i] = x;
                }
            }
            s.tk[i] = k;
        }
        __syncthreads();
        for (uint32_t k = tid; k < slots; k += 1024)
            if (s.kkey[k]) {
                const uint32_t h = s.kcls[k];
                if (s.cch[h] == s.csize[h]) atomicMax(&s.cbest[h], ((unsigned long long)s.kcnt[k] << 32) | k);
            }
        __syncthreads();
        // an id for every group: the class's own for the group that keeps it
        for (uint32_t k = tid; k < slots; k += 1024)
            if (s.kkey[k]) {
                const uint32_t h = s.kcls[k], c = s.ckey[h];
                const bool all = s.cch[h] == s.csize[h];
                if (all && (uint32_t)s.cbest[h] == k) {
                    s.kid[k] = c;
                    a.size[c] = s.kcnt[k];
                } else {
                    s.kid[k] = s.kcnt[k] == 1u ? kSingleton : atomicAdd(&s.nid, 1u);  // a class of one: by its node
                    if (s.kcnt[k] > 1u) a.size[s.kid[k]] = s.kcnt[k];
                    atomicAdd(&s.nnew, 1u);
                }
            }
        for (uint32_t h = tid; h < slots; h += 1024)
            if (s.ckey[h] != 0xffffffffu && s.cch[h] != s.csize[h]) a.size[s.ckey[h]] = s.csize[h] - s.cch[h];
        __syncthreads();
        for (uint32_t i = tid; i < nt; i += 1024) {
            const uint32_t k = s.tk[i];
            if (k == kIncSlots) continue;
            const uint32_t id = s.kid[k], u = s.tu[cur][i], c = s.ckey[s.kcls[k]];
            if (id & kSingleton) {
                a.col[u] = kSingleton | u;
                a.tflag[u] = 0xffffffffu;  // never in T again
            } else {
                a.S[id] = s.ts[i];
                if (id != c) a.col[u] = id;
            }
            if (id != c) s.wl[atomicAdd(&s.nw, 1u)] = i;
        }
        __syncthreads();
        const uint32_t nnew = s.nnew, nw = s.nw;
        ++round;
        blocks += nnew;
        if (tid == 0 && round < (uint32_t)kRoundLog) a.res->round_blocks[round] = blocks;
        if (nnew == 0u) {
            done = 1;
            break;
        }
        // the predecessors of the nodes that changed class: a warp per node
        for (uint32_t q = warp; q < nw; q += 32) {
            const uint32_t i = s.wl[q], u = s.tu[cur][i], k = s.tk[i], id = s.kid[k];
            const uint64_t d = fu_term((id & kSingleton) ? (kSingleton | u) : id, a.salt) - fu_term(s.ckey[s.kcls[k]], a.salt);
            const uint32_t b = s.tb[i], e = s.te[i];
            for (uint32_t j = b + lane; j < e; j += 32) {
                const uint32_t v = __ldg(a.tsrc + j);
                atomicAdd(a.sig + v, WEIGHTED ? d * __ldg(reinterpret_cast<const unsigned long long*>(a.twt) + j) : (unsigned long long)d);
                if (atomicMax(a.tflag + v, stamp) < stamp) {
                    const uint32_t p = atomicAdd(&s.nnext, 1u);
                    if (p < kIncCap) s.tu[cur ^ 1u][p] = v;
                }
            }
        }
        __threadfence();
        __syncthreads();
        clear();
        nt = s.nnext;
        cur ^= 1u;
        __syncthreads();
    }
    if (!done && round >= a.max_rounds) over = 1;  // (a wide last pass ends the loop before the test in it)
    if (tid == 0) {
        a.ctr->done = done;
        a.ctr->rounds = round;
        a.ctr->blocks = blocks;
        a.ctr->over = over;
    }
}

}  // namespace rbsc
