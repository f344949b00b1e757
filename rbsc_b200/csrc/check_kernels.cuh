// check_kernels.cuh -- the rows that a one-launch refinement's exact check left
// undecided (fused_kernels.cuh, list_kernels.cuh): those with more colours than
// a block's table in shared memory holds, or more arcs than it may count.
//
// They are few and long (both copies of a hub of a lifted skewed graph, pages
// with the same list of thousands of links), so all warps share their arcs:
// each row and its class's smallest member count into a table of their own in
// global memory, + for the member's arcs and - for the node's, and every count
// must end at 0.  Any doubt (a table that is too full) counts as a difference:
// the caller then refines launch by launch, whose check decides.
//
// Bound by the random sectors of the gathers and counts.  A double cover of
// R-MAT-18 with 14.3 M arcs (1,976 rows above 1,024 arcs), resident from one
// class, whole call: 1.85 ms; launch by launch, whose check sorts such rows,
// 5.25, after one or two refinements for nothing 19.6.  Weighted 2.61 / 23.9 /
// 37.2 ms.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "common.cuh"
#include "fused_kernels.cuh"
#include "list_kernels.cuh"

namespace rbsc {

constexpr uint32_t kCkChunk = 512;    // arcs of a warp's piece of a row
constexpr uint32_t kCkProbes = 1024;  // the tables are at most half full

struct CheckRow {
    uint32_t u, r;      // the node, its class's smallest member
    uint32_t du, dr;    // their arcs
    uint32_t first;     // the row's first piece: the member's, then the node's
    uint32_t mask;      // of its table
    uint64_t base;      // the table's place
};

// The marked nodes of a check's list.
static __global__ void k_check_rows(const FusedArgs a, uint32_t nlist, const uint32_t* __restrict__ col, CheckRow* __restrict__ rows,
                                    uint32_t* __restrict__ count)
{
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nlist; i += gridDim.x * blockDim.x) {
        const uint32_t e = a.list[i];
        if (!(e & kSingleton)) continue;
        CheckRow x{};
        x.u = e & ~kSingleton;
        x.r = a.minm[col[x.u] & ~kSlotBit];
        x.du = (uint32_t)(fu_end(a, x.u) - fu_off(a, x.u));
        x.dr = (uint32_t)(fu_end(a, x.r) - fu_off(a, x.r));
        rows[atomicAdd(count, 1u)] = x;
    }
}

template <bool WEIGHTED>
static __global__ void __launch_bounds__(256) k_check_count(const FusedArgs a, const uint32_t* __restrict__ col,
                                                            const CheckRow* __restrict__ rows, uint32_t nrows, uint32_t pieces,
                                                            uint32_t* __restrict__ keys, unsigned long long* __restrict__ vals,
                                                            uint32_t* __restrict__ bad)
{
    const int lane = threadIdx.x & 31;
    for (uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < pieces; p += (gridDim.x * blockDim.x) >> 5) {
        uint32_t lo = 0, hi = nrows - 1;  // the row of piece p
        while (lo < hi) {
            const uint32_t mid = lo + ((hi - lo + 1) >> 1);
            if (rows[mid].first <= p) lo = mid;
            else hi = mid - 1;
        }
        const CheckRow x = rows[lo];
        const uint32_t k = p - x.first, kr = (x.dr + kCkChunk - 1) / kCkChunk;
        const bool member = k < kr;
        const uint64_t row = fu_off(a, member ? x.r : x.u), b = row + (uint64_t)(member ? k : k - kr) * kCkChunk;
        const uint64_t e = min(row + (member ? x.dr : x.du), b + kCkChunk);
        for (uint64_t i0 = b; i0 < e; i0 += 32) {
            const bool in = i0 + lane < e;
            const uint32_t c = in ? col[a.idx[i0 + lane]] : 0xffffffffu;
            unsigned long long v = !in ? 0ull : WEIGHTED ? a.wt[i0 + lane] : 1ull;
            if (!member) v = 0ull - v;
            // a hub of one colour: one atomic for the warp
            int same = 0;
            __match_all_sync(0xffffffffu, c, &same);
            if (same) v = fu_warp_sum(v, 32);
            if (!in || (same && lane)) continue;
            uint32_t h = (uint32_t)((uint64_t)c * kGolden >> 32) & x.mask, left = kCkProbes;
            for (; left; --left, h = (h + 1u) & x.mask) {
                uint32_t o = __ldcg(keys + x.base + h);
                if (o == 0xffffffffu) o = atomicCAS(keys + x.base + h, 0xffffffffu, c);
                if (o == 0xffffffffu || o == c) break;
            }
            if (left) atomicAdd(vals + x.base + h, v);
            else atomicOr(bad, 1u);
        }
        __syncwarp();
    }
}

static __global__ void __launch_bounds__(256) k_check_zero(uint64_t slots, const unsigned long long* __restrict__ vals, uint32_t* __restrict__ bad)
{
    bool diff = false;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < slots; i += (uint64_t)gridDim.x * blockDim.x) diff |= vals[i] != 0ull;
    if (__any_sync(0xffffffffu, diff) && (threadIdx.x & 31) == 0) atomicOr(bad, 1u);
}

}  // namespace rbsc
