// Batches of small graphs: the graphs are refined together as one resident
// graph (their disjoint union, so the colours form one namespace), then the
// per-graph results are taken out of the union's colouring on the device.
//
// Graphs of at most kBatchNodes nodes: one block per graph groups its nodes by
// colour in shared memory, which gives its histogram entries (colours
// increasing), their counts and smallest nodes, every node's local label, the
// block count and the fingerprint; a scan over the block counts and a copy put
// the entries of all graphs side by side (100,000 graphs of 10 to 500 nodes:
// 0.7 ms, against 4.7 ms for the global sort below and its passes).
//
// A batch with a larger graph:
//   key(u) = (graph of u) << 32 | colour(u)   for every node, value u
//   stable radix sort by key                  -> nodes grouped by graph, then
//                                                by colour, then by node id
//   segment heads + exclusive scan            -> one histogram entry per
//                                                (graph, colour): its colour,
//                                                first position, smallest node
//   per entry                                 -> count, graph fingerprint
//   per node                                  -> local canonical label
//
// A graph's local canonical label of u is the smallest node of u's block in
// u's graph (minus the graph's first node): the same label a refinement of
// that graph alone gives, since the union's coarsest stable partition
// restricted to one graph is that graph's own coarsest stable partition.
#include <algorithm>
#include <chrono>
#include <cstring>

#include <cuda_runtime.h>

#include "../../include/rbsc.h"
#include "common.cuh"
#include "radix.cuh"
#include "scan.cuh"
#include "internal.h"

using namespace rbsc;

namespace {

// The term of one histogram entry in its graph's fingerprint.
__device__ __forceinline__ unsigned long long entry_mix(uint32_t color, uint32_t count)
{
    return fmix64(((uint64_t)color << 32 | count) * kGolden + 0x2545f4914f6cdd1dull);
}

// graph of node u: the largest i with graph_nodes[i] <= u
__global__ void k_batch_keys(uint32_t n, const uint64_t* __restrict__ gn, uint32_t G, const uint32_t* __restrict__ col,
                             unsigned long long* __restrict__ keys, uint32_t* __restrict__ vals)
{
    const uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n) return;
    uint32_t lo = 0, hi = G - 1;
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo + 1) >> 1);
        if (gn[mid] <= u) lo = mid;
        else hi = mid - 1;
    }
    keys[u] = ((unsigned long long)lo << 32) | col[u];
    vals[u] = u;
}

__global__ void k_batch_heads(uint32_t n, const unsigned long long* __restrict__ keys, uint32_t* __restrict__ head)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) head[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

// One histogram entry per segment of equal keys.  ex = exclusive scan of the
// heads; entry of sorted position i = ex[i] + head[i] - 1.
__global__ void k_batch_entries(uint32_t n, const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ vals,
                                const uint32_t* __restrict__ head, const uint32_t* __restrict__ ex,
                                uint32_t* __restrict__ ecolor, uint32_t* __restrict__ estart, uint32_t* __restrict__ emin,
                                uint64_t* __restrict__ hoff)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !head[i]) return;
    const uint32_t e = ex[i];
    const unsigned long long k = keys[i];
    ecolor[e] = (uint32_t)k;
    estart[e] = i;
    emin[e] = vals[i];  // the sort is stable and the values started in node order
    const uint32_t g = (uint32_t)(k >> 32);
    if (i == 0 || (uint32_t)(keys[i - 1] >> 32) != g) hoff[g] = e;
}

// Entry counts and the per-graph fingerprint: the sum over its entries of a
// mix of (colour, count), which does not depend on the order of the entries.
__global__ void k_batch_counts(uint32_t H, uint32_t n, const uint32_t* __restrict__ estart, const uint32_t* __restrict__ ecolor,
                               const unsigned long long* __restrict__ keys, uint32_t* __restrict__ ecount,
                               unsigned long long* __restrict__ fp)
{
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= H) return;
    const uint32_t s = estart[e];
    const uint32_t c = (e + 1 < H ? estart[e + 1] : n) - s;
    ecount[e] = c;
    const uint32_t g = (uint32_t)(keys[s] >> 32);
    atomicAdd(&fp[g], entry_mix(ecolor[e], c));
}

__global__ void k_batch_local(uint32_t n, const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ vals,
                              const uint32_t* __restrict__ head, const uint32_t* __restrict__ ex,
                              const uint32_t* __restrict__ emin, const uint64_t* __restrict__ gn, uint32_t* __restrict__ local)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t e = ex[i] + head[i] - 1u;
    const uint32_t g = (uint32_t)(keys[i] >> 32);
    local[vals[i]] = emin[e] - (uint32_t)gn[g];
}

__global__ void k_batch_blocks(uint32_t G, const uint64_t* __restrict__ hoff, uint32_t* __restrict__ blocks)
{
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g < G) blocks[g] = (uint32_t)(hoff[g + 1] - hoff[g]);
}

constexpr uint32_t kBatchNodes = 2048;
constexpr int kBatchThreads = 256;

// One block per graph (see the top of the file).  A colour is the smallest
// node of its class over the batch, so a node whose colour is a node of its own
// graph needs no sorting: its entry is that node's, and those entries come in
// node order.  Only the nodes whose class starts in an earlier graph are
// sorted; their colours are smaller, so their entries come first.  (Sorting
// every node took 1.27 ms on the 100,000 graphs, this 0.51: most nodes of that
// batch start a class.)  Entries go to the graph's own stretch [gn[g], ...) of
// ecolor / ecount.
__global__ void __launch_bounds__(kBatchThreads) k_batch_graph(const uint64_t* __restrict__ gn, const uint32_t* __restrict__ col,
                                                               uint32_t* __restrict__ local, uint32_t* __restrict__ blocks,
                                                               unsigned long long* __restrict__ fp, uint32_t* __restrict__ ecolor,
                                                               uint32_t* __restrict__ ecount)
{
    __shared__ unsigned long long s_key[kBatchNodes];   // colour << 32 | node, of classes from earlier graphs
    __shared__ uint32_t s_start[kBatchNodes + 1];       // where each of their entries starts
    __shared__ uint32_t s_cnt[kBatchNodes];             // nodes of the class that starts at this node
    __shared__ uint32_t s_far, s_total;
    __shared__ unsigned long long s_fp;
    const uint64_t b = gn[blockIdx.x];
    const uint32_t n = (uint32_t)(gn[blockIdx.x + 1] - b);
    for (uint32_t i = threadIdx.x; i < n; i += kBatchThreads) s_cnt[i] = 0u;
    if (threadIdx.x == 0) {
        s_far = 0u;
        s_fp = 0ull;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += kBatchThreads) {
        const uint32_t c = col[b + i];
        if (c >= (uint32_t)b) {
            local[b + i] = c - (uint32_t)b;
            atomicAdd(&s_cnt[c - (uint32_t)b], 1u);
        } else {
            s_key[atomicAdd(&s_far, 1u)] = (unsigned long long)c << 32 | i;
        }
    }
    __syncthreads();
    const uint32_t far = s_far;
    uint32_t size = 2;
    while (size < far) size <<= 1;
    for (uint32_t i = far + threadIdx.x; i < size; i += kBatchThreads) s_key[i] = ~0ull;
    __syncthreads();
    if (far > 1)
        for (uint32_t k = 2; k <= size; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t t = threadIdx.x; t < size / 2; t += kBatchThreads) {
                    const uint32_t lo = (t & (j - 1)) | (t & ~(j - 1)) << 1, hi = lo | j;
                    const unsigned long long x = s_key[lo], y = s_key[hi];
                    if ((x > y) == ((lo & k) == 0u)) {
                        s_key[lo] = y;
                        s_key[hi] = x;
                    }
                }
                __syncthreads();
            }
    // the sorted ones' entries: each thread looks at consecutive positions
    const uint32_t per = (far + kBatchThreads - 1) / kBatchThreads;
    const uint32_t i0 = min(far, threadIdx.x * per), i1 = min(far, i0 + per);
    auto starts = [&](uint32_t i) { return i == 0 || (uint32_t)(s_key[i] >> 32) != (uint32_t)(s_key[i - 1] >> 32); };
    uint32_t heads = 0;
    for (uint32_t i = i0; i < i1; ++i) heads += starts(i) ? 1u : 0u;
    const uint32_t e0 = block_excl_scan<uint32_t>(heads, &s_total);
    const uint32_t nfar = s_total;
    uint32_t e = e0;
    for (uint32_t i = i0; i < i1; ++i)
        if (starts(i)) s_start[e++] = i;
    if (threadIdx.x == 0) s_start[nfar] = far;
    __syncthreads();
    e = e0;
    for (uint32_t i = i0; i < i1; ++i) {
        if (starts(i)) ++e;
        // the entry's first node: the pairs are in node order inside an entry
        local[b + (uint32_t)s_key[i]] = (uint32_t)s_key[s_start[e - 1]];
    }
    unsigned long long f = 0;
    for (uint32_t x = threadIdx.x; x < nfar; x += kBatchThreads) {
        const uint32_t at = s_start[x], c = (uint32_t)(s_key[at] >> 32), cnt = s_start[x + 1] - at;
        ecolor[b + x] = c;
        ecount[b + x] = cnt;
        f += entry_mix(c, cnt);
    }
    // then the classes that start in this graph, in node order
    uint32_t base = nfar;
    for (uint32_t i = 0; i < n; i += kBatchThreads) {
        const uint32_t u = i + threadIdx.x, cnt = u < n ? s_cnt[u] : 0u;
        const uint32_t at = base + block_excl_scan<uint32_t>(cnt ? 1u : 0u, &s_total);
        if (cnt) {
            ecolor[b + at] = (uint32_t)b + u;
            ecount[b + at] = cnt;
            f += entry_mix((uint32_t)b + u, cnt);
        }
        base += s_total;
        __syncthreads();
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) f += __shfl_xor_sync(0xffffffffu, f, d);
    if ((threadIdx.x & 31) == 0 && f) atomicAdd(&s_fp, f);
    __syncthreads();
    if (threadIdx.x == 0) {
        blocks[blockIdx.x] = base;
        fp[blockIdx.x] = s_fp;
    }
}

// The graphs' entries side by side.
__global__ void __launch_bounds__(kBatchThreads) k_batch_join(const uint64_t* __restrict__ gn, const uint64_t* __restrict__ hoff,
                                                              const uint32_t* __restrict__ ecolor, const uint32_t* __restrict__ ecount,
                                                              uint32_t* __restrict__ hcolor, uint32_t* __restrict__ hcount)
{
    const uint64_t b = gn[blockIdx.x], h = hoff[blockIdx.x];
    const uint32_t k = (uint32_t)(hoff[blockIdx.x + 1] - h);
    for (uint32_t x = threadIdx.x; x < k; x += kBatchThreads) {
        hcolor[h + x] = ecolor[b + x];
        hcount[h + x] = ecount[b + x];
    }
}

unsigned grid_of(uint64_t n) { return (unsigned)std::max<uint64_t>(1, (n + 255) / 256); }

}  // namespace

#define BK(call)                                                                     \
    do {                                                                             \
        cudaError_t e_ = (call);                                                     \
        if (e_ != cudaSuccess) { st = rbsc_cuda_fail(ctx, e_, #call, __LINE__); goto done; } \
    } while (0)
#define BKS(call)                              \
    do {                                       \
        st = (call);                           \
        if (st != RBSC_OK) goto done;          \
    } while (0)

extern "C" rbsc_status rbsc_graph_batch_refine(rbsc_ctx* ctx, rbsc_graph* g, const uint64_t* graph_nodes, uint32_t num_graphs,
                                               const uint32_t* init_colors, rbsc_batch_result* out, rbsc_stats* stats)
{
    if (!ctx || !g || !graph_nodes || !out) return rbsc_fail(ctx, RBSC_ERR_INVALID, "null argument");
    if (num_graphs == 0) return rbsc_fail(ctx, RBSC_ERR_INVALID, "empty batch");
    if (graph_nodes[0] != 0 || graph_nodes[num_graphs] != g->n)
        return rbsc_fail(ctx, RBSC_ERR_INVALID, "graph_nodes must start at 0 and end at N");
    uint64_t largest = 0;
    for (uint32_t i = 0; i < num_graphs; ++i) {
        if (graph_nodes[i + 1] <= graph_nodes[i]) return rbsc_fail(ctx, RBSC_ERR_INVALID, "graph %u has no node", i);
        largest = std::max(largest, graph_nodes[i + 1] - graph_nodes[i]);
    }
    const bool small = largest <= kBatchNodes;
    rbsc_status st = RBSC_OK;
    auto t0 = std::chrono::steady_clock::now();
    cudaStream_t s = ctx->stream;
    const uint32_t n = g->n, G = num_graphs;
    int gbits = 0;
    while (gbits < 32 && (1ull << gbits) < G) ++gbits;
    unsigned long long *keys = nullptr, *keys2 = nullptr, *fp = nullptr;
    uint32_t *vals = nullptr, *vals2 = nullptr, *head = nullptr, *ex = nullptr, *ecolor = nullptr, *estart = nullptr,
             *emin = nullptr, *ecount = nullptr, *local = nullptr, *blocks = nullptr;
    uint64_t* gn = nullptr;
    uint64_t* hoff = nullptr;
    void* tmp = nullptr;
    bool alt = false;
    uint32_t H = 0;
    uint64_t hH = 0;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    float batch_ms = 0.f;
    std::chrono::steady_clock::time_point c0;  // the first result copy
    // the refinement of the union
    BKS(rbsc_graph_refine(ctx, g, init_colors, nullptr, stats));
    BK(cudaEventCreate(&e0));
    BK(cudaEventCreate(&e1));
    BK(cudaEventRecord(e0, s));
    BKS(dev_alloc(ctx, (void**)&gn, 8 * ((size_t)G + 1)));
    BKS(dev_alloc(ctx, (void**)&hoff, 8 * ((size_t)G + 1)));
    BKS(dev_alloc(ctx, (void**)&fp, 8 * (size_t)G));
    BKS(dev_alloc(ctx, (void**)&local, 4 * (size_t)n));
    BKS(dev_alloc(ctx, (void**)&blocks, 4 * (size_t)G));
    BK(cudaMemcpyAsync(gn, graph_nodes, 8 * ((size_t)G + 1), cudaMemcpyHostToDevice, s));
    if (small) {
        BKS(dev_alloc(ctx, (void**)&head, 4 * (size_t)n));
        BKS(dev_alloc(ctx, (void**)&ex, 4 * (size_t)n));
        BKS(dev_alloc(ctx, (void**)&ecount, 4 * (size_t)n));
        BKS(dev_alloc(ctx, (void**)&vals, 4 * (size_t)n));
        BKS(dev_alloc(ctx, &tmp, scan_temp_bytes<uint64_t>((uint64_t)G + 1) + 1024));
        ++rbsc::launch_counter();
        k_batch_graph<<<G, kBatchThreads, 0, s>>>(gn, g->d_out, local, blocks, fp, head, ex);
        BK(cudaGetLastError());
        BK((exclusive_scan<uint32_t, uint64_t>(blocks, hoff, G, hoff + G, tmp, s)));
        ++rbsc::launch_counter();
        ecolor = vals;
        k_batch_join<<<G, kBatchThreads, 0, s>>>(gn, hoff, head, ex, ecolor, ecount);
        BK(cudaGetLastError());
        BK(cudaEventRecord(e1, s));
        BK(cudaMemcpyAsync(&hH, hoff + G, 8, cudaMemcpyDeviceToHost, s));
        // the colours (final already) travel beside these kernels
        c0 = std::chrono::steady_clock::now();
        if (out->colors) BKS(copy_out(ctx, out->colors, g->d_out, 4 * (size_t)n, ctx->side));
        BK(cudaStreamSynchronize(s));
        H = (uint32_t)hH;
    } else {
        BKS(dev_alloc(ctx, (void**)&keys, 8 * (size_t)n));
        BKS(dev_alloc(ctx, (void**)&keys2, 8 * (size_t)n));
        BKS(dev_alloc(ctx, (void**)&vals, 4 * (size_t)n));
        BKS(dev_alloc(ctx, (void**)&vals2, 4 * (size_t)n));
        BKS(dev_alloc(ctx, (void**)&head, 4 * (size_t)n));
        BKS(dev_alloc(ctx, (void**)&ex, 4 * ((size_t)n + 1)));
        BKS(dev_alloc(ctx, &tmp, std::max(radix_temp_bytes(n), scan_temp_bytes<uint32_t>((uint64_t)n + 1)) + 1024));
        ++rbsc::launch_counter();
        k_batch_keys<<<grid_of(n), 256, 0, s>>>(n, gn, G, g->d_out, keys, vals);
        BK(cudaGetLastError());
        BK(radix_sort<uint32_t>(keys, keys2, vals, vals2, n, 0, 32 + gbits, tmp, s, &alt));
        if (alt) {
            std::swap(keys, keys2);
            std::swap(vals, vals2);
        }
        ++rbsc::launch_counter();
        k_batch_heads<<<grid_of(n), 256, 0, s>>>(n, keys, head);
        BK(cudaGetLastError());
        BK((exclusive_scan<uint32_t, uint32_t>(head, ex, n, ex + n, tmp, s)));
        BK(cudaMemcpyAsync(&H, ex + n, 4, cudaMemcpyDeviceToHost, s));
        BK(cudaStreamSynchronize(s));
        // entries reuse the second sort buffers (free after the sort)
        ecolor = vals2;
        estart = reinterpret_cast<uint32_t*>(keys2);
        emin = estart + n;
        BKS(dev_alloc(ctx, (void**)&ecount, 4 * ((size_t)H + 1)));
        BK(cudaMemsetAsync(fp, 0, 8 * (size_t)G, s));
        hH = H;
        BK(cudaMemcpyAsync(hoff + G, &hH, 8, cudaMemcpyHostToDevice, s));
        ++rbsc::launch_counter();
        k_batch_entries<<<grid_of(n), 256, 0, s>>>(n, keys, vals, head, ex, ecolor, estart, emin, hoff);
        ++rbsc::launch_counter();
        k_batch_counts<<<grid_of(H), 256, 0, s>>>(H, n, estart, ecolor, keys, ecount, fp);
        ++rbsc::launch_counter();
        k_batch_local<<<grid_of(n), 256, 0, s>>>(n, keys, vals, head, ex, emin, gn, local);
        ++rbsc::launch_counter();
        k_batch_blocks<<<grid_of(G), 256, 0, s>>>(G, hoff, blocks);
        BK(cudaGetLastError());
        BK(cudaEventRecord(e1, s));
        BK(cudaStreamSynchronize(s));
        c0 = std::chrono::steady_clock::now();
        if (out->colors) BKS(copy_out(ctx, out->colors, g->d_out, 4 * (size_t)n, s));
    }
    if (out->local) BKS(copy_out(ctx, out->local, local, 4 * (size_t)n, s));
    if (out->blocks) BK(cudaMemcpyAsync(out->blocks, blocks, 4 * (size_t)G, cudaMemcpyDeviceToHost, s));
    if (out->fingerprint) BK(cudaMemcpyAsync(out->fingerprint, fp, 8 * (size_t)G, cudaMemcpyDeviceToHost, s));
    if (out->hist_offsets) BK(cudaMemcpyAsync(out->hist_offsets, hoff, 8 * ((size_t)G + 1), cudaMemcpyDeviceToHost, s));
    if (out->hist_colors) BKS(copy_out(ctx, out->hist_colors, ecolor, 4 * (size_t)H, s));
    if (out->hist_counts) BKS(copy_out(ctx, out->hist_counts, ecount, 4 * (size_t)H, s));
    BK(cudaStreamSynchronize(ctx->side));
    BK(cudaStreamSynchronize(s));
    cudaEventElapsedTime(&batch_ms, e0, e1);
    if (stats) {
        stats->device_ms += batch_ms;
        if (out->colors) stats->d2h_bytes = 4ull * n;
        stats->d2h_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - c0).count();
        stats->time_s += std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    }
done:
    cudaStreamSynchronize(s);
    cudaStreamSynchronize(ctx->side);
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    dev_free(ctx, (void*&)gn);
    dev_free(ctx, (void*&)keys);
    dev_free(ctx, (void*&)keys2);
    dev_free(ctx, (void*&)vals);
    dev_free(ctx, (void*&)vals2);
    dev_free(ctx, (void*&)head);
    dev_free(ctx, (void*&)ex);
    dev_free(ctx, tmp);
    dev_free(ctx, (void*&)ecount);
    dev_free(ctx, (void*&)hoff);
    dev_free(ctx, (void*&)fp);
    dev_free(ctx, (void*&)local);
    dev_free(ctx, (void*&)blocks);
    return st;
}

extern "C" rbsc_status rbsc_batch_refine(rbsc_ctx* ctx, const rbsc_csr* graphs, const uint64_t* graph_nodes, uint32_t num_graphs,
                                         const uint32_t* init_colors, rbsc_batch_result* out, rbsc_stats* stats)
{
    if (!ctx) return rbsc_fail(nullptr, RBSC_ERR_INVALID, "null context");
    auto t0 = std::chrono::steady_clock::now();
    rbsc_graph* g = nullptr;
    rbsc_status st = graph_upload_oneshot(ctx, graphs, init_colors, &g, nullptr, nullptr);
    if (st != RBSC_OK) return st;
    st = rbsc_graph_batch_refine(ctx, g, graph_nodes, num_graphs, init_colors, out, stats);
    rbsc_graph_free(g);
    if (st == RBSC_OK && stats) stats->time_s = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    return st;
}
