// noalloc.cu -- refinement of a small graph without any device allocation.
//
// Some callers cannot call cudaMalloc at all: code that runs while another
// framework owns the device memory pool, real-time paths that must not take
// the implicit device synchronisation an allocation can cause, or hosts that
// hand this library only pointers into memory they manage themselves.  For
// them rbsc_refine_noalloc refines a small graph (N <= 16384 nodes) in ONE
// kernel launch on the caller's stream.  Inputs and outputs are the caller's
// device buffers; every other byte the kernel needs lives in one file-scope
// __device__ array (g_noalloc_scratch, about 5 MB), which every GPU that loads
// this library holds until the process exits.
//
// The kernel is the one-launch refinement (fused_kernels.cuh), in one thread
// block for the smallest graphs and one cluster of eight otherwise: the same hashed passes, exact check and repair as the
// multi-kernel path, so its labels and counts equal those of rbsc_refine on
// the same graph.
//
// Sharing rules: all calls share the scratch array.  The kernel clears what it
// needs at the start of every call; two calls whose kernels overlap on the GPU
// (different streams, no ordering between them) race on it and give wrong
// results.  The first call on a device resolves the array's device address with
// cudaGetSymbolAddress (with that device current) and keeps it until the
// process exits; make that first call before any stream capture that would
// include it, and make no call on a device after cudaDeviceReset on it.
//
// Unlike the reference (which trusts its input, rbsc.cu:156-180), the kernel
// checks the graph before its first indexed read, as the regular path's
// k_validate does: a malformed graph returns RBSC_ERR_INVALID in d_result.
#include <cstring>
#include <mutex>

#include <cuda_runtime.h>

#include "../../include/rbsc.h"
#include "common.cuh"
#include "refine_kernels.cuh"
#include "fused_kernels.cuh"

using namespace rbsc;

namespace {

constexpr uint32_t kNaMaxNodes = RBSC_NOALLOC_MAX_NODES;
// One cluster: its blocks are resident together without a cooperative launch,
// and its barrier is a hardware one.  Eight blocks is the portable size.
constexpr unsigned kNaBlocks = 8;
constexpr size_t kNaWork = 2u << 20;  // fused_layout of the largest graph: 2,048,000 bytes
constexpr size_t kNaInit = kNaWork + (size_t)kNaBlocks * kFuWideSlots * 12;  // initial colours that the labels overwrite
constexpr size_t kNaBytes = kNaInit + 4 * (size_t)kNaMaxNodes;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNaBytes];

std::mutex g_na_mutex;
unsigned char* g_na_ptr[64] = {};

}  // namespace

rbsc_status rbsc_fail(rbsc_ctx* ctx, rbsc_status code, const char* fmt, ...);

extern "C" rbsc_status rbsc_refine_noalloc(const rbsc_csr* g, const uint32_t* d_init_colors, uint32_t* d_out_labels,
                                           rbsc_noalloc_result* d_result, const rbsc_opts* opts, void* stream)
{
    if (!g || !d_out_labels || !d_result) return rbsc_fail(nullptr, RBSC_ERR_INVALID, "null argument");
    if (g->n > kNaMaxNodes)
        return rbsc_fail(nullptr, RBSC_ERR_TOO_LARGE, "rbsc_refine_noalloc: N = %u exceeds the limit of %u nodes", g->n,
                         kNaMaxNodes);
    if (g->m > RBSC_NOALLOC_MAX_ARCS)
        return rbsc_fail(nullptr, RBSC_ERR_TOO_LARGE, "rbsc_refine_noalloc: M = %llu exceeds the limit of %u arcs",
                         (unsigned long long)g->m, (unsigned)RBSC_NOALLOC_MAX_ARCS);
    if (g->offset_bytes != 4 && g->offset_bytes != 8) return rbsc_fail(nullptr, RBSC_ERR_INVALID, "offset_bytes must be 4 or 8");
    if (!g->offsets || (g->m && !g->indices)) return rbsc_fail(nullptr, RBSC_ERR_INVALID, "null graph array");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return rbsc_fail(nullptr, RBSC_ERR_CUDA, "no current CUDA device");
    unsigned char* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_na_mutex);
        if (!g_na_ptr[dev]) {
            // once per device, with that device current: the device address of
            // the scratch array (its host-side name is not a device address)
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess)
                return rbsc_fail(nullptr, RBSC_ERR_CUDA, "cudaGetSymbolAddress(scratch) failed: %s", cudaGetErrorString(e));
            for (const void* k : {(const void*)k_refine_block<false>, (const void*)k_refine_block<true>}) {
                e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFuBlockSmem);
                if (e != cudaSuccess)
                    return rbsc_fail(nullptr, RBSC_ERR_CUDA, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(e));
            }
            g_na_ptr[dev] = static_cast<unsigned char*>(p);
        }
        scratch = g_na_ptr[dev];
    }
    rbsc_opts o;
    if (opts) o = *opts;
    else rbsc_opts_default(&o);
    const FusedLayout l = fused_layout(g->n, g->m);
    if (l.bytes > kNaWork) return rbsc_fail(nullptr, RBSC_ERR_DEVICE, "rbsc_refine_noalloc: scratch layout");
    FusedArgs a{};
    fused_bind(a, l, scratch);
    a.wide = scratch + kNaWork;
    a.n = g->n;
    a.m = g->m;
    fused_csr(a, g->offsets, g->offset_bytes == 8);
    a.idx = g->indices;
    a.wt = g->weights;
    a.init = d_init_colors;
    a.out = d_out_labels;
    a.na_res = d_result;
    a.validate = 1;
    a.verify = 1;
    a.seed = o.seed;
    a.max_rounds = o.max_rounds ? o.max_rounds : g->n + 1u;
    a.hash_bits = o.test_hash_bits < 0 ? 64u : (uint32_t)o.test_hash_bits;
    ++launch_counter();
    cudaLaunchConfig_t cfg{};
    if (fused_fits_block(a, l)) {
        cfg.gridDim = 1;
        cfg.blockDim = kFuThreads;
        cfg.dynamicSmemBytes = fused_block_smem(a, l);
        cfg.stream = static_cast<cudaStream_t>(stream);
        e = a.wt ? cudaLaunchKernelEx(&cfg, k_refine_block<true>, a, l) : cudaLaunchKernelEx(&cfg, k_refine_block<false>, a, l);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return rbsc_fail(nullptr, RBSC_ERR_CUDA, "k_refine_block launch failed: %s", cudaGetErrorString(e));
        }
        return RBSC_OK;
    }
    if (labels_over_init(d_init_colors, d_out_labels, g->n)) {
        // (one block has them in its shared memory)
        e = cudaMemcpyAsync(scratch + kNaInit, d_init_colors, 4 * (size_t)g->n, cudaMemcpyDeviceToDevice, static_cast<cudaStream_t>(stream));
        if (e != cudaSuccess) {
            cudaGetLastError();
            return rbsc_fail(nullptr, RBSC_ERR_CUDA, "copy of the initial colours failed: %s", cudaGetErrorString(e));
        }
        a.init = reinterpret_cast<const uint32_t*>(scratch + kNaInit);
    }
    cfg.gridDim = kNaBlocks;
    cfg.blockDim = kFuThreads;
    cfg.stream = static_cast<cudaStream_t>(stream);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kNaBlocks;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    e = a.wt ? cudaLaunchKernelEx(&cfg, k_refine_fused<kFuCluster, true>, a) : cudaLaunchKernelEx(&cfg, k_refine_fused<kFuCluster, false>, a);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return rbsc_fail(nullptr, RBSC_ERR_CUDA, "k_refine_fused launch failed: %s", cudaGetErrorString(e));
    }
    return RBSC_OK;
}
