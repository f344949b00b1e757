// hostcopy.cu -- copies between the device and pageable host memory.
//
// cudaMemcpyAsync moves pageable memory through a pinned buffer of the driver,
// filled by the calling thread alone: 12-16 GB/s on a link of 55.  Large
// copies go through this context's own pinned slots instead, filled (or
// emptied) by several threads, each with slots of its own, so that the link is
// the bound and an output's first-touch page faults are shared out.  Order on
// the stream and the meaning of the call stay those of a pageable
// cudaMemcpyAsync: the source may change when copy_in returns, the data is
// there when copy_out returns.  The threads are started with the first such
// copy, sleep between copies and end with the context.
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <functional>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/rbsc.h"
#include "internal.h"

namespace {

constexpr size_t kSlot = 1u << 20;       // bytes of a slot: the largest chunk
// Smaller copies stay with the driver, whose one thread keeps up while the
// array is in cache (upload of 14 MB 0.92 ms, by threads 1.45; 32 MB 1.8 / 2.2;
// 60 MB 3.8 / 2.9; 200 MB 15 / 5).
constexpr size_t kWorth = 40u << 20;
constexpr unsigned kMaxThreads = 8;

struct Chunk {
    char* dev;
    char* host;
    size_t bytes;
};

}  // namespace

// The pinned slots of a context: two per thread, each with the event of the
// copy that last used it; and its threads.
struct HostCopier {
    unsigned threads = 0;  // the caller is thread 0
    char* mem = nullptr;
    cudaEvent_t ev[kMaxThreads * 2] = {};
    std::vector<std::thread> ts;
    std::mutex mu;
    std::condition_variable wake, idle;
    const std::function<void(unsigned)>* job = nullptr;
    uint64_t gen = 0;
    unsigned running = 0;
    bool stop = false;

    void main(unsigned t)
    {
        std::unique_lock<std::mutex> lk(mu);
        for (uint64_t seen = 0;;) {
            wake.wait(lk, [&] { return stop || gen != seen; });
            if (stop) return;
            seen = gen;
            const auto* f = job;
            lk.unlock();
            (*f)(t);
            lk.lock();
            if (--running == 0) idle.notify_one();
        }
    }

    // Starts the threads; those that cannot be started are done without.
    void start(unsigned want)
    {
        threads = 1;
        try {
            ts.reserve(want);
            while (threads < want) {
                ts.emplace_back(&HostCopier::main, this, threads);
                ++threads;
            }
        } catch (const std::system_error&) {
        } catch (const std::bad_alloc&) {
        }
    }

    // f(t) on every thread t; returns when all are done.
    void run(const std::function<void(unsigned)>& f)
    {
        {
            std::lock_guard<std::mutex> lk(mu);
            job = &f;
            running = (unsigned)ts.size();
            ++gen;
        }
        wake.notify_all();
        f(0);
        std::unique_lock<std::mutex> lk(mu);
        idle.wait(lk, [&] { return running == 0; });
    }

    ~HostCopier()
    {
        {
            std::lock_guard<std::mutex> lk(mu);
            stop = true;
        }
        wake.notify_all();
        for (auto& t : ts) t.join();
    }
};

static bool pageable(const void* p)
{
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

void copier_release(rbsc_ctx* ctx)
{
    HostCopier* c = ctx->copier;
    if (!c) return;
    for (auto& e : c->ev)
        if (e) cudaEventDestroy(e);
    host_free(ctx, (void*&)c->mem);
    delete c;
    ctx->copier = nullptr;
}

// False when the slots cannot be had (no pinned memory): plain copies then.
static bool ensure_copier(rbsc_ctx* ctx)
{
    if (ctx->copier) return true;
    HostCopier* c = new (std::nothrow) HostCopier();
    if (!c) return false;
    ctx->copier = c;
    // beside other contexts' threads (a server's executors) fewer
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    c->start(std::max(1u, std::min(ctx->shared_gpu ? kMaxThreads / 2 : kMaxThreads, hw / 2)));
    bool ok = host_alloc(ctx, (void**)&c->mem, kSlot * 2 * c->threads) == RBSC_OK;
    for (unsigned i = 0; ok && i < c->threads * 2; ++i) ok = cudaEventCreateWithFlags(&c->ev[i], cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        copier_release(ctx);
    }
    return ok;
}

static rbsc_status run_chunks(rbsc_ctx* ctx, const std::vector<Chunk>& chunks, cudaStream_t s, bool in)
{
    HostCopier* c = ctx->copier;
    std::atomic<size_t> next{0};
    std::atomic<int> err{(int)cudaSuccess};
    auto work = [&](unsigned t) {
        cudaError_t e = cudaSetDevice(ctx->device);
        Chunk pend[2] = {};  // out: what each slot holds once its copy is done
        unsigned k = 0;
        for (; e == cudaSuccess && err.load(std::memory_order_relaxed) == (int)cudaSuccess; ++k) {
            const size_t i = next.fetch_add(1);
            const unsigned slot = k & 1u;
            char* p = c->mem + (2 * t + slot) * kSlot;
            cudaEvent_t ev = c->ev[2 * t + slot];
            e = cudaEventSynchronize(ev);  // an earlier copy (of an earlier call, too) may still use the slot
            if (e != cudaSuccess) break;
            if (pend[slot].host) std::memcpy(pend[slot].host, p, pend[slot].bytes);
            pend[slot] = Chunk{};
            if (i >= chunks.size()) break;
            const Chunk& x = chunks[i];
            if (in) std::memcpy(p, x.host, x.bytes);
            e = in ? cudaMemcpyAsync(x.dev, p, x.bytes, cudaMemcpyHostToDevice, s)
                   : cudaMemcpyAsync(p, x.dev, x.bytes, cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaEventRecord(ev, s);
            if (!in) pend[slot] = x;
        }
        for (unsigned slot = 0; slot < 2 && e == cudaSuccess; ++slot)
            if (pend[slot].host) {
                e = cudaEventSynchronize(c->ev[2 * t + slot]);
                if (e == cudaSuccess) std::memcpy(pend[slot].host, c->mem + (2 * t + slot) * kSlot, pend[slot].bytes);
            }
        if (e != cudaSuccess) err.store((int)e);
    };
    c->run(std::ref(work));  // (a copy of it would be allocated, which can throw)
    const cudaError_t e = (cudaError_t)err.load();
    if (e != cudaSuccess) return rbsc_cuda_fail(ctx, e, "host copy", __LINE__);
    return RBSC_OK;
}

static rbsc_status copy(rbsc_ctx* ctx, void* dev, void* host, size_t bytes, cudaStream_t s, bool in)
{
    if (!bytes) return RBSC_OK;
    if (bytes >= kWorth && pageable(host) && ensure_copier(ctx)) {
        std::vector<Chunk> chunks;
        try {
            chunks.reserve(bytes / kSlot + 1);
        } catch (const std::bad_alloc&) {
            return rbsc_fail(ctx, RBSC_ERR_OOM, "out of host memory");
        }
        for (size_t a = 0; a < bytes; a += kSlot)
            chunks.push_back(Chunk{static_cast<char*>(dev) + a, static_cast<char*>(host) + a, std::min(kSlot, bytes - a)});
        return run_chunks(ctx, chunks, s, in);
    }
    EK(in ? cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, s) : cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, s));
    return RBSC_OK;
}

rbsc_status copy_in(rbsc_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t s)
{
    return copy(ctx, dst, const_cast<void*>(src), bytes, s, true);
}

rbsc_status copy_out(rbsc_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t s)
{
    return copy(ctx, const_cast<void*>(src), dst, bytes, s, false);
}
