/*
 * gexs_upload.cpp — host-to-device copies from pageable memory through a
 * ring of pinned buffers filled by several host threads.
 *
 * cudaMemcpyAsync from pageable memory goes through the driver's own
 * staging on the calling thread, about 10 GB/s on the measured host.  Here
 * worker threads copy chunks of at most kSlotBytes into pinned slots while
 * the calling thread queues the device copies in order: a manager pass over
 * 3e6 lines (132 MB of arrays) 13.7 against 20.4 ms.
 * The bound is the host's memory and the PCIe link (55 GB/s from pinned
 * memory).  As with the driver's staging, a pageable source has been read
 * when the call returns; pinned sources are copied directly and must stay
 * valid until the stream has passed the copy.
 */
#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>
#include <cuda_runtime.h>
#include "../csrc/gexs_internal.h"

namespace gexs {

namespace {
constexpr size_t kSlotBytes = (size_t)512 << 10;
constexpr int kSlots = 16;
constexpr int kThreads = 8;
/* below this the threads' start (~0.2 ms) costs more than it saves */
constexpr size_t kMinStaged = (size_t)4 << 20;

bool pageable(const void* p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return true; }
    return a.type == cudaMemoryTypeUnregistered;
}
}  // namespace

namespace {
/* The ring, 8 MiB for all contexts of the process: pinning it takes longer
 * than many uploads (0.7 ms per MiB), so a context created later finds it.
 * Allocated by the first upload that uses it, freed with the last context.
 * An upload holds `use` throughout; another at the same time does without. */
struct Ring {
    std::mutex mu;                       /* contexts, pinned */
    int contexts = 0;
    unsigned char* pinned = nullptr;
    bool tried = false;
    std::mutex use;
    cudaEvent_t last[kSlots] = {};       /* the slot's last device copy */
} g_ring;
}  // namespace

/* a context's events on its own device */
struct Uploader {
    int device = 0;
    cudaEvent_t ev[kSlots] = {};
    bool tried = false, ok = false;

    /* with g_ring.use held */
    bool ready()
    {
        if (!tried) {
            tried = ok = true;
            for (cudaEvent_t& e : ev)
                if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) ok = false;
            if (!ok) cudaGetLastError();
        }
        std::lock_guard<std::mutex> g(g_ring.mu);
        if (!g_ring.tried) {
            g_ring.tried = true;
            void* p = nullptr;
            if (cudaHostAlloc(&p, kSlotBytes * kSlots, cudaHostAllocPortable) == cudaSuccess)
                g_ring.pinned = static_cast<unsigned char*>(p);
            else
                cudaGetLastError();
        }
        return ok && g_ring.pinned;
    }
};

Uploader* uploader_create(int device)
{
    Uploader* u = new Uploader();
    u->device = device;
    std::lock_guard<std::mutex> g(g_ring.mu);
    ++g_ring.contexts;
    return u;
}

void uploader_destroy(Uploader* u)
{
    if (!u) return;
    {
        std::lock_guard<std::mutex> use(g_ring.use);
        for (int k = 0; k < kSlots; ++k)
            if (u->ev[k]) {
                if (g_ring.last[k] == u->ev[k]) {
                    cudaEventSynchronize(u->ev[k]);
                    g_ring.last[k] = nullptr;
                }
                cudaEventDestroy(u->ev[k]);
            }
        std::lock_guard<std::mutex> g(g_ring.mu);
        if (--g_ring.contexts == 0) {
            if (g_ring.pinned) cudaFreeHost(g_ring.pinned);
            g_ring.pinned = nullptr;
            g_ring.tried = false;
        }
    }
    delete u;
}

/* Waits poll for kPoll and then sleep: a chunk takes some 25 us, and a sleep
 * and wake-up at every chunk made the manager pass 24 ms long (13.5 with
 * polling, 20.3 with the driver's staging); but the stream may have other
 * work before the copies, and the host's cores may be fewer than the
 * threads (a quota). */
constexpr std::chrono::microseconds kPoll(1000);

template <typename F>
static bool poll(const F& done)
{
    const auto end = std::chrono::steady_clock::now() + kPoll;
    do {
        if (done()) return true;
        std::this_thread::yield();
    } while (std::chrono::steady_clock::now() < end);
    return false;
}

struct Waiters {
    std::mutex mu;
    std::condition_variable cv;
    std::atomic<int> asleep{0};
    template <typename F>
    void wait(const F& done)
    {
        if (poll(done)) return;
        std::unique_lock<std::mutex> g(mu);
        asleep.fetch_add(1);
        cv.wait(g, done);
        asleep.fetch_sub(1);
    }
    /* after the change that a waiter looks for: a waiter counts itself before
     * it looks for the last time, so one of the two sees the other */
    void wake()
    {
        if (asleep.load() == 0) return;
        { std::lock_guard<std::mutex> g(mu); }
        cv.notify_all();
    }
};

/* the event's work is done (waited for) */
static bool passed(cudaEvent_t e)
{
    cudaError_t r = cudaErrorNotReady;
    int n = 0;
    poll([&] { return n++ % 32 == 0 && (r = cudaEventQuery(e)) != cudaErrorNotReady; });
    while (r == cudaErrorNotReady) {
        std::this_thread::sleep_for(std::chrono::microseconds(200));
        r = cudaEventQuery(e);
    }
    return r == cudaSuccess;
}

cudaError_t upload(Uploader* u, const gexs_upload_piece* pieces, int n, cudaStream_t s)
{
    struct Chunk { void* dst; const void* src; size_t bytes; cudaEvent_t after; bool staged; };
    std::vector<Chunk> chunks;
    std::vector<size_t> staged;            /* indices of the chunks that go through a slot */
    size_t total = 0;
    std::vector<char> pg(n, 0);
    for (int i = 0; i < n; ++i)
        if (pieces[i].bytes && pageable(pieces[i].src)) { pg[i] = 1; total += pieces[i].bytes; }
    if (total) {
        /* a captured copy would read its source, or the slot, at each replay */
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(s, &cap) != cudaSuccess) cudaGetLastError();
        if (cap != cudaStreamCaptureStatusNone) return cudaErrorStreamCaptureUnsupported;
    }
    std::unique_lock<std::mutex> lock(g_ring.use, std::defer_lock);
    const unsigned hw = std::thread::hardware_concurrency();
    const int nt = (int)std::min<size_t>(kThreads, hw > 1 ? hw - 1 : 1);
    bool use = total >= kMinStaged && nt > 1;
    if (use) use = lock.try_lock() && u->ready();
    for (int i = 0; i < n; ++i) {
        const gexs_upload_piece& p = pieces[i];
        const bool st = use && pg[i];
        size_t o = 0;
        do {
            const size_t m = st ? std::min(kSlotBytes, p.bytes - o) : p.bytes;
            if (st) staged.push_back(chunks.size());
            chunks.push_back({(unsigned char*)p.dst + o, (const unsigned char*)p.src + o, m,
                              o + m >= p.bytes ? (cudaEvent_t)p.event : nullptr, st});
            o += m;
        } while (o < p.bytes);
    }
    /* staged chunk k uses slot k % kSlots: filled once chunk k - kSlots has
     * been queued and its device copy has finished */
    std::vector<std::atomic<int>> filled(staged.size());
    for (auto& f : filled) f.store(0, std::memory_order_relaxed);
    std::atomic<size_t> next{0}, queued{0};
    std::atomic<bool> stop{false};
    Waiters room, ready;
    auto work = [&]() {
        cudaSetDevice(u->device);
        for (;;) {
            const size_t k = next.fetch_add(1);
            if (k >= staged.size()) return;
            room.wait([&] { return stop.load() || queued.load() + kSlots > k; });
            if (stop.load()) return;
            const int slot = (int)(k % kSlots);
            const cudaEvent_t last = g_ring.last[slot];
            const bool ok = !last || passed(last);
            const Chunk& c = chunks[staged[k]];
            if (ok) std::memcpy(g_ring.pinned + slot * kSlotBytes, c.src, c.bytes);
            filled[k].store(ok ? 1 : -1);
            ready.wake();
            if (!ok) return;
        }
    };
    std::vector<std::thread> th;
    if (!staged.empty()) {
        try {
            for (int t = 0; t < nt; ++t) th.emplace_back(work);
        } catch (...) {
            /* fewer threads; with none, the driver stages */
        }
    }
    cudaError_t e = cudaSuccess;
    size_t k = 0;
    for (const Chunk& c : chunks) {
        const void* src = c.src;
        if (c.staged && !th.empty()) {
            ready.wait([&] { return filled[k].load() != 0; });
            if (filled[k].load() < 0) { e = cudaErrorUnknown; break; }
            src = g_ring.pinned + (k % kSlots) * kSlotBytes;
        }
        if (c.bytes) e = cudaMemcpyAsync(c.dst, src, c.bytes, cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess && c.staged && !th.empty()) {
            e = cudaEventRecord(u->ev[k % kSlots], s);
            g_ring.last[k % kSlots] = u->ev[k % kSlots];
            queued.store(++k);
            room.wake();
        }
        if (e == cudaSuccess && c.after) e = cudaEventRecord(c.after, s);
        if (e != cudaSuccess) break;
    }
    stop.store(true);
    room.wake();
    for (std::thread& t : th) t.join();
    return e;
}

}  // namespace gexs

extern "C" int gexs_ctx_upload(gexs_ctx* ctx, const gexs_upload_piece* pieces, int n, void* stream)
{
    using namespace gexs;
    if (!ctx || n < 0 || (n > 0 && !pieces)) return set_error(GEXS_ERR_INVALID, "gexs_ctx_upload: arguments");
    for (int i = 0; i < n; ++i)
        if (pieces[i].bytes && (!pieces[i].dst || !pieces[i].src))
            return set_error(GEXS_ERR_INVALID, "gexs_ctx_upload: NULL array");
    cudaSetDevice(ctx_device(ctx));
    try {
        const cudaError_t e = upload(ctx_uploader(ctx), pieces, n, (cudaStream_t)stream);
        return e == cudaSuccess ? GEXS_OK : cuda_error(e, "gexs_ctx_upload");
    } catch (...) {
        return set_error(GEXS_ERR_OOM, "gexs_ctx_upload: host memory");
    }
}
