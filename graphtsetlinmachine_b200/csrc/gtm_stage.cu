// Copy threads, page-locked staging buffers and copy streams behind the host side of the engine (gtm_stage.h).
#include "gtm_stage.h"

#include <stdint.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <mutex>
#include <new>
#include <thread>

#if defined(__x86_64__)
#include <immintrin.h>
#endif

#include "gtm_host.cuh"

// ---------------------------------------------------------------------------------------------- copy threads
// One job at a time.  The job's ticket word holds its number of items (bits 24..47) and the next item (bits 0..23): a
// thread takes an item with one fetch_add and sees from the same word whether the item exists, so that a thread that
// comes late to a finished job reads nothing of it.  The job's function and context are written before the ticket and
// stay until every existing item is done.
namespace {

constexpr int kCopyThreads = 7;                 // beside the calling thread; 8 threads saturate the host's memory
constexpr int kCountShift = 24;
constexpr uint64_t kIndexMask = ((uint64_t)1 << kCountShift) - 1;

struct CopyPool {
    std::mutex user;                            // held by the caller whose job runs
    std::mutex lock;
    std::condition_variable wake;
    std::atomic<uint64_t> ticket{0};
    std::atomic<int> done{0}, sleeping{0};
    std::atomic<bool> stop{false};
    void (*fn)(void *, int) = nullptr;
    void *ctx = nullptr;
    std::thread threads[kCopyThreads];
    pid_t owner = getpid();                     // a forked child has the pool but not its threads

    bool open() const
    {
        const uint64_t t = ticket.load(std::memory_order_acquire);
        return (t & kIndexMask) < (t >> kCountShift);
    }
    void work()
    {
        while (true) {
            const uint64_t t = ticket.fetch_add(1, std::memory_order_acq_rel);
            if ((t & kIndexMask) >= (t >> kCountShift)) return;
            fn(ctx, (int)(t & kIndexMask));
            done.fetch_add(1, std::memory_order_release);
        }
    }
    // A worker looks for the next job for a while before it sleeps: the pieces of one call come every few tens of
    // microseconds, and waking a sleeping thread takes about as long as copying a piece.  Whoever waits gives its processor
    // away at every look: a worker that is woken may start on the processor of the caller or of another worker, and would hold
    // its piece there until the one that only waits has used up its 3 to 4 ms.
    void loop()
    {
        while (!stop.load(std::memory_order_relaxed)) {
            const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(60);
            while (!open() && std::chrono::steady_clock::now() < until) std::this_thread::yield();
            if (open()) { work(); continue; }
            std::unique_lock<std::mutex> hold(lock);
            sleeping.fetch_add(1);
            wake.wait(hold, [&] { return open() || stop.load(); });
            sleeping.fetch_sub(1);
        }
    }
    void run(int count, void (*f)(void *, int), void *c)
    {
        fn = f; ctx = c;
        done.store(0, std::memory_order_relaxed);
        ticket.store((uint64_t)count << kCountShift, std::memory_order_seq_cst);
        if (sleeping.load() > 0) {
            { std::lock_guard<std::mutex> hold(lock); }
            wake.notify_all();
        }
        work();
        while (done.load(std::memory_order_acquire) < count) std::this_thread::yield();
    }
    ~CopyPool()
    {
        { std::lock_guard<std::mutex> hold(lock); stop.store(true); }
        wake.notify_all();
        for (std::thread &t : threads) if (t.joinable()) t.join();
    }
};

constexpr int kLanesKept = 2;

std::mutex g_lock;                               // guards what follows
int g_users = 0, g_device = -1;
CopyPool *g_pool = nullptr;                      // plain pointers: nothing is torn down behind a process that just exits
StageLane *g_lanes = nullptr;                    // free lanes

CopyPool *pool_get()
{
    std::lock_guard<std::mutex> hold(g_lock);
    if (!g_pool && g_users > 0) {
        CopyPool *p = new (std::nothrow) CopyPool();
        const int n = std::min(kCopyThreads, (int)std::thread::hardware_concurrency() - 1);
        try {
            for (int i = 0; p && i < n; ++i) p->threads[i] = std::thread([p] { p->loop(); });
        } catch (const std::exception &) {}             // what threads there are, or the caller alone
        g_pool = p;
    }
    return g_pool && g_pool->owner == getpid() ? g_pool : nullptr;
}

void lane_destroy(StageLane *l)
{
    cudaSetDevice(l->device);
    for (int i = 0; i < kStageSlots; ++i) {
        if (l->up[i].host) cudaFreeHost(l->up[i].host);
        if (l->down[i].host) cudaFreeHost(l->down[i].host);
        if (l->up[i].done) cudaEventDestroy(l->up[i].done);
        if (l->down[i].done) cudaEventDestroy(l->down[i].done);
    }
    for (cudaEvent_t e : l->event) if (e) cudaEventDestroy(e);
    if (l->in) cudaStreamDestroy(l->in);
    if (l->back) cudaStreamDestroy(l->back);
    if (l->aux) cudaStreamDestroy(l->aux);
    if (l->small) cudaFreeHost(l->small);
    for (char *p : l->scratch) if (p) cudaFree(p);
    delete l;
}

int lane_fill(StageLane *l)
{
    GTM_CU(cudaStreamCreateWithFlags(&l->in, cudaStreamNonBlocking));
    GTM_CU(cudaStreamCreateWithFlags(&l->back, cudaStreamNonBlocking));
    GTM_CU(cudaStreamCreateWithFlags(&l->aux, cudaStreamNonBlocking));
    for (cudaEvent_t &e : l->event) GTM_CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (int i = 0; i < kStageSlots; ++i) {
        GTM_CU(cudaEventCreateWithFlags(&l->up[i].done, cudaEventDisableTiming));
        GTM_CU(cudaEventCreateWithFlags(&l->down[i].done, cudaEventDisableTiming));
    }
    GTM_CU(cudaMallocHost((void **)&l->small, 2 * kStageSmall));
    return GTM_OK;
}

// The slot's buffer; nothing of the slot is in flight.
int slot_reserve(StageSlot &slot)
{
    if (!slot.host) GTM_CU(cudaMallocHost((void **)&slot.host, kStagePiece));
    return GTM_OK;
}

}  // namespace

void host_parallel(int count, void (*fn)(void *ctx, int i), void *ctx)
{
    CopyPool *p = count > 1 ? pool_get() : nullptr;
    if (p && p->user.try_lock()) {
        p->run(count, fn, ctx);
        p->user.unlock();
        return;
    }
    for (int i = 0; i < count; ++i) fn(ctx, i);
}

// Copy into a staging buffer (64-byte aligned) with stores that leave no lines in the caches: the copy engine reads lines
// that eight cores hold modified at 30 GB/s, memory at 50.
static void copy_past_caches(char *dst, const char *src, size_t bytes)
{
#if defined(__x86_64__)
    size_t at = 0;
    for (; at + 64 <= bytes; at += 64) {
        const __m128i *s = (const __m128i *)(src + at);
        const __m128i a = _mm_loadu_si128(s), b = _mm_loadu_si128(s + 1), c = _mm_loadu_si128(s + 2), d = _mm_loadu_si128(s + 3);
        __m128i *t = (__m128i *)(dst + at);
        _mm_stream_si128(t, a); _mm_stream_si128(t + 1, b); _mm_stream_si128(t + 2, c); _mm_stream_si128(t + 3, d);
    }
    memcpy(dst + at, src + at, bytes - at);
    _mm_sfence();
#else
    memcpy(dst, src, bytes);
#endif
}

void host_copy(void *dst, const void *src, size_t bytes, bool past_caches)
{
    struct Job { char *dst; const char *src; size_t bytes, piece; bool past; } job;
    job.dst = (char *)dst; job.src = (const char *)src; job.bytes = bytes; job.past = past_caches;
    // below 256 KB one thread is done (10 GB/s) before the others have taken their share
    if (bytes < ((size_t)256 << 10)) {
        if (past_caches) copy_past_caches(job.dst, job.src, bytes);
        else memcpy(dst, src, bytes);
        return;
    }
    const size_t parts = std::min<size_t>(16, bytes / ((size_t)64 << 10));
    job.piece = ((bytes + parts - 1) / parts + 4095) & ~(size_t)4095;
    host_parallel((int)((bytes + job.piece - 1) / job.piece), [](void *c, int i) {
        const Job *j = (const Job *)c;
        const size_t at = (size_t)i * j->piece;
        const size_t n = std::min(j->piece, j->bytes - at);
        if (j->past) copy_past_caches(j->dst + at, j->src + at, n);
        else memcpy(j->dst + at, j->src + at, n);
    }, &job);
}

// ------------------------------------------------------------------------------------------------------ lanes
int lane_acquire(int device, StageLane **out)
{
    *out = nullptr;
    {
        std::lock_guard<std::mutex> hold(g_lock);
        for (StageLane **at = &g_lanes; *at; at = &(*at)->next)
            if ((*at)->device == device) {
                *out = *at;
                *at = (*at)->next;
                return GTM_OK;
            }
    }
    StageLane *l = new (std::nothrow) StageLane();
    if (!l) return fail(GTM_ERR_OOM, "host allocation failed");
    l->device = device;
    const int st = lane_fill(l);
    if (st != GTM_OK) { lane_destroy(l); return st; }
    *out = l;
    return GTM_OK;
}

void lane_release(StageLane *lane)
{
    {
        std::lock_guard<std::mutex> hold(g_lock);
        int kept = 0;
        for (const StageLane *l = g_lanes; l; l = l->next) kept += l->device == lane->device;
        if (kept < kLanesKept && g_users > 0) { lane->next = g_lanes; g_lanes = lane; return; }
    }
    lane_destroy(lane);
}

int lane_scratch(StageLane *lane, int i, size_t bytes)
{
    if (bytes <= lane->scratch_bytes[i]) return GTM_OK;
    char *old = lane->scratch[i];
    lane->scratch[i] = nullptr;
    lane->scratch_bytes[i] = 0;
    GTM_CU(cudaFree(old));
    GTM_TRY(dev_alloc(&lane->scratch[i], bytes));
    lane->scratch_bytes[i] = bytes;
    return GTM_OK;
}

void stage_retain(int device)
{
    std::lock_guard<std::mutex> hold(g_lock);
    ++g_users;
    if (device >= 0) g_device = device;
}

int stage_device()
{
    std::lock_guard<std::mutex> hold(g_lock);
    return g_device;
}

void stage_drop()
{
    StageLane *lanes;
    CopyPool *pool;
    {
        std::lock_guard<std::mutex> hold(g_lock);
        if (--g_users > 0) return;
        lanes = g_lanes;
        g_lanes = nullptr;
        pool = g_pool;
        g_pool = nullptr;
    }
    while (lanes) {
        StageLane *l = lanes;
        lanes = l->next;
        lane_destroy(l);
    }
    if (pool && pool->owner == getpid()) delete pool;     // in a forked child there is nothing to join
}

bool host_is_pinned(const void *p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return at.type == cudaMemoryTypeHost;
}

int stage_up(StageLane *lane, void *dst, const void *src, size_t bytes, bool pinned, cudaStream_t s)
{
    if (bytes == 0) return GTM_OK;
    if (pinned) { GTM_CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s)); return GTM_OK; }
    for (size_t at = 0; at < bytes; at += kStagePiece) {
        const size_t n = std::min(kStagePiece, bytes - at);
        StageSlot &slot = lane->up[lane->up_next];
        lane->up_next = (lane->up_next + 1) % kStageSlots;
        if (slot.busy) GTM_CU(cudaEventSynchronize(slot.done));
        slot.busy = false;
        GTM_TRY(slot_reserve(slot));
        host_copy(slot.host, (const char *)src + at, n, true);
        GTM_CU(cudaMemcpyAsync((char *)dst + at, slot.host, n, cudaMemcpyHostToDevice, s));
        GTM_CU(cudaEventRecord(slot.done, s));
        slot.busy = true;
    }
    return GTM_OK;
}

static int slot_land(StageSlot &slot)
{
    if (!slot.busy) return GTM_OK;
    GTM_CU(cudaEventSynchronize(slot.done));
    slot.busy = false;
    if (slot.dst) host_copy(slot.dst, slot.host, slot.bytes, false);
    slot.dst = nullptr;
    return GTM_OK;
}

int stage_down(StageLane *lane, void *dst, const void *src, size_t bytes, bool pinned, cudaStream_t s)
{
    if (bytes == 0) return GTM_OK;
    if (pinned) {
        GTM_CU(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s));
        GTM_CU(cudaEventRecord(lane->event[3], s));       // stage_down_finish waits for the last of these
        return GTM_OK;
    }
    // the host copies a piece while the copy engine brings the next
    for (size_t at = 0; at < bytes; at += kStagePiece) {
        const size_t n = std::min(kStagePiece, bytes - at);
        StageSlot &slot = lane->down[lane->down_next];
        lane->down_next = (lane->down_next + 1) % kStageSlots;
        GTM_TRY(slot_land(slot));
        GTM_TRY(slot_reserve(slot));
        GTM_CU(cudaMemcpyAsync(slot.host, (const char *)src + at, n, cudaMemcpyDeviceToHost, s));
        GTM_CU(cudaEventRecord(slot.done, s));
        slot.busy = true;
        slot.dst = (char *)dst + at;
        slot.bytes = n;
    }
    return GTM_OK;
}

int stage_down_finish(StageLane *lane)
{
    for (int i = 0; i < kStageSlots; ++i) GTM_TRY(slot_land(lane->down[(lane->down_next + i) % kStageSlots]));   // oldest first
    GTM_CU(cudaEventSynchronize(lane->event[3]));         // complete at once when no page-locked copy was queued
    return GTM_OK;
}

void stage_abandon(StageLane *lane)
{
    cudaStreamSynchronize(lane->in);
    cudaStreamSynchronize(lane->back);
    cudaStreamSynchronize(lane->aux);
    for (int i = 0; i < kStageSlots; ++i) {
        if (lane->up[i].busy) cudaEventSynchronize(lane->up[i].done);
        if (lane->down[i].busy) cudaEventSynchronize(lane->down[i].done);
        lane->up[i].busy = lane->down[i].busy = false;
        lane->down[i].dst = nullptr;
    }
}
