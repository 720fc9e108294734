// Page-locked staging buffers and copy streams behind the host side of the engine (gtm_stage.h).
#include "gtm_stage.h"

#include <algorithm>
#include <cstring>
#include <mutex>
#include <new>

#include "gtm_host.cuh"

namespace {

constexpr int kLanesKept = 2;

std::mutex g_lock;                               // guards what follows
int g_users = 0, g_device = -1;
StageLane *g_lanes = nullptr;                    // free lanes; a plain list: nothing is torn down behind a process that just exits

void lane_destroy(StageLane *l)
{
    cudaSetDevice(l->device);
    for (int i = 0; i < kStageSlots; ++i) {
        if (l->down[i].host) cudaFreeHost(l->down[i].host);
        if (l->down[i].done) cudaEventDestroy(l->down[i].done);
    }
    for (cudaEvent_t e : l->event) if (e) cudaEventDestroy(e);
    if (l->in) cudaStreamDestroy(l->in);
    if (l->back) cudaStreamDestroy(l->back);
    if (l->aux) cudaStreamDestroy(l->aux);
    if (l->small) cudaFreeHost(l->small);
    delete l;
}

int lane_fill(StageLane *l)
{
    GTM_CU(cudaStreamCreateWithFlags(&l->in, cudaStreamNonBlocking));
    GTM_CU(cudaStreamCreateWithFlags(&l->back, cudaStreamNonBlocking));
    GTM_CU(cudaStreamCreateWithFlags(&l->aux, cudaStreamNonBlocking));
    for (cudaEvent_t &e : l->event) GTM_CU(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (StageSlot &slot : l->down) GTM_CU(cudaEventCreateWithFlags(&slot.done, cudaEventDisableTiming));
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

void stage_retain(int device)
{
    std::lock_guard<std::mutex> hold(g_lock);
    ++g_users;
    g_device = device;
}

int stage_device()
{
    std::lock_guard<std::mutex> hold(g_lock);
    return g_device;
}

void stage_drop()
{
    StageLane *lanes;
    {
        std::lock_guard<std::mutex> hold(g_lock);
        if (--g_users > 0) return;
        lanes = g_lanes;
        g_lanes = nullptr;
    }
    while (lanes) {
        StageLane *l = lanes;
        lanes = l->next;
        lane_destroy(l);
    }
}

bool host_is_pinned(const void *p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) { cudaGetLastError(); return false; }
    return at.type == cudaMemoryTypeHost;
}

static int slot_land(StageSlot &slot)
{
    if (!slot.busy) return GTM_OK;
    GTM_CU(cudaEventSynchronize(slot.done));
    slot.busy = false;
    if (slot.dst) memcpy(slot.dst, slot.host, slot.bytes);
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
        if (lane->down[i].busy) cudaEventSynchronize(lane->down[i].done);
        lane->down[i].busy = false;
        lane->down[i].dst = nullptr;
    }
}
