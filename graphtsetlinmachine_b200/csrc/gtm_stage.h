// Host side of the copies from the device to a caller's arrays: page-locked buffers, copy streams and events, kept between
// calls (gtm_stage.cu).
//
// A copy to pageable memory holds the calling thread until it has ended, so that nothing further is queued meanwhile.  Here the
// copy engine fills page-locked pieces, and the calling thread copies a piece out while it brings the next.  Copies to the
// device are left to the driver (18 GB/s from pageable memory on the host of one B200; through pieces of our own 13).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

// Bytes of one piece.  Page-locking takes 0.6 ms per MB, which a program's first large result pays.
constexpr size_t kStagePiece = (size_t)256 << 10;
constexpr int kStageSlots = 4;                       // pieces in flight
constexpr size_t kStageSmall = (size_t)256 << 10;    // sets and results up to this size go through the small buffer

struct StageSlot {
    char *host = nullptr;        // page-locked, made on first use
    cudaEvent_t done = nullptr;
    bool busy = false;
    void *dst = nullptr;         // a piece on its way down: where it goes once it has landed
    size_t bytes = 0;
};

// What one call borrows: copy streams, events, staging buffers.  Lives on one device.
struct StageLane {
    StageLane *next = nullptr;   // on the free list
    int device = -1;
    cudaStream_t in = nullptr, back = nullptr, aux = nullptr;    // copies up, copies down, a second stream for kernels
    cudaEvent_t event[4] = {};   // free for the borrower's use
    char *small = nullptr;       // [2][kStageSmall] page-locked: packed inputs, results
    StageSlot down[kStageSlots];
    int down_next = 0;
};

// A lane of the device, from the free list or new.  At most kLanesKept lanes per device stay on the list; all of them are
// given back when the last model is destroyed (stage_retain / stage_drop).  stage_device: the device of the model made
// last, -1 before the first.
int lane_acquire(int device, StageLane **out);
void lane_release(StageLane *lane);
void stage_retain(int device);
void stage_drop();
int stage_device();

struct LaneGuard {
    StageLane *lane = nullptr;
    ~LaneGuard() { if (lane) lane_release(lane); }
};

bool host_is_pinned(const void *p);

// Queues a copy of `bytes` to the host on stream s; dst holds them once stage_down_finish has returned.
int stage_down(StageLane *lane, void *dst, const void *src, size_t bytes, bool pinned, cudaStream_t s);
int stage_down_finish(StageLane *lane);

// After an error: waits until nothing of the lane is in flight and forgets it.
void stage_abandon(StageLane *lane);
