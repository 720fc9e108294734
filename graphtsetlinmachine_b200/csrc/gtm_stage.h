// Host side of the copies between a caller's pageable arrays and the device: a few copy threads, page-locked staging
// buffers, copy streams and events, all kept between calls (gtm_stage.cu).
//
// A cudaMemcpyAsync from or to pageable memory is one host thread copying through a small buffer of the driver: 6 to
// 12 GB/s, with the copy engine idle most of the time, and a fresh result array costs that thread a page fault every
// 4 KB on top.  Here a few threads copy pieces to or from page-locked buffers while the copy engine moves the pieces
// before: 120,000 images of 32 bytes up and their 4.8 MB of class sums down took 0.9 ms through pageable copies.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

// Bytes of one staging buffer.  Page-locking takes 0.5 ms per MB, which the first call pays: four buffers of 4 MB in each
// direction made the first 120,000 images of a program 23 ms instead of 4.  Steady copies are as fast with 0.5 MB as with 4
// (two sets of 120,000 images: 1.16 ms a pass with 0.5 MB, 1.24 with 1, 1.40 with 4).
constexpr size_t kStagePiece = (size_t)512 << 10;
constexpr int kStageSlots = 4;                       // staging buffers per direction
constexpr size_t kStageSmall = (size_t)256 << 10;    // sets and results up to this size go through the small buffer

// Runs fn(ctx, i) for i in [0, count) on the copy threads and the calling thread; returns when all are done.  When the
// threads are busy with another caller's work, the calling thread does everything itself.
void host_parallel(int count, void (*fn)(void *ctx, int i), void *ctx);

// memcpy by several threads when it is large enough to pay; `past_caches` (64-byte aligned dst): with streaming stores.
void host_copy(void *dst, const void *src, size_t bytes, bool past_caches);

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
    char *scratch[2] = {};       // device memory for the kernels on the borrower's stream and on `aux`
    size_t scratch_bytes[2] = {};
    StageSlot up[kStageSlots], down[kStageSlots];
    int up_next = 0, down_next = 0;
};

// A lane of the device, from the free list or new.  At most kLanesKept lanes per device stay on the list; all of them,
// and the copy threads, are given back when the last model is destroyed (stage_retain / stage_drop).  stage_device: the
// device of the model made last, -1 before the first; stage_retain(-1) names no device.
int lane_acquire(int device, StageLane **out);
void lane_release(StageLane *lane);
void stage_retain(int device);
void stage_drop();
int stage_device();

struct LaneGuard {
    StageLane *lane = nullptr;
    ~LaneGuard() { if (lane) lane_release(lane); }
};

// Makes scratch block i of the lane at least this large.  Only the borrower's kernels use it, and they have ended when the lane
// is released.  (Blocks of hundreds of MB that every call took from the memory pool broke up between the graph sets that come
// and go there: two sets of 6,000 multigraphs 7 to 13 ms a pass, 7.1 with blocks that stay, one B200.)
int lane_scratch(StageLane *lane, int i, size_t bytes);

bool host_is_pinned(const void *p);

// Queues a copy of `bytes` to the device on stream s.  The source may be reused when the call returns, unless it is
// page-locked memory of the caller: then it must stay until the stream has passed the copy.
int stage_up(StageLane *lane, void *dst, const void *src, size_t bytes, bool pinned, cudaStream_t s);

// Queues a copy of `bytes` to the host on stream s; dst holds them once stage_down_finish has returned.
int stage_down(StageLane *lane, void *dst, const void *src, size_t bytes, bool pinned, cudaStream_t s);
int stage_down_finish(StageLane *lane);

// After an error: waits until nothing of the lane is in flight and forgets it.
void stage_abandon(StageLane *lane);
