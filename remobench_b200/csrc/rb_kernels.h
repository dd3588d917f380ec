// Kernel launch wrappers shared by the stage translation units and the host
// orchestration (rb_capi.cu). Host code never sees a kernel symbol directly.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "rb_state.h"

namespace rb {

// Per-frame render parameters (the subset of SharedUniforms,
// include/remo/HostDeviceCommon.h:28-60, that the LOD cut and splat read).
struct Frame {
    float width, height;
    float transform[16];        // row-major, clip = M (x, y, z, 1)
    float transformFrozen[16];  // LOD-selection and frustum transform
    float boxMin[3], boxMax[3];
    float lodPixelBudget;
    int32_t pointSize;
    int32_t colorMode;          // 0 rgb, 1 by node, 2 by level, 3 white
    uint32_t showBoundingBox;
};

// The draw list's cursor and the samples its items hold, points and voxels as
// counted (rb_render_result). cursor: items emitted in the low kDrawCountBits
// bits (a node is emitted at most once, and there are at most 2^21), the stored
// samples of the items so far above them.
struct RenderScratch {
    unsigned long long cursor;
    unsigned long long samples;
};
constexpr uint32_t kDrawCountBits = 24;
constexpr unsigned long long kDrawCountMask = (1ull << kDrawCountBits) - 1ull;

// A draw list entry: the node in the low kDrawNodeBits bits (ids are below 2^21),
// the stored samples of the items before it above them. Together they can pass
// 2^32: past an arena overflow points without a chunk count too.
struct DrawItem {
    unsigned long long bits;
};
constexpr uint32_t kDrawNodeBits = 21;
__host__ __device__ inline DrawItem drawItem(uint32_t node, unsigned long long first) {
    return DrawItem{first << kDrawNodeBits | node};
}
__host__ __device__ inline uint32_t itemNode(DrawItem it) { return (uint32_t)it.bits & ((1u << kDrawNodeBits) - 1u); }
__host__ __device__ inline unsigned long long itemFirst(DrawItem it) { return it.bits >> kDrawNodeBits; }

// The samples [begin, end) of a frame's `total` that warp w of `warps` draws.
struct DrawShare {
    unsigned long long begin, end;
};
__host__ __device__ inline DrawShare drawShare(unsigned long long total, uint32_t warps, uint32_t w) {
    const unsigned long long share = ((total + warps - 1u) / warps + 31ull) & ~31ull, begin = w * share;
    return begin >= total ? DrawShare{total, total} : DrawShare{begin, total - begin < share ? total : begin + share};
}
// The first sample of an item of n that a share ending at `end` leaves.
__host__ __device__ inline uint32_t itemStop(DrawItem it, uint32_t n, unsigned long long end) {
    return end - itemFirst(it) < n ? (uint32_t)(end - itemFirst(it)) : n;
}

// What a render reports, in pinned host memory that k_raster writes.
struct RenderResult {
    uint32_t numItems;
    uint32_t overflow;
    unsigned long long samples;
};

// Update
void launchBatchBegin(const Dev& d, cudaStream_t s);
// One batch at the device cursor as an instantiated graph (see rb_update.cu).
cudaError_t captureBatchGraph(const Dev& d, int pointGrid, int fixedGrid, int restGrid, cudaGraphExec_t* out);
// The cooperative expand-pass kernel: its grid, and one launch.
cudaError_t expandRestGrid(int numSMs, int* grid);
cudaError_t launchExpandRest(const Dev& d, int grid, cudaStream_t s);
void launchCountFirst(const Dev& d, const Point* pts, uint32_t n, int grid, cudaStream_t s);
void launchRecount(const Dev& d, const Point* pts, uint32_t n, uint32_t prevStamp, int grid, cudaStream_t s);
void launchSplit(const Dev& d, uint32_t stamp, cudaStream_t s);
void launchZeroGrids(const Dev& d, int grid, cudaStream_t s);
// the expand round (rb_update.cu): book the first count's splits, bin the
// points below them, make every split the counts decide, move the points
void launchDeepBook(const Dev& d, cudaStream_t s);
void launchDeepBin(const Dev& d, const Point* pts, uint32_t n, int grid, cudaStream_t s);
void launchDeepSplit(const Dev& d, cudaStream_t s);
void launchDeepMove(const Dev& d, const Point* pts, uint32_t n, int grid, cudaStream_t s);
void launchExpandCond(const Dev& d, cudaStream_t s);
void launchSpillCopy(const Dev& d, int grid, cudaStream_t s);
void launchVoxSample(const Dev& d, const Point* pts, uint32_t n, int grid, cudaStream_t s);
void launchVoxLift(const Dev& d, int grid, cudaStream_t s);
void launchVoxSampleLevels(const Dev& d, const Point* pts, uint32_t n, int grid, cudaStream_t s);
void launchDeepenBegin(const Dev& d, const uint32_t* queue, uint32_t queueLen, uint32_t budget, uint32_t minPoints,
                       cudaStream_t s);
void launchDeepenEnd(const Dev& d, cudaStream_t s);
void launchCollapse(const Dev& d, uint32_t count, uint32_t maxPoints, int grid, cudaStream_t s);
void launchVoxCommit(const Dev& d, int grid, cudaStream_t s);
void launchFinishLeaves(const Dev& d, const Point* pts, uint32_t n, int grid, cudaStream_t s);
void launchAllocPoints(const Dev& d, int grid, cudaStream_t s);
void launchAllocVoxels(const Dev& d, int grid, cudaStream_t s);
void launchInsert(const Dev& d, const Point* pts, uint32_t n, int grid, cudaStream_t s);
void launchVoxStore(const Dev& d, int grid, cudaStream_t s);
void launchBatchEnd(const Dev& d, uint32_t n, cudaStream_t s);
void launchSweep(const Dev& d, int grid, cudaStream_t s);
void launchResetRoot(const Dev& d, int grid, cudaStream_t s);

// Accumulate
// atCursor: Counters::batchletIndex takes batchIndex's place.
void launchAccumulate(const Dev& d, uint32_t batchIndex, bool atCursor, int useList, int grid, cudaStream_t s);
void launchAccumVerify(const Dev& d, int grid, cudaStream_t s);

// Rasterize
void launchFbClear(unsigned long long* fb, uint64_t npx, int grid, cudaStream_t s);
// The draw list of a frame and its cleared framebuffer.
void launchCut(const Dev& d, const Frame& f, unsigned long long* fb, uint64_t npx, const uint8_t* force,
               RenderScratch* rs, DrawItem* items, uint32_t cap, int grid, cudaStream_t s);
void launchRaster(const Dev& d, const Frame& f, unsigned long long* fb, const RenderScratch* rs,
                  const DrawItem* items, uint32_t cap, RenderResult* host, int grid, cudaStream_t s);
void launchRasterFlat(const Frame& f, unsigned long long* fb, const Point* pts, uint64_t n, int grid,
                      cudaStream_t s);
// EDL in place; rgba (optional) receives the resolved colours.
void launchEdl(unsigned long long* fb, uint32_t* rgba, uint32_t w, uint32_t h, float strength, cudaStream_t s);
void launchResolve(const unsigned long long* fb, uint32_t* rgba, uint64_t npx, int grid, cudaStream_t s);
// The draw items' bounding boxes as lines (remo_lines.cuh:120-137), after EDL.
void launchWireframe(const Dev& d, const Frame& f, unsigned long long* fb, const RenderScratch* rs,
                     const DrawItem* items, uint32_t cap, int grid, cudaStream_t s);

}  // namespace rb
