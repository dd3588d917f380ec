// Refinement passes beyond the LOD-cut mask (rb_refine.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "rb_state.h"

namespace rb {

struct RefineCounters {
    uint32_t nodes;               // queue prefix filtered
    uint32_t voxels;              // accumulator entries in use
    unsigned long long points;    // (point, filtered ancestor) pairs
    unsigned long long pairs;     // those whose ancestor has voxels
    uint32_t units;               // units of points the gathering pass takes
    uint32_t pad;
};

// Colour filtering's scratch, sized at allocation: one accumulator entry per
// voxel being filtered (capacity), a (node slot, cell) -> entry table of twice
// that, and per node its slot in the call (kNone outside a call).
struct RefineScratch {
    uint32_t* refSlot;            // [maxNodes]
    uint32_t* voxNode;            // [maxNodes + 1] filtered node per slot
    uint32_t* voxBase;            // [maxNodes + 1] first entry per slot, then the total
    ulonglong4* acc;              // [capacity] r, g, b sums and the count of the points gathered here
    ulonglong4* up;               // [capacity] the same of the points gathered in filtered nodes below
    uint32_t* entrySlot;          // [capacity] the entry's table slot
    uint2* upSlot;                // [maxNodes + 1] per slot, the next filtered node up that has voxels and its level
    ulonglong2* hash;             // [hashMask + 1] (key, entry), key ~0: free
    RefineCounters* ctr;
    uint32_t capacity;
    uint32_t hashMask;
};

__device__ uint32_t blockExclusiveScanRefine(uint32_t v, uint32_t* total, uint32_t* s_warp);

void launchRefineColors(const Dev& d, const RefineScratch& r, const uint32_t* queue, uint32_t queueLen,
                        uint32_t budget, int grid, cudaStream_t s);

}  // namespace rb
