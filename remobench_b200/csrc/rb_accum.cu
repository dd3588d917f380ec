// Accumulate stage: per-leaf running sums behind a watermark, restating
// kernels/remolod/remolod_accum.cu:47-233. A plan splits every dirty leaf's
// new points into fixed-size work items spread over the whole grid.
//
// The reference sums node-local coordinates in [0, 1] as doubles, so its sums
// depend on the order the points are folded in. Here each point is quantised
// to its 28-bit octree coordinate P (the reference's MAX_DEPTH_GRIDSIZE grid,
// remolod_octree.cu:167-169) and taken relative to its leaf,
//   q = clamp(P - (N << (28 - L)), 0, 2^(28 - L))   per axis,
// and Σq (u64) and Σqqᵀ (128-bit) are exact integers: any fold order gives the
// same bits. Colour sums are exact integers of the 8-bit channels.
//
// Bound: reading 16 B per new point (plus its chunk-table entry). The watermark
// `count` makes the pass incremental: only [count, numPoints) is read.
#include <cuda_runtime.h>

#include "rb_kernels.h"
#include "rb_launch.h"
#include "rb_state.h"

namespace rb {

// remoMortonSpread / remoMortonCode (remolod_accum.cu:24-36)
__device__ __forceinline__ unsigned long long mortonSpread(uint32_t v) {
    unsigned long long x = (unsigned long long)v & 0xFFFFFull;
    x = (x | (x << 32)) & 0x001F00000000FFFFull;
    x = (x | (x << 16)) & 0x001F0000FF0000FFull;
    x = (x | (x << 8)) & 0x100F00F00F00F00Full;
    x = (x | (x << 4)) & 0x10C30C30C30C30C3ull;
    x = (x | (x << 2)) & 0x1249249249249249ull;
    return x;
}

// The watermark is the largest 60-bit Morton code of the folded points.
// Codes are compared without building them: the dimension whose coordinates
// differ in the highest bit decides (x before y before z at the same bit, the
// order of the interleave), found with the test "msb(p) < msb(q)" =
// p < q && p < (p ^ q) (Chan, "Closest-point problems simplified on the RAM",
// SODA 2002). Only the block's largest point is spread into a code.
__device__ __forceinline__ bool msbLess(uint32_t p, uint32_t q) { return p < q && p < (p ^ q); }

__device__ __forceinline__ bool mortonLess(uint32_t ax, uint32_t ay, uint32_t az, uint32_t bx, uint32_t by,
                                           uint32_t bz) {
    const uint32_t dx = ax ^ bx, dy = ay ^ by, dz = az ^ bz;
    uint32_t da = dx, a = ax, b = bx;
    if (msbLess(da, dy)) {
        da = dy;
        a = ay;
        b = by;
    }
    if (msbLess(da, dz)) {
        a = az;
        b = bz;
    }
    return a < b;
}

__device__ __forceinline__ void add128(unsigned long long& lo, unsigned long long& hi,
                                       unsigned long long v) {
    const unsigned long long o = lo;
    lo = o + v;
    hi += (lo < o) ? 1ull : 0ull;
}

__device__ __forceinline__ bool leafRow(const Dev& d, uint32_t node) {
    const int4* row = reinterpret_cast<const int4*>(d.child + node * 8u);
    const int4 a = row[0], b = row[1];
    return (a.x & a.y & a.z & a.w & b.x & b.y & b.z & b.w) == -1;
}

constexpr int kAccumThreads = 256;

// 128-bit atomic add on a (lo, hi) pair: the add that wraps lo carries into hi.
__device__ __forceinline__ void atomicAdd128(unsigned long long* lo, unsigned long long* hi,
                                             unsigned long long vlo, unsigned long long vhi) {
    const unsigned long long old = atomicAdd(lo, vlo);
    const unsigned long long carry = (old + vlo < old) ? 1ull : 0ull;
    if (vhi + carry) atomicAdd(hi, vhi + carry);
}

// The fold whose items, point chunks, are cut into kAccumParts parts, a warp each:
// of fewer new points than kAccumFine whole chunks hold, and with at least a warp's
// width of points a part. A warp per whole chunk leaves most of the 3,552 resident
// warps without work below that (100,000 points in chunks of 1,000: 18.2 us whole,
// 8.3 in quarters); above, and in small chunks, an item's reduction, about 20
// points' worth, is better spent on a whole one (2M points in chunks of 7: 540 us
// whole, 1,817 in quarters).
constexpr uint32_t kAccumFine = 3000;
constexpr uint32_t kAccumParts = 4;
static_assert(kAccumThreads / 32 % kAccumParts == 0, "a block's warps count the parts off");

// Starts a fold: its counters to zero (RemolodPipeline.cpp:251-256 restarts the
// globals per launch), and how its chunks are cut, from the points that came in
// since the last one.
__global__ void k_accum_begin(Dev d) {
    follow();
    Counters* c = d.ctr;
    AccumGlobals* g = d.accumGlobals;
    g->sumLeafCounts = 0;
    g->pointsFolded = 0;
    g->numLeavesFolded = 0;
    g->innerWithSums = 0;
    const unsigned long long seen = c->numPointsProcessed + c->spilledPointsTotal;
    const bool fine = d.ppc >= 32u * kAccumParts && seen - c->accumMark < (unsigned long long)kAccumFine * d.ppc;
    c->accumParts = fine ? kAccumParts : 1u;
    c->accumMark = seen;
    c->accumItems = 0;
    c->mortonBound = 0;
}

__device__ __forceinline__ unsigned long long mortonCode(uint32_t x, uint32_t y, uint32_t z) {
    return (mortonSpread(x) << 2) | (mortonSpread(y) << 1) | mortonSpread(z);
}

// The fold's plan: the nodes to visit (the dirty list, or every node), each
// leaf's new range [count, min(numPoints, capacity)) read before any fold
// updates count, and each node's work items. An inner node with sums is one
// item (cleared); a leaf with new points one item per point chunk its new range
// touches. Sums are exact, so the order of items is free: each block claims a
// contiguous run of item indices with one atomic (Counters::accumItems) and
// writes every item's plan entry, so a warp of the fold finds its item with one
// load. The parts of an item (Counters::accumParts) are not listed: the fold's
// warps count them off, and a part without a new point is skipped. Items can pass
// accumUnitCap (every live point chunk plus every node) only once the arena
// has run out (RB_OVF_ARENA): those are not folded. Folded-leaf and point
// totals are added per block. The watermark needs only the leaves that can hold
// the largest Morton code: a code grows with each coordinate, so a point's is at
// least its leaf's lower corner's (clamping only raises a coordinate), and the
// largest lower corner of the leaves with new points bounds it from below.
__global__ void __launch_bounds__(256) k_accum_plan(Dev d, int useList) {
    follow();
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_base, s_leaves;
    __shared__ unsigned long long s_points, s_bound;
    Counters* c = d.ctr;
    const uint32_t total = useList ? (c->numDirty < d.maxNodes ? c->numDirty : d.maxNodes) : c->numNodes;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        s_leaves = 0;
        s_points = 0;
        s_bound = 0;
    }
    __syncthreads();
    // the same number of steps in every thread of the block
    for (uint32_t w0 = blockIdx.x * blockDim.x; w0 < total; w0 += gridDim.x * blockDim.x) {
        const uint32_t w = w0 + threadIdx.x;
        uint32_t items = 0, from = 0, to = 0;
        if (w < total) {
            const uint32_t node = useList ? d.dirtyList[w] : w;
            if (!leafRow(d, node)) {
                items = d.accum[node].count != 0u ? 1u : 0u;
            } else {
                from = d.accum[node].count;
                const uint32_t cap = d.numPointChunks[node] * d.ppc;
                const uint32_t np = d.numPoints[node];
                to = np < cap ? np : cap;
                if (to > from) {
                    items = (to - 1u) / d.ppc - from / d.ppc + 1u;
                    const uint32_t sh = (uint32_t)kMaxDepth - d.level[node];
                    atomicMax(&s_bound, mortonCode(d.nodeX[node] << sh, d.nodeY[node] << sh, d.nodeZ[node] << sh));
                    atomicAdd(&s_leaves, 1u);
                    atomicAdd(&s_points, (unsigned long long)(to - from));
                } else {
                    to = from;
                }
            }
            d.accumFrom[w] = from;
            d.accumTo[w] = to;
        }
        // block-wide exclusive scan of the item counts
        uint32_t x = items;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        if (lane == 31u) s_warp[warp] = x;
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t run = 0;
            for (uint32_t k = 0; k < blockDim.x / 32u; k++) {
                const uint32_t t = s_warp[k];
                s_warp[k] = run;
                run += t;
            }
            s_base = run ? atomicAdd(&c->accumItems, run) : 0u;
        }
        __syncthreads();
        const uint32_t first = s_base + s_warp[warp] + x - items;
        if (w < total) {
            d.accumItem[w] = first;
            for (uint32_t u = first; u < first + items && u < d.accumUnitCap; u++) d.accumUnitW[u] = w;
        }
        __syncthreads();
    }
    __syncthreads();
    if (threadIdx.x == 0 && s_leaves) {
        atomicAdd(&d.accumGlobals->numAccumulated, s_points);
        atomicAdd(&d.accumGlobals->pointsFolded, (uint32_t)s_points);
        atomicAdd(&d.accumGlobals->numLeavesFolded, s_leaves);
        // past an arena overflow a chunk may be missing, and its points with it
        if (!(c->overflowFlags & (uint32_t)kOvfArena)) atomicMax(&c->mortonBound, s_bound);
    }
}

// 128-bit sum of two (lo, hi) pairs.
__device__ __forceinline__ void add128pair(unsigned long long& lo, unsigned long long& hi, unsigned long long olo,
                                           unsigned long long ohi) {
    const unsigned long long nl = lo + olo;
    hi += ohi + (nl < lo ? 1ull : 0ull);
    lo = nl;
}

// Folds the plan's work items, one warp per item: an item is the part of one
// leaf's new range inside one point chunk (at most ppc points, one chunk-table
// read), its partial sums added atomically into the leaf's exact sums -- any
// order gives the same bits -- or an inner node's sums cleared. Lane k of the
// warp issues the atomic of sum k, so an item's 21 updates go out together.
// The watermark is merged per block in shared memory, one global atomic per
// block. Three blocks per SM (80 registers, a few bytes spilled) fold 9% faster
// than the two that 93 registers allow. Bound by instruction issue: 20M points
// took 108 us with a division per coordinate, 64-bit clamps and a Morton
// comparison per point, 77 us without (4.2 TB/s of the points read).
__global__ void __launch_bounds__(kAccumThreads, 3) k_accumulate(Dev d, uint32_t batchIndex, bool atCursor,
                                                                int useList) {
    follow();
    __shared__ unsigned long long s_morton;
    const Counters* c = d.ctr;
    const uint32_t items = c->accumItems;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t ppc = d.ppc, parts = c->accumParts, step = (ppc + parts - 1u) / parts;
    const unsigned long long bound = c->mortonBound;
    if (atCursor) batchIndex = c->batchletIndex;
    if (threadIdx.x == 0) s_morton = 0ull;
    __syncthreads();
    // a block's warps, and so the grid's, are a multiple of the parts
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5, warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t part = warp % parts;
    unsigned long long blockMax = 0ull;  // lane 0's running watermark
    for (uint32_t it = warp / parts; it < items; it += warps / parts) {
        if (it >= d.accumUnitCap) break;  // only past an arena overflow (see k_accum_plan)
        const uint32_t w = d.accumUnitW[it];
        const uint32_t node = useList ? d.dirtyList[w] : w;
        AccumI* a = &d.accum[node];
        const uint32_t from0 = d.accumFrom[w], to = d.accumTo[w];
        if (to == from0) {  // an inner node holding sums
            if (lane == 0 && part == 0u) {
                AccumI z = {};
                *a = z;
            }
            continue;
        }
        const uint32_t ci = from0 / ppc + (it - d.accumItem[w]), lo = ci * ppc + part * step;
        const uint32_t from = max(from0, lo);
        const uint32_t end = min(to, min(lo + step, (ci + 1u) * ppc));
        if (from >= end) continue;
        const uint32_t lv = d.level[node];
        const uint32_t sh = 28u - lv;
        const uint32_t lim = 1u << sh;
        const uint32_t origin[3] = {d.nodeX[node] << sh, d.nodeY[node] << sh, d.nodeZ[node] << sh};
        const uint32_t phys = d.tablePool[d.ptTableOff[node] + ci];
        // whether a point of this leaf can hold the watermark (k_accum_plan)
        const uint32_t sh20 = (uint32_t)kMaxDepth - lv, corner = (1u << sh20) - 1u;
        const bool candidate = mortonCode((d.nodeX[node] << sh20) | corner, (d.nodeY[node] << sh20) | corner,
                                          (d.nodeZ[node] << sh20) | corner) >= bound;

        // Per lane at most ppc / 32 + 1 points: Σq < 2^28 · 32 needs u64, Σq·q <
        // 32 · 2^56 fits u64 without carries, colour sums fit u32; the 128-bit
        // carries start at the warp reduction.
        unsigned long long s1[3] = {0, 0, 0};
        unsigned long long p2[6] = {0, 0, 0, 0, 0, 0};
        uint32_t c1[3] = {0, 0, 0}, c2[3] = {0, 0, 0};
        uint32_t mx = 0, my = 0, mz = 0;  // the largest point in Morton order so far
        if (phys != kNone) {
            const float4* cp = reinterpret_cast<const float4*>(chunkPoints(d, phys));
            const uint32_t base = ci * ppc;
            for (uint32_t s0 = from + lane; s0 < end; s0 += 4u * 32u) {
                // four points per step: their loads in flight together
                float4 v4[4];
                bool ok[4];
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const uint32_t sidx = s0 + (uint32_t)h * 32u;
                    ok[h] = sidx < end;
                    if (ok[h]) v4[h] = __ldg(cp + (sidx - base));
                }
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    if (!ok[h]) continue;
                    const float4 v = v4[h];
                    const uint32_t P[3] = {quant28(d, v.x, 0), quant28(d, v.y, 1), quant28(d, v.z, 2)};
                    // clamped to [0, 2^(28 - level)]: 32-bit values, 64-bit products
                    uint32_t q[3];
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        q[k] = min(max(P[k], origin[k]) - origin[k], lim);
                        s1[k] += q[k];
                    }
                    p2[0] += (unsigned long long)q[0] * q[0];
                    p2[1] += (unsigned long long)q[0] * q[1];
                    p2[2] += (unsigned long long)q[0] * q[2];
                    p2[3] += (unsigned long long)q[1] * q[1];
                    p2[4] += (unsigned long long)q[1] * q[2];
                    p2[5] += (unsigned long long)q[2] * q[2];
                    const uint32_t col = __float_as_uint(v.w);
                    const uint32_t ch[3] = {col & 255u, (col >> 8) & 255u, (col >> 16) & 255u};
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        c1[k] += ch[k];
                        c2[k] += ch[k] * ch[k];
                    }
                    // only where it can be the largest: in the last leaves in Morton
                    // order, or past the box, where a leaf's cube says nothing of it
                    if (candidate || max(max(P[0], P[1]), P[2]) >= (1u << 28)) {
                        // the 20-bit coordinate is the 28-bit one shifted (power-of-two scaling
                        // commutes with round-to-nearest); only a saturated conversion differs
                        uint32_t X = P[0] < 0xFFFFFF00u ? P[0] >> 8 : quant20(d, v.x, 0);
                        uint32_t Y = P[1] < 0xFFFFFF00u ? P[1] >> 8 : quant20(d, v.y, 1);
                        uint32_t Z = P[2] < 0xFFFFFF00u ? P[2] >> 8 : quant20(d, v.z, 2);
                        X = X < 1048575u ? X : 1048575u;
                        Y = Y < 1048575u ? Y : 1048575u;
                        Z = Z < 1048575u ? Z : 1048575u;
                        if (mortonLess(mx, my, mz, X, Y, Z)) {
                            mx = X;
                            my = Y;
                            mz = Z;
                        }
                    }
                }
            }
        }
        // the warp's sums: 21 values (s1 x3, s2 lo/hi x6, c1 x3, c2 x3) and the watermark
        unsigned long long wm = mortonCode(mx, my, mz);
        unsigned long long lo2[6], hi2[6] = {0, 0, 0, 0, 0, 0};
        unsigned long long c1w[3], c2w[3];
#pragma unroll
        for (int k = 0; k < 6; k++) lo2[k] = p2[k];
#pragma unroll
        for (int k = 0; k < 3; k++) {
            c1w[k] = c1[k];
            c2w[k] = c2[k];
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                s1[k] += __shfl_xor_sync(0xFFFFFFFFu, s1[k], off);
                c1w[k] += __shfl_xor_sync(0xFFFFFFFFu, c1w[k], off);
                c2w[k] += __shfl_xor_sync(0xFFFFFFFFu, c2w[k], off);
            }
#pragma unroll
            for (int k = 0; k < 6; k++) {
                const unsigned long long ol = __shfl_xor_sync(0xFFFFFFFFu, lo2[k], off);
                const unsigned long long oh = __shfl_xor_sync(0xFFFFFFFFu, hi2[k], off);
                add128pair(lo2[k], hi2[k], ol, oh);
            }
            const unsigned long long om = __shfl_xor_sync(0xFFFFFFFFu, wm, off);
            wm = om > wm ? om : wm;
        }
        // every lane holds the totals: lane k issues sum k's atomic (values
        // picked by unrolled selects, so the arrays stay in registers)
        if (lane < 3u) {
            unsigned long long v1 = 0, vc1 = 0, vc2 = 0;
#pragma unroll
            for (int k = 0; k < 3; k++) {
                if (lane == (uint32_t)k) {
                    v1 = s1[k];
                    vc1 = c1w[k];
                    vc2 = c2w[k];
                }
            }
            atomicAdd(&a->s1[lane], v1);
            atomicAdd(&a->c1[lane], vc1);
            atomicAdd(&a->c2[lane], vc2);
        } else if (lane < 9u) {
            unsigned long long vlo = 0, vhi = 0;
#pragma unroll
            for (int k = 0; k < 6; k++) {
                if (lane == 3u + (uint32_t)k) {
                    vlo = lo2[k];
                    vhi = hi2[k];
                }
            }
            atomicAdd128(&a->s2lo[lane - 3u], &a->s2hi[lane - 3u], vlo, vhi);
        } else if (lane == 9u) {
            // every item of a leaf writes the same watermark and batch
            a->count = to;
            a->lastTouchedBatch = batchIndex;
        }
        if (wm > blockMax) blockMax = wm;
    }
    if (lane == 0 && blockMax != 0ull) atomicMax(&s_morton, blockMax);
    __syncthreads();
    if (threadIdx.x == 0 && s_morton != 0ull) atomicMax(&d.accumGlobals->mortonWatermark, s_morton);
}

// kernel_accum_verify (remolod_accum.cu:214-233). One thread restarts the dirty
// list, which names the nodes touched since this fold (nothing here reads it).
__global__ void __launch_bounds__(256) k_accum_verify(Dev d) {
    follow();
    const uint32_t nn = d.ctr->numNodes;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        d.ctr->buildStamp += 1u;
        d.ctr->numDirty = 0;
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        const uint32_t cnt = d.accum[i].count;
        if (leafRow(d, i)) {
            if (cnt) atomicAdd(&d.accumGlobals->sumLeafCounts, (unsigned long long)cnt);
        } else if (cnt != 0) {
            atomicAdd(&d.accumGlobals->innerWithSums, 1u);
        }
    }
}

void launchAccumulate(const Dev& d, uint32_t batchIndex, bool atCursor, int useList, int grid, cudaStream_t s) {
    k_accum_begin<<<1, 1, 0, s>>>(d);
    launchBehind(k_accum_plan, grid / 4 + 1, 256, 0, s, d, useList);
    launchBehind(k_accumulate, grid, kAccumThreads, 0, s, d, batchIndex, atCursor, useList);
}
void launchAccumVerify(const Dev& d, int grid, cudaStream_t s) { launchBehind(k_accum_verify, grid, 256, 0, s, d); }

}  // namespace rb
