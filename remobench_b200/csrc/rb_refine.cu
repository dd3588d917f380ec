// Refinement's colour filtering (wiki/02_KernelPipeline.md:228-243: "average
// colour across a node's samples", listed by the reference and not built
// there): a voxel's colour becomes the mean colour of the points below its
// node that fall in its cell, instead of one representative point's.
//
// The reference's notes rule out a dense per-node colour grid (128^3 RGBA
// sums would be ~16 MB per node) and ask for a sparse accumulator keyed off
// the voxels. Here the accumulator has one entry per voxel being filtered,
// found through a table keyed by (filtered node, cell):
//   k_cf_plan   the queue prefix whose voxels fit the capacity, each node's
//               first entry (one block);
//   k_cf_units  the leaves below a filtered node, cut into units of points;
//   k_cf_index  every entry's cell from its voxel's centre into the table;
//   k_cf_gather a unit's points summed per cell of the deepest filtered node
//               above them, first in shared memory, then into its entries (or,
//               with few points a voxel, every point into its entries: perPoint);
//   k_cf_roll   every entry's sums into the entries of the filtered nodes above:
//               a point's cell in an ancestor is a prefix of its cell below;
//   k_cf_apply  means (rounded half up, alpha kept) written into the voxels,
//               the table and the node marks cleared for the next call.
// So the table is probed once per cell of a unit and once per (entry, ancestor),
// not once per (point, ancestor), which took four 64-bit atomics each: with 4M
// points, 64 filtered nodes and 18.1M such pairs, gathering by a block per leaf
// took 1,560 us; units, gather and roll take 6 + 84 + 42 us. Bound by the point
// pass: its quantisation, its shared atomics and the latency of the flush.
// Integer sums: the result does not depend on the order points arrive in.
#include <cuda_runtime.h>

#include "rb_kernels.h"
#include "rb_refine.h"
#include "rb_state.h"

namespace rb {

namespace {

__device__ __forceinline__ uint32_t cellOf(uint32_t x28, uint32_t y28, uint32_t z28, uint32_t level) {
    const uint32_t sh = (uint32_t)kMaxDepth + 1u - level;
    return ((x28 >> sh) & 127u) + ((y28 >> sh) & 127u) * 128u + ((z28 >> sh) & 127u) * 16384u;
}

// The table's home slot of a (node slot << 21 | cell) key: 2 x 2 x 2 cells share
// a 128-byte line (eight 16-byte slots), hashed together, the place within the
// line mixed with the hash so that flat surfaces fill all eight; probing goes
// from line to line at the same place (nextSlot).
__device__ __forceinline__ uint32_t slotOf(unsigned long long key, uint32_t mask) {
    const uint32_t cell = (uint32_t)key & 0x1FFFFFu;
    const uint32_t place = (cell & 1u) | ((cell >> 6) & 2u) | ((cell >> 12) & 4u);
    unsigned long long h = (key & ~0x4081ull) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 31;
    h *= 0xBF58476D1CE4E5B9ull;
    return (((uint32_t)(h >> 32) & ~7u) | (((uint32_t)(h >> 24) ^ place) & 7u)) & mask;
}

// The cell a voxel of node `node` stands for, from its centre
// nodeMin + size (c + 0.5) / 128 (half a cell from either boundary).
__device__ __forceinline__ uint32_t voxelCell(const Dev& d, uint32_t node, const Point& v) {
    const float size = __fdiv_rn(d.octreeSize, __int_as_float((int)((127u + d.level[node]) << 23)));
    const float scale = __fdiv_rn(128.0f, size);
    const float mn[3] = {__fmaf_rn((float)d.nodeX[node], size, d.boxMin[0]),
                         __fmaf_rn((float)d.nodeY[node], size, d.boxMin[1]),
                         __fmaf_rn((float)d.nodeZ[node], size, d.boxMin[2])};
    const float pv[3] = {v.x, v.y, v.z};
    uint32_t c[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
        const int q = __float2int_rd(__fmul_rn(__fsub_rn(pv[a], mn[a]), scale));
        c[a] = (uint32_t)min(max(q, 0), 127);
    }
    return c[0] + 128u * c[1] + 16384u * c[2];
}

__global__ void __launch_bounds__(1024) k_cf_plan(Dev d, RefineScratch r, const uint32_t* queue, uint32_t queueLen,
                                                  uint32_t budget) {
    __shared__ uint32_t s_warp[32];
    __shared__ uint32_t s_run, s_stop;
    const uint32_t n = queueLen < budget ? queueLen : budget;
    if (threadIdx.x == 0) {
        s_run = 0;
        s_stop = n;
    }
    __syncthreads();
    for (uint32_t k0 = 0; k0 < n; k0 += blockDim.x) {
        const uint32_t k = k0 + threadIdx.x;
        uint32_t nv = 0, node = 0;
        if (k < n) {
            node = queue[k];
            nv = d.numVoxels[node];
            const uint32_t stored = d.numVoxelsStored[node], cap = d.numVoxelChunks[node] * d.ppc;
            nv = nv < stored ? nv : stored;
            nv = nv < cap ? nv : cap;
        }
        uint32_t tot;
        const uint32_t pre = blockExclusiveScanRefine(nv, &tot, s_warp);
        const uint32_t base = s_run + pre;
        // the prefix that fits: every node whose voxels end within the capacity
        if (k < n && base + nv > r.capacity) atomicMin(&s_stop, k);
        __syncthreads();
        if (k < n && k < s_stop) {
            r.voxNode[k] = node;
            r.voxBase[k] = base;
            r.refSlot[node] = k;
        }
        __syncthreads();
        if (threadIdx.x == 0) s_run += tot;
        __syncthreads();
        if (s_stop < n) break;
    }
    if (threadIdx.x == 0) {
        const uint32_t m = s_stop;
        uint32_t total = 0;
        if (m > 0) {
            const uint32_t last = r.voxNode[m - 1];
            uint32_t nv = d.numVoxels[last];
            const uint32_t stored = d.numVoxelsStored[last], cap = d.numVoxelChunks[last] * d.ppc;
            nv = nv < stored ? nv : stored;
            nv = nv < cap ? nv : cap;
            total = r.voxBase[m - 1] + nv;
        }
        r.voxBase[m] = total;
        r.ctr->nodes = m;
        r.ctr->voxels = total;
        r.ctr->points = 0;
        r.ctr->pairs = 0;
        r.ctr->units = 0;
    }
}

// Whether the call adds each point to its entries one by one: with few points a
// voxel, as in a cloud that fills its volume, most cells hold one, and summing them
// per cell first, then upwards, is only more work. 2M points spread evenly, 1.6M
// voxels, 1.2 points each: 358 us per cell, 275 per point; 1.3M voxels, 4.6 points
// each: 315 and 300; 2.1M and 5.0: 634 and 697; the filter of a scan's queue, 20
// each: 168 and 439.
constexpr unsigned long long kCfPairs = 4ull;
__device__ __forceinline__ bool perPoint(const RefineScratch& r) { return r.ctr->pairs < kCfPairs * r.ctr->voxels; }

__global__ void __launch_bounds__(256) k_cf_index(Dev d, RefineScratch r) {
    const uint32_t nodes = r.ctr->nodes, total = r.ctr->voxels;
    const bool direct = perPoint(r);
    // each filtered node's next filtered node up that has voxels
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nodes; k += gridDim.x * blockDim.x) {
        const uint32_t node = r.voxNode[k];
        uint2 up = make_uint2(kNone, 0u);
        for (uint32_t l = d.level[node]; l-- > 0u && up.x == kNone;) {
            const uint32_t q = r.refSlot[d.anc[(size_t)node * kMaxDepth + l].x];
            if (q != kNone && r.voxBase[q + 1u] != r.voxBase[q]) up = make_uint2(q, l);
        }
        r.upSlot[k] = up;
    }
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = nodes;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (r.voxBase[mid] <= e) lo = mid;
            else hi = mid;
        }
        const uint32_t node = r.voxNode[lo], s = e - r.voxBase[lo];
        const uint32_t phys = d.tablePool[d.vxTableOff[node] + s / d.ppc];
        Point v = {0.f, 0.f, 0.f, 0u};
        if (phys != kNone) v = reinterpret_cast<const Point*>(d.arena + (uint64_t)phys * 16u)[s % d.ppc];
        const unsigned long long key = ((unsigned long long)lo << 21) | voxelCell(d, node, v);
        r.acc[e] = make_ulonglong4(0ull, 0ull, 0ull, 0ull);
        if (!direct) r.up[e] = make_ulonglong4(0ull, 0ull, 0ull, 0ull);
        r.entrySlot[e] = kNone;
        if (phys == kNone) continue;
        uint32_t slot = slotOf(key, r.hashMask);
        for (uint32_t probe = 0; probe <= r.hashMask; probe++) {
            const unsigned long long prev = atomicCAS(&r.hash[slot].x, ~0ull, key);
            if (prev == ~0ull) {
                r.hash[slot].y = e;
                r.entrySlot[e] = slot;
                break;
            }
            if (prev == key) break;  // one voxel per cell: not reached
            slot = nextSlot(slot, r.hashMask);
        }
    }
}

__device__ __forceinline__ uint32_t findEntry(const RefineScratch& r, unsigned long long key) {
    uint32_t slot = slotOf(key, r.hashMask);
    for (uint32_t probe = 0; probe <= r.hashMask; probe++) {
        const ulonglong2 kv = __ldg(&r.hash[slot]);
        if (kv.x == key) return (uint32_t)kv.y;
        if (kv.x == ~0ull) return kNone;
        slot = nextSlot(slot, r.hashMask);
    }
    return kNone;
}

// The points of one unit: whole chunks, about kCfUnit points, so that a leaf
// has no more units than chunks; of larger chunks no more than the 32-bit sums of
// one cell hold (255 a point).
constexpr uint32_t kCfUnit = 2048, kCfUnitMax = 1u << 24;
__device__ __forceinline__ uint32_t unitPoints(uint32_t ppc) {
    return ppc >= kCfUnit ? min(ppc, kCfUnitMax) : kCfUnit / ppc * ppc;
}

// Per node: a leaf with points below (or itself) a filtered node adds its
// (point, filtered ancestor) pairs to the count and, where one of those has
// voxels, its units to the list: Dev::accumUnitW names each unit's leaf,
// Dev::accumItem the leaf's first unit (Accumulate's plan, free between folds).
__global__ void __launch_bounds__(256) k_cf_units(Dev d, RefineScratch r) {
    const uint32_t nn = d.ctr->numNodes, unit = unitPoints(d.ppc);
    const bool arenaFull = (d.ctr->overflowFlags & (uint32_t)kOvfArena) != 0u;
    unsigned long long visited = 0, pairs = 0;
    for (uint32_t leaf = blockIdx.x * blockDim.x + threadIdx.x; leaf < nn; leaf += gridDim.x * blockDim.x) {
        const uint32_t np = min(d.numPoints[leaf], d.numPointChunks[leaf] * d.ppc);
        if (np == 0u) continue;
        const int4* row = reinterpret_cast<const int4*>(d.child + leaf * 8u);
        const int4 a = row[0], b = row[1];
        if ((a.x & a.y & a.z & a.w & b.x & b.y & b.z & b.w) != -1) continue;
        const uint32_t lv = d.level[leaf];
        uint32_t m = 0, withVoxels = 0;  // filtered nodes, and those with voxels
        for (uint32_t l = 0; l <= lv; l++) {
            const uint32_t k = r.refSlot[l < lv ? d.anc[(size_t)leaf * kMaxDepth + l].x : leaf];
            if (k == kNone) continue;
            m++;
            withVoxels += r.voxBase[k + 1u] != r.voxBase[k];
        }
        uint32_t held = np;
        if (arenaFull && m > 0u) {  // points whose chunk the arena had no room for are not there
            const uint32_t off = d.ptTableOff[leaf];
            for (uint32_t k = 0; k <= (np - 1u) / d.ppc; k++)
                if (d.tablePool[off + k] == kNone) held -= min(d.ppc, np - k * d.ppc);
        }
        visited += (unsigned long long)held * m;
        pairs += (unsigned long long)held * withVoxels;
        if (withVoxels == 0u) continue;
        const uint32_t units = (np + unit - 1u) / unit, first = atomicAdd(&r.ctr->units, units);
        d.accumItem[leaf] = first;
        for (uint32_t u = first; u < first + units && u < d.accumUnitCap; u++) d.accumUnitW[u] = leaf;
    }
    for (int o = 16; o > 0; o >>= 1) {
        visited += __shfl_xor_sync(0xFFFFFFFFu, visited, o);
        pairs += __shfl_xor_sync(0xFFFFFFFFu, pairs, o);
    }
    if ((threadIdx.x & 31u) == 0 && visited) {
        atomicAdd(&r.ctr->points, visited);
        atomicAdd(&r.ctr->pairs, pairs);
    }
}

__device__ __forceinline__ void addSums(ulonglong4* to, unsigned long long cr, unsigned long long cg,
                                        unsigned long long cb, unsigned long long n) {
    atomicAdd(&to->x, cr);
    atomicAdd(&to->y, cg);
    atomicAdd(&to->z, cb);
    atomicAdd(&to->w, n);
}

// One block per unit (grid-stride). The filtered nodes above the unit's leaf,
// deepest first; the points' sums per cell of the deepest in a shared table
// (kCfTable cells, open addressing; a crowded one falls back to the entries),
// then per cell into that node's entry, or, where its voxel is missing, into
// the next filtered node's that has one. A point with a coordinate outside the
// box (past 2^28) has no common prefix with its node's cells: it goes to every
// filtered node's entry by itself (RefineScratch::up, which k_cf_roll does not
// carry further).
constexpr uint32_t kCfTable = 2048;

__global__ void __launch_bounds__(256) k_cf_gather(Dev d, RefineScratch r) {
    __shared__ uint32_t s_key[kCfTable];
    __shared__ uint32_t s_sum[4][kCfTable];
    __shared__ uint32_t s_slot[kMaxDepth + 1], s_lv[kMaxDepth + 1];
    __shared__ uint32_t s_m;
    const uint32_t ppc = d.ppc, unit = unitPoints(ppc);
    const uint32_t units = min(r.ctr->units, d.accumUnitCap);
    const bool direct = perPoint(r);
    ulonglong4* alone = direct ? r.acc : r.up;  // where a point goes by itself
    for (uint32_t u = blockIdx.x; u < units; u += gridDim.x) {
        const uint32_t leaf = d.accumUnitW[u];
        const uint32_t lv = d.level[leaf];
        for (uint32_t i = threadIdx.x; i < kCfTable && !direct; i += blockDim.x) {
            s_key[i] = kNone;
#pragma unroll
            for (int k = 0; k < 4; k++) s_sum[k][i] = 0;
        }
        if (threadIdx.x < 32u) {
            // lane l: the node at level lv - l
            const uint32_t l = threadIdx.x;
            uint32_t k = kNone;
            if (l <= lv) {
                k = r.refSlot[l == 0u ? leaf : d.anc[(size_t)leaf * kMaxDepth + lv - l].x];
                if (k != kNone && r.voxBase[k + 1u] == r.voxBase[k]) k = kNone;
            }
            const unsigned mask = __ballot_sync(0xFFFFFFFFu, k != kNone);
            if (k != kNone) {
                const uint32_t at = __popc(mask & ((1u << l) - 1u));
                s_slot[at] = k;
                s_lv[at] = lv - l;
            }
            if (l == 0u) s_m = __popc(mask);
        }
        __syncthreads();
        const uint32_t m = s_m, top = s_lv[0];
        const uint32_t np = min(d.numPoints[leaf], d.numPointChunks[leaf] * ppc);
        const uint32_t first = (u - d.accumItem[leaf]) * unit, last = min(np, first + unit);
        const uint32_t off = d.ptTableOff[leaf];
        // a cell's sums into the entries: the deepest filtered node's cell at
        // full coordinates (7 + level bits), shortened for the ones above
        const uint32_t X = d.nodeX[leaf] >> (lv - top), Y = d.nodeY[leaf] >> (lv - top), Z = d.nodeZ[leaf] >> (lv - top);
        auto addCell = [&](uint32_t cell, uint32_t cr, uint32_t cg, uint32_t cb, uint32_t n) {
            const uint32_t px = (X << 7) | (cell & 127u), py = (Y << 7) | ((cell >> 7) & 127u), pz = (Z << 7) | (cell >> 14);
            for (uint32_t j = 0; j < m; j++) {
                const uint32_t sh = top - s_lv[j];
                const uint32_t c = ((px >> sh) & 127u) + ((py >> sh) & 127u) * 128u + ((pz >> sh) & 127u) * 16384u;
                const uint32_t e = findEntry(r, ((unsigned long long)s_slot[j] << 21) | c);
                if (e == kNone) continue;
                addSums(&r.acc[e], cr, cg, cb, n);
                break;
            }
        };
        // four points a thread a step, each step's loads issued for all four
        for (uint32_t s0 = first + threadIdx.x; s0 - threadIdx.x < last; s0 += 4u * blockDim.x) {
            float4 v[4];
            bool ok[4];
#pragma unroll
            for (uint32_t j = 0; j < 4u; j++) {
                const uint32_t s = s0 + j * blockDim.x;
                uint32_t within = 0;
                const uint32_t chunk = s < last ? chunkOf(d, s, within) : 0u;
                const uint32_t phys = s < last ? d.tablePool[off + chunk] : kNone;
                ok[j] = phys != kNone;
                v[j] = ok[j] ? __ldg(reinterpret_cast<const float4*>(d.arena + (uint64_t)phys * 16u) + within)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll 1
            for (uint32_t j = 0; j < 4u; j++) {
                const float4 p = j == 0u ? v[0] : (j == 1u ? v[1] : (j == 2u ? v[2] : v[3]));
                const bool there = j == 0u ? ok[0] : (j == 1u ? ok[1] : (j == 2u ? ok[2] : ok[3]));
                const uint32_t x = quant28(d, p.x, 0),
                               y = quant28(d, p.y, 1),
                               z = quant28(d, p.z, 2);
                const uint32_t color = __float_as_uint(p.w);
                uint32_t cr = color & 255u, cg = (color >> 8) & 255u, cb = (color >> 16) & 255u, n = 1u;
                const bool regular = !direct && max(max(x, y), z) <= (1u << 28);
                if (there && !regular) {
                    for (uint32_t q = 0; q < m; q++) {
                        const uint32_t e = findEntry(r, ((unsigned long long)s_slot[q] << 21) | cellOf(x, y, z, s_lv[q]));
                        if (e != kNone) addSums(&alone[e], cr, cg, cb, 1ull);
                    }
                }
                if (direct) continue;
                uint32_t cell = there && regular ? cellOf(x, y, z, top) : kNone;
                // a warp whose points share one cell (a coarse ancestor's) adds once
                const uint32_t cell0 = __shfl_sync(0xFFFFFFFFu, cell, 0);
                if (__all_sync(0xFFFFFFFFu, cell == cell0)) {
                    cr = __reduce_add_sync(0xFFFFFFFFu, cr);
                    cg = __reduce_add_sync(0xFFFFFFFFu, cg);
                    cb = __reduce_add_sync(0xFFFFFFFFu, cb);
                    n = 32u;
                    if ((threadIdx.x & 31u) != 0u) cell = kNone;
                }
                if (cell == kNone) continue;
                uint32_t h = (cell * 0x9E3779B1u) >> 21;
                bool done = false;
                for (uint32_t probe = 0; probe < 16u && !done; probe++) {
                    uint32_t cur = s_key[h];
                    if (cur == kNone) cur = atomicCAS(&s_key[h], kNone, cell);
                    if (cur == kNone || cur == cell) {
                        atomicAdd(&s_sum[0][h], cr);
                        atomicAdd(&s_sum[1][h], cg);
                        atomicAdd(&s_sum[2][h], cb);
                        atomicAdd(&s_sum[3][h], n);
                        done = true;
                    }
                    h = (h + 1u) & (kCfTable - 1u);
                }
                if (!done) addCell(cell, cr, cg, cb, n);
            }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < kCfTable && !direct; i += blockDim.x)
            if (s_key[i] != kNone) addCell(s_key[i], s_sum[0][i], s_sum[1][i], s_sum[2][i], s_sum[3][i]);
        __syncthreads();
    }
}

// Every entry's own sums into the entries of all filtered nodes above its node,
// found by following each filtered node's next one up (RefineScratch::upSlot),
// four lookups in flight. Latency bound: a walk over all levels with one lookup
// at a time took 61 us for 209k entries, 42 us so.
__global__ void __launch_bounds__(256) k_cf_roll(Dev d, RefineScratch r) {
    constexpr uint32_t kAhead = 4;
    const uint32_t total = r.ctr->voxels;
    if (perPoint(r)) return;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const uint32_t slot = r.entrySlot[e];
        const ulonglong4 a = r.acc[e];
        if (slot == kNone || a.w == 0ull) continue;
        const unsigned long long key = __ldg(&r.hash[slot].x);
        uint32_t k = (uint32_t)(key >> 21);
        const uint32_t node = r.voxNode[k], cell = (uint32_t)(key & 0x1FFFFFull);
        const uint32_t lv = d.level[node];
        const uint32_t px = (d.nodeX[node] << 7) | (cell & 127u), py = (d.nodeY[node] << 7) | ((cell >> 7) & 127u),
                       pz = (d.nodeZ[node] << 7) | (cell >> 14);
        uint2 up = r.upSlot[k];  // (slot, level) of the next filtered node up
        while (up.x != kNone) {
            unsigned long long keys[kAhead];
            ulonglong2 kv[kAhead];
            uint32_t n = 0;
#pragma unroll
            for (uint32_t j = 0; j < kAhead; j++) {
                keys[j] = 0ull;
                if (up.x != kNone) {
                    const uint32_t sh = lv - up.y;
                    const uint32_t c = ((px >> sh) & 127u) + ((py >> sh) & 127u) * 128u + ((pz >> sh) & 127u) * 16384u;
                    keys[j] = ((unsigned long long)up.x << 21) | c;
                    up = r.upSlot[up.x];
                    n = j + 1u;
                }
            }
#pragma unroll
            for (uint32_t j = 0; j < kAhead; j++)
                kv[j] = j < n ? __ldg(&r.hash[slotOf(keys[j], r.hashMask)]) : make_ulonglong2(0ull, 0ull);
#pragma unroll
            for (uint32_t j = 0; j < kAhead; j++) {
                if (j >= n) continue;
                const uint32_t to = kv[j].x == keys[j] ? (uint32_t)kv[j].y : findEntry(r, keys[j]);
                if (to != kNone) addSums(&r.up[to], a.x, a.y, a.z, a.w);
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_cf_apply(Dev d, RefineScratch r) {
    const uint32_t nodes = r.ctr->nodes, total = r.ctr->voxels;
    const bool direct = perPoint(r);
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = nodes;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (r.voxBase[mid] <= e) lo = mid;
            else hi = mid;
        }
        const uint32_t node = r.voxNode[lo], s = e - r.voxBase[lo];
        ulonglong4 a = r.acc[e];
        if (!direct) {
            const ulonglong4 up = r.up[e];
            a.x += up.x;
            a.y += up.y;
            a.z += up.z;
            a.w += up.w;
        }
        const uint32_t phys = d.tablePool[d.vxTableOff[node] + s / d.ppc];
        if (a.w > 0 && phys != kNone) {
            Point* v = reinterpret_cast<Point*>(d.arena + (uint64_t)phys * 16u) + s % d.ppc;
            const unsigned long long half = a.w / 2u;
            const uint32_t cr = (uint32_t)((a.x + half) / a.w), cg = (uint32_t)((a.y + half) / a.w),
                           cb = (uint32_t)((a.z + half) / a.w);
            v->color = (v->color & 0xFF000000u) | cr | (cg << 8) | (cb << 16);
        }
        if (r.entrySlot[e] != kNone) r.hash[r.entrySlot[e]].x = ~0ull;
    }
    // every planned node's mark, voxels or not, for the next call
    for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nodes; k += gridDim.x * blockDim.x)
        r.refSlot[r.voxNode[k]] = kNone;
}

}  // namespace

__device__ uint32_t blockExclusiveScanRefine(uint32_t v, uint32_t* total, uint32_t* s_warp) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < (blockDim.x >> 5) ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, w, o);
            if (lane >= (uint32_t)o) w += y;
        }
        s_warp[lane] = w;
    }
    __syncthreads();
    const uint32_t prefix = (warp > 0 ? s_warp[warp - 1] : 0u) + x - v;
    *total = s_warp[(blockDim.x >> 5) - 1];
    __syncthreads();
    return prefix;
}

void launchRefineColors(const Dev& d, const RefineScratch& r, const uint32_t* queue, uint32_t queueLen,
                        uint32_t budget, int grid, cudaStream_t s) {
    k_cf_plan<<<1, 1024, 0, s>>>(d, r, queue, queueLen, budget);
    k_cf_units<<<grid, 256, 0, s>>>(d, r);
    k_cf_index<<<grid, 256, 0, s>>>(d, r);
    k_cf_gather<<<grid, 256, 0, s>>>(d, r);
    k_cf_roll<<<grid, 256, 0, s>>>(d, r);
    k_cf_apply<<<grid, 256, 0, s>>>(d, r);
}

}  // namespace rb
