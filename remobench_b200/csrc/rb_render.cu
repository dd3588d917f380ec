// Rasterize stage: frustum test, pixel-budget LOD cut, the visible nodes' samples
// split over warps, 64-bit depth|colour atomicMin splatting into a headless
// framebuffer.
//
// Restates kernels/remolod/remolod_render.cu:30-198 and
// kernels/shared/remo_{math,framebuffer,draw}.cuh. The framebuffer packs
// (float_bits(depth) << 32) | rgba, so atomicMin keeps the nearest sample and,
// on a depth tie, the smaller colour: the result does not depend on the order
// samples arrive in, which is what makes it bit-comparable with the CPU oracle.
//
// This file is compiled with -fmad=false: every float operation below rounds
// once, as in the oracle (compiled with -ffp-contract=off).
#include <cuda_runtime.h>

#include "rb_kernels.h"
#include "rb_launch.h"
#include "rb_state.h"

namespace rb {

constexpr unsigned long long kFbClear = 0x7f80000000332211ull;  // REMO_FB_CLEAR

struct F4 {
    float x, y, z, w;
};

// remoMatMul (remo_math.cuh:25-32)
__device__ __forceinline__ F4 matmul(const float* m, float x, float y, float z, float w) {
    F4 r;
    r.x = m[0] * x + m[1] * y + m[2] * z + m[3] * w;
    r.y = m[4] * x + m[5] * y + m[6] * z + m[7] * w;
    r.z = m[8] * x + m[9] * y + m[10] * z + m[11] * w;
    r.w = m[12] * x + m[13] * y + m[14] * z + m[15] * w;
    return r;
}

struct Plane {
    float nx, ny, nz, d;
};

// Frustum::fromViewProj (remo_math.cuh:52-67)
__device__ void frustumPlanes(const float* m, Plane pl[6]) {
    float v[6][4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        v[0][k] = m[12 + k] - m[k];
        v[1][k] = m[12 + k] + m[k];
        v[2][k] = m[12 + k] + m[4 + k];
        v[3][k] = m[12 + k] - m[4 + k];
        v[4][k] = m[12 + k] - m[8 + k];
        v[5][k] = m[12 + k] + m[8 + k];
    }
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const float a = v[i][0], b = v[i][1], c = v[i][2], dd = v[i][3];
        const float len = sqrtf(a * a + b * b + c * c);
        const float inv = len > 0.0f ? 1.0f / len : 0.0f;
        pl[i].nx = a * inv;
        pl[i].ny = b * inv;
        pl[i].nz = c * inv;
        pl[i].d = dd * inv;
    }
}

__device__ __forceinline__ bool frustumBox(const Plane* pl, const float mn[3], const float mx[3]) {
#pragma unroll
    for (int i = 0; i < 6; i++) {
        const float px = pl[i].nx > 0.0f ? mx[0] : mn[0];
        const float py = pl[i].ny > 0.0f ? mx[1] : mn[1];
        const float pz = pl[i].nz > 0.0f ? mx[2] : mn[2];
        if (pl[i].nx * px + pl[i].ny * py + pl[i].nz * pz + pl[i].d < 0.0f) return false;
    }
    return true;
}

__device__ __forceinline__ bool leafRowR(const Dev& d, uint32_t node) {
    const int4* row = reinterpret_cast<const int4*>(d.child + node * 8u);
    const int4 a = row[0], b = row[1];
    return (a.x & a.y & a.z & a.w & b.x & b.y & b.z & b.w) == -1;
}

// remoDrawPoint (remo_framebuffer.cuh:33-61): the sample's pixel and packed
// value; false when it lies behind the camera or its splat of half-width `half`
// misses the frame.
__device__ __forceinline__ bool project(const Frame& f, float x, float y, float z, uint32_t color, int32_t half,
                                        int32_t W, int32_t H, int32_t& ix, int32_t& iy, unsigned long long& packed) {
    const F4 clip = matmul(f.transform, x, y, z, 1.0f);
    if (clip.w <= 0.0f) return false;
    const float invW = 1.0f / clip.w;
    const float ndcX = clip.x * invW;
    const float ndcY = clip.y * invW;
    const float px = (ndcX * 0.5f + 0.5f) * f.width;
    const float py = (ndcY * 0.5f + 0.5f) * f.height;
    ix = __float2int_rz(px);
    iy = __float2int_rz(py);
    packed = ((unsigned long long)__float_as_uint(clip.w) << 32) | (unsigned long long)color;
    if (half == 0) return (uint32_t)ix < (uint32_t)W && (uint32_t)iy < (uint32_t)H;
    return (long long)ix + half >= 0 && (long long)iy + half >= 0 && (long long)ix - half < W &&
           (long long)iy - half < H;
}

// Pixels a block knows an upper bound of: a direct-mapped table of pixel index
// << 32 | depth bits, each entry read and written whole. A thread that lowers a
// pixel, or reads it, notes the depth it then has at most, so a later sample
// further away needs neither the read nor the atomic.
constexpr uint32_t kSeenBits = 11;  // 16 KB a block
struct SeenPixels {
    unsigned long long e[1u << kSeenBits];
};

// Draws up to kDraw samples a thread (ok: which there are). One-pixel splats,
// the usual size, read their pixels together before the first atomic; with
// `seen`, only those the block's table does not settle. Wider splats read four
// pixels of a row together: with a read and an atomic at a time, 81 pixels a splat
// took 284 us in the frame of a 2M-point tree at 1920 x 1080 and 1,435 of 8M flat
// points, 195 and 740 so, and 100 flat points, a chain of round trips, 38 and 20
// (6 by atomics alone, which take 1,394 and 8,450 for the other two).
template <bool kOnePixel, bool kSeen, uint32_t kDraw>
__device__ __forceinline__ void drawPoints(unsigned long long* fb, const Frame& f, const float4 (&v)[kDraw],
                                           const bool (&ok)[kDraw], bool rgb, uint32_t fixed,
                                           volatile unsigned long long* seen) {
    const int32_t half = kOnePixel ? 0 : f.pointSize / 2;
    const int32_t W = __float2int_rz(f.width), H = __float2int_rz(f.height);
    int32_t ix[kDraw], iy[kDraw];
    unsigned long long packed[kDraw];
    bool in[kDraw];
#pragma unroll
    for (uint32_t j = 0; j < kDraw; j++)
        in[j] = ok[j] && project(f, v[j].x, v[j].y, v[j].z, rgb ? __float_as_uint(v[j].w) : fixed, half, W, H, ix[j],
                                 iy[j], packed[j]);
    if (kOnePixel) {
        unsigned long long* px[kDraw];
        unsigned long long cur[kDraw];
        uint32_t tag[kDraw], slot[kDraw];
#pragma unroll
        for (uint32_t j = 0; j < kDraw; j++) {
            const unsigned long long at =
                in[j] ? (unsigned long long)(uint32_t)iy[j] * (uint32_t)W + (uint32_t)ix[j] : 0ull;
            px[j] = fb + at;
            if (kSeen) {
                tag[j] = (uint32_t)at;
                slot[j] = (tag[j] * 0x9E3779B1u) >> (32u - kSeenBits);
                const unsigned long long e = seen[slot[j]];
                in[j] = in[j] && !((uint32_t)(e >> 32) == tag[j] && (uint32_t)e < (uint32_t)(packed[j] >> 32));
            }
            cur[j] = in[j] ? __ldcg(px[j]) : 0ull;
        }
#pragma unroll
        for (uint32_t j = 0; j < kDraw; j++) {
            if (!in[j]) continue;
            if (cur[j] > packed[j]) atomicMin(px[j], packed[j]);
            if (kSeen) seen[slot[j]] = ((unsigned long long)tag[j] << 32) | (min(cur[j], packed[j]) >> 32);
        }
        return;
    }
    if (half < 0) return;  // a negative size draws nothing
    constexpr uint32_t kRow = 4;
#pragma unroll
    for (uint32_t j = 0; j < kDraw; j++) {
        if (!in[j]) continue;
        // not empty: project() saw the splat meet the frame
        const uint32_t x0 = (uint32_t)max((long long)ix[j] - half, 0ll), x1 = (uint32_t)min((long long)ix[j] + half, W - 1ll);
        const uint32_t y0 = (uint32_t)max((long long)iy[j] - half, 0ll), y1 = (uint32_t)min((long long)iy[j] + half, H - 1ll);
        for (uint32_t y = y0; y <= y1; y++) {
            unsigned long long* row = fb + (unsigned long long)y * (uint32_t)W;
            for (uint32_t x = x0; x <= x1; x += kRow) {
                // a pixel only ever decreases, so a sample no lower than what a plain
                // read returns (stale or not) needs no atomic
                unsigned long long cur[kRow];
#pragma unroll
                for (uint32_t k = 0; k < kRow; k++) cur[k] = x + k <= x1 ? __ldcg(row + x + k) : 0ull;
#pragma unroll
                for (uint32_t k = 0; k < kRow; k++)
                    if (cur[k] > packed[j]) atomicMin(row + x + k, packed[j]);
            }
        }
    }
}

__global__ void __launch_bounds__(256) k_fb_clear(unsigned long long* fb, uint64_t npx) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < npx;
         i += (uint64_t)gridDim.x * blockDim.x)
        fb[i] = kFbClear;
}

// The projected extent of a node's box above the pixel budget
// (projectedExtent, remolod_render.cu:40-70), or the node forced open.
__device__ __forceinline__ bool nodeLarge(const Frame& f, const uint8_t* forceLarge, uint32_t node, const float mn[3],
                                          const float mx[3]) {
    float minX = 1e30f, minY = 1e30f, maxX = -1e30f, maxY = -1e30f;
    bool any = false;
#pragma unroll
    for (int corner = 0; corner < 8; corner++) {
        const float x = (corner & 1) ? mx[0] : mn[0];
        const float y = (corner & 2) ? mx[1] : mn[1];
        const float z = (corner & 4) ? mx[2] : mn[2];
        const F4 clip = matmul(f.transformFrozen, x, y, z, 1.0f);
        if (clip.w <= 0.0f) continue;
        const float invW = 1.0f / clip.w;
        const float sx = (clip.x * invW * 0.5f + 0.5f) * f.width;
        const float sy = (clip.y * invW * 0.5f + 0.5f) * f.height;
        minX = fminf(minX, sx);
        maxX = fmaxf(maxX, sx);
        minY = fminf(minY, sy);
        maxY = fmaxf(maxY, sy);
        any = true;
    }
    float dx = 0.0f, dy = 0.0f;
    if (any) {
        dx = maxX - minX;
        dy = maxY - minY;
    }
    return dx > f.lodPixelBudget || dy > f.lodPixelBudget || (forceLarge && forceLarge[node]);
}

__device__ __forceinline__ void nodeBox(const Frame& f, float cube, uint32_t level, uint32_t X, uint32_t Y, uint32_t Z,
                                        float mn[3], float mx[3]) {
    const float s = cube / __int_as_float((int)((127u + level) << 23));
    mn[0] = f.boxMin[0] + (float)X * s;
    mn[1] = f.boxMin[1] + (float)Y * s;
    mn[2] = f.boxMin[2] + (float)Z * s;
    mx[0] = mn[0] + s;
    mx[1] = mn[1] + s;
    mx[2] = mn[2] + s;
}

// What is stored of a node's points and voxels.
__device__ __forceinline__ uint32_t storedPoints(const Dev& d, uint32_t node) {
    return min(d.numPoints[node], d.numPointChunks[node] * d.ppc);
}
__device__ __forceinline__ uint32_t storedVoxels(const Dev& d, uint32_t node) {
    return min(min(d.numVoxels[node], d.numVoxelsStored[node]), d.numVoxelChunks[node] * d.ppc);
}

// The LOD cut (both passes of remolod_render.cu:113-178) and the framebuffer's
// clear, which it does not depend on, in one launch. The disjoint frontier: a
// large inner node emits its visible children that are not large, a large
// visible leaf emits itself. Asked from the emitted node's side -- visible, and
// either not large below a large parent, or a large leaf -- it needs no flags of
// other nodes: the parent's box follows from the node's, so its test is redone
// with the same arithmetic where it matters. Each emitted item gets its place in
// the draw list and the samples before it in the list from one 64-bit atomic per
// warp (RenderScratch::cursor), so that k_raster can split the samples, not the
// items, over its warps. Bound at 7680 x 4320 by the clear (265 MB, 43 us), at
// 1920 x 1080 by the chain of one node's loads: 6.4 us, against 11.6 for clear,
// flags and frontier as three launches with their gaps besides.
__global__ void __launch_bounds__(256) k_cut(Dev d, Frame f, unsigned long long* fb, uint64_t npx,
                                             const uint8_t* forceLarge, RenderScratch* rs, DrawItem* items,
                                             uint32_t cap) {
    follow();
    __shared__ Plane s_pl[6];
    if (threadIdx.x == 0) {
        Plane pl[6];
        frustumPlanes(f.transformFrozen, pl);
        for (int i = 0; i < 6; i++) s_pl[i] = pl[i];
    }
    __syncthreads();
    uint32_t nn = d.ctr->numNodes;
    if (nn > d.maxNodes) nn = d.maxNodes;
    const float cube = fmaxf(fmaxf(f.boxMax[0] - f.boxMin[0], f.boxMax[1] - f.boxMin[1]),
                             f.boxMax[2] - f.boxMin[2]);
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < nn; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + lane;
        bool emit = false;
        uint32_t np = 0, nv = 0;
        if (i < nn) {
            np = d.numPoints[i];
            nv = d.numVoxels[i];
            const uint32_t lv = d.level[i], X = d.nodeX[i], Y = d.nodeY[i], Z = d.nodeZ[i];
            const uint32_t parent = lv > 0u ? d.parent[i].x : kNone;
            float mn[3], mx[3];
            nodeBox(f, cube, lv, X, Y, Z, mn, mx);
            if ((np > 0u || nv > 0u) && frustumBox(s_pl, mn, mx)) {
                if (nodeLarge(f, forceLarge, i, mn, mx)) {
                    emit = leafRowR(d, i);
                } else if (parent != kNone &&
                           d.child[parent * 8u + (((X & 1u) << 2) | ((Y & 1u) << 1) | (Z & 1u))] == (int32_t)i) {
                    nodeBox(f, cube, lv - 1u, X >> 1, Y >> 1, Z >> 1, mn, mx);
                    emit = nodeLarge(f, forceLarge, parent, mn, mx);
                }
            }
        }
        const unsigned em = __ballot_sync(0xFFFFFFFFu, emit);
        if (em == 0u) continue;
        const uint32_t work = emit ? storedPoints(d, i) + storedVoxels(d, i) : 0u;
        unsigned long long pre = work;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xFFFFFFFFu, pre, o);
            if (lane >= o) pre += y;
        }
        unsigned long long at = 0;
        if (lane == 31u) at = atomicAdd(&rs->cursor, (pre << kDrawCountBits) | (unsigned long long)__popc(em));
        at = __shfl_sync(0xFFFFFFFFu, at, 31);
        const uint32_t idx = (uint32_t)(at & kDrawCountMask) + (uint32_t)__popc(em & ((1u << lane) - 1u));
        const bool listed = emit && idx < cap;
        if (listed) items[idx] = drawItem(i, (at >> kDrawCountBits) + pre - work);
        unsigned long long drawn = listed ? (unsigned long long)np + nv : 0ull;
#pragma unroll
        for (uint32_t o = 16; o > 0u; o >>= 1) drawn += __shfl_xor_sync(0xFFFFFFFFu, drawn, o);
        if (lane == 0u && drawn) atomicAdd(&rs->samples, drawn);
    }
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < npx; i += (uint64_t)gridDim.x * blockDim.x)
        fb[i] = kFbClear;
}

// remoHashColor (kernels/shared/remo_prelude.cuh:87-97): a splitmix-style
// hash of the key, each channel mapped to [96, 255], alpha 255.
__device__ __forceinline__ uint32_t hashColor(unsigned long long key) {
    unsigned long long h = (key + 0x9E3779B97F4A7C15ull) * 0x9E3779B97F4A7C15ull;
    h ^= h >> 29;
    h *= 0xBF58476D1CE4E5B9ull;
    h ^= h >> 32;
    const uint32_t r = 96u + (((uint32_t)h & 0xFFu) * 159u) / 255u;
    const uint32_t g = 96u + (((uint32_t)(h >> 8) & 0xFFu) * 159u) / 255u;
    const uint32_t b = 96u + (((uint32_t)(h >> 16) & 0xFFu) * 159u) / 255u;
    return r | (g << 8) | (b << 16) | (255u << 24);
}

// remoSampleColor (remo_draw.cuh:104-116): the colour every sample of a draw
// item takes in the non-RGB modes; the item key is the node's pool index.
__device__ __forceinline__ uint32_t itemColor(int32_t mode, uint32_t node, uint32_t level) {
    if (mode == 3) return 0xFFFFFFFFu;
    if (mode == 1) return hashColor(node);
    return hashColor((unsigned long long)level * 2654435761ull);
}

__device__ __forceinline__ uint32_t listedItems(const RenderScratch* rs, uint32_t cap) {
    return (uint32_t)min(rs->cursor & kDrawCountMask, (unsigned long long)cap);
}

// remoRasterizeDrawList (remo_draw.cuh:118-167). The frame's samples, in draw
// list order, are split evenly over the grid's warps: a warp finds the item its
// share begins in by a 32-ary search of the items' running sample counts and
// walks on from there, its lanes on consecutive samples (one chunk's loads
// coalesce), kDraw samples a lane with each step's loads issued for all. The
// block-per-item form this replaces left most of the chip waiting for the blocks
// that drew the largest items (14.6% of warps active at 1080p): 102 us there for
// 8M points, 13 so; 142 and 43 at 7680 x 4320. Bound by the latency of the chunk,
// sample and pixel reads: two samples a lane at six blocks per SM (13.0 us) beat
// four at four (15.2). The counts the host reads go straight to its pinned copy.
template <bool kOnePixel>
__global__ void __launch_bounds__(256, 6) k_raster(Dev d, Frame f, unsigned long long* fb,
                                                const RenderScratch* rs, const DrawItem* items,
                                                uint32_t cap, RenderResult* host) {
    follow();
    constexpr uint32_t kDraw = 2;
    const uint32_t ni = listedItems(rs, cap);
    const uint32_t lane = threadIdx.x & 31u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        host->numItems = (uint32_t)(rs->cursor & kDrawCountMask);
        host->overflow = host->numItems > cap ? 1u : 0u;
        host->samples = rs->samples;
    }
    if (ni == 0u) return;
    unsigned long long total = rs->cursor >> kDrawCountBits;
    if ((rs->cursor & kDrawCountMask) > cap) {  // the list is full: its last item ends the work
        const DrawItem last = items[ni - 1u];
        total = itemFirst(last) + storedPoints(d, itemNode(last)) + storedVoxels(d, itemNode(last));
    }
    const DrawShare mine =
        drawShare(total, (gridDim.x * blockDim.x) >> 5, (blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (mine.begin >= mine.end) return;
    const unsigned long long begin = mine.begin, end = mine.end;
    // the last item that starts at or before `begin`: [lo, hi) narrows 32-fold a round
    uint32_t lo = 0, hi = ni;
    while (hi - lo > 1u) {
        const uint32_t step = (hi - lo + 31u) >> 5;
        const uint32_t p = lo + lane * step;
        const bool le = p < hi && itemFirst(items[p]) <= begin;
        const uint32_t k = 31u - (uint32_t)__clz((int)__ballot_sync(0xFFFFFFFFu, le));
        lo += k * step;
        hi = min(hi, lo + step);
    }
    const bool rgb = f.colorMode < 1 || f.colorMode > 3;
    for (unsigned long long s = begin; s < end; lo++) {
        const DrawItem it = items[lo];
        const uint32_t node = itemNode(it);
        const uint32_t np = storedPoints(d, node), n = np + storedVoxels(d, node);
        const uint32_t poff = d.ptTableOff[node], voff = d.vxTableOff[node];
        const uint32_t fixed = rgb ? 0u : itemColor(f.colorMode, node, d.level[node]);
        const uint32_t stop = itemStop(it, n, end);
        for (uint32_t k0 = (uint32_t)(s - itemFirst(it)); k0 < stop; k0 += 32u * kDraw) {
            float4 v[kDraw];
            bool ok[kDraw];
#pragma unroll
            for (uint32_t j = 0; j < kDraw; j++) {
                const uint32_t k = k0 + j * 32u + lane;
                const bool pt = k < np;
                uint32_t within;
                const uint32_t chunk = chunkOf(d, pt ? k : k - np, within);
                const uint32_t phys = k < stop ? d.tablePool[(pt ? poff : voff) + chunk] : kNone;
                ok[j] = phys != kNone;
                v[j] = ok[j] ? __ldg(reinterpret_cast<const float4*>(chunkPoints(d, phys) + within))
                             : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            drawPoints<kOnePixel, false, kDraw>(fb, f, v, ok, rgb, fixed, nullptr);
        }
        s = itemFirst(it) + stop;
    }
}

// remoClipSegment2D (remo_lines.cuh:30-55): Liang-Barsky against
// [0, xmax] x [0, ymax]; false when the segment misses.
__device__ __forceinline__ bool clipTest(float p, float q, float& t0, float& t1) {
    if (p == 0.0f) return q >= 0.0f;
    const float r = q / p;
    if (p < 0.0f) {
        if (r > t1) return false;
        if (r > t0) t0 = r;
    } else {
        if (r < t0) return false;
        if (r < t1) t1 = r;
    }
    return true;
}

// remoDrawSegment (remo_lines.cuh:57-117): near-plane clip in clip space at
// w = 1e-6, screen clip, then one sample per step along the longer axis with
// depth from the interpolated 1/w.
__device__ void drawSegment(unsigned long long* fb, const Frame& f, float ax0, float ay0, float az0, float bx0,
                            float by0, float bz0, uint32_t color) {
    F4 c0 = matmul(f.transform, ax0, ay0, az0, 1.0f);
    F4 c1 = matmul(f.transform, bx0, by0, bz0, 1.0f);
    const float kMinW = 1.0e-6f;
    if (c0.w < kMinW && c1.w < kMinW) return;
    if (c0.w < kMinW) {
        const float t = (kMinW - c0.w) / (c1.w - c0.w);
        c0 = F4{c0.x + t * (c1.x - c0.x), c0.y + t * (c1.y - c0.y), c0.z + t * (c1.z - c0.z), kMinW};
    } else if (c1.w < kMinW) {
        const float t = (kMinW - c1.w) / (c0.w - c1.w);
        c1 = F4{c1.x + t * (c0.x - c1.x), c1.y + t * (c0.y - c1.y), c1.z + t * (c0.z - c1.z), kMinW};
    }
    const float invW0 = 1.0f / c0.w, invW1 = 1.0f / c1.w;
    const float sx0 = (c0.x * invW0 * 0.5f + 0.5f) * f.width;
    const float sy0 = (c0.y * invW0 * 0.5f + 0.5f) * f.height;
    const float sx1 = (c1.x * invW1 * 0.5f + 0.5f) * f.width;
    const float sy1 = (c1.y * invW1 * 0.5f + 0.5f) * f.height;
    const int32_t W = __float2int_rz(f.width), H = __float2int_rz(f.height);
    if (W <= 0 || H <= 0) return;
    const float dx = sx1 - sx0, dy = sy1 - sy0;
    float t0 = 0.0f, t1 = 1.0f;
    if (!clipTest(-dx, sx0, t0, t1) || !clipTest(dx, (float)(W - 1) - sx0, t0, t1) || !clipTest(-dy, sy0, t0, t1) ||
        !clipTest(dy, (float)(H - 1) - sy0, t0, t1))
        return;
    const float ax = sx0 + t0 * (sx1 - sx0), ay = sy0 + t0 * (sy1 - sy0);
    const float bx = sx0 + t1 * (sx1 - sx0), by = sy0 + t1 * (sy1 - sy0);
    const int32_t steps = __float2int_rz(fmaxf(fabsf(bx - ax), fabsf(by - ay))) + 1;
    const float invSteps = 1.0f / (float)steps;
    for (int32_t st = 0; st <= steps; ++st) {
        const float q = (float)st * invSteps;
        const int32_t ix = __float2int_rz(ax + q * (bx - ax));
        const int32_t iy = __float2int_rz(ay + q * (by - ay));
        if (ix < 0 || iy < 0 || ix >= W || iy >= H) continue;
        const float sT = t0 + q * (t1 - t0);
        const float invW = invW0 + sT * (invW1 - invW0);
        if (!(invW > 0.0f)) continue;
        const float depth = 1.0f / invW;
        atomicMin(&fb[(unsigned long long)iy * (unsigned long long)W + (unsigned long long)ix],
                  ((unsigned long long)__float_as_uint(depth) << 32) | (unsigned long long)color);
    }
}

// remoDrawListWireframe (remo_lines.cuh:120-137): the 12 edges of every draw
// item's node box (remoBoxEdge, :11-27: edge / 4 is the axis the edge runs
// along, edge % 4 picks the offsets on the other two), coloured by level.
__global__ void __launch_bounds__(256) k_wireframe(Dev d, Frame f, unsigned long long* fb,
                                                   const RenderScratch* rs, const DrawItem* items, uint32_t cap) {
    const uint32_t ni = listedItems(rs, cap);
    const float cube = fmaxf(fmaxf(f.boxMax[0] - f.boxMin[0], f.boxMax[1] - f.boxMin[1]), f.boxMax[2] - f.boxMin[2]);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < (uint64_t)ni * 12u;
         i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t node = itemNode(items[i / 12u]);
        const uint32_t edge = (uint32_t)(i % 12u);
        const uint32_t lv = d.level[node];
        const float size = cube / __int_as_float((int)((127u + lv) << 23));
        if (!(size > 0.0f)) continue;
        const float mn[3] = {f.boxMin[0] + (float)d.nodeX[node] * size, f.boxMin[1] + (float)d.nodeY[node] * size,
                             f.boxMin[2] + (float)d.nodeZ[node] * size};
        const uint32_t axis = edge / 4u, rest = edge % 4u;
        float off[3] = {0.0f, 0.0f, 0.0f};
        off[(axis + 1u) % 3u] = (rest & 1u) ? size : 0.0f;
        off[(axis + 2u) % 3u] = (rest & 2u) ? size : 0.0f;
        const float a[3] = {mn[0] + off[0], mn[1] + off[1], mn[2] + off[2]};
        off[axis] = size;
        drawSegment(fb, f, a[0], a[1], a[2], mn[0] + off[0], mn[1] + off[1], mn[2] + off[2],
                    hashColor((unsigned long long)lv * 2654435761ull));
    }
}

// flat_render.cu:9-76: every point of a resident cloud. A scan puts most of its
// points on few pixels (88% of 8M on 10,000 of a 1080p frame), so an atomic a
// point queues up on them: 125 us. A block takes one contiguous run of points,
// one wave of blocks, and remembers the pixels it has met; what is left is the
// latency of the point loads, hence many warps (32 registers) with two points
// each in flight: 47 us, against 77 with four points at four blocks per SM.
template <bool kOnePixel, bool kSeen>
__global__ void __launch_bounds__(256, 8) k_raster_flat(Frame f, unsigned long long* fb,
                                                     const Point* __restrict__ pts, uint64_t n) {
    constexpr uint32_t kDraw = 2;
    __shared__ SeenPixels s_seen;
    if (kSeen)  // ~0 marks no pixel: no depth is above its own
        for (uint32_t i = threadIdx.x; i < (1u << kSeenBits); i += blockDim.x) s_seen.e[i] = ~0ull;
    __syncthreads();
    const uint64_t share = (n / gridDim.x + 32u) & ~31ull;
    const uint64_t begin = blockIdx.x * share, end = begin + share < n ? begin + share : n;
    for (uint64_t b = begin + threadIdx.x; b < end; b += (uint64_t)blockDim.x * kDraw) {
        float4 v[kDraw];
        bool ok[kDraw];
#pragma unroll
        for (uint32_t j = 0; j < kDraw; j++) {
            const uint64_t i = b + (uint64_t)j * blockDim.x;
            ok[j] = i < end;
            v[j] = ok[j] ? __ldg(reinterpret_cast<const float4*>(pts + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        drawPoints<kOnePixel, kSeen, kDraw>(fb, f, v, ok, true, 0u, s_seen.e);
    }
}

__device__ __forceinline__ float fbDepth(unsigned long long px) {
    return __uint_as_float((uint32_t)(px >> 32));
}

// remoApplyEDL (remo_framebuffer.cuh:78-122); libm log2f/expf in place of the
// reference's __log2f/__expf. In place: a pixel reads its neighbours' depths
// only and rewrites its own colour half only, so the result does not depend on
// which neighbours were already shaded. rgba, when given, receives the resolved
// colours (remoResolve, :63-76) in the same pass over the framebuffer.
//
// A block shades a 64 x (4 kEdlRows) tile: the log depths of the tile and its one-pixel
// rim go to shared memory once (1.1 to 1.2 logarithms a pixel instead of 5;
// NaN where there is no surface), then each thread shades the pixels of its part
// of a column. A pixel
// whose colour does not change is not written back. Bound by instruction issue
// and, at 7680 x 4320, the bytes: EDL took 78 us there and the resolve, which
// read the framebuffer again, 76; 80 us together.
constexpr int kEdlW = 64;

template <int kEdlRows>
__global__ void __launch_bounds__(256) k_edl(unsigned long long* fb, uint32_t* rgba, uint32_t width, uint32_t height,
                                             float strength) {
    follow();
    constexpr int kEdlH = 4 * kEdlRows;
    __shared__ float s_log[kEdlH + 2][kEdlW + 2];
    const int w = (int)width, h = (int)height;
    const int tx = (int)(threadIdx.x & (kEdlW - 1u)), ty = (int)(threadIdx.x / kEdlW) * kEdlRows;
    const int x0 = (int)blockIdx.x * kEdlW, x = x0 + tx;
    const float none = __int_as_float(0x7fc00000);
    auto logAt = [&](unsigned long long px) {
        const float depth = fbDepth(px);
        return depth < 3.0e38f ? log2f(depth) : none;
    };
    for (int y0 = (int)blockIdx.y * kEdlH; y0 < h; y0 += (int)gridDim.y * kEdlH) {
        const uint64_t at = (uint64_t)(y0 + ty) * width + (uint32_t)x;
        const int rows = x < w ? min(kEdlRows, h - (y0 + ty)) : 0;
        unsigned long long px[kEdlRows];
#pragma unroll
        for (int j = 0; j < kEdlRows; j++) px[j] = j < rows ? fb[at + (uint64_t)j * width] : kFbClear;
        // the rim: the rows above and below, the columns left and right
        int sx = -1, sy = 0;
        unsigned long long rim = kFbClear;
        if (threadIdx.x < 2u * kEdlW + 2u * kEdlH) {
            const int t = (int)threadIdx.x, u = t - 2 * kEdlW;
            sx = u < 0 ? tx + 1 : (u < kEdlH ? 0 : kEdlW + 1);
            sy = u < 0 ? (t < kEdlW ? 0 : kEdlH + 1) : u % kEdlH + 1;
            const int gx = x0 + sx - 1, gy = y0 + sy - 1;
            if (gx >= 0 && gy >= 0 && gx < w && gy < h) rim = fb[(uint64_t)gy * width + (uint32_t)gx];
        }
        __syncthreads();  // the last tile's logs are read
#pragma unroll
        for (int j = 0; j < kEdlRows; j++) s_log[ty + j + 1][tx + 1] = logAt(px[j]);
        if (sx >= 0) s_log[sy][sx] = logAt(rim);
        __syncthreads();
        float up = s_log[ty][tx + 1], ld = s_log[ty + 1][tx + 1];
#pragma unroll
        for (int j = 0; j < kEdlRows; j++) {
            if (j >= rows) break;
            const float down = s_log[ty + j + 2][tx + 1];
            uint32_t c = (uint32_t)px[j];
            if (ld == ld) {
                const float n[4] = {s_log[ty + j + 1][tx], s_log[ty + j + 1][tx + 2], up, down};
                float resp = 0.0f;
                int taps = 0;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (n[k] == n[k]) {
                        resp += fmaxf(0.0f, ld - n[k]);
                        taps++;
                    }
                }
                if (taps) {
                    // the mean of the taps; a power of two's quotient is its reciprocal's product
                    resp = taps == 3 ? resp / 3.0f : resp * (taps == 4 ? 0.25f : (taps == 2 ? 0.5f : 1.0f));
                    const float shade = expf(-resp * 24.0f * strength);
                    const uint32_t r = (uint32_t)((float)(c & 255u) * shade);
                    const uint32_t g = (uint32_t)((float)((c >> 8) & 255u) * shade);
                    const uint32_t b = (uint32_t)((float)((c >> 16) & 255u) * shade);
                    const uint32_t shaded = r | (g << 8) | (b << 16) | (255u << 24);
                    if (shaded != c) {
                        c = shaded;
                        // the colour half only (little-endian: the low word)
                        reinterpret_cast<uint32_t*>(fb + at + (uint64_t)j * width)[0] = c;
                    }
                }
            }
            if (rgba) rgba[at + (uint64_t)j * width] = c;
            up = ld;
            ld = down;
        }
    }
}

// remoResolve (remo_framebuffer.cuh:63-76) into a plain RGBA buffer.
__global__ void __launch_bounds__(256) k_resolve(const unsigned long long* fb, uint32_t* rgba, uint64_t npx) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < npx;
         i += (uint64_t)gridDim.x * blockDim.x)
        rgba[i] = (uint32_t)fb[i];
}

void launchFbClear(unsigned long long* fb, uint64_t npx, int grid, cudaStream_t s) {
    k_fb_clear<<<grid, 256, 0, s>>>(fb, npx);
}
void launchCut(const Dev& d, const Frame& f, unsigned long long* fb, uint64_t npx, const uint8_t* force,
               RenderScratch* rs, DrawItem* items, uint32_t cap, int grid, cudaStream_t s) {
    cudaMemsetAsync(rs, 0, sizeof(RenderScratch), s);
    k_cut<<<grid, 256, 0, s>>>(d, f, fb, npx, force, rs, items, cap);
}
void launchRaster(const Dev& d, const Frame& f, unsigned long long* fb, const RenderScratch* rs,
                  const DrawItem* items, uint32_t cap, RenderResult* host, int grid, cudaStream_t s) {
    if (f.pointSize / 2 == 0) launchBehind(k_raster<true>, grid, 256, 0, s, d, f, fb, rs, items, cap, host);
    else launchBehind(k_raster<false>, grid, 256, 0, s, d, f, fb, rs, items, cap, host);
}
void launchRasterFlat(const Frame& f, unsigned long long* fb, const Point* pts, uint64_t n, int grid,
                      cudaStream_t s) {
    // the table of seen pixels names a pixel by 32 bits of its index: one-pixel
    // splats in larger frames go without it
    const bool indexed = (uint64_t)f.width * (uint64_t)f.height <= 1ull << 32;
    // no more blocks than have points: each of the others would clear its table
    const int blocks = (int)min((n + 255u) / 256u, (uint64_t)grid);
    if (f.pointSize / 2 != 0) k_raster_flat<false, false><<<blocks, 256, 0, s>>>(f, fb, pts, n);
    else if (indexed) k_raster_flat<true, true><<<blocks, 256, 0, s>>>(f, fb, pts, n);
    else k_raster_flat<true, false><<<blocks, 256, 0, s>>>(f, fb, pts, n);
}
void launchEdl(unsigned long long* fb, uint32_t* rgba, uint32_t w, uint32_t h, float strength, cudaStream_t s) {
    // 32-row tiles while they are many waves of blocks, else 16-row ones: at
    // 1920 x 1080 (1,020 tiles of 32 rows) 9.1 us against 8.1, at 7680 x 4320 80 against 100
    const bool tall = (uint64_t)w * h >= (4ull << 20);
    const uint32_t rows = tall ? 32u : 16u;
    const dim3 grid((w + kEdlW - 1u) / kEdlW, min((h + rows - 1u) / rows, 65535u));
    if (tall) launchBehind(k_edl<8>, grid, 256, 0, s, fb, rgba, w, h, strength);
    else launchBehind(k_edl<4>, grid, 256, 0, s, fb, rgba, w, h, strength);
}
void launchResolve(const unsigned long long* fb, uint32_t* rgba, uint64_t npx, int grid, cudaStream_t s) {
    k_resolve<<<grid, 256, 0, s>>>(fb, rgba, npx);
}
void launchWireframe(const Dev& d, const Frame& f, unsigned long long* fb, const RenderScratch* rs,
                     const DrawItem* items, uint32_t cap, int grid, cudaStream_t s) {
    k_wireframe<<<grid, 256, 0, s>>>(d, f, fb, rs, items, cap);
}

}  // namespace rb
