// Analysis stage: roll the leaves' exact sums up the tree, finalise each
// node's centred covariance, solve the 3x3 symmetric eigenproblem, score each
// node by surface variation x screen coverage, and rebuild the per-frame
// priority queue.
//
// The reference specifies this stage in prose only (wiki/02_KernelPipeline.md:204-224,
// README.md:30-48, plans/01_NoveltyAssessment.md:44-46); there is no kernel to
// follow. Conventions fixed here: eigenvalues are descending, l1 >= l2 >= l3,
// in units of (node size)^2; surface variation = l3 / (l1 + l2 + l3);
// planarity = (l2 - l3) / l1; closure = the node's subtree received no point
// for `closure_margin` batches (lastTouchedBatch plus a batch-age margin,
// wiki/02_KernelPipeline.md:215-221; the Morton watermark is not a closure
// test because no reader emits Morton order).
//
// Arithmetic: the roll-up is exact (64/128-bit integers, children re-based to
// the parent's origin); the centred scatter n*Sxx - Sx*Sx is exact in 128 bits
// and is converted to FP64 once; the eigen-solve is the closed-form
// trigonometric method (O. K. Smith, "Eigenvalues of a symmetric 3x3 matrix",
// CACM 4(4):168, 1961) in FP32, with a cyclic Jacobi in FP64 for near-degenerate
// matrices (l3 < 1e-3 * l1, or a nearly diagonal matrix).
#include <cuda_runtime.h>

#include "rb_analysis.h"
#include "rb_kernels.h"
#include "rb_launch.h"
#include "rb_state.h"

namespace rb {

typedef unsigned __int128 u128;
typedef __int128 i128;

__device__ __forceinline__ bool leafA(const Dev& d, uint32_t node) {
    const int4* row = reinterpret_cast<const int4*>(d.child + node * 8u);
    const int4 a = row[0], b = row[1];
    return (a.x & a.y & a.z & a.w & b.x & b.y & b.z & b.w) == -1;
}

// The roll-up: every node's sums over its subtree's leaves. With coordinates
// taken from the root's origin they are plain additions, so a leaf's sums are
// first re-based by its own origin O in the 2^28 grid: S1 += n O,
// S2_ab += O_a S1_b + O_b S1_a + n O_a O_b, and k_analyze re-bases each node's
// total back to the node's origin. Integers modulo 2^64 and 2^128: any order of
// additions gives the same bits, and the totals fit.
//
// One launch for every level. A split hands its children eight consecutive ids
// in octant order, so sibling group g is nodes 1 + 8 g .. 8 + 8 g and eight
// lanes hold one group, each its node's sums. They go through shared memory so
// that each lane adds up a share of the parent's words and writes it (a
// butterfly of shuffles moves every word three times). A group whose members
// are all leaves goes on to its parent's group; elsewhere the last of the
// group's own leaves and its inner members to arrive does (rollArrive counts
// them, and the one that goes on clears it). No block waits for another. Bound
// by the longest chain of dependent round trips, one arrival and one read per
// level of the tree, not by bytes (184 B read and written per node). Measured
// at 31,497 nodes: 232 us as a launch per level (a pass over all nodes for each
// of the 21, whatever the tree's depth), 38 us so; at 2,000 nodes 120 and
// 23 us. Re-basing at every step of the chain instead: 59 and 33 us.
constexpr uint32_t kRollThreads = 128;
constexpr uint32_t kRollWords = sizeof(RollSum) / 8u;

// r, relative to the origin of the node at `level` with coordinates N, to the
// root's origin (up) or back (down).
template <bool up>
__device__ __forceinline__ void rollRebase(RollSum& r, uint32_t level, uint32_t X, uint32_t Y, uint32_t Z) {
    const uint32_t sh = 28u - level;
    const unsigned long long o[3] = {(unsigned long long)X << sh, (unsigned long long)Y << sh,
                                     (unsigned long long)Z << sh};
    const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
    for (int k = 0; k < 6; k++) {
        u128 s2 = ((u128)r.s2[2 * k + 1] << 64) | r.s2[2 * k];
        const u128 cross = (u128)o[pa[k]] * r.s1[pb[k]] + (u128)o[pb[k]] * r.s1[pa[k]];
        const u128 square = (u128)(o[pa[k]] * o[pb[k]]) * r.n;
        s2 = up ? s2 + cross + square : s2 - cross + square;
        r.s2[2 * k] = (unsigned long long)s2;
        r.s2[2 * k + 1] = (unsigned long long)(s2 >> 64);
    }
#pragma unroll
    for (int k = 0; k < 3; k++) r.s1[k] = up ? r.s1[k] + r.n * o[k] : r.s1[k] - r.n * o[k];
}

__device__ __forceinline__ RollSum leafSums(const AccumI& a) {
    RollSum r;
    r.n = a.count;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        r.s1[k] = a.s1[k];
        r.c1[k] = a.c1[k];
        r.c2[k] = a.c2[k];
    }
#pragma unroll
    for (int k = 0; k < 6; k++) {
        r.s2[2 * k] = a.s2lo[k];
        r.s2[2 * k + 1] = a.s2hi[k];
    }
    r.lastTouched = a.count ? a.lastTouchedBatch : 0u;
    r.pad = 0;
    return r;
}

// One more arrival: what the group's lanes wrote before it is visible to the
// one that sees the last.
__device__ __forceinline__ uint32_t arriveAcqRel(uint32_t* p) {
    uint32_t old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
    return old;
}

__global__ void __launch_bounds__(kRollThreads) k_roll(Dev d, RollSum* roll, uint32_t* rollArrive,
                                                       AnalysisCounters* ac) {
    follow();
    __shared__ unsigned long long s_words[kRollThreads / 8][8][kRollWords];
    const uint32_t nn = d.ctr->numNodes;
    const uint32_t oct = threadIdx.x & 7u;
    const unsigned gmask = 0xFFu << (threadIdx.x & 24u);
    unsigned long long(*words)[kRollWords] = s_words[threadIdx.x >> 3];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *ac = AnalysisCounters{};
        ac->numNodes = nn;
        if (leafA(d, 0)) roll[0] = leafSums(d.accum[0]);  // its origin is the root's
    }
    // the words this lane adds up: lanes 0..5 a 128-bit sum of s2 and one of
    // {n, s1}; lanes 6 and 7 the three of c1 or c2
    const bool pair = oct < 6u;
    const uint32_t w0 = pair ? 4u + 2u * oct : (oct == 6u ? 16u : 19u), w1 = w0 + 1u;
    const uint32_t w2 = oct < 4u ? oct : w0 + 2u;
    const bool third = oct < 4u || !pair;
    const uint32_t groups = nn / 8u;  // the root, then eight nodes per split
    for (uint32_t g0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 3; g0 < groups; g0 += (gridDim.x * blockDim.x) >> 3) {
        uint32_t g = g0, node = 1u + 8u * g + oct;
        bool leaf = leafA(d, node);
        uint32_t parent = d.parent[node].x;
        RollSum r = {};
        if (leaf) {
            r = leafSums(d.accum[node]);
            rollRebase<true>(r, d.level[node], d.nodeX[node], d.nodeY[node], d.nodeZ[node]);
            roll[node] = r;
        }
        // a collapsed node's former children hang off nothing
        const bool attached = d.child[parent * 8u + oct] == (int32_t)node;
        if (__ballot_sync(gmask, attached) != gmask) continue;
        __syncwarp(gmask);
        const bool whole = __ballot_sync(gmask, leaf) == gmask;
        for (bool start = true;; start = false) {
            if (start && whole) {
                const unsigned long long* q = reinterpret_cast<const unsigned long long*>(&r);
#pragma unroll
                for (uint32_t k = 0; k < kRollWords; k++) words[oct][k] = q[k];
            } else {
                uint32_t arrived = 0;
                if (oct == 0u) arrived = arriveAcqRel(&rollArrive[g]) + 1u;
                arrived = __shfl_sync(gmask, arrived, 0, 8);
                const uint32_t inner = __popc(__ballot_sync(gmask, !leaf));
                if (arrived != inner + 1u) break;
                if (oct == 0u) rollArrive[g] = 0u;
                __syncwarp(gmask);  // lane 0's acquire, for the others' reads
                const unsigned long long* p = reinterpret_cast<const unsigned long long*>(&roll[node]);
#pragma unroll
                for (uint32_t k = 0; k < kRollWords; k++) words[oct][k] = __ldcg(p + k);
            }
            __syncwarp(gmask);
            unsigned long long a = 0, b = 0, e = 0, lt = 0;
            // half unrolled: a climb runs this cold, and eight copies cost more in
            // instruction fetches than they save (27 against 23 us at 2,000 nodes)
#pragma unroll 2
            for (uint32_t m = 0; m < 8u; m++) {
                const unsigned long long va = words[m][w0];
                a += va;
                b += words[m][w1] + (pair && a < va ? 1ull : 0ull);
                e += words[m][w2];
                lt = max(lt, words[m][22]);
            }
            unsigned long long* out = reinterpret_cast<unsigned long long*>(&roll[parent]);
            out[w0] = a;
            out[w1] = b;
            if (third) out[w2] = e;
            if (oct == 5u) out[22] = lt;  // the newest batch; pad is zero
            if (parent == 0u) break;
            // the group above: what does not depend on its other members
            g = (parent - 1u) >> 3;
            node = 1u + 8u * g + oct;
            leaf = leafA(d, node);
            parent = d.parent[node].x;
            __syncwarp(gmask);
        }
        __syncwarp(gmask);  // the words are read before the next group's are written
    }
}

__device__ __forceinline__ double i128ToDouble(i128 v) {
    const bool neg = v < 0;
    const u128 m = neg ? (u128)(-v) : (u128)v;
    const double hi = (double)(unsigned long long)(m >> 64);
    const double lo = (double)(unsigned long long)m;
    const double r = hi * 18446744073709551616.0 + lo;
    return neg ? -r : r;
}

// Cyclic Jacobi on a symmetric 3x3 in FP64; eigenvalues descending, the
// eigenvector of the smallest in vmin.
__device__ void jacobi3(const double ain[6], double eig[3], double vmin[3]) {
    double a[3][3] = {{ain[0], ain[1], ain[2]}, {ain[1], ain[3], ain[4]}, {ain[2], ain[4], ain[5]}};
    double v[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
    for (int sweep = 0; sweep < 32; sweep++) {
        const double off = a[0][1] * a[0][1] + a[0][2] * a[0][2] + a[1][2] * a[1][2];
        const double diag = a[0][0] * a[0][0] + a[1][1] * a[1][1] + a[2][2] * a[2][2];
        if (off <= 1e-36 * diag || off == 0.0) break;
        for (int p = 0; p < 2; p++)
            for (int q = p + 1; q < 3; q++) {
                if (a[p][q] == 0.0) continue;
                const double th = (a[q][q] - a[p][p]) / (2.0 * a[p][q]);
                const double t = (th >= 0 ? 1.0 : -1.0) / (fabs(th) + sqrt(th * th + 1.0));
                const double c = 1.0 / sqrt(t * t + 1.0), s = t * c;
                for (int k = 0; k < 3; k++) {
                    const double akp = a[k][p], akq = a[k][q];
                    a[k][p] = c * akp - s * akq;
                    a[k][q] = s * akp + c * akq;
                }
                for (int k = 0; k < 3; k++) {
                    const double apk = a[p][k], aqk = a[q][k];
                    a[p][k] = c * apk - s * aqk;
                    a[q][k] = s * apk + c * aqk;
                }
                for (int k = 0; k < 3; k++) {
                    const double vkp = v[k][p], vkq = v[k][q];
                    v[k][p] = c * vkp - s * vkq;
                    v[k][q] = s * vkp + c * vkq;
                }
            }
    }
    int o[3] = {0, 1, 2};
    const double dg[3] = {a[0][0], a[1][1], a[2][2]};
    for (int i = 0; i < 3; i++)
        for (int j = i + 1; j < 3; j++)
            if (dg[o[j]] > dg[o[i]]) {
                const int t = o[i];
                o[i] = o[j];
                o[j] = t;
            }
    for (int i = 0; i < 3; i++) eig[i] = dg[o[i]];
    for (int k = 0; k < 3; k++) vmin[k] = v[k][o[2]];
}

// Smith's closed form in FP32. Returns false when the matrix is too close to
// degenerate for it (the caller then takes the FP64 branch).
__device__ bool smith3(const float a[6], float eig[3]) {
    const float p1 = a[1] * a[1] + a[2] * a[2] + a[4] * a[4];
    const float q = (a[0] + a[3] + a[5]) * (1.0f / 3.0f);
    const float b00 = a[0] - q, b11 = a[3] - q, b22 = a[5] - q;
    const float p2 = b00 * b00 + b11 * b11 + b22 * b22 + 2.0f * p1;
    if (!(p2 > 0.0f)) return false;
    const float p = sqrtf(p2 * (1.0f / 6.0f));
    if (p1 < 1e-12f * p2) return false;  // nearly diagonal
    const float ip = 1.0f / p;
    const float c00 = b00 * ip, c11 = b11 * ip, c22 = b22 * ip;
    const float c01 = a[1] * ip, c02 = a[2] * ip, c12 = a[4] * ip;
    const float det = c00 * (c11 * c22 - c12 * c12) - c01 * (c01 * c22 - c12 * c02) + c02 * (c01 * c12 - c11 * c02);
    float r = 0.5f * det;
    r = fminf(fmaxf(r, -1.0f), 1.0f);
    const float phi = acosf(r) * (1.0f / 3.0f);
    const float l1 = q + 2.0f * p * cosf(phi);
    const float l3 = q + 2.0f * p * cosf(phi + 2.0943951023931953f);
    const float l2 = 3.0f * q - l1 - l3;
    eig[0] = l1;
    eig[1] = l2;
    eig[2] = l3;
    return l3 >= 1e-3f * l1;
}

struct F4a {
    float x, y, z, w;
};

__device__ __forceinline__ F4a mat(const float* m, float x, float y, float z) {
    F4a r;
    r.x = m[0] * x + m[1] * y + m[2] * z + m[3];
    r.y = m[4] * x + m[5] * y + m[6] * z + m[7];
    r.z = m[8] * x + m[9] * y + m[10] * z + m[11];
    r.w = m[12] * x + m[13] * y + m[14] * z + m[15];
    return r;
}

// Per node: covariance, eigen-solve, metrics, screen coverage, score, queue key.
__global__ void __launch_bounds__(256) k_analyze(Dev d, RollSum* roll, NodeAnalysis* out,
                                                 float* features, AnalysisParams prm, Frame f,
                                                 AnalysisCounters* ac) {
    follow();
    const uint32_t nn = d.ctr->numNodes;
    const float cube = fmaxf(fmaxf(f.boxMax[0] - f.boxMin[0], f.boxMax[1] - f.boxMin[1]), f.boxMax[2] - f.boxMin[2]);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        // from the root's origin (k_roll) to the node's
        RollSum r = roll[i];
        rollRebase<false>(r, d.level[i], d.nodeX[i], d.nodeY[i], d.nodeZ[i]);
        roll[i] = r;
        NodeAnalysis o;
        o.count = r.n;
        o.lastTouched = r.lastTouched;
        o.flags = 0;
        for (int k = 0; k < 3; k++) {
            o.eig[k] = 0.0f;
            o.normal[k] = 0.0f;
        }
        o.surfaceVariation = 0.0f;
        o.planarity = 0.0f;
        const uint32_t lv = d.level[i];
        if (r.n >= 3) {
            const u128 n = r.n;
            const i128 s1[3] = {(i128)r.s1[0], (i128)r.s1[1], (i128)r.s1[2]};
            const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {0, 1, 2, 1, 2, 2};
            double cov[6];
            const double nd = (double)r.n;
            const double unit = ldexp(1.0, (int)(28u - lv));
            const double scale = 1.0 / (nd * nd * unit * unit);
            for (int k = 0; k < 6; k++) {
                const u128 s2 = ((u128)r.s2[2 * k + 1] << 64) | r.s2[2 * k];
                const i128 c = (i128)(n * s2) - s1[pa[k]] * s1[pb[k]];
                cov[k] = i128ToDouble(c) * scale;
            }
            float cf[6];
            for (int k = 0; k < 6; k++) cf[k] = (float)cov[k];
            float e[3];
            if (smith3(cf, e)) {
                for (int k = 0; k < 3; k++) o.eig[k] = e[k];
                // normal: the row cross product of (A - l3 I) with the largest norm
                const float m00 = cf[0] - e[2], m11 = cf[3] - e[2], m22 = cf[5] - e[2];
                const float r0[3] = {m00, cf[1], cf[2]}, r1[3] = {cf[1], m11, cf[4]}, r2[3] = {cf[2], cf[4], m22};
                float c0[3] = {r0[1] * r1[2] - r0[2] * r1[1], r0[2] * r1[0] - r0[0] * r1[2], r0[0] * r1[1] - r0[1] * r1[0]};
                float c1[3] = {r0[1] * r2[2] - r0[2] * r2[1], r0[2] * r2[0] - r0[0] * r2[2], r0[0] * r2[1] - r0[1] * r2[0]};
                float c2[3] = {r1[1] * r2[2] - r1[2] * r2[1], r1[2] * r2[0] - r1[0] * r2[2], r1[0] * r2[1] - r1[1] * r2[0]};
                const float n0 = c0[0] * c0[0] + c0[1] * c0[1] + c0[2] * c0[2];
                const float n1 = c1[0] * c1[0] + c1[1] * c1[1] + c1[2] * c1[2];
                const float n2 = c2[0] * c2[0] + c2[1] * c2[1] + c2[2] * c2[2];
                const float* best = n0 >= n1 && n0 >= n2 ? c0 : (n1 >= n2 ? c1 : c2);
                const float nb = fmaxf(fmaxf(n0, n1), n2);
                const float inv = nb > 0.0f ? rsqrtf(nb) : 0.0f;
                for (int k = 0; k < 3; k++) o.normal[k] = best[k] * inv;
            } else {
                double ed[3], vd[3];
                jacobi3(cov, ed, vd);
                for (int k = 0; k < 3; k++) {
                    o.eig[k] = (float)ed[k];
                    o.normal[k] = (float)vd[k];
                }
                o.flags |= kAnalysisFp64;
                atomicAdd(&ac->fp64Branch, 1u);
            }
            const float tr = o.eig[0] + o.eig[1] + o.eig[2];
            o.surfaceVariation = tr > 0.0f ? fmaxf(o.eig[2], 0.0f) / tr : 0.0f;
            o.planarity = o.eig[0] > 0.0f ? (o.eig[1] - o.eig[2]) / o.eig[0] : 0.0f;
        }
        // screen coverage of the node's box at this frame (projectedExtent, remolod_render.cu:40-70)
        float ext[2][4];
        bool anyv[2] = {false, false};
        for (int which = 0; which < 2; which++) {
            const uint32_t L = which == 0 ? lv : (lv > 0 ? lv - 1u : 0u);
            const uint32_t sh = which == 0 ? 0u : (lv > 0 ? 1u : 0u);
            const float s = cube / __int_as_float((int)((127u + L) << 23));
            const float mn[3] = {f.boxMin[0] + (float)(d.nodeX[i] >> sh) * s, f.boxMin[1] + (float)(d.nodeY[i] >> sh) * s,
                                 f.boxMin[2] + (float)(d.nodeZ[i] >> sh) * s};
            float minX = 1e30f, minY = 1e30f, maxX = -1e30f, maxY = -1e30f;
            for (int corner = 0; corner < 8; corner++) {
                const F4a c = mat(f.transformFrozen, (corner & 1) ? mn[0] + s : mn[0], (corner & 2) ? mn[1] + s : mn[1],
                                  (corner & 4) ? mn[2] + s : mn[2]);
                if (c.w <= 0.0f) continue;
                const float iw = 1.0f / c.w;
                const float sx = (c.x * iw * 0.5f + 0.5f) * f.width, sy = (c.y * iw * 0.5f + 0.5f) * f.height;
                minX = fminf(minX, sx);
                maxX = fmaxf(maxX, sx);
                minY = fminf(minY, sy);
                maxY = fmaxf(maxY, sy);
                anyv[which] = true;
            }
            ext[which][0] = minX;
            ext[which][1] = maxX;
            ext[which][2] = minY;
            ext[which][3] = maxY;
        }
        float cov2d = 0.0f;
        bool large = false, parentLarge = lv == 0;
        if (anyv[0]) {
            const float x0 = fmaxf(ext[0][0], 0.0f), x1 = fminf(ext[0][1], f.width);
            const float y0 = fmaxf(ext[0][2], 0.0f), y1 = fminf(ext[0][3], f.height);
            if (x1 > x0 && y1 > y0) cov2d = (x1 - x0) * (y1 - y0) / (f.width * f.height);
            large = (ext[0][1] - ext[0][0]) > prm.pixelBudget || (ext[0][3] - ext[0][2]) > prm.pixelBudget;
        }
        if (lv > 0 && anyv[1])
            parentLarge = (ext[1][1] - ext[1][0]) > prm.pixelBudget || (ext[1][3] - ext[1][2]) > prm.pixelBudget;
        const bool inner = !leafA(d, i);
        if (large) o.flags |= kAnalysisLarge;
        if (inner && !large && parentLarge) o.flags |= kAnalysisFrontier;
        o.coverage = cov2d;
        o.closed = (prm.currentBatch >= o.lastTouched + prm.closureMargin && r.n > 0) ? 1u : 0u;
        o.score = 0.0f;
        out[i] = o;
        // the learned scorer's inputs (the training-data logger records these)
        float* ft = features + (size_t)i * kNumFeatures;
        const double nd = r.n ? (double)r.n : 1.0;
        const double unit = ldexp(1.0, (int)(28u - lv));
        ft[0] = log2f(1.0f + (float)r.n) * (1.0f / 24.0f);
        ft[1] = (float)lv * (1.0f / 20.0f);
        for (int k = 0; k < 3; k++) ft[2 + k] = r.n ? (float)((double)r.s1[k] / (nd * unit)) : 0.0f;
        {
            // normalised centred second moments (a uniform cube has 1/12 on the diagonal)
            const int pa[6] = {0, 0, 0, 1, 1, 2}, pb[6] = {0, 1, 2, 1, 2, 2};
            for (int k = 0; k < 6; k++) {
                float v = 0.0f;
                if (r.n >= 2) {
                    const u128 s2 = ((u128)r.s2[2 * k + 1] << 64) | r.s2[2 * k];
                    const i128 c = (i128)((u128)r.n * s2) - (i128)r.s1[pa[k]] * (i128)r.s1[pb[k]];
                    v = (float)(i128ToDouble(c) / (nd * nd * unit * unit) * 12.0);
                }
                ft[5 + k] = v;
            }
        }
        ft[11] = o.surfaceVariation * 3.0f;
        ft[12] = o.planarity;
        const bool leafNode = !inner;
        const float fill = leafNode ? (float)d.numPoints[i] * (1.0f / 50000.0f) : (float)d.numVoxels[i] * (1.0f / 16384.0f);
        ft[13] = fminf(fill, 4.0f);
        float cvar = 0.0f;
        if (r.n >= 2) {
            for (int k = 0; k < 3; k++) {
                const double m = (double)r.c1[k] / nd;
                cvar += (float)(((double)r.c2[k] / nd - m * m) / (255.0 * 255.0));
            }
        }
        ft[14] = cvar * (4.0f / 3.0f);
        const float age = prm.currentBatch > o.lastTouched ? (float)(prm.currentBatch - o.lastTouched) : 0.0f;
        ft[15] = fminf(age / (float)(prm.closureMargin ? prm.closureMargin : 1u), 2.0f);
    }
}

// Score x coverage, the queue key, per node. In the learned mode an open
// node's surface variation is its partial one plus the network's predicted
// correction (output 0, x 1/300).
__global__ void __launch_bounds__(256) k_score(Dev d, NodeAnalysis* out, const float* pred, unsigned long long* keys,
                                               uint32_t* hist, AnalysisParams prm, AnalysisCounters* ac) {
    follow();
    const uint32_t nn = d.ctr->numNodes;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        NodeAnalysis o = out[i];
        float sv = o.surfaceVariation;
        if (prm.scoreMode == kScoreClosed && !o.closed) sv = 0.0f;
        // the network predicts the change from the partial surface variation to the final one
        if (prm.scoreMode == kScoreLearned && !o.closed && pred)
            sv = fminf(fmaxf(sv + pred[2 * i] * (1.0f / 300.0f), 0.0f), 1.0f / 3.0f);
        float score = sv * o.coverage;
        if (o.count < prm.minPoints) score = 0.0f;
        out[i].score = score;
        const bool eligible = score > 0.0f && (prm.frontierOnly == 0u || (o.flags & kAnalysisFrontier));
        keys[i] = eligible ? (((unsigned long long)__float_as_uint(score) << 32) | (0xFFFFFFFFu - i)) : 0ull;
        if (eligible) {
            atomicAdd(&ac->eligible, 1u);
            atomicAdd(&hist[__float_as_uint(score) >> 16], 1u);
        }
    }
}

// Radix select of the queue, over k_score's 65536-bin histogram of the keys'
// top 16 bits: the lowest bin b such that the bins >= b hold at least K keys.
// One block; warp w owns 2,048 consecutive bins counted from the top, read as
// 16 coalesced rows of 16 bytes a lane, all in flight. Only the warp in which
// the count reaches K looks closer. Bound by one SM reading 256 KB: 77 us with
// a load per bin and a scan by one thread, 21 us with 16 loads a thread at a
// stride of 256 B, 5 us so.
__global__ void __launch_bounds__(1024) k_queue_threshold(const uint32_t* hist, uint32_t K, AnalysisCounters* ac) {
    follow();
    __shared__ uint32_t s_warp[32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // row j, lane l: bins top - 128 j - 4 l - 3 .. top - 128 j - 4 l
    const uint32_t top = 65535u - warp * 2048u;
    uint4 v[16];
#pragma unroll
    for (uint32_t j = 0; j < 16u; j++)
        v[j] = __ldcg(reinterpret_cast<const uint4*>(hist + (top - 128u * j - 4u * lane - 3u)));
    uint32_t local = 0;
#pragma unroll
    for (uint32_t j = 0; j < 16u; j++) local += v[j].x + v[j].y + v[j].z + v[j].w;
    const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, local);
    if (lane == 0u) s_warp[warp] = sum;
    __syncthreads();
    uint32_t above = 0;
    for (uint32_t w = 0; w < warp; w++) above += s_warp[w];
    // fewer than K keys: the threshold stays 0, all of them
    if (above >= K || above + sum < K) return;
#pragma unroll
    for (uint32_t j = 0; j < 16u; j++) {
        const uint32_t row = v[j].x + v[j].y + v[j].z + v[j].w;
        uint32_t x = row;
#pragma unroll
        for (uint32_t o = 1; o < 32u; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= o) x += y;
        }
        uint32_t acc = above + x - row;
        if (acc < K && acc + row >= K) {
            uint32_t bin = top - 128u * j - 4u * lane;
            const uint32_t c[4] = {v[j].w, v[j].z, v[j].y, v[j].x};
            for (uint32_t k = 0; k < 3u && (acc += c[k]) < K; k++) bin--;
            ac->thresholdBin = bin;
        }
        above += __shfl_sync(0xFFFFFFFFu, x, 31);
    }
}

__global__ void __launch_bounds__(256) k_queue_collect(const Dev d, const unsigned long long* keys,
                                                       unsigned long long* cand, uint32_t cap, uint32_t* hist,
                                                       AnalysisCounters* ac) {
    follow();
    const uint32_t nn = d.ctr->numNodes;
    const uint32_t thr = ac->thresholdBin;
    // the histogram back to zero for the next call
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 65536u / 4u; i += gridDim.x * blockDim.x)
        reinterpret_cast<uint4*>(hist)[i] = make_uint4(0, 0, 0, 0);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x) {
        const unsigned long long k = keys[i];
        if (k && (uint32_t)(k >> 48) >= thr) {
            const uint32_t slot = atomicAdd(&ac->numCandidates, 1u);
            if (slot < cap) cand[slot] = k;
        }
    }
}

// One block: descending bitonic sort of the candidates in shared memory; the
// first K become the queue (node ids).
__global__ void __launch_bounds__(1024) k_queue_sort(const unsigned long long* cand, uint32_t cap, uint32_t K,
                                                     uint32_t* queue, AnalysisCounters* ac, AnalysisCounters* host) {
    follow();
    extern __shared__ unsigned long long s_k[];
    uint32_t n = ac->numCandidates;
    if (n > cap) {
        if (threadIdx.x == 0) ac->overflow = 1;
        n = cap;
    }
    uint32_t m = 1;
    while (m < n) m <<= 1;
    for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) s_k[i] = i < n ? cand[i] : 0ull;
    __syncthreads();
    for (uint32_t k = 2; k <= m; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
                const uint32_t l = i ^ j;
                if (l > i) {
                    const unsigned long long a = s_k[i], b = s_k[l];
                    const bool desc = (i & k) == 0;
                    if ((a < b) == desc) {
                        s_k[i] = b;
                        s_k[l] = a;
                    }
                }
            }
            __syncthreads();
        }
    }
    const uint32_t q = n < K ? n : K;
    for (uint32_t i = threadIdx.x; i < q; i += blockDim.x)
        queue[i] = 0xFFFFFFFFu - (uint32_t)(s_k[i] & 0xFFFFFFFFull);
    // the call's counters, complete now, into the host's pinned copy
    if (threadIdx.x == 0) {
        ac->queueLength = q;
        *host = *ac;
    }
}

// Refinement's budgeted pass: the first `budget` queue entries become forced
// splits of the LOD cut (rb_render's force-large mask). The queue is in
// descending key order and keys differ, so its prefix is the nodes whose key is
// at least the last taken entry's: one pass over the nodes writes the mask (a
// node made since Analysis has no key).
__global__ void __launch_bounds__(256) k_refine_mask(const Dev d, const uint32_t* queue, const unsigned long long* keys,
                                                     const AnalysisCounters* ac, uint32_t budget, uint8_t* mask) {
    const uint32_t nn = d.ctr->numNodes;
    const uint32_t q = ac->queueLength < budget ? ac->queueLength : budget;
    const unsigned long long last = q ? keys[queue[q - 1u]] : ~0ull;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nn; i += gridDim.x * blockDim.x)
        mask[i] = i < ac->numNodes && keys[i] >= last ? 1 : 0;
}

// The same after a queue whose candidates overflowed its sort (it then holds
// the highest of those that were kept): entry by entry, over a cleared mask.
__global__ void __launch_bounds__(256) k_refine_set(const uint32_t* queue, const AnalysisCounters* ac,
                                                    uint32_t budget, uint8_t* mask) {
    const uint32_t q = ac->queueLength < budget ? ac->queueLength : budget;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < q; i += gridDim.x * blockDim.x) mask[queue[i]] = 1;
}

void launchRoll(const Dev& d, RollSum* roll, uint32_t* rollArrive, AnalysisCounters* ac, int grid, cudaStream_t s) {
    k_roll<<<grid, kRollThreads, 0, s>>>(d, roll, rollArrive, ac);
}
void launchAnalyze(const Dev& d, RollSum* roll, NodeAnalysis* out, float* features,
                   const AnalysisParams& p, const Frame& f, AnalysisCounters* ac, int grid, cudaStream_t s) {
    launchBehind(k_analyze, grid, 256, 0, s, d, roll, out, features, p, f, ac);
}
void launchScore(const Dev& d, NodeAnalysis* out, const float* predictions, unsigned long long* keys, uint32_t* hist,
                 const AnalysisParams& p, AnalysisCounters* ac, int grid, cudaStream_t s) {
    launchBehind(k_score, grid, 256, 0, s, d, out, predictions, keys, hist, p, ac);
}
void launchQueue(const Dev& d, const unsigned long long* keys, uint32_t* hist, unsigned long long* cand,
                 uint32_t candCap, uint32_t K, uint32_t* queue, AnalysisCounters* ac, AnalysisCounters* host, int grid,
                 cudaStream_t s) {
    launchBehind(k_queue_threshold, 1, 1024, 0, s, hist, K, ac);
    launchBehind(k_queue_collect, grid, 256, 0, s, d, keys, cand, candCap, hist, ac);
    uint32_t m = 1;
    while (m < candCap) m <<= 1;
    launchBehind(k_queue_sort, 1, 1024, (size_t)m * 8, s, cand, candCap, K, queue, ac, host);
}
void launchRefineMask(const Dev& d, const uint32_t* queue, const unsigned long long* keys, const AnalysisCounters* ac,
                      uint32_t budget, bool overflowed, uint8_t* mask, int grid, cudaStream_t s) {
    k_refine_mask<<<grid, 256, 0, s>>>(d, queue, keys, ac, overflowed ? 0u : budget, mask);
    if (overflowed) k_refine_set<<<grid, 256, 0, s>>>(queue, ac, budget, mask);
}
cudaError_t configureQueueSort(uint32_t candCap) {
    uint32_t m = 1;
    while (m < candCap) m <<= 1;
    return cudaFuncSetAttribute(k_queue_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(m * 8));
}

}  // namespace rb
