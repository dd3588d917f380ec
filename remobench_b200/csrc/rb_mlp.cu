// The learned scorer: a 16 -> 64 -> 64 -> 2 MLP with GELU, BF16 weights and
// activations, FP32 accumulation; inference, the gradient of the training loss,
// and Adam. The reference has no learned component (plans/04_NeuralPass.md is
// empty); the network, its inputs and targets are this project's.
//
// Outputs: y0 = predicted (final - partial) surface variation x 300, y1 = closure logit.
// Loss per sample: (y0 - t0)^2 + BCE(sigmoid(y1), t1), averaged over the batch.
// GELU is the tanh form (Hendrycks & Gimpel, arXiv:1606.08415):
//   gelu(z) = 0.5 z (1 + tanh(c (z + 0.044715 z^3))), c = sqrt(2 / pi).
// Adam: Kingma & Ba, arXiv:1412.6980, with bias correction.
//
// Every contraction runs on the tensor cores as mma.sync.m16n8k16 (BF16 in,
// FP32 accumulate). A warp takes 16 samples: the layers are GEMMs of the
// warp's [16 x K] activations with the [K x N] weights, and a layer's FP32
// result tile, rounded to BF16, is already laid out as the next layer's A
// operand, so activations never leave registers. The backward pass computes
// dA1 = dZ2 W2 per warp the same way; the weight gradients dW2 = dZ2^T A1 and
// dW1 = dZ1^T X are contractions over samples, so each block stages its 64
// samples' dZ2, A1, dZ1 and X in shared memory, sample by sample as the
// fragments hold them, ldmatrix reads them transposed, and each warp
// accumulates one 16-row slice of dW2 and dW1 across the block's samples.
// Bias gradients, the 64 x 2 output layer and its gradient are FP32 sums and
// dot products with 2 outputs: kept per lane until the end, not GEMMs.
//
// Fragment layouts (PTX ISA, mma.m16n8k16 with .bf16): lane = 4 g + t;
// A (16 x 16, row-major): {a0, a1, a2, a3} = rows {g, g + 8, g, g + 8}, columns
// {2t, 2t + 1} (+ 8 for a2, a3); B (16 x 8): {b0, b1} = rows {2t, 2t + 1}
// (+ 8 for b1), column g; C (16 x 8): {c0, c1, c2, c3} = (row g, columns 2t,
// 2t + 1), (row g + 8, the same columns).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "rb_mlp.h"
#include "rb_launch.h"

namespace rb {

constexpr int kWarps = 4;                  // warps per block
constexpr int kTile = 16;                  // samples per warp and tile
constexpr int kBlockSamples = kWarps * kTile;
// shared-memory row strides in BF16 elements, padded so that the 8 rows a
// fragment load touches fall in different banks
constexpr int kW1Row = 24;                 // W1 [64][16]
constexpr int kW2Row = 72;                 // W2 and W2^T [64][64]
constexpr int kW3Row = 72;                 // W3 padded to [8][64]
constexpr int kSRow = 72;                  // per-sample columns of the staged transposes [.][64]

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
}

// The forward-only form, as inference has always computed it.
__device__ __forceinline__ float gelu(float z) {
    const float c = 0.7978845608028654f;
    const float u = c * (z + 0.044715f * z * z * z);
    return 0.5f * z * (1.0f + tanhf(u));
}

// With its derivative, through (1 + tanh(u)) / 2 = 1 / (1 + e^(-2u)): with
// p = e^(-2|u|), s = 1 / (1 + p) and r = 1 - s = p s,
//   gelu(z) = max(z, 0) - |z| r,  gelu'(z) = (z > 0 ? s : r) + 2 z s r u'.
// No difference of near-equal numbers, so its rms error against FP64 is at or
// below the tanhf form's (9.3e-9 against 1.8e-8 on [-3, 0), 4.5e-8 against
// 5.9e-8 on [0, 3); derivative 1.6e-8 against 3.7e-8, 5.7e-8 against 5.2e-8,
// and 4.5e-8 against 1.9e-7 on [3, 6)), at half the instructions: the two GELUs
// were most of the gradient kernel's. +infinity (a sum past FP32's range) is taken
// as the largest float, which the caller's rounding to BF16 makes +infinity again,
// as the tanhf form gives; |z| r would be infinity times zero. A NaN stays one.
__device__ __forceinline__ float geluGrad(float z, float& dgelu) {
    const float c = 0.7978845608028654f;
    asm("min.NaN.f32 %0, %0, 0f7F7FFFFF;" : "+f"(z));
    const float zz = z * z;
    const float u = c * (z + 0.044715f * zz * z);
    const float p = expf(-2.0f * fabsf(u));
    const float s = __fdividef(1.0f, 1.0f + p);
    const float r = p * s;
    const float du = c * (1.0f + 3.0f * 0.044715f * zz);
    dgelu = (z > 0.0f ? s : r) + 2.0f * z * (s * r) * du;
    return fmaf(-fabsf(z), r, fmaxf(z, 0.0f));
}

// D += A B on the tensor cores.
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t lds32(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }

struct __align__(16) SmemWeights {
    __nv_bfloat16 w1[kHidden * kW1Row];   // W1[n][k]
    __nv_bfloat16 w2[kHidden * kW2Row];   // W2[n][k]
    __nv_bfloat16 w3[8 * kW3Row];         // W3[n][k], rows 2..7 zero
    float b1[kHidden], b2[kHidden], b3[8];
    float w3f[kOut][kHidden];             // W3 as FP32 values of its BF16 copy (backward dot products)
};

// 16 bytes at a time: the BF16 copies start at multiples of eight elements, and
// every row here and there is one.
__device__ void loadWeights(SmemWeights& s, const __nv_bfloat16* wq, const float* params) {
    static_assert(kQW1 % 8 == 0 && kQW2 % 8 == 0 && kQW3 % 8 == 0 && kIn % 8 == 0 && kHidden % 8 == 0 &&
                      kW1Row % 8 == 0 && kW2Row % 8 == 0 && kW3Row % 8 == 0, "16-byte rows");
    const uint4* q = reinterpret_cast<const uint4*>(wq);
    for (int i = threadIdx.x; i < kHidden * kIn / 8; i += blockDim.x)
        *reinterpret_cast<uint4*>(&s.w1[(i / (kIn / 8)) * kW1Row + i % (kIn / 8) * 8]) = q[kQW1 / 8 + i];
    for (int i = threadIdx.x; i < kHidden * kHidden / 8; i += blockDim.x)
        *reinterpret_cast<uint4*>(&s.w2[(i / (kHidden / 8)) * kW2Row + i % (kHidden / 8) * 8]) = q[kQW2 / 8 + i];
    for (int i = threadIdx.x; i < 8 * kHidden / 8; i += blockDim.x) {
        const int n = i / (kHidden / 8), k = i % (kHidden / 8) * 8;
        const uint4 w = n < kOut ? q[kQW3 / 8 + i] : make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(&s.w3[n * kW3Row + k]) = w;
        if (n < kOut) {
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
            for (int e = 0; e < 4; e++) {
                s.w3f[n][k + 2 * e] = __low2float(h[e]);
                s.w3f[n][k + 2 * e + 1] = __high2float(h[e]);
            }
        }
    }
    for (int i = threadIdx.x; i < kHidden; i += blockDim.x) {
        s.b1[i] = params[kPB1 + i];
        s.b2[i] = params[kPB2 + i];
    }
    if (threadIdx.x < 8) s.b3[threadIdx.x] = threadIdx.x < kOut ? params[kPB3 + threadIdx.x] : 0.0f;
}

// One warp's forward pass over samples [base, base + 16) (rows past n are
// zeros). Leaves the layers' values in fragment layout.
struct Fwd {
    uint32_t xa[4];        // X rounded to BF16: A operand of layer 1
    uint32_t a1[4][4];     // A1 rounded to BF16: A operand of layer 2, per k-step
    uint32_t a2[4][4];     // A2 rounded to BF16: A operand of layer 3
    float dg1[8][4];       // gelu'(Z1) per C element of layer 1
    float dg2[8][4];       // gelu'(Z2)
    float y[4];            // layer 3's C tile: (row g, outputs 2t, 2t + 1), (row g + 8, ...)
};

template <bool kGrad>
__device__ __forceinline__ void forwardTile(const SmemWeights& s, const float* __restrict__ x, uint32_t n,
                                            uint32_t base, Fwd& f) {
    const uint32_t lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u;
    // layer 1: X [16 x 16] x W1^T
    {
        const uint32_t r0 = base + g, r1 = base + g + 8;
        float2 v00 = make_float2(0.f, 0.f), v01 = v00, v10 = v00, v11 = v00;
        if (r0 < n) {
            v00 = *reinterpret_cast<const float2*>(x + (size_t)r0 * kIn + 2 * t);
            v01 = *reinterpret_cast<const float2*>(x + (size_t)r0 * kIn + 2 * t + 8);
        }
        if (r1 < n) {
            v10 = *reinterpret_cast<const float2*>(x + (size_t)r1 * kIn + 2 * t);
            v11 = *reinterpret_cast<const float2*>(x + (size_t)r1 * kIn + 2 * t + 8);
        }
        f.xa[0] = pack2(v00.x, v00.y);
        f.xa[1] = pack2(v10.x, v10.y);
        f.xa[2] = pack2(v01.x, v01.y);
        f.xa[3] = pack2(v11.x, v11.y);
    }
    float c[8][4];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int col = 8 * i + 2 * t;
        c[i][0] = s.b1[col];
        c[i][1] = s.b1[col + 1];
        c[i][2] = s.b1[col];
        c[i][3] = s.b1[col + 1];
        const __nv_bfloat16* w = s.w1 + (8 * i + g) * kW1Row + 2 * t;
        mma(c[i], f.xa, lds32(w), lds32(w + 8));
    }
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) c[i][e] = kGrad ? geluGrad(c[i][e], f.dg1[i][e]) : gelu(c[i][e]);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        f.a1[j][0] = pack2(c[2 * j][0], c[2 * j][1]);
        f.a1[j][1] = pack2(c[2 * j][2], c[2 * j][3]);
        f.a1[j][2] = pack2(c[2 * j + 1][0], c[2 * j + 1][1]);
        f.a1[j][3] = pack2(c[2 * j + 1][2], c[2 * j + 1][3]);
    }
    // layer 2: A1 [16 x 64] x W2^T
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int col = 8 * i + 2 * t;
        c[i][0] = s.b2[col];
        c[i][1] = s.b2[col + 1];
        c[i][2] = s.b2[col];
        c[i][3] = s.b2[col + 1];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const __nv_bfloat16* w = s.w2 + (8 * i + g) * kW2Row + 16 * j + 2 * t;
            mma(c[i], f.a1[j], lds32(w), lds32(w + 8));
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) c[i][e] = kGrad ? geluGrad(c[i][e], f.dg2[i][e]) : gelu(c[i][e]);
#pragma unroll
    for (int j = 0; j < 4; j++) {
        f.a2[j][0] = pack2(c[2 * j][0], c[2 * j][1]);
        f.a2[j][1] = pack2(c[2 * j][2], c[2 * j][3]);
        f.a2[j][2] = pack2(c[2 * j + 1][0], c[2 * j + 1][1]);
        f.a2[j][3] = pack2(c[2 * j + 1][2], c[2 * j + 1][3]);
    }
    // layer 3: A2 [16 x 64] x W3^T, the two outputs padded to an 8-wide tile
    f.y[0] = s.b3[2 * t];
    f.y[1] = s.b3[2 * t + 1];
    f.y[2] = s.b3[2 * t];
    f.y[3] = s.b3[2 * t + 1];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const __nv_bfloat16* w = s.w3 + g * kW3Row + 16 * j + 2 * t;
        mma(f.y, f.a2[j], lds32(w), lds32(w + 8));
    }
}

__global__ void __launch_bounds__(kWarps * 32) k_mlp_predict(const __nv_bfloat16* wq, const float* params,
                                                             const float* __restrict__ x, uint32_t n,
                                                             const uint32_t* nDev, float* y) {
    __shared__ SmemWeights s;
    if (nDev) n = *nDev;
    loadWeights(s, wq, params);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3u;
    for (uint32_t base = (blockIdx.x * kWarps + warp) * kTile; base < n; base += gridDim.x * kBlockSamples) {
        Fwd f;
        forwardTile<false>(s, x, n, base, f);
        if (t == 0) {
            if (base + g < n) *reinterpret_cast<float2*>(y + 2 * (size_t)(base + g)) = make_float2(f.y[0], f.y[1]);
            if (base + g + 8 < n)
                *reinterpret_cast<float2*>(y + 2 * (size_t)(base + g + 8)) = make_float2(f.y[2], f.y[3]);
        }
    }
}

// The block's values for the weight-gradient GEMMs, per sample.
struct __align__(16) SmemStage {
    __nv_bfloat16 dz2[kBlockSamples * kSRow];  // dZ2 [sample][layer-2 neuron]
    __nv_bfloat16 a1[kBlockSamples * kSRow];   // A1  [sample][layer-1 neuron]
    __nv_bfloat16 dz1[kBlockSamples * kSRow];  // dZ1 [sample][layer-1 neuron]
    __nv_bfloat16 x[kBlockSamples * kW1Row];   // X   [sample][input]
};

// Fragments of stored matrices read transposed. A (16 x 16) from rows that are
// A's columns: matrices (rows 0-7, cols 0-7), (8-15, 0-7), (0-7, 8-15), (8-15,
// 8-15) of A, i.e. of the stored matrix its transposes. B (16 x 8) from rows
// that are B's rows.
__device__ __forceinline__ void ldmatrixA(uint32_t (&a)[4], const __nv_bfloat16* rows, int stride, int col) {
    const uint32_t lane = threadIdx.x & 31u, m = lane >> 3, r = lane & 7u;
    const uint32_t p = (uint32_t)__cvta_generic_to_shared(rows + (r + (m >> 1) * 8) * stride + col + (m & 1) * 8);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(p) : "memory");
}
// Two neighbouring B tiles (columns col .. col + 15) over 16 rows.
__device__ __forceinline__ void ldmatrixB2(uint32_t (&b)[4], const __nv_bfloat16* rows, int stride, int col) {
    const uint32_t lane = threadIdx.x & 31u, m = lane >> 3, r = lane & 7u;
    const uint32_t p = (uint32_t)__cvta_generic_to_shared(rows + (r + (m & 1) * 8) * stride + col + (m >> 1) * 8);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(b[0]), "=r"(b[1]), "=r"(b[2]), "=r"(b[3]) : "r"(p) : "memory");
}

__device__ __forceinline__ void sts32(__nv_bfloat16* p, uint32_t v) { *reinterpret_cast<uint32_t*>(p) = v; }

// Sum of v over the 8 row groups of a fragment (lanes with equal t).
__device__ __forceinline__ float sumRows(float v) {
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 4);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 8);
    v += __shfl_xor_sync(0xFFFFFFFFu, v, 16);
    return v;
}

// Gradient of the mean loss over n samples, added into grad (kNumParams floats
// and the loss sum after them, zero before the launch).
//
// Bound by instruction issue, half of it the 128 GELUs of a sample with their
// derivatives; the tensor cores idle (12.6 GFLOP at 400k samples, 8 us of their
// peak). At 400,003 samples: 463 us with tanhf, transposes staged two bytes at a
// time, the FP32 sums reduced by shuffles in every tile and one block per SM;
// 127 us so, at two (141 at three, which spill). At 2,048 samples 16.1 and 9.9 us.
__global__ void __launch_bounds__(kWarps * 32, 2) k_mlp_grad(const __nv_bfloat16* wq, const float* params,
                                                             const float* __restrict__ x,
                                                             const float* __restrict__ tgt, uint32_t n, float* grad) {
    follow();
    extern __shared__ __align__(16) unsigned char s_raw[];
    SmemWeights& s = *reinterpret_cast<SmemWeights*>(s_raw);
    SmemStage& st = *reinterpret_cast<SmemStage*>(s_raw + sizeof(SmemWeights));
    loadWeights(s, wq, params);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3u;
    const float invN = 1.0f / (float)n;
    // this warp's slices of the weight gradients: rows 16 warp .. +15 of dW2 (8 column tiles) and dW1 (2)
    float dw2[8][4], dw1[2][4];
    // this lane's FP32 sums over its rows g, g + 8 of every tile: per column pair
    // (8 i + 2 t, + 1) db2, db1 and dW3's two rows; db3 and the loss on lanes t == 0
    float db2[8][2], db1[8][2], dw3[2][8][2], db3[2] = {0.0f, 0.0f}, loss = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
#pragma unroll
        for (int e = 0; e < 4; e++) dw2[i][e] = 0.0f;
#pragma unroll
        for (int e = 0; e < 2; e++) db2[i][e] = db1[i][e] = dw3[0][i][e] = dw3[1][i][e] = 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) dw1[i][e] = 0.0f;
    for (uint32_t block0 = blockIdx.x * kBlockSamples; block0 < n; block0 += gridDim.x * kBlockSamples) {
        const uint32_t base = block0 + warp * kTile;
        const uint32_t row0 = warp * kTile + g;  // this lane's first staged sample; the other is row0 + 8
        Fwd f;
        forwardTile<true>(s, x, n, base, f);
        // A1 and X as they are
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) sts32(&st.a1[(row0 + 8 * (q & 1)) * kSRow + 16 * j + 2 * t + 8 * (q >> 1)], f.a1[j][q]);
#pragma unroll
        for (int q = 0; q < 4; q++) sts32(&st.x[(row0 + 8 * (q & 1)) * kW1Row + 2 * t + 8 * (q >> 1)], f.xa[q]);
        // the loss and dY per sample (lanes t == 0 hold the outputs of rows g and g + 8)
        float dy[2][2] = {{0.f, 0.f}, {0.f, 0.f}};
        if (t == 0) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint32_t r = base + g + 8 * h;
                if (r >= n) continue;
                const float y0 = f.y[2 * h], y1 = f.y[2 * h + 1];
                const float2 tv = *reinterpret_cast<const float2*>(tgt + 2 * (size_t)r);
                const float e = y0 - tv.x;
                const float sig = 1.0f / (1.0f + expf(-y1));
                // BCE with logits, stable form: max(y,0) - y t + log(1 + exp(-|y|))
                loss += e * e + fmaxf(y1, 0.0f) - y1 * tv.y + log1pf(expf(-fabsf(y1)));
                dy[h][0] = 2.0f * e * invN;
                dy[h][1] = (sig - tv.y) * invN;
            }
            db3[0] += dy[0][0] + dy[1][0];
            db3[1] += dy[0][1] + dy[1][1];
        }
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int o = 0; o < 2; o++) dy[h][o] = __shfl_sync(0xFFFFFFFFu, dy[h][o], lane & ~3u);
        // layer 3 backward: dW3 += dY^T A2, dA2 = dY W3, dZ2 = dA2 gelu'(Z2);
        // dZ2 rounded to BF16 is the A operand of dA1 = dZ2 W2, and staged
        uint32_t dza[4][4];
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const float2 w0 = *reinterpret_cast<const float2*>(&s.w3f[0][8 * i + 2 * t]);
            const float2 w1 = *reinterpret_cast<const float2*>(&s.w3f[1][8 * i + 2 * t]);
            float dz2[4];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                dz2[2 * h] = (dy[h][0] * w0.x + dy[h][1] * w1.x) * f.dg2[i][2 * h];
                dz2[2 * h + 1] = (dy[h][0] * w0.y + dy[h][1] * w1.y) * f.dg2[i][2 * h + 1];
                // A2's values of this row (BF16 as stored in the fragments)
                const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&f.a2[i >> 1][(i & 1) * 2 + h]);
                const float vx = __low2float(v), vy = __high2float(v);
#pragma unroll
                for (int o = 0; o < 2; o++) {
                    dw3[o][i][0] += dy[h][o] * vx;
                    dw3[o][i][1] += dy[h][o] * vy;
                }
                db2[i][0] += dz2[2 * h];
                db2[i][1] += dz2[2 * h + 1];
                const uint32_t packed = pack2(dz2[2 * h], dz2[2 * h + 1]);
                dza[i >> 1][(i & 1) * 2 + h] = packed;
                sts32(&st.dz2[(row0 + 8 * h) * kSRow + 8 * i + 2 * t], packed);
            }
        }
        // layer 2 backward: dA1 = dZ2 W2 (W2's rows are the contraction's), dZ1 = dA1 gelu'(Z1)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int j = 0; j < 4; j++) {
                uint32_t b[4];
                ldmatrixB2(b, s.w2 + 16 * j * kW2Row, kW2Row, 16 * i);
                mma(c[0], dza[j], b[0], b[1]);
                mma(c[1], dza[j], b[2], b[3]);
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int k = 2 * i + u;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const float d0 = c[u][2 * h] * f.dg1[k][2 * h], d1 = c[u][2 * h + 1] * f.dg1[k][2 * h + 1];
                    db1[k][0] += d0;
                    db1[k][1] += d1;
                    sts32(&st.dz1[(row0 + 8 * h) * kSRow + 8 * k + 2 * t], pack2(d0, d1));
                }
            }
        }
        __syncthreads();
        // the weight gradients over the block's 64 samples: this warp's 16 rows
        const int m0 = 16 * (int)warp;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            uint32_t a[4], b[4];
            ldmatrixA(a, st.dz2 + 16 * k * kSRow, kSRow, m0);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                ldmatrixB2(b, st.a1 + 16 * k * kSRow, kSRow, 16 * i);
                mma(dw2[2 * i], a, b[0], b[1]);
                mma(dw2[2 * i + 1], a, b[2], b[3]);
            }
            ldmatrixA(a, st.dz1 + 16 * k * kSRow, kSRow, m0);
            ldmatrixB2(b, st.x + 16 * k * kW1Row, kW1Row, 0);
            mma(dw1[0], a, b[0], b[1]);
            mma(dw1[1], a, b[2], b[3]);
        }
        __syncthreads();
    }
    // this warp's slices of dW2 and dW1 into the global gradient
    const int m0 = 16 * (int)warp;
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int row = m0 + g + 8 * (e >> 1), col = 8 * i + 2 * t + (e & 1);
            atomicAdd(&grad[kPW2 + row * kHidden + col], dw2[i][e]);
        }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int row = m0 + g + 8 * (e >> 1), col = 8 * i + 2 * t + (e & 1);
            atomicAdd(&grad[kPW1 + row * kIn + col], dw1[i][e]);
        }
    // the FP32 sums: over the lanes of equal t by shuffles, over the warps in
    // shared memory (the staging is done with), one atomic per block and entry
    float* red = reinterpret_cast<float*>(&st);  // [warp][dW3 | db2 | db1 | db3, loss]
    constexpr int kRed = kOut * kHidden + 2 * kHidden + kOut + 1;
    static_assert(sizeof(SmemStage) >= kWarps * kRed * sizeof(float), "reduction scratch");
    float* mine = red + warp * kRed;
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int e = 0; e < 2; e++) {
            const int col = 8 * i + 2 * t + e;
            const float w30 = sumRows(dw3[0][i][e]), w31 = sumRows(dw3[1][i][e]);
            const float s2 = sumRows(db2[i][e]), s1 = sumRows(db1[i][e]);
            if (g == 0) {
                mine[col] = w30;
                mine[kHidden + col] = w31;
                mine[kOut * kHidden + col] = s2;
                mine[(kOut + 1) * kHidden + col] = s1;
            }
        }
    const float s30 = sumRows(db3[0]), s31 = sumRows(db3[1]), sl = sumRows(loss);
    if (lane == 0) {
        mine[kRed - 3] = s30;
        mine[kRed - 2] = s31;
        mine[kRed - 1] = sl;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kRed; i += blockDim.x) {
        float v = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; w++) v += red[w * kRed + i];
        int to;
        if (i < kOut * kHidden) to = kPW3 + i;
        else if (i < (kOut + 1) * kHidden) to = kPB2 + i - kOut * kHidden;
        else if (i < (kOut + 2) * kHidden) to = kPB1 + i - (kOut + 1) * kHidden;
        else to = kPB3 + i - (kOut + 2) * kHidden;  // b3, then the loss at kNumParams
        atomicAdd(&grad[to], v);
    }
}

// One Adam step; leaves the gradient and the loss sum at zero for the next one
// and the sum in hostLoss (pinned).
__global__ void k_mlp_adam(float* params, float* grad, float* m, float* v, __nv_bfloat16* wq, AdamStep a,
                           float* hostLoss) {
    follow();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kNumParams; i += gridDim.x * blockDim.x) {
        const float g = grad[i];
        grad[i] = 0.0f;
        const float mi = a.beta1 * m[i] + (1.0f - a.beta1) * g;
        const float vi = a.beta2 * v[i] + (1.0f - a.beta2) * g * g;
        m[i] = mi;
        v[i] = vi;
        const float mh = mi / a.bc1, vh = vi / a.bc2;
        const float w = params[i] - a.lr * mh / (sqrtf(vh) + a.eps);
        params[i] = w;
        const int q = quantIndex(i);
        if (q >= 0) wq[q] = __float2bfloat16_rn(w);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *hostLoss = grad[kNumParams];
        grad[kNumParams] = 0.0f;
    }
}

__global__ void k_mlp_quantize(const float* params, __nv_bfloat16* wq) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kNumParams; i += gridDim.x * blockDim.x) {
        const int q = quantIndex(i);
        if (q >= 0) wq[q] = __float2bfloat16_rn(params[i]);
    }
}

void launchMlpPredict(const MlpState& st, const float* x, uint32_t n, float* y, int grid, cudaStream_t s) {
    if (n == 0) return;
    const uint32_t tiles = (n + kBlockSamples - 1) / kBlockSamples;
    k_mlp_predict<<<tiles < (uint32_t)grid ? (int)tiles : grid, kWarps * 32, 0, s>>>(st.wq, st.params, x, n, nullptr, y);
}

void launchMlpPredictCounted(const MlpState& st, const float* x, const uint32_t* nDev, float* y, int grid,
                             cudaStream_t s) {
    k_mlp_predict<<<grid, kWarps * 32, 0, s>>>(st.wq, st.params, x, 0u, nDev, y);
}

constexpr size_t kGradSmem = sizeof(SmemWeights) + sizeof(SmemStage);

cudaError_t configureMlp() {
    return cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGradSmem);
}

void launchMlpGrad(const MlpState& st, const float* x, const float* t, uint32_t n, int grid, cudaStream_t s) {
    if (n == 0) return;
    const uint32_t tiles = (n + kBlockSamples - 1) / kBlockSamples;
    k_mlp_grad<<<tiles < (uint32_t)grid ? (int)tiles : grid, kWarps * 32, kGradSmem, s>>>(st.wq, st.params, x, t, n,
                                                                                           st.grad);
}

void launchMlpAdam(const MlpState& st, const AdamStep& a, float* hostLoss, cudaStream_t s) {
    launchBehind(k_mlp_adam, (kNumParams + 255) / 256, 256, 0, s, st.params, st.grad, st.m, st.v, st.wq, a, hostLoss);
}

void launchMlpQuantize(const MlpState& st, cudaStream_t s) {
    k_mlp_quantize<<<(kNumParams + 255) / 256, 256, 0, s>>>(st.params, st.wq);
}

}  // namespace rb
