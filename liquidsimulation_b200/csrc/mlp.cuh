// Per-particle MLP of the learned PCISPH warm start: 8 features -> 32 -> 32 -> 1, SiLU,
// BF16 operands on the tensor cores with FP32 accumulation. This header holds the training
// side (warp-level mma.sync m16n8k16, whose fragments the backward pass reuses); inference
// runs on tcgen05 (mlp_tc.cuh).
//
// A warp evaluates 32 particles as two 16-row tiles. The accumulator fragment of one
// layer (rows g, g+8; columns 2q, 2q+1 of each 8-column tile; g = lane/4, q = lane%4)
// is exactly the A-operand fragment of the next layer's 16-column k-tile, so hidden
// activations never leave registers. Weights live in shared memory already split into
// per-lane B fragments (MlpPacked), one 32-bit word per lane per register.
//
// Parameter vector (FP32 master copy, 1377 floats):
//   W1[8][32] @0, b1[32] @256, W2[32][32] @288, b2[32] @1312, W3[32] @1344, b3 @1376
#pragma once

#include <cstdint>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace lsp {

constexpr int kMlpIn = 8;
constexpr int kMlpHidden = 32;
constexpr int kMlpParams = 8 * 32 + 32 + 32 * 32 + 32 + 32 + 1;   // 1377
constexpr int kOffW1 = 0, kOffB1 = 256, kOffW2 = 288, kOffB2 = 1312, kOffW3 = 1344, kOffB3 = 1376;

// Fragment-ordered BF16 weights (bf16x2 words) and FP32 biases.
struct MlpPacked {
    uint32_t l1[4][32];          // layer 1 B fragment b0 per n-tile (b1 is the zero padding of K 8->16)
    uint32_t l2[4][2][2][32];    // layer 2 [n-tile][k-tile][reg]
    uint32_t l3[2][2][32];       // layer 3 [k-tile][reg], output column 0 only
    uint32_t l2t[4][2][2][32];   // W2 transposed, for the backward pass dh1 = dz2 W2^T
    float b1[32], b2[32], w3[32], b3, pad[3];   // w3: BF16-rounded W3 as float (backward)
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// D = A * B + D, A 16x16 bf16 (row), B 16x8 bf16 (col), D 16x8 fp32.
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The network's activations use the hardware approximations (__expf, __fdividef): the
// library is compiled for IEEE-exact division and square roots (the physics needs them),
// which the activations do not, and their error (a few ulp) is far below the BF16
// rounding of every activation. For z < -87, __expf(-z) overflows and the quotient is 0.
__device__ __forceinline__ float sigmoidf(float z) { return __fdividef(1.f, 1.f + __expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigmoidf(z); }
// silu'(z) from s = sigmoid(z).
__device__ __forceinline__ float silu_grad(float z, float s) { return s * (1.f + z * (1.f - s)); }

// Forward of one 16-particle tile. a1: layer-1 A fragment (features). Returns the output
// of rows g (in y[0]) and g+8 (in y[1]), valid in lanes with q == 0, and the activations' slopes
// s1 = silu'(z1), s2 = silu'(z2) (fragment layout) for the backward pass.
__device__ __forceinline__ void mlp_tile_forward(const MlpPacked& w, const uint32_t (&a1)[4], float (&s1)[4][4],
                                                 float (&s2)[4][4], uint32_t (&h1)[2][4], uint32_t (&h2)[2][4],
                                                 float (&y)[2])
{
    const int lane = threadIdx.x & 31, q = lane & 3;
    // z -> silu(z), with the slope from the same sigmoid.
    auto activate = [](float& z, float& slope) {
        const float s = sigmoidf(z);
        slope = silu_grad(z, s);
        z *= s;
    };
#pragma unroll
    for (int t = 0; t < 4; t++) {
        float c0 = w.b1[8 * t + 2 * q], c1 = w.b1[8 * t + 2 * q + 1];
        float z[4] = {c0, c1, c0, c1};
        mma16816(z, a1, w.l1[t][lane], 0u);
#pragma unroll
        for (int e = 0; e < 4; e++) activate(z[e], s1[t][e]);
        h1[t >> 1][(t & 1) * 2] = pack_bf16(z[0], z[1]);
        h1[t >> 1][(t & 1) * 2 + 1] = pack_bf16(z[2], z[3]);
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
        float c0 = w.b2[8 * t + 2 * q], c1 = w.b2[8 * t + 2 * q + 1];
        float z[4] = {c0, c1, c0, c1};
#pragma unroll
        for (int k = 0; k < 2; k++) mma16816(z, h1[k], w.l2[t][k][0][lane], w.l2[t][k][1][lane]);
#pragma unroll
        for (int e = 0; e < 4; e++) activate(z[e], s2[t][e]);
        h2[t >> 1][(t & 1) * 2] = pack_bf16(z[0], z[1]);
        h2[t >> 1][(t & 1) * 2 + 1] = pack_bf16(z[2], z[3]);
    }
    float o[4] = {w.b3, 0.f, w.b3, 0.f};
#pragma unroll
    for (int k = 0; k < 2; k++) mma16816(o, h2[k], w.l3[k][0][lane], w.l3[k][1][lane]);
    y[0] = o[0];
    y[1] = o[2];
}

// Sums in row order. A sum of 2,048 partial rows in order is a chain of additions (4.2 us); a plain
// loop, one thread per column, waited for a load every few rows and took most of a training
// iteration (118 us; 32 us now, 14 of them here). Here a block of 256 threads
// takes kSumCols columns, so that all SMs load: chunks of kSumRows rows go through shared memory,
// transposed, the next one in flight in registers while a lane per column adds the current one four
// rows per read. (32 columns per block on 44 SMs with cp.async of 4 bytes: 45 us.)
constexpr int kSumCols = 8, kSumRows = 256, kSumThreads = 256;
constexpr int kSumPitch = kSumRows + 4;
struct alignas(16) SumBuffer {
    float v[kSumCols][kSumPitch];
};
// sum + v[0..n-1] in order (v 16-byte aligned, shared memory).
__device__ __forceinline__ float add_in_order(float sum, const float* v, int n)
{
    int k = 0;
    for (; k + 32 <= n; k += 32) {
        float4 b[8];   // all reads in flight before the chain of additions
#pragma unroll
        for (int u = 0; u < 8; u++) b[u] = *reinterpret_cast<const float4*>(v + k + 4 * u);
#pragma unroll
        for (int u = 0; u < 8; u++) {
            sum += b[u].x;
            sum += b[u].y;
            sum += b[u].z;
            sum += b[u].w;
        }
    }
    for (; k < n; k++) sum += v[k];
    return sum;
}
// Column c0 + t of the row-major matrix m (rows x width), summed in row order, in thread t < kSumCols.
__device__ __forceinline__ float ordered_column_sum(const float* __restrict__ m, int rows, int width, int c0,
                                                    SumBuffer& buf)
{
    constexpr int kLoads = kSumRows * kSumCols / kSumThreads;
    const int c = threadIdx.x % kSumCols, r0 = threadIdx.x / kSumCols;
    const float* column = m + min(c0 + c, width - 1);
    float next[kLoads];
    auto fetch = [&](int base) {
#pragma unroll
        for (int k = 0; k < kLoads; k++)
            next[k] = __ldcg(column + (int64_t)min(base + r0 + k * (kSumThreads / kSumCols), rows - 1) * width);
    };
    float sum = 0.f;
    fetch(0);
    for (int base = 0; base < rows; base += kSumRows) {
        __syncthreads();   // the chunk before has been added
#pragma unroll
        for (int k = 0; k < kLoads; k++) buf.v[c][r0 + k * (kSumThreads / kSumCols)] = next[k];
        __syncthreads();
        if (base + kSumRows < rows) fetch(base + kSumRows);
        if (threadIdx.x < kSumCols) sum = add_in_order(sum, buf.v[threadIdx.x], min(rows - base, kSumRows));
    }
    return sum;
}
// v[0..n-1] summed in order, in thread 0.
__device__ __forceinline__ float ordered_sum(const float* __restrict__ v, int n, SumBuffer& buf)
{
    float* to = &buf.v[0][0];
    constexpr int kBuf = kSumCols * kSumPitch;
    float sum = 0.f;
    for (int base = 0; base < n; base += kBuf) {
        const int m = min(n - base, kBuf);
        for (int k = threadIdx.x; k < m; k += blockDim.x) to[k] = v[base + k];
        __syncthreads();
        if (threadIdx.x == 0) sum = add_in_order(sum, to, m);
        __syncthreads();
    }
    return sum;
}
// Blocks of a grid that sums `width` columns and, in its last block, one more vector.
constexpr int sum_blocks(int width) { return (width + kSumCols - 1) / kSumCols + 1; }

}  // namespace lsp
