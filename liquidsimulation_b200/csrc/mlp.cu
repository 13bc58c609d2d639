// Training and inference kernels of the warm-start MLP (see mlp.cuh for the layout).
//
//   k_mlp_pack   FP32 master parameters -> BF16 fragment-ordered weights + FP32 biases
//   k_mlp_grad   forward + backward on the tensor cores for a batch, MSE loss; the data
//                gradients use the register-resident fragments, the weight gradients
//                (reductions over particles) are MMAs whose operands are the transposed
//                activation tiles read back from shared memory. Each warp writes its own
//                partial gradient row, so the reduction order is fixed.
//   k_mlp_adam   sums the warp partials in order, applies Adam to the FP32 master and writes each
//                parameter's places in the packed weights.
#include "mlp.cuh"
#include "mlp_tc.cuh"
#include "lsp_kernels.h"

namespace lsp {

constexpr int kMlpThreads = 256;
constexpr int kMlpWarps = kMlpThreads / 32;

__device__ __forceinline__ float bf16_to_float(uint16_t b)
{
    return __uint_as_float(((uint32_t)b) << 16);
}
__global__ void k_mlp_pack(const float* __restrict__ m, MlpPacked* __restrict__ out)
{
    const float* W1 = m + kOffW1;
    const float* W2 = m + kOffW2;
    const float* W3 = m + kOffW3;
    for (int idx = threadIdx.x; idx < 32 * 4; idx += blockDim.x) {
        const int t = idx / 32, lane = idx % 32, g = lane >> 2, q = lane & 3;
        out->l1[t][lane] = pack_bf16(W1[(2 * q) * 32 + 8 * t + g], W1[(2 * q + 1) * 32 + 8 * t + g]);
    }
    for (int idx = threadIdx.x; idx < 4 * 2 * 2 * 32; idx += blockDim.x) {
        const int lane = idx % 32, r = (idx / 32) % 2, k = (idx / 64) % 2, t = idx / 128;
        const int g = lane >> 2, q = lane & 3;
        const int kk = 16 * k + 8 * r + 2 * q, n = 8 * t + g;
        out->l2[t][k][r][lane] = pack_bf16(W2[kk * 32 + n], W2[(kk + 1) * 32 + n]);
        // W2 transposed: B'[k = m][n = c] = W2[c][m].
        out->l2t[t][k][r][lane] = pack_bf16(W2[n * 32 + kk], W2[n * 32 + kk + 1]);
    }
    for (int idx = threadIdx.x; idx < 2 * 2 * 32; idx += blockDim.x) {
        const int lane = idx % 32, r = (idx / 32) % 2, k = idx / 64;
        const int g = lane >> 2, q = lane & 3;
        const int kk = 16 * k + 8 * r + 2 * q;
        out->l3[k][r][lane] = g == 0 ? pack_bf16(W3[kk], W3[kk + 1]) : 0u;
    }
    for (int c = threadIdx.x; c < 32; c += blockDim.x) {
        out->b1[c] = m[kOffB1 + c];
        out->b2[c] = m[kOffB2 + c];
        out->w3[c] = bf16_round(W3[c]);
    }
    if (threadIdx.x == 0) {
        out->b3 = m[kOffB3];
        out->pad[0] = out->pad[1] = out->pad[2] = 0.f;
    }
}

__device__ __forceinline__ void load_packed(MlpPacked& s, const MlpPacked* g)
{
    const uint32_t* src = reinterpret_cast<const uint32_t*>(g);
    uint32_t* dst = reinterpret_cast<uint32_t*>(&s);
    for (int i = threadIdx.x; i < (int)(sizeof(MlpPacked) / 4); i += blockDim.x) dst[i] = src[i];
}

// Row-major 16 x 32 bf16 tile in shared memory, rows padded to 20 words so that the eight 16-byte
// rows of an ldmatrix fall in different banks.
constexpr int kTilePitch = 20;
// Stores the D-layout fragments of a 16 x 32 activation tile as bf16 words, row-major.
__device__ __forceinline__ void store_tile(uint32_t* t, const uint32_t (&h)[2][4])
{
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int k = 0; k < 2; k++) {
        t[g * kTilePitch + 8 * k + q] = h[k][0];
        t[(g + 8) * kTilePitch + 8 * k + q] = h[k][1];
        t[g * kTilePitch + 8 * k + 4 + q] = h[k][2];
        t[(g + 8) * kTilePitch + 8 * k + 4 + q] = h[k][3];
    }
}
// Four transposed 8 x 8 blocks: lane 8 b + r gives the address of row r of block b; r[b] then holds
// elements [2 q][g] and [2 q + 1][g] of block b.
__device__ __forceinline__ void load_transposed(uint32_t (&r)[4], const uint32_t* row)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"((uint32_t)__cvta_generic_to_shared(row))
                 : "memory");
}
// Rows 8 (b >> 1) and columns 8 (b & 1) after `col` of a stored tile for block b (the A operand of a
// reduction over the tile's rows), and the same with the roles of the bits swapped (two column
// tiles' B operands).
__device__ __forceinline__ void load_tile_a(uint32_t (&r)[4], const uint32_t* t, int col)
{
    const int lane = threadIdx.x & 31, b = lane >> 3;
    load_transposed(r, t + ((lane & 7) + 8 * (b >> 1)) * kTilePitch + (col + 8 * (b & 1)) / 2);
}
__device__ __forceinline__ void load_tile_b(uint32_t (&r)[4], const uint32_t* t, int col)
{
    const int lane = threadIdx.x & 31, b = lane >> 3;
    load_transposed(r, t + ((lane & 7) + 8 * (b & 1)) * kTilePitch + (col + 8 * (b >> 1)) / 2);
}

// Batch row t drawn uniformly from [0, n) by a counter-based hash of (seed, t).
__device__ __forceinline__ int random_row(uint64_t seed, int t, int n)
{
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * (uint64_t)(t + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (int)(z % (uint64_t)n);
}

// Bound by its shared-memory reads (43 % of the L1 data pipe) and each warp's chain of MMAs and
// activations, one or two warps per scheduler: the transposed operands of the weight gradients come by
// ldmatrix (7 loads a tile where single elements took about 50, four-way conflicted), an activation
// and its slope share one sigmoid, and two blocks per SM at 128 registers take a batch of 65,536 in
// one wave (23 -> 18 us a batch; 19.5 with 176 registers, one block per SM and two waves).
// With draw > 0 the batch's rows are drawn from the first `draw` rows (random_row), else they are
// rows 0..nb-1.
template <bool kVector>   // the feature rows are 16-byte aligned
__global__ void __launch_bounds__(kMlpThreads, 2) k_mlp_grad(const MlpPacked* __restrict__ wg,
                                                         const float* __restrict__ feat,
                                                         const float* __restrict__ target,
                                                         int draw, uint64_t seed, int nb, float inv_batch,
                                                         float over_w, float* __restrict__ partial,
                                                         float* __restrict__ loss_partial)
{
    __shared__ MlpPacked w;
    __shared__ alignas(16) uint32_t stage[kMlpWarps][32 * 4];
    __shared__ alignas(16) uint32_t th1[kMlpWarps][16 * kTilePitch], tdz2[kMlpWarps][16 * kTilePitch],
        tdz1[kMlpWarps][16 * kTilePitch];
    load_packed(w, wg);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int gw = blockIdx.x * kMlpWarps + warp;
    const int nwarps = gridDim.x * kMlpWarps;

    float dW2[2][4][4] = {}, dW1[4][4] = {};
    float dW3[4][2] = {}, db2[4][2] = {}, db1[4][2] = {};
    float db3 = 0.f, loss = 0.f;

    for (int base = gw * 32; base < nb; base += nwarps * 32) {
        const int bi = base + lane;
        const bool valid = bi < nb;
        const int i = valid ? (draw > 0 ? random_row(seed, bi, draw) : bi) : 0;
        float f[kMlpIn];
        if (kVector) {
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            const float4* row = reinterpret_cast<const float4*>(feat) + 2 * (int64_t)i;
            const float4 u = valid ? row[0] : zero, v = valid ? row[1] : zero;
            f[0] = u.x, f[1] = u.y, f[2] = u.z, f[3] = u.w, f[4] = v.x, f[5] = v.y, f[6] = v.z, f[7] = v.w;
        } else {
#pragma unroll
            for (int c = 0; c < kMlpIn; c++) f[c] = valid ? feat[(int64_t)i * kMlpIn + c] : 0.f;
        }
        const float tgt = valid ? target[i] : 0.f;
        uint32_t* st = stage[warp];
        *reinterpret_cast<uint4*>(st + lane * 4) = make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]),
                                                              pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
        __syncwarp();
#pragma unroll
        for (int m = 0; m < 2; m++) {
            uint32_t a1[4] = {st[(16 * m + g) * 4 + q], st[(16 * m + g + 8) * 4 + q], 0u, 0u};
            float s1[4][4], s2[4][4], y[2];
            uint32_t h1[2][4], h2[2][4];
            mlp_tile_forward(w, a1, s1, s2, h1, h2, y);
            // Output gradient of rows g and g+8 (valid in lanes q == 0), then broadcast.
            const float t0 = __shfl_sync(0xffffffffu, tgt, 16 * m + g);
            const float t1 = __shfl_sync(0xffffffffu, tgt, 16 * m + g + 8);
            const bool v0 = base + 16 * m + g < nb, v1 = base + 16 * m + g + 8 < nb;
            // Loss 1/(2n) sum w(r) r^2 with r = y - t, w = over_w when the guess is too high.
            const float r0 = y[0] - t0, r1 = y[1] - t1;
            const float w0 = r0 > 0.f ? over_w : 1.f, w1 = r1 > 0.f ? over_w : 1.f;
            float dy0 = v0 ? w0 * r0 * inv_batch : 0.f;
            float dy1 = v1 ? w1 * r1 * inv_batch : 0.f;
            if (q == 0) {
                loss += (v0 ? 0.5f * w0 * r0 * r0 : 0.f) + (v1 ? 0.5f * w1 * r1 * r1 : 0.f);
                db3 += dy0 + dy1;
            }
            dy0 = __shfl_sync(0xffffffffu, dy0, 4 * g);
            dy1 = __shfl_sync(0xffffffffu, dy1, 4 * g);
            // Layer 3: dW3[c] += sum_rows h2[row][c] dy[row]; dz2 = dy W3 silu'(z2).
            float dz2[4][4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                const uint32_t r0 = h2[t >> 1][(t & 1) * 2], r1 = h2[t >> 1][(t & 1) * 2 + 1];
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int c = 8 * t + 2 * q + j;
                    const float hr0 = bf16_to_float(j ? (uint16_t)(r0 >> 16) : (uint16_t)(r0 & 0xffffu));
                    const float hr1 = bf16_to_float(j ? (uint16_t)(r1 >> 16) : (uint16_t)(r1 & 0xffffu));
                    dW3[t][j] += hr0 * dy0 + hr1 * dy1;
                    dz2[t][j] = dy0 * w.w3[c] * s2[t][j];
                    dz2[t][2 + j] = dy1 * w.w3[c] * s2[t][2 + j];
                    db2[t][j] += dz2[t][j] + dz2[t][2 + j];
                }
            }
            uint32_t dz2p[2][4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                dz2p[k][0] = pack_bf16(dz2[2 * k][0], dz2[2 * k][1]);
                dz2p[k][1] = pack_bf16(dz2[2 * k][2], dz2[2 * k][3]);
                dz2p[k][2] = pack_bf16(dz2[2 * k + 1][0], dz2[2 * k + 1][1]);
                dz2p[k][3] = pack_bf16(dz2[2 * k + 1][2], dz2[2 * k + 1][3]);
            }
            // Layer 2 data gradient: dh1 = dz2 W2^T, dz1 = dh1 silu'(z1).
            float dz1[4][4];
#pragma unroll
            for (int t = 0; t < 4; t++) {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = 0; k < 2; k++) mma16816(acc, dz2p[k], w.l2t[t][k][0][lane], w.l2t[t][k][1][lane]);
#pragma unroll
                for (int e = 0; e < 4; e++) dz1[t][e] = acc[e] * s1[t][e];
#pragma unroll
                for (int j = 0; j < 2; j++) db1[t][j] += dz1[t][j] + dz1[t][2 + j];
            }
            uint32_t dz1p[2][4];
#pragma unroll
            for (int k = 0; k < 2; k++) {
                dz1p[k][0] = pack_bf16(dz1[2 * k][0], dz1[2 * k][1]);
                dz1p[k][1] = pack_bf16(dz1[2 * k][2], dz1[2 * k][3]);
                dz1p[k][2] = pack_bf16(dz1[2 * k + 1][0], dz1[2 * k + 1][1]);
                dz1p[k][3] = pack_bf16(dz1[2 * k + 1][2], dz1[2 * k + 1][3]);
            }
            // Weight gradients: reductions over the 16 rows as MMAs with K = rows.
            store_tile(th1[warp], h1);
            store_tile(tdz2[warp], dz2p);
            store_tile(tdz1[warp], dz1p);
            __syncwarp();
            // dW2[k][c] = sum_r h1[r][k] dz2[r][c]: A[m = k][kk = r] = h1[r][k], B[kk = r][n = c] = dz2[r][c].
            {
                uint32_t a0[4], a1t[4], b0[4], b1[4];
                load_tile_a(a0, th1[warp], 0);
                load_tile_a(a1t, th1[warp], 16);
                load_tile_b(b0, tdz2[warp], 0);
                load_tile_b(b1, tdz2[warp], 16);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const uint32_t(&b)[4] = t < 2 ? b0 : b1;
                    mma16816(dW2[0][t], a0, b[2 * (t & 1)], b[2 * (t & 1) + 1]);
                    mma16816(dW2[1][t], a1t, b[2 * (t & 1)], b[2 * (t & 1) + 1]);
                }
            }
            // dW1[f][c] = sum_r x[r][f] dz1[r][c] (features padded to 16 rows of A).
            {
                uint32_t x[4], b0[4], b1[4];
                // Blocks 0 and 1: rows 0-7 and 8-15 of the tile's features (2 and 3 repeat them).
                load_transposed(x, st + (16 * m + (lane & 15)) * 4);
                const uint32_t a[4] = {x[0], 0u, x[1], 0u};
                load_tile_b(b0, tdz1[warp], 0);
                load_tile_b(b1, tdz1[warp], 16);
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const uint32_t(&b)[4] = t < 2 ? b0 : b1;
                    mma16816(dW1[t], a, b[2 * (t & 1)], b[2 * (t & 1) + 1]);
                }
            }
            __syncwarp();
        }
        __syncwarp();
    }
    // Reduce the per-lane column partials over the 8 row groups (lanes with equal q).
#pragma unroll
    for (int t = 0; t < 4; t++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int off = 4; off < 32; off <<= 1) {
                dW3[t][j] += __shfl_xor_sync(0xffffffffu, dW3[t][j], off);
                db2[t][j] += __shfl_xor_sync(0xffffffffu, db2[t][j], off);
                db1[t][j] += __shfl_xor_sync(0xffffffffu, db1[t][j], off);
            }
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) {
        db3 += __shfl_xor_sync(0xffffffffu, db3, off);
        loss += __shfl_xor_sync(0xffffffffu, loss, off);
    }
    float* row = partial + (int64_t)gw * kMlpParams;
#pragma unroll
    for (int mu = 0; mu < 2; mu++)
#pragma unroll
        for (int t = 0; t < 4; t++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int k = 16 * mu + g + (e >= 2 ? 8 : 0), c = 8 * t + 2 * q + (e & 1);
                row[kOffW2 + k * 32 + c] = dW2[mu][t][e];
            }
#pragma unroll
    for (int t = 0; t < 4; t++)
#pragma unroll
        for (int e = 0; e < 2; e++) row[kOffW1 + g * 32 + 8 * t + 2 * q + e] = dW1[t][e];
    if (g == 0) {
#pragma unroll
        for (int t = 0; t < 4; t++)
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int c = 8 * t + 2 * q + j;
                row[kOffW3 + c] = dW3[t][j];
                row[kOffB2 + c] = db2[t][j];
                row[kOffB1 + c] = db1[t][j];
            }
    }
    if (lane == 0) {
        row[kOffB3] = db3;
        loss_partial[gw] = loss;
    }
}

__device__ __forceinline__ uint16_t bf16_bits(float x)
{
    const __nv_bfloat16 v = __float2bfloat16_rn(x);
    return *reinterpret_cast<const uint16_t*>(&v);
}

// Writes parameter p's value to its places in both packed images (k_mlp_pack, k_mlp_pack_umma;
// what holds no parameter stays as those left it).
__device__ __forceinline__ void pack_parameter(int p, float v, MlpPacked* f, MlpUmma* u)
{
    const uint16_t h = bf16_bits(v);
    auto half = [&](uint32_t* words, int word, int odd) { reinterpret_cast<uint16_t*>(words)[2 * word + odd] = h; };
    if (p < kOffB1) {
        const int k = p / 32, n = p % 32;   // W1[k][n]
        half(&f->l1[0][0], (n / 8) * 32 + (n % 8) * 4 + k / 2, k & 1);
        u->w1t[umma_kmajor_offset(n, k, 256) / 2] = h;
    } else if (p < kOffW2) {
        f->b1[p - kOffB1] = u->b1[p - kOffB1] = v;
    } else if (p < kOffB2) {
        const int k = (p - kOffW2) / 32, n = (p - kOffW2) % 32;   // W2[k][n]
        // Fragment word of element (row of the contraction, column) in [n-tile][k-tile][reg][lane].
        auto word = [](int kk, int nn) {
            return (((nn / 8) * 2 + kk / 16) * 2 + (kk % 16) / 8) * 32 + (nn % 8) * 4 + (kk % 8) / 2;
        };
        half(&f->l2[0][0][0][0], word(k, n), k & 1);
        half(&f->l2t[0][0][0][0], word(n, k), n & 1);
        u->w2t[umma_kmajor_offset(n, k, 512) / 2] = h;
    } else if (p < kOffW3) {
        f->b2[p - kOffB2] = u->b2[p - kOffB2] = v;
    } else if (p < kOffB3) {
        const int c = p - kOffW3;
        half(&f->l3[0][0][0], ((c / 16) * 2 + (c % 16) / 8) * 32 + (c % 8) / 2, c & 1);
        f->w3[c] = u->w3[c] = bf16_round(v);
    } else {
        f->b3 = u->b3 = v;
    }
}

// Sums the warp partials in row order (kSumCols parameters per block; the last block sums the losses) and,
// with apply, takes one Adam step and repacks the parameter. Latency-bound: of 14 us for
// 2,048 rows (a batch of 65,536) the chain of additions takes 4.2; most of the rest goes into the block
// barriers between a chunk's arrival and its addition (12 of the stalled warps per issue wait there).
__global__ void __launch_bounds__(kSumThreads) k_mlp_adam(const float* __restrict__ partial,
                                                         const float* __restrict__ loss_partial, int rows,
                                                         float* __restrict__ master, float* __restrict__ m1,
                                                         float* __restrict__ m2, float* __restrict__ grad_out,
                                                         float* __restrict__ loss_out, MlpPacked* packed, MlpUmma* umma,
                                                         float lr, float beta1, float beta2, float eps, float bc1,
                                                         float bc2, int apply)
{
    __shared__ SumBuffer buf;
    if (blockIdx.x == gridDim.x - 1) {
        const float l = ordered_sum(loss_partial, rows, buf);
        if (threadIdx.x == 0 && loss_out) *loss_out = l;
        return;
    }
    const float gsum = ordered_column_sum(partial, rows, kMlpParams, blockIdx.x * kSumCols, buf);
    const int p = blockIdx.x * kSumCols + (int)threadIdx.x;
    if (threadIdx.x >= kSumCols || p >= kMlpParams) return;
    if (grad_out) grad_out[p] = gsum;
    if (!apply) return;
    float a = beta1 * m1[p] + (1.f - beta1) * gsum;
    float b = beta2 * m2[p] + (1.f - beta2) * gsum * gsum;
    m1[p] = a;
    m2[p] = b;
    const float w = master[p] - lr * (a / bc1) / (sqrtf(b / bc2) + eps);
    master[p] = w;
    pack_parameter(p, w, packed, umma);
}

void launch_mlp_pack(const float* master, MlpPacked* packed, cudaStream_t s)
{
    k_mlp_pack<<<1, 256, 0, s>>>(master, packed);
}


int mlp_grad_rows(int nb)
{
    int blocks = (nb + kMlpThreads - 1) / kMlpThreads;
    blocks = blocks < 1 ? 1 : (blocks > 296 ? 296 : blocks);
    return blocks * kMlpWarps;
}

static void launch_grad(const MlpPacked* packed, const float* feat, const float* target, int draw, uint64_t seed, int nb,
                        int blocks, float over_weight, float* partial, float* loss_partial, cudaStream_t s)
{
    const float inv = 1.f / (float)nb;
    // Callers' device buffers may start anywhere a float may.
    if ((uintptr_t)feat % sizeof(float4) == 0)
        k_mlp_grad<true><<<blocks, kMlpThreads, 0, s>>>(packed, feat, target, draw, seed, nb, inv, over_weight, partial,
                                                        loss_partial);
    else
        k_mlp_grad<false><<<blocks, kMlpThreads, 0, s>>>(packed, feat, target, draw, seed, nb, inv, over_weight, partial,
                                                         loss_partial);
}

void launch_mlp_grad(const MlpPacked* packed, const float* feat, const float* target, int draw, uint64_t seed, int nb,
                     float over_weight, float* partial, float* loss_partial, cudaStream_t s)
{
    launch_grad(packed, feat, target, draw, seed, nb, mlp_grad_rows(nb) / kMlpWarps, over_weight, partial, loss_partial,
                s);
}

void launch_mlp_grad_blocks(const MlpPacked* packed, const float* feat, const float* target, int nb, int blocks,
                            float* partial, float* loss_partial, cudaStream_t s)
{
    launch_grad(packed, feat, target, 0, 0, nb, blocks, 1.f, partial, loss_partial, s);
}

void launch_mlp_adam(const float* partial, const float* loss_partial, int rows, float* master, float* m1, float* m2,
                     float* grad_out, float* loss_out, MlpPacked* packed, MlpUmma* umma, float lr, int step, int apply,
                     cudaStream_t s)
{
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    float bc1 = 1.f - powf(beta1, (float)step), bc2 = 1.f - powf(beta2, (float)step);
    k_mlp_adam<<<sum_blocks(kMlpParams), kSumThreads, 0, s>>>(partial, loss_partial, rows, master, m1, m2, grad_out,
                                                                  loss_out, packed, umma, lr, beta1, beta2, eps, bc1,
                                                                  bc2, apply);
}

}  // namespace lsp
