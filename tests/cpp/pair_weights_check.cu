// GPU check of the kernel weights by arithmetic (weight_w, weight_sdw, NonpressureWeights and
// their two-pair forms in liquidsimulation_b200/csrc/lsp_device.cuh) against the tables they
// restate, bit for bit. The tables and slot thresholds are built here as HostKernels::build
// builds them; the expected weight of a distance d is tab[(int)(d / step)] below h (IEEE
// division and square root on the host side of the tables, by the thresholds on the device:
// tests/cpp/lookup_exhaustive.cu proves those equal), else 0.
//   1. every float s (squared distance) in [0, 1.1 cut2], and infinities, NaN and far values:
//      poly6 W, gradient and Laplacian and the viscosity Laplacian;
//   2. every float d in [0, 1.05 h] and the same special values but NaN: the spiky gradient.
//   3. the two-pair distance and direction against IEEE square root and division on 77 million
//      random difference vectors.
// The second half of each two-pair call takes another float, so that both halves see every
// value. Prints the mismatch counts; exit status 0 when all are zero.
//   usage: pair_weights_check <particle radius> <kernel radius factor>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <vector>
#include <cuda_runtime.h>
#include "lsp_device.cuh"

using namespace lsp;

__device__ unsigned long long g_bad[5];
__device__ unsigned int g_first[5];

__device__ void differ(int what, float x, float got, float want)
{
    if (__float_as_uint(got) != __float_as_uint(want) && atomicAdd(&g_bad[what], 1ull) == 0)
        g_first[what] = __float_as_uint(x);
}
__device__ float expect_sq(const float* tab, const float* tables, float s, const DevParams& P)
{
    const float w = tab[table_slot_sq_from(s, __fsqrt_rn(s), P.inv_step, tables + kThresh2Offset)];
    return !(s >= P.cut2) ? w : 0.f;
}
__device__ void check_sq(const DevParams& P, const float* t, float s, float s2)
{
    const F2 both = f2(-s, -s2), w = weight_w(both, P, t);
    const NonpressureWeights n(s, P, t);
    const NonpressureWeights2 n2(both, P, t);
    const float *W = t, *DW = t + kTableSize, *D2W = t + 2 * kTableSize, *VD2W = t + 4 * kTableSize;
    differ(0, s, weight_w(s, P, t), expect_sq(W, t, s, P));
    differ(0, s, lo(w), expect_sq(W, t, s, P));
    differ(0, s2, hi(w), expect_sq(W, t, s2, P));
    differ(1, s, n.dw, expect_sq(DW, t, s, P));
    differ(1, s, n.d2w, expect_sq(D2W, t, s, P));
    differ(1, s, n.vd2w, expect_sq(VD2W, t, s, P));
    differ(2, s, lo(n2.dw), n.dw);
    differ(2, s, lo(n2.d2w), n.d2w);
    differ(2, s, lo(n2.vd2w), n.vd2w);
    differ(2, s2, hi(n2.dw), expect_sq(DW, t, s2, P));
    differ(2, s2, hi(n2.d2w), expect_sq(D2W, t, s2, P));
    differ(2, s2, hi(n2.vd2w), expect_sq(VD2W, t, s2, P));
}
__device__ float expect_d(const float* t, float d, const DevParams& P)
{
    return !(d >= P.h) ? t[3 * kTableSize + table_slot(d, P.inv_step, t + kThreshOffset)] : 0.f;
}
__device__ void check_d(const DevParams& P, const float* t, float d, float d2)
{
    const F2 w = weight_sdw(f2(-d, -d2), P, t);
    differ(3, d, weight_sdw(d, P, t), expect_d(t, d, P));
    differ(3, d, lo(w), expect_d(t, d, P));
    differ(3, d2, hi(w), expect_d(t, d2, P));
}
// The two-pair vector operations against the scalar ones on random neighbour-like differences.
__device__ uint64_t mix(uint64_t x)
{
    x += 0x9e3779b97f4a7c15ull;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ull;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}
__global__ void k_ops(float h)
{
    const uint64_t me = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    for (int r = 0; r < 256; r++) {
        float v[6];
        for (int c = 0; c < 6; c++) v[c] = ((float)(mix(me * 4096 + r * 6 + c) >> 40) * 0x1p-24f - 0.5f) * 2.f * h;
        const F2 x = f2(v[0], v[3]), y = f2(v[1], v[4]), z = f2(v[2], v[5]);
        const F2 nd = neg_sqrt_rn(neg_sqmag(x, y, z)), q = div_by(x, nd, recip_rn(nd));
        for (int k = 0; k < 2; k++) {
            const V3 a = v3(v[3 * k], v[3 * k + 1], v[3 * k + 2]);
            const float d = mag(a);
            differ(4, v[3 * k], k ? hi(nd) : lo(nd), -d);
            differ(4, v[3 * k], k ? hi(q) : lo(q), a.x / d);
        }
    }
}
__global__ void k_all(DevParams P, const float* t, uint32_t sq_end, uint32_t d_end)
{
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x, me = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    for (uint64_t b = me; b <= sq_end; b += step)
        check_sq(P, t, __uint_as_float((uint32_t)b), __uint_as_float(sq_end - (uint32_t)b));
    for (uint64_t b = me; b <= d_end; b += step)
        check_d(P, t, __uint_as_float((uint32_t)b), __uint_as_float(d_end - (uint32_t)b));
    // Exponents up to the largest, infinity and (squared distances only) NaN.
    for (uint32_t b = (uint32_t)me; b < 8192; b += (uint32_t)step) {
        const float x = __uint_as_float(sq_end + (uint32_t)(((uint64_t)(0x7f800000u - sq_end) * b) / 8191));
        check_sq(P, t, x, P.cut2);
        if (x >= P.h) check_d(P, t, x, P.h);
    }
    if (me == 0) check_sq(P, t, __uint_as_float(0x7fffffffu), 0.f);
}

int main(int argc, char** argv)
{
    const float radius = argc > 1 ? std::strtof(argv[1], nullptr) : 0.0125f;
    const float factor = argc > 2 ? std::strtof(argv[2], nullptr) : 3.2f;
    const int sub = kTableSize - 1;
    const float h = factor * radius;
    float r2 = h * h, r3 = r2 * h, r4 = r3 * h, r5 = r4 * h, r6 = r5 * h, r9 = r6 * r3;
    const float step = h / sub;
    const double pi = 3.14159265358979323846;
    DevParams P{};
    P.h = h;
    P.h2 = h * h;
    P.step = step;
    P.inv_step = 1.f / step;
    P.kw = (float)(315.0 / (64.0 * pi * (double)r9));
    P.kdw = (float)(-945.0 / (32.0 * pi * (double)r9));
    P.kd2w = P.kdw;
    P.ksdw = (float)(-45.0 / (pi * (double)r6));
    P.kvd2w = (float)(45.0 / (pi * (double)r6));
    std::vector<float> t(kTableFloats, 0.f);
    for (int i = 0; i <= sub; i++) {
        float d = i * step;
        float q = r2 - d * d;
        t[0 * kTableSize + i] = P.kw * q * q * q;
        t[1 * kTableSize + i] = P.kdw * q * q;
        t[2 * kTableSize + i] = P.kd2w * (r2 - d * d) * (3.f * r2 - 7.f * d * d);
        float s = h - d;
        t[3 * kTableSize + i] = P.ksdw * s * s;
        t[4 * kTableSize + i] = P.kvd2w * (h - d);
    }
    auto smallest = [](float top, auto pred) {   // smallest float in [0, top] with pred (monotone)
        uint32_t a = 0, b;
        std::memcpy(&b, &top, 4);
        while (a < b) {
            const uint32_t m = a + (b - a) / 2;
            float x;
            std::memcpy(&x, &m, 4);
            if (pred(x)) b = m; else a = m + 1;
        }
        float x;
        std::memcpy(&x, &a, 4);
        return x;
    };
    float *thr = t.data() + kThreshOffset, *thr2 = t.data() + kThresh2Offset;
    for (int k = 1; k <= sub; k++) {
        thr[k] = smallest(2.f * h, [&](float d) { return (int)(d / step) >= k; });
        thr2[k] = smallest(4.f * thr[k] * thr[k] + 1.f, [&](float s) { return std::sqrt(s) >= thr[k]; });
    }
    thr[kTableSize] = thr2[kTableSize] = std::numeric_limits<float>::infinity();
    P.cut2 = smallest(4.f * h * h + 1.f, [&](float s) { return std::sqrt(s) >= h; });

    float* dt = nullptr;
    cudaMalloc((void**)&dt, t.size() * sizeof(float));
    cudaMemcpy(dt, t.data(), t.size() * sizeof(float), cudaMemcpyHostToDevice);
    const float s_end = 1.1f * P.cut2, d_end = 1.05f * h;
    uint32_t sb, db;
    std::memcpy(&sb, &s_end, 4);
    std::memcpy(&db, &d_end, 4);
    k_all<<<148 * 8, 256>>>(P, dt, sb, db);
    k_ops<<<148 * 8, 256>>>(h);
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        std::printf("cuda error %s\n", cudaGetErrorString(e));
        return 2;
    }
    unsigned long long bad[5];
    unsigned int first[5];
    cudaMemcpyFromSymbol(bad, g_bad, sizeof(bad));
    cudaMemcpyFromSymbol(first, g_first, sizeof(first));
    const char* name[5] = {"poly6 W", "non-pressure weights", "non-pressure weights of two pairs", "spiky gradient",
                           "distance and direction of two pairs"};
    bool ok = true;
    for (int k = 0; k < 5; k++) {
        std::printf("%s: %llu mismatches\n", name[k], bad[k]);
        if (bad[k]) std::printf("  first at 0x%08x\n", first[k]);
        ok = ok && bad[k] == 0;
    }
    cudaFree(dt);
    return ok ? 0 : 1;
}
