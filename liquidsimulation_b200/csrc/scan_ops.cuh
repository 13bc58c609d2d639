// Block-wide exclusive scan, shared by the grid build (grid.cu) and the one-launch step
// (small_step.cu).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace lsp {

constexpr int kScanItems = 8;

// Exclusive scan of one value per thread over the block, warp shuffles inside each warp, then
// the warp totals.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* warp_sums, uint32_t* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        uint32_t w = lane < nw ? warp_sums[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) warp_sums[lane] = w;
    }
    __syncthreads();
    uint32_t warp_prefix = warp ? warp_sums[warp - 1] : 0u;
    if (total) *total = warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

// The histogram and the cell table are padded with zeros to a multiple of 8 entries
// (scan_entries): each thread moves its 8 consecutive entries as two 16-byte vectors. n8 is
// the padded count.
__device__ __forceinline__ void load8(const uint32_t* p, uint32_t (&v)[kScanItems])
{
    const uint4 a = *reinterpret_cast<const uint4*>(p);
    const uint4 b = *reinterpret_cast<const uint4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

__device__ __forceinline__ void clear8(uint32_t* p)
{
    *reinterpret_cast<uint4*>(p) = make_uint4(0u, 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(p + 4) = make_uint4(0u, 0u, 0u, 0u);
}

// Writes the exclusive scan of v, starting at ex, to out[0..7] and clears hist[0..7] (hist: may be
// null).
__device__ __forceinline__ void store8_scan(uint32_t* out, uint32_t* hist, const uint32_t (&v)[kScanItems], uint32_t ex)
{
    uint32_t o[kScanItems];
#pragma unroll
    for (int j = 0; j < kScanItems; j++) {
        o[j] = ex;
        ex += v[j];
    }
    *reinterpret_cast<uint4*>(out) = make_uint4(o[0], o[1], o[2], o[3]);
    *reinterpret_cast<uint4*>(out + 4) = make_uint4(o[4], o[5], o[6], o[7]);
    if (hist) clear8(hist);
}

}  // namespace lsp
