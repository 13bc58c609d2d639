// Uniform-grid build: cell keys, counting sort by (cell, caller id), particle reorder,
// dense cell table, and the start-of-step neighbour lists.
//
// Replaces the reference's per-step grid build, both its CPU hash grid
// (SPHSpatialGrid.cpp:19-90, via SPHSolver.cpp:431-440) and its OpenCL grid
// (calcGridIndices / countDigitsInBuckets / permuteParticles / buildCellList,
// SPHKernels.cl:66-186 with the host scan at SPHSolver.cpp:1052-1119).
//
// Cells are the CPU grid's cells, c = (int)(x / h) per axis, inside a fixed grid box;
// the key orders them x slowest, z fastest, which is the order in which the CPU's
// neighbour search visits cells. Sorting by (key, caller id) therefore lays out every
// 3-cell z-run of the 3x3 row neighbourhood as one contiguous range, in exactly the
// CPU's visiting order, so neighbour lists come out in the reference's order.
//
// The sort is a counting sort (a radix sort whose single digit is the whole cell key):
//   k_keys_hist   key per particle; warp-aggregated histogram (__match_any_sync) with slots
//   k_scan_*      exclusive scan of the histogram = dense cell table (lower bounds)
//   k_scatter     particle -> (cell start + slot)
//   k_rank_gather deterministic rank by caller id inside each cell, then one gather of
//                 the 64-byte persistent state into the new order
//   k_neighbors_density  the start-of-step neighbour lists, reference order, with the density
//                 and pressure summed over the accepted pairs
#include "chained.cuh"
#include "lsp_kernels.h"
#include "particle_ops.cuh"
#include "scan_ops.cuh"

namespace lsp {

constexpr int kScanThreads = 256;
constexpr int kScanTile = kScanThreads * kScanItems;

__global__ void k_keys_hist(DevParams P, const float4* __restrict__ pos, uint32_t* __restrict__ key,
                            uint32_t* __restrict__ slot, uint32_t* __restrict__ hist, DevStatus* st)
{
    const int i = chained((int)(blockIdx.x * blockDim.x + threadIdx.x));
    const bool valid = i < P.n;
    uint32_t k = 0xffffffffu;
    bool escaped = false, bad = false;
    if (valid) k = cell_key(P, pos[i], escaped, bad);
    const uint32_t sl = hist_slot(k, valid, hist);
    if (valid) {
        key[i] = k;
        slot[i] = sl;
    }
    record_key_flags(valid, escaped, bad, st);
}

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const uint32_t* __restrict__ in, int64_t n8,
                                                             uint32_t* __restrict__ tile_sums)
{
    __shared__ uint32_t ws[32];
    const int64_t base = (int64_t)chained(blockIdx.x * kScanThreads + threadIdx.x) * kScanItems;
    uint32_t s = 0;
    if (base < n8) {
        uint32_t v[kScanItems];
        load8(in + base, v);
#pragma unroll
        for (int j = 0; j < kScanItems; j++) s += v[j];
    }
    uint32_t total;
    block_exclusive_scan(s, ws, &total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// One block scans the tile sums in place (exclusive), chunk by chunk with a carry; only
// launched when there are more than kFoldTiles tiles.
__global__ void __launch_bounds__(1024) k_scan_top(uint32_t* tile_sums, int tiles)
{
    __shared__ uint32_t ws[32];
    uint32_t carry = 0;
    const int t = chained((int)threadIdx.x);
    for (int b = 0; b < tiles; b += blockDim.x) {
        int i = b + t;
        uint32_t v = i < tiles ? tile_sums[i] : 0u;
        uint32_t total;
        uint32_t ex = block_exclusive_scan(v, ws, &total);
        if (i < tiles) tile_sums[i] = carry + ex;
        carry += total;
        __syncthreads();
    }
}

// Exclusive scan of the histogram into the dense cell table; clears the histogram for the
// next step. With fold, the block sums the tile totals before its own tile (up to kFoldTiles
// of them) itself; otherwise k_scan_top has turned tile_sums into those prefixes.
constexpr int kFoldTiles = 4096;
__global__ void __launch_bounds__(kScanThreads) k_scan_apply(uint32_t* __restrict__ hist, int64_t n8,
                                                             const uint32_t* __restrict__ tile_sums, int fold,
                                                             uint32_t* __restrict__ out)
{
    __shared__ uint32_t ws[32];
    const int g = chained((int)(blockIdx.x * kScanThreads + threadIdx.x));
    const int tile = g / kScanThreads;
    uint32_t prefix;
    if (fold) {
        uint32_t s = 0;
        for (int k = g % kScanThreads; k < tile; k += kScanThreads) s += tile_sums[k];
        block_exclusive_scan(s, ws, &prefix);
    } else {
        prefix = tile_sums[tile];
    }
    const int64_t base = (int64_t)g * kScanItems;
    uint32_t v[kScanItems] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (base < n8) load8(hist + base, v);
    uint32_t s = 0;
#pragma unroll
    for (int j = 0; j < kScanItems; j++) s += v[j];
    uint32_t ex = block_exclusive_scan(s, ws, nullptr) + prefix;
    if (base < n8) store8_scan(out + base, hist + base, v, ex);
}

__global__ void k_scatter(DevParams P, const float4* __restrict__ pos, const uint32_t* __restrict__ key,
                          const uint32_t* __restrict__ slot, const uint32_t* __restrict__ cell_start,
                          int2* __restrict__ tmp)
{
    const int i = chained((int)(blockIdx.x * blockDim.x + threadIdx.x));
    if (i >= P.n) return;
    uint32_t k = key[i];
    tmp[cell_start[k] + slot[i]] = make_int2(i, id_of(pos[i]));
}

// rank_gather_one (particle_ops.cuh) for every sorted slot.
__global__ void k_rank_gather(GridBuildArgs g)
{
    const int p = chained((int)(blockIdx.x * blockDim.x + threadIdx.x));
    if (p < g.P.n) rank_gather_one(g, p);
}

// Start-of-step neighbour lists (neighbors_one) plus the start-of-step density
// and pressure (SPHSolver::calcParticleDensityPressure,
// SPHSolver.cpp:442-463), summed while the list is built: a pass over the stored list and
// its position gathers would cost more. (A list that
// overflows its capacity raises the overflow flag and the step is redone, so the sum over
// every accepted pair never differs from the stored list's.)
__global__ void k_neighbors_density(DevParams P, const float4* __restrict__ pos,
                                    const uint32_t* __restrict__ cell_start, int32_t* __restrict__ nbr,
                                    int32_t* __restrict__ count, DevStatus* st, const float* __restrict__ tables,
                                    float* __restrict__ rho, float* __restrict__ pres,
                                    const float4* __restrict__ vel, float4* __restrict__ vrho,
                                    float4* __restrict__ xpf)
{
    extern __shared__ uint2 masks[];
    const int i = chained((int)(blockIdx.x * blockDim.x + threadIdx.x));
    const bool valid = i < P.n;
    float* stage = reinterpret_cast<float*>(masks + blockDim.x * kScanChunks) + (threadIdx.x >> 5) * kStageFloats;
    float sum;
    const int c = neighbors_one<true>(P, pos, cell_start, nbr, min(i, P.n - 1), tables, masks + threadIdx.x, blockDim.x, &sum,
                                      stage, valid);
    if (valid) {
        store_density(P, i, c, sum, pos, vel, count, rho, pres, vrho, xpf, st);
    }
    record_neighbor_count(P, c, valid, st);
}

// ------------------------------------------------------------------ launchers

static inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

int launch_grid_keys(const GridBuildArgs& a, cudaStream_t s)
{
    if (a.P.n <= 0) return 0;
    launch_chained(k_keys_hist, blocks_for(a.P.n, 256), 256, 0, s, a.P, a.pos_in, a.key, a.slot, a.hist, a.status);
    return 1;
}

int launch_grid_scan(const GridBuildArgs& a, cudaStream_t s)
{
    const int64_t n8 = scan_entries((int64_t)a.P.cells + 1);
    const int tiles = (int)scan_tiles((int64_t)a.P.cells + 1);
    launch_chained(k_scan_tiles, tiles, kScanThreads, 0, s, a.hist, n8, a.tile_sums);
    const int fold = tiles <= kFoldTiles ? 1 : 0;
    if (!fold) launch_chained(k_scan_top, 1, 1024, 0, s, a.tile_sums, tiles);
    launch_chained(k_scan_apply, tiles, kScanThreads, 0, s, a.hist, n8, a.tile_sums, fold, a.cell_start);
    return fold ? 2 : 3;
}

int launch_grid_scatter(const GridBuildArgs& a, cudaStream_t s)
{
    if (a.P.n <= 0) return 0;
    launch_chained(k_scatter, blocks_for(a.P.n, 256), 256, 0, s, a.P, a.pos_in, a.key, a.slot, a.cell_start, a.tmp);
    return 1;
}

int launch_grid_gather(const GridBuildArgs& a, cudaStream_t s)
{
    if (a.P.n <= 0) return 0;
    launch_chained(k_rank_gather, blocks_for(a.P.n, 256), 256, 0, s, a);
    return 1;
}

int launch_grid_order(const GridBuildArgs& a, cudaStream_t s)
{
    const int T = 256;
    const DevParams& P = a.P;
    int launches = launch_grid_scan(a, s);
    if (P.n > 0) {
        launch_chained(k_scatter, blocks_for(P.n, T), T, 0, s, P, a.pos_in, a.key, a.slot, a.cell_start, a.tmp);
        launch_chained(k_rank_gather, blocks_for(P.n, T), T, 0, s, a);
        launches += 2;
    }
    return launches;
}

int launch_neighbors(const GridBuildArgs& a, cudaStream_t s)
{
    const int T = 128;
    if (a.P.n <= 0) return 0;
    launch_chained(k_neighbors_density, blocks_for(a.P.n, T), T, scan_smem(T), s, a.P, a.pos_out, a.cell_start, a.nbr,
                   a.nbr_count, a.status, a.tables, a.rho, a.pres, a.vel_out, a.vrho, a.xpf);
    return 1;
}

}  // namespace lsp
