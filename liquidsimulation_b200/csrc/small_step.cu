// The whole step of a small scene, or of a batch of small scenes, in one cooperative launch: grid build, neighbour lists,
// non-pressure forces, the pressure (SPH force or the PCISPH loop) and the integration, separated
// by grid barriers, with a group of L lanes per particle where a neighbour list is walked
// (group_ops.cuh). Each result carries the bits of the separate kernels (grid.cu, sph.cu,
// pcisph.cu), which larger scenes use.
//
// What bounds a small scene is latency: at 1,200 particles the separate kernels took 134 us of
// device time for a four-iteration step, in which the chip did about 2 us of work; a third of it
// went into launches and memsets, the rest into serial walks. Here a group keeps its particle's
// list and state in registers for the whole step, so a pass is one dependent fetch (the neighbours'
// positions) and a barrier. A PCISPH step with 4 iterations, wall clock, separate kernels -> this:
// 1,200 particles 89 -> 42 us, 4,700 145 -> 73, 9,400 156 -> 93, 18,900 177 -> 118, 30,000 203 ->
// 180, 37,800 219 -> 188 us. About 1.2 us of it is each grid barrier (6 + 2 per iteration, 7 in a
// large grid).
//
//   keys | (scan sums |) scan | scatter | rank + gather | lists + density |
//   non-pressure + predict(0), then the loop of k_pci_loop       (PCISPH)
//   all forces | integrate                                       (SPH)
//
// Everything one phase writes and a later one reads goes through plain or L2 loads; the grid
// barrier orders them.
#include "group_ops.cuh"
#include "host_util.h"
#include "loop_sync.cuh"
#include "scan_ops.cuh"
#include "small_step.h"

#include <algorithm>
#include <atomic>
#include <cstddef>
#include <mutex>

namespace lsp {

// 512 threads per SM leave each 128 registers: the groups keep their particle's list and state there.
constexpr int kMaxThreads = 512;
// Rounds of the block over the counts that cost less than the barrier they save. A step of 12,000
// particles in 4,000 cells takes 1.7 us less, 1,200 in 15,600 cells 1.5 us less (4 rounds: not taken).
constexpr int kFewRounds = 12;
// A batch's blocks: small, so that a scene's last one wastes little. 16 scenes, 20,071 particles, four
// steps with their transfers: 464 us with 128 threads, 475 with 256, 495 with 64.
constexpr int kBatchThreads = 128;
// Shared memory of a group in the build: one row of terms and the list.
template <int L>
constexpr int build_words()
{
    return group_pitch(L) + kGroupList;
}

// The blocks of one scene: this block's place among them, and what they share.
struct SceneBlocks {
    int block, blocks;
    LoopSync* sync;
    uint32_t* maxerr;
    uint32_t* tile_sums;
    DevStatus* host;
    uint32_t stalled;   // BarrierStall::barrier of this scene
};

// The step of one scene by its blocks. kBatch: the scene's particles start at slot P.base and its
// cells at P.cell_base, a multiple of 8.
template <int L, bool kBatch>
__device__ __forceinline__ void small_step(const DevParams& P, const GridBuildArgs& g, const StepBuffers& b, float4* ppos_alt,
                                           int pcisph, const SceneBlocks& own_blocks)
{
    extern __shared__ float4 dyn[];   // the groups' terms; in the build also their lists
    __shared__ uint32_t ws[32];
    __shared__ Collider cols[kMaxColliders];
    __shared__ uint32_t block_max;
    DevStatus* st = b.status;
    const int block = own_blocks.block, blocks = own_blocks.blocks;
    uint32_t* const maxerr = own_blocks.maxerr;
    const int tid = block * blockDim.x + threadIdx.x;
    const int n = P.n;
    const int base = kBatch ? P.base : 0;
    uint32_t epoch = 0;
    // A barrier that gave up tells the host in a word of its own, which the status copy at the end of
    // a block that got further leaves alone. The step's buffers are unfinished then, and the counts
    // may not be cleared: the host goes back to the buffers that the step read (abandon_step).
    auto barrier = [&]() {
        const bool ok = blocks_barrier(own_blocks.sync, st, epoch, (uint32_t)blocks, own_blocks.stalled);
        if (!ok && threadIdx.x == 0) own_blocks.host->gave_up = 1u;
        return ok;
    };
    // The status over PCIe, in as few stores as leave that word out.
    auto report = [&]() {
        static_assert(sizeof(DevStatus) == 64 && offsetof(DevStatus, gave_up) == 60, "gave_up is the last word");
        const uint32_t* from = reinterpret_cast<const uint32_t*>(st);
        uint4* to = reinterpret_cast<uint4*>(own_blocks.host);
#pragma unroll
        for (int q = 0; q < 3; q++) to[q] = make_uint4(from[4 * q], from[4 * q + 1], from[4 * q + 2], from[4 * q + 3]);
        *reinterpret_cast<uint2*>(to + 3) = make_uint2(from[12], from[13]);
        reinterpret_cast<uint32_t*>(to)[14] = from[14];
    };
    for (int w = threadIdx.x; w < P.ncoll * (int)(sizeof(Collider) / 4); w += blockDim.x)
        reinterpret_cast<uint32_t*>(cols)[w] = reinterpret_cast<const uint32_t*>(b.colliders + P.coll_off)[w];

    // ---- cell keys and histogram (k_keys_hist); thread t holds particle t until the gather
    const bool mine = tid < n;
    uint32_t key = 0xffffffffu;
    float4 x4 = make_float4(0.f, 0.f, 0.f, 0.f);
    bool escaped = false, bad = false;
    if (mine) {
        x4 = __ldg(g.pos_in + base + tid);
        key = cell_key(P, x4, escaped, bad);
    }
    const uint32_t slot = hist_slot(key, mine, g.hist);
    record_key_flags(mine, escaped, bad, st);
    if (!barrier()) return;

    // ---- scan: each block owns a contiguous run of the scene's cells
    uint32_t* const hist = kBatch ? g.hist + P.cell_base : g.hist;
    uint32_t* const cell_start = kBatch ? g.cell_start + P.cell_base : g.cell_start;
    const int64_t n8 = scan_entries((int64_t)P.cells + 1);
    const int64_t per = (n8 / kScanItems + blocks - 1) / blocks * kScanItems;
    const int64_t c0 = min((int64_t)block * per, n8), c1 = min(c0 + per, n8);
    const int64_t stride = (int64_t)blockDim.x * kScanItems, own = (int64_t)threadIdx.x * kScanItems;
    auto sum_of = [&](int64_t from, int64_t to) {
        uint32_t s = 0;
#pragma unroll 4
        for (int64_t e = from + own; e < to; e += stride) {
            uint32_t v[kScanItems];
            load8(hist + e, v);
#pragma unroll
            for (int j = 0; j < kScanItems; j++) s += v[j];
        }
        return s;
    };
    // Few cells: each block adds up the counts before its run itself, which saves a barrier; the counts
    // are then cleared once every block has read them.
    const bool few = n8 <= kFewRounds * stride;
    uint32_t carry;
    if (few) {
        block_exclusive_scan(sum_of(0, c0), ws, &carry);
    } else {
        uint32_t total;
        block_exclusive_scan(sum_of(c0, c1), ws, &total);
        if (threadIdx.x == 0) own_blocks.tile_sums[block] = total;
        if (!barrier()) return;
        uint32_t s = 0;
        for (int k = threadIdx.x; k < block; k += blockDim.x) s += __ldcg(own_blocks.tile_sums + k);
        block_exclusive_scan(s, ws, &carry);
    }
    carry += (uint32_t)base;
    for (int64_t e0 = c0; e0 < c1; e0 += stride) {
        const int64_t e = e0 + own;
        uint32_t v[kScanItems] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (e < c1) load8(hist + e, v);
        uint32_t sum = 0, total;
#pragma unroll
        for (int j = 0; j < kScanItems; j++) sum += v[j];
        const uint32_t ex = block_exclusive_scan(sum, ws, &total) + carry;
        if (e < c1) store8_scan(cell_start + e, few ? nullptr : hist + e, v, ex);
        carry += total;
    }
    if (!barrier()) return;
    if (few)
        for (int64_t e = c0 + own; e < c1; e += stride) clear8(hist + e);

    // ---- scatter (k_scatter), then rank by caller id inside the cell and move the state
    // (rank_gather_one, from the particle's side)
    uint32_t beg = 0, end = 0;
    if (mine) {
        beg = __ldcg(g.cell_start + key);
        end = __ldcg(g.cell_start + key + 1);
        g.tmp[beg + slot] = make_int2(base + tid, id_of(x4));
    }
    if (!barrier()) return;
    if (mine) {
        const int from = base + tid;
        const float4 v4 = __ldg(g.vel_in + from), h4 = __ldg(g.half_in + from), o4 = __ldg(g.old_in + from);
        const int id = id_of(x4);
        uint32_t rank = 0;
        if (end - beg <= (uint32_t)kMaxCellOccupancy) {
            for (uint32_t q = beg; q < end; q++) rank += __ldcg(g.tmp + q).y < id ? 1u : 0u;
        } else {
            rank = slot;   // order inside an overfull cell is not the reference's
            atomicOr(&st->error_flags, kErrScan);
        }
        const uint32_t dest = beg + rank;
        store_sorted(g, dest, id, key, x4, v4, h4, o4);
        if (g.hist_out) g.hist_out[dest] = __ldg(g.hist_in + from);
    }
    if (!barrier()) return;

    // ---- neighbour lists, density, pressure (k_neighbors_density); from here a group holds
    // sorted particle i
    const int i = base + min(tid / L, n - 1);
    const bool valid = tid / L < n;
    {
        Group<L> own(reinterpret_cast<float*>(dyn));
        own.row = reinterpret_cast<float*>(dyn) + (threadIdx.x / L) * build_words<L>();
        int* list = reinterpret_cast<int*>(own.row + group_pitch(L));
        float sum;
        const int c = group_neighbors(own, P, b.pos, b.tables, g.cell_start, g.nbr, i, valid, list, &sum);
        const bool first = valid && own.lane == 0;
        if (first) store_density(P, i, c, sum, b.pos, b.vel, g.nbr_count, g.rho, g.pres, g.vrho, g.xpf, st);
        record_neighbor_count(P, c, first, st);
    }
    if (threadIdx.x == 0) block_max = 0u;
    if (!barrier()) return;

    const Group<L> grp(reinterpret_cast<float*>(dyn));
    const HeldList<L> list(grp, P, b, i, valid);
    const float4 p4 = b.pos[i], v4 = b.vel[i], h4 = b.half[i], o4 = b.old[i];
    const float rho = b.rho[i];
    const V3 x0 = v3(p4), half0 = v3(h4);
    V3 v = v3(v4);
    const bool lead = valid && grp.lane == 0;   // the lane that stores the particle's results
    V3 F = pcisph ? group_nonpressure(grp, P, b, i, x0, v, rho, list) : group_sph_forces(grp, P, b, i, x0, v, rho, list);
    auto integrate = [&](V3 total, float p) {
        V3 x = x0, half = half0, old;
        float first = v4.w;
        integrate_motion(P, cols, total, rho, x, v, first, half, old);
        if (!lead) return;
        b.pos[i] = f4(x, p4.w);
        b.vel[i] = f4(v, first);
        b.half[i] = f4(half, h4.w);
        b.old[i] = f4(old, o4.w);
        if (b.hist) {
            // Warm-start pressure history: (p_n, p_{n-1}, p_{n-2}) for the next step's features.
            const float4 hs = b.hist[i];
            b.hist[i] = make_float4(p, hs.x, hs.y, 0.f);
        }
    };

    if (!pcisph) {
        const float pres = b.pres[i];
        if (!barrier()) return;   // the positions are read by other groups until here
        integrate(F, pres);
        if (tid == 0) report();
        return;
    }

    // ---- PCISPH: the loop of k_pci_loop from zero pressure. All lanes follow the particle's
    // predicted state.
    auto pp = [&](int parity) { return parity ? ppos_alt : b.ppos; };
    V3 px, ph;
    predict_motion(P, cols, st, F, v3(0.f, 0.f, 0.f), rho, x0, v, v4.w, half0, px, ph);
    if (lead) pp(0)[i] = f4(px, 0.f);
    if (!P.keep_initial_velocity) v = (v3(o4) + half0) / 2.f;
    float p = 0.f;
    if (!barrier()) return;
    for (int k = 0;; k++) {
        const float sum = group_density_sum(grp, P, b.tables, pp(k & 1), px, list.cnt, list.most, list);
        float pd, er;
        pressure_update(P, sum, pd, er, p);
        const float tf = p / (pd * pd);
        if (lead) reinterpret_cast<float*>(pp(k & 1) + i)[3] = tf;
        // Maximum of non-negative floats: their bit patterns order like the values.
        const uint32_t mb = __reduce_max_sync(kFullWarp, lead ? __float_as_uint(error_magnitude(er)) : 0u);
        if ((threadIdx.x & 31) == 0 && mb) atomicMax(&block_max, mb);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (block_max) atomicMax(&maxerr[k], block_max);
            block_max = 0u;
        }
        if (!barrier()) return;
        const uint32_t me = ld_volatile(&maxerr[k]);
        // PCISPHSolver.cpp:152-162: ratio = max|e| / rho0 in float, exit when below eta.
        const bool conv = fabsf(__uint_as_float(me) / P.rho0) < P.eta;
        const bool done = (conv && k + 1 >= P.min_it) || k + 1 >= P.max_it;
        const V3 Fp = group_pci_force(grp, P, b, i, pp(k & 1), px, tf, rho, list);
        if (done) {
            if (lead) {
                b.prho[i] = pd;
                b.err[i] = er;
                b.pres[i] = p;
                b.phalf[i] = f4(ph, 0.f);
                b.pforce[i] = f4(Fp, 0.f);
            }
            F += Fp;
            integrate(F, p);
            if (tid == 0) {
                st->iterations = k + 1;
                st->converged = conv ? 1 : 0;
                st->max_err_bits = me;
                st->warm_used = 0;
                st->last_k = k;
                report();
            }
            return;
        }
        predict_motion(P, cols, st, F, Fp, rho, x0, v, v4.w, half0, px, ph);
        if (lead) pp((k + 1) & 1)[i] = f4(px, 0.f);
        if (!barrier()) return;
    }
}

template <int L>
__global__ void __launch_bounds__(kMaxThreads, 1) k_small_step(SmallStepArgs a)
{
    small_step<L, false>(a.g.P, a.g, a.b, a.ppos_alt, a.pcisph,
                         {(int)blockIdx.x, (int)gridDim.x, reinterpret_cast<LoopSync*>(a.sync), a.maxerr, a.g.tile_sums, a.host,
                          a.stall.barrier});
}

// The same for a batch of scenes in one launch. A scene has blocks and a barrier of its own, so it
// takes its iterations without waiting for the others. Four steps of 16 scenes (20,071 particles)
// with their transfers: 650 us as separate kernels over all scenes, whose loop runs in lockstep
// rounds with one thread per particle; 464 us here.
template <int L>
__global__ void __launch_bounds__(kBatchThreads, kMaxThreads / kBatchThreads) k_small_batch(SmallStepArgs a, SmallBatchArgs sb)
{
    __shared__ DevParams P;
    const SmallBatchBlock me = sb.blocks[blockIdx.x];
    const uint32_t* from = reinterpret_cast<const uint32_t*>(sb.sp + me.scene);
    for (int w = threadIdx.x; w < (int)(sizeof(DevParams) / 4); w += blockDim.x) reinterpret_cast<uint32_t*>(&P)[w] = from[w];
    __syncthreads();
    GridBuildArgs g = a.g;
    StepBuffers b = a.b;
    b.status += me.scene;
    g.status = b.status;
    b.tables += (size_t)me.scene * sb.table_stride;
    small_step<L, true>(P, g, b, a.ppos_alt, a.pcisph,
                        {(int)blockIdx.x - me.first, me.count, reinterpret_cast<LoopSync*>(a.sync) + me.scene,
                         a.maxerr + (size_t)me.scene * sb.mstride, g.tile_sums + me.first, a.host + me.scene,
                         me.scene == a.stall.scene ? a.stall.barrier : 0u});
}

// ------------------------------------------------------------------ launch

constexpr int kMaxDevices = 64;
constexpr int kLaneChoices = 4;   // 16, 8, 4 and 2 lanes
static const void* const g_kernel[kLaneChoices] = {(const void*)k_small_step<16>, (const void*)k_small_step<8>,
                                                   (const void*)k_small_step<4>, (const void*)k_small_step<2>};
template <int L>
static size_t lanes_smem(int threads)
{
    const size_t walk = group_smem(threads, L), build = (size_t)(threads / L) * build_words<L>() * sizeof(float);
    return walk > build ? walk : build;
}
static size_t step_smem(int choice, int threads)
{
    return choice == 0   ? lanes_smem<16>(threads)
           : choice == 1 ? lanes_smem<8>(threads)
           : choice == 2 ? lanes_smem<4>(threads)
                         : lanes_smem<2>(threads);
}
// Whether a block of each choice fits an SM (asked once per device, under a lock: solvers on
// different host threads may launch at once).
static bool g_fits[kMaxDevices][kLaneChoices], g_ready[kMaxDevices];
static std::mutex g_mutex;

// A scene's blocks scan its cells; a block's share of a single scene's largest box.
constexpr int64_t kBatchBlockCells = kSmallStepCells / 128;

// As many lanes per particle as the threads allow: fewer lanes take longer walks (12,000 particles:
// 93 us a step with 4 lanes). Beyond two lanes per particle the separate kernels, with one thread
// per particle and full occupancy, are as fast (45,000 particles: 252 us either way).
int small_step_lanes(int64_t n, int64_t cells)
{
    if (n <= 0 || cells > kSmallStepCells) return 0;
    const int64_t threads = (int64_t)device_sm_count() * kMaxThreads;
    for (int lanes = 16; lanes >= 2; lanes /= 2)
        if (n * lanes <= threads) return lanes;
    return 0;
}

// One group per particle in one block per SM, as evenly as whole warps allow.
static void small_shape(int64_t n, int lanes, int* block, int* grid)
{
    const int sms = device_sm_count();
    const int64_t threads = n * lanes;
    const int64_t per_sm = (threads + sms - 1) / sms;
    *block = (int)((per_sm + 63) / 64 * 64 < 128 ? 128 : (per_sm + 63) / 64 * 64);
    *grid = (int)((threads + *block - 1) / *block);
}

static int64_t chip_threads() { return (int64_t)device_sm_count() * kMaxThreads; }

int64_t step_threads(int64_t n, int lanes)
{
    if (!lanes) return std::min(n, chip_threads()) / 2;
    int block, grid;
    small_shape(n, lanes, &block, &grid);
    return (int64_t)block * grid;
}

int64_t batch_step_threads(int64_t n, int small_blocks)
{
    return small_blocks ? (int64_t)small_blocks * kBatchThreads : std::min(n, chip_threads()) / 2;
}

// Threads of the steps in flight per device. Separate kernels count half of theirs: they leave places
// free at their ends and between them. us a step of a small and of a large solver stepped at once,
// the small one in one launch / in separate kernels: PCISPH of 1,200 particles beside SPH of 250,047
// 73 and 178 / 135 and 153; 12,167 beside the same 97 and 208 / 151 and 165; 29,791 122 and 358 / 167
// and 172, beside PCISPH of 417,792 161 and 812 / 420 and 499.
static std::atomic<int64_t> g_in_flight[kMaxDevices];

// An eighth more than fits still counts as fitting: the last blocks then wait for the end of another
// step, which costs less than the separate kernels do. us a step, T threads stepping a PCISPH (SPH)
// solver each, one launch / separate kernels: 1,200 particles T = 4, 1.01 of the chip, 22.7 / 28.5 (16.3 /
// 18.1); 4,913, T = 2, 1.04 of the chip, 46.3 / 54.7 (30.5 / 31.0); 12,167, T = 2, 1.29, 58.4 / 57.2 (36.0 /
// 31.6); 29,791, T = 2, 1.6, 81.8 / 64.9 (46.3 / 34.6); 12,167, T = 8, 57.1 / 19.9 (36.2 / 12.6). A step of a
// quarter of the chip, one block of 128 threads per SM, runs beside three like it and takes one launch
// whatever is in flight: 512 particles T = 16 5.8 / 10.9 (4.3 / 10.2), 1,100 particles T = 24 11.9 / 11.8
// (8.4 / 9.8); with 150 blocks, 1,200 particles, T = 16, it is 22.4 / 11.2 (15.6 / 9.7).
StepInFlight::StepInFlight(int device, int64_t threads) : dev_(device), threads_(threads)
{
    if (dev_ < 0 || dev_ >= kMaxDevices) return;
    const int64_t others = g_in_flight[dev_].fetch_add(threads_, std::memory_order_relaxed);
    if (others == 0) return;
    fits_ = threads_ * 4 <= chip_threads() || others + threads_ <= chip_threads() * 9 / 8;
}

StepInFlight::~StepInFlight()
{
    if (dev_ >= 0 && dev_ < kMaxDevices) g_in_flight[dev_].fetch_sub(threads_, std::memory_order_relaxed);
}

bool launch_small_step(const SmallStepArgs& a, int lanes, cudaStream_t s)
{
    const int c = lanes == 16 ? 0 : lanes == 8 ? 1 : lanes == 4 ? 2 : 3;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return false;
    bool fits;
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        if (!g_ready[dev]) {
            int coop = 0;
            cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
            for (int k = 0; k < kLaneChoices; k++) {
                int per = 0;
                const size_t smem = step_smem(k, kMaxThreads);
                g_fits[dev][k] =
                    coop &&
                    cudaFuncSetAttribute(g_kernel[k], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) ==
                        cudaSuccess &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, g_kernel[k], kMaxThreads, smem) == cudaSuccess &&
                    per > 0;
            }
            g_ready[dev] = true;
        }
        fits = g_fits[dev][c];
    }
    if (!fits) return false;
    int block, grid;
    small_shape(a.g.P.n, lanes, &block, &grid);
    if (block > kMaxThreads) return false;
    SmallStepArgs ac = a;
    void* args[] = {&ac};
    return cudaLaunchCooperativeKernel(g_kernel[c], dim3(grid), dim3(block), args, step_smem(c, block), s) ==
           cudaSuccess;
}

static const void* const g_batch_kernel[kLaneChoices] = {(const void*)k_small_batch<16>, (const void*)k_small_batch<8>,
                                                         (const void*)k_small_batch<4>, (const void*)k_small_batch<2>};

// Resident blocks of a choice's batch kernel on the current device, 0 when it cannot run.
static int64_t batch_block_limit(int c)
{
    int dev = 0, coop = 0, per = 0;
    const size_t smem = step_smem(c, kBatchThreads);
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
        !coop ||
        cudaFuncSetAttribute(g_batch_kernel[c], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, g_batch_kernel[c], kBatchThreads, smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return (int64_t)per * device_sm_count();
}

// The rule of small_step_lanes for all scenes together, in whole blocks. A PCISPH step, separate
// kernels -> one launch: 4 scenes of 250 particles 99 -> 52 us, 48 of 71 104 -> 58, 16 of 500
// 113 -> 103, 16 of 1,040 115 -> 79, 16 of 2,070 116 -> 96, 2 of 17,400 122 -> 106 us.
int small_batch_plan(const std::vector<int64_t>& n, const std::vector<int64_t>& cells, std::vector<SmallBatchBlock>* blocks)
{
    blocks->clear();
    for (int c = 0; c < kLaneChoices; c++) {
        const int64_t lanes = 16 >> c;
        int64_t total = 0;
        bool fits = true;
        for (size_t s = 0; s < n.size() && fits; s++) {
            const int64_t count = (n[s] * lanes + kBatchThreads - 1) / kBatchThreads;
            total += count;
            fits = n[s] > 0 && cells[s] <= count * kBatchBlockCells;
        }
        if (!fits || total > (int64_t)device_sm_count() * (kMaxThreads / kBatchThreads) || total > batch_block_limit(c)) continue;
        for (size_t s = 0; s < n.size(); s++) {
            const int count = (int)((n[s] * lanes + kBatchThreads - 1) / kBatchThreads), first = (int)blocks->size();
            for (int q = 0; q < count; q++) blocks->push_back({(int)s, first, count, 0});
        }
        return (int)lanes;
    }
    return 0;
}

bool launch_small_batch(const SmallStepArgs& a, const SmallBatchArgs& sb, int lanes, int blocks, cudaStream_t s)
{
    const int c = lanes == 16 ? 0 : lanes == 8 ? 1 : lanes == 4 ? 2 : 3;
    SmallStepArgs ac = a;
    SmallBatchArgs bc = sb;
    void* args[] = {&ac, &bc};
    return cudaLaunchCooperativeKernel(g_batch_kernel[c], dim3(blocks), dim3(kBatchThreads), args,
                                       step_smem(c, kBatchThreads), s) == cudaSuccess;
}

}  // namespace lsp
