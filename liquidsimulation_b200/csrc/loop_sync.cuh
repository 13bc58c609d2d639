// Grid-wide barrier of the cooperative persistent kernels (the PCISPH loop of one scene
// and of a batch of scenes). Every block of the grid is resident (cooperative launch).
// The spin is bounded: past the limit it raises kErrTimeout and an abort word that makes
// every block leave, and the host reports LSP_ERR_TIMEOUT.
#pragma once

#include "lsp_device.cuh"

namespace lsp {

constexpr unsigned long long kBarrierSpinLimit = 1ull << 25;
constexpr unsigned long long kStallSpinLimit = 1ull << 14;   // some 10 ms

struct LoopSync {
    uint32_t count;   // barrier arrivals since the launch
    uint32_t abort;
    uint32_t pad[2];
};

static __device__ __forceinline__ uint32_t ld_volatile(const uint32_t* p) { return *(const volatile uint32_t*)p; }
static __device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p)
{
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
static __device__ __forceinline__ void add_release(uint32_t* p)
{
    asm volatile("red.add.release.gpu.global.u32 [%0], 1;" : : "l"(p) : "memory");
}

// Thread 0's bounded wait for the arrival counter to reach target; false when it, or another
// block, gave up. The first polls come without a pause: a small scene's phases are about as long
// as one.
static __device__ __forceinline__ bool barrier_wait(LoopSync* sy, DevStatus* st, uint32_t target,
                                                    unsigned long long spin_limit)
{
    unsigned long long spins = 0;
    while ((int)(ld_acquire(&sy->count) - target) < 0) {
        if (++spins < 64) continue;
        if (ld_volatile(&sy->abort)) return false;
        if (spins > spin_limit) {
            atomicExch(&sy->abort, 1u);
            atomicOr(&st->error_flags, kErrTimeout);
            return false;
        }
        __nanosleep(64);
    }
    return ld_volatile(&sy->abort) == 0u;
}

// Barrier of the `blocks` blocks that share sy. Returns false when the loop must stop (a barrier
// gave up somewhere). The arrival counter only grows during a launch (the host clears it before each
// one): the e-th barrier of a launch is over when the counter reaches e times the number of blocks,
// so one reduction per block and barrier is all the traffic; epoch counts the barriers this block
// has passed. The arrival releases and the last poll acquires at device scope; block barriers on
// both sides carry that to the other threads. stalled: the barrier (from 1) that waits, for a short time, for
// an arrival that does not come, 0: none.
static __device__ bool blocks_barrier(LoopSync* sy, DevStatus* st, uint32_t& epoch, uint32_t blocks, uint32_t stalled = 0)
{
    __shared__ int ok;
    const uint32_t target = ++epoch * blocks + (stalled && epoch == stalled ? 1u : 0u);
    __syncthreads();
    if (threadIdx.x == 0) {
        add_release(&sy->count);
        ok = barrier_wait(sy, st, target, stalled ? kStallSpinLimit : kBarrierSpinLimit) ? 1 : 0;
    }
    __syncthreads();
    return ok != 0;
}

static __device__ __forceinline__ bool grid_barrier(LoopSync* sy, DevStatus* st, uint32_t& epoch)
{
    return blocks_barrier(sy, st, epoch, gridDim.x);
}

}  // namespace lsp
