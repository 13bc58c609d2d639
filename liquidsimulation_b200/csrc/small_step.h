// Launch interface of the one-launch step of small scenes (small_step.cu).
#pragma once

#include <vector>

#include "lsp_kernels.h"

namespace lsp {

// A step made to give up (lsp_stalled_step): its `barrier`-th barrier (from 1; 0: none) of scene
// `scene` waits for an arrival that does not come.
struct BarrierStall {
    uint32_t barrier;
    int scene;
};

struct SmallStepArgs {
    GridBuildArgs g;
    StepBuffers b;       // the buffers the grid build gathers into
    float4* ppos_alt;
    void* sync;          // 16 zeroed bytes
    uint32_t* maxerr;    // max_it zeroed words
    DevStatus* host;     // pinned: the step's status, written at its end
    int pcisph;
    BarrierStall stall;
};

// Largest grid box of the one-launch step, whose blocks scan a contiguous share of the cells each:
// 1,200 particles take 42 us a step in 15,600 cells and 49 us in 1,000,000 (separate kernels 89).
constexpr int64_t kSmallStepCells = 1 << 20;
// Entries of tile_sums the one-launch step needs (one per block).
constexpr int kSmallStepTiles = 1024;

// Lanes per particle of the one-launch step for n particles in a grid of `cells`, 0 when the
// separate kernels are used.
int small_step_lanes(int64_t n, int64_t cells);
// Threads that a step counts for (StepInFlight): those of its one launch, else half of one per particle
// (of no more than fit).
int64_t step_threads(int64_t n, int lanes);   // lanes: of the one launch, 0: separate kernels
int64_t batch_step_threads(int64_t n, int small_blocks);   // small_blocks: of a one-launch step, 0: separate

// A step in flight on a device, for the solvers that other host threads step there at the same time: a
// one-launch step takes all its blocks' places at once and keeps them to its end, so steps that do
// not fit beside each other would run one after the other, where separate kernels share the chip.
class StepInFlight {
public:
    StepInFlight(int device, int64_t threads);
    ~StepInFlight();
    StepInFlight(const StepInFlight&) = delete;
    StepInFlight& operator=(const StepInFlight&) = delete;
    // Whether the step fits beside those that were in flight when it began.
    bool fits() const { return fits_; }

private:
    const int dev_;
    const int64_t threads_;
    bool fits_ = true;
};

// False when the device refuses the launch (the caller then runs the separate kernels).
bool launch_small_step(const SmallStepArgs& a, int lanes, cudaStream_t s);

// The one-launch step of a batch: block q of the launch belongs to blocks[q].scene, whose blocks are
// [first, first + count).
struct SmallBatchBlock {
    int scene, first, count, pad;
};
struct SmallBatchArgs {
    const DevParams* sp;             // [scenes]
    const SmallBatchBlock* blocks;   // device
    int mstride;                     // words of maxerr per scene
    int table_stride;                // floats of tables per scene
};

// Lanes per particle of a batch's one-launch step, and its blocks; 0 (and no blocks) when the
// separate kernels are used. n, cells: particles and grid cells of each scene.
int small_batch_plan(const std::vector<int64_t>& n, const std::vector<int64_t>& cells, std::vector<SmallBatchBlock>* blocks);
// a: b.status and host hold an entry per scene, sync 16 zeroed bytes per scene, g.tile_sums a word
// per block. False when the device refuses the launch.
bool launch_small_batch(const SmallStepArgs& a, const SmallBatchArgs& sb, int lanes, int blocks, cudaStream_t s);

}  // namespace lsp
