// Passes over the start-of-step neighbour lists: non-pressure forces (gravity, surface tension,
// viscosity) of PCISPH, all forces of SPH, and the fused leapfrog integration + collision pass (the density and pressure are summed in the neighbour build, grid.cu).
//
// Thread per particle; each thread walks its own neighbour list in the reference's
// order, so its sums round exactly as the reference CPU solver's do.
#include "chained.cuh"
#include "lsp_device.cuh"
#include "lsp_kernels.h"
#include "particle_ops.cuh"

namespace lsp {

constexpr int kThreads = 256;

// SPHSolver::accumulateNonPressureForces, CPU branch (SPHSolver.cpp:201-248). The
// reference walks the list up to three times (normal, colour Laplacian when the normal
// exceeds the threshold, viscosity); each sum is independent, so one walk computes all
// three with the same per-sum rounding.
template <bool kGrad>
__global__ void __launch_bounds__(kThreads) k_nonpressure(DevParams P, StepBuffers b)
{
    const int i = chained((int)(blockIdx.x * blockDim.x + threadIdx.x));
    if (i < P.n) nonpressure_one<kGrad>(P, b, i);
}

// All forces of SPH (sph_forces_walk).
constexpr int kForceThreads = 128;
__global__ void __launch_bounds__(kForceThreads) k_sph_forces(DevParams P, StepBuffers b)
{
    const int i = chained((int)(blockIdx.x * blockDim.x + threadIdx.x));
    if (i < P.n) sph_forces_one(P, b, i);
}

// SPHParticle::integrate (SPHParticle.cpp:30-44) then SPHSolver::handleCollisions
// (SPHSolver.cpp:337-355) for one particle. With add_pforce the PCISPH pressure force is
// added first (PCISPHSolver.cpp:166-169).
__global__ void __launch_bounds__(kThreads) k_integrate_collide(DevParams P, StepBuffers b, int add_pforce)
{
    const int i = chained((int)(blockIdx.x * blockDim.x + threadIdx.x));
    if (i >= P.n) return;
    integrate_one(P, b, i, add_pforce);
}

static inline unsigned blocks_for(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

void launch_nonpressure(const DevParams& P, const StepBuffers& b, cudaStream_t s)
{
    if (!P.n) return;
    if (b.gradrho)
        launch_chained(k_nonpressure<true>, blocks_for(P.n, kThreads), kThreads, 0, s, P, b);
    else
        launch_chained(k_nonpressure<false>, blocks_for(P.n, kThreads), kThreads, 0, s, P, b);
}
void launch_sph_forces(const DevParams& P, const StepBuffers& b, cudaStream_t s)
{
    if (P.n) launch_chained(k_sph_forces, blocks_for(P.n, kForceThreads), kForceThreads, 0, s, P, b);
}
void launch_integrate_collide(const DevParams& P, const StepBuffers& b, bool add_pforce, cudaStream_t s)
{
    if (P.n) launch_chained(k_integrate_collide, blocks_for(P.n, kThreads), kThreads, 0, s, P, b, add_pforce ? 1 : 0);
}

}  // namespace lsp
