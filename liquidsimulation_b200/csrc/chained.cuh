// Kernels of a step that overlap the tail of the kernel before them on the stream (programmatic
// dependent launch): the next kernel's blocks take their places while the last blocks of the
// current one still run, and wait there for its end and its memory operations. That hides about a
// microsecond of launch latency per kernel: 1,178 -> 1,127 us for four SPH steps of 250,000 particles
// with their transfers (8 kernels a step), 951 -> 945 us for four PCISPH steps of 102,400, whose loop
// is a cooperative launch and waits for the whole kernel before it.
#pragma once

#include <cuda_runtime.h>

namespace lsp {

// First thing in a kernel launched with launch_chained. Returns v, a value that all addresses of the
// kernel's loads have to depend on: no load, not even one through the read-only path, can then move
// before the wait.
template <typename T>
__device__ __forceinline__ T chained(T v)
{
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    asm volatile("" : "+r"(v) : : "memory");
    return v;
}

template <typename... Params, typename... Args>
void launch_chained(void (*kernel)(Params...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t s, Args... args)
{
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace lsp
