// launch.cuh -- launches of the kernels of a step, which follow one another on
// one stream with nothing in between.  A kernel launched by launch_next may be
// placed on the SMs while the one before it drains (programmatic dependent
// launch); it begins with wait_for_previous, which returns when every earlier
// kernel has finished and its writes are visible.  The next kernel's blocks are
// admitted only when all blocks of this one have started, so they never take
// the place of one of them.  Saves about two microseconds per kernel boundary
// (4,096-body direct steps 13.5 -> 11.6 us; the nine kernels of a 100,003-body
// tree step 258 -> 245 us).
//
// Such a kernel exists while earlier ones still write what it will read.  So it
// reads their results with plain loads (or past L1, __ldcg): read-only loads
// (__ldg, const __restrict__ parameters) are for memory that nothing writes as long
// as the kernel exists, and may be moved above the wait.  Tables the host wrote
// before the step (the prefixes of a batch) may be read so.
//
// Blocks placed early go where there is room, not evenly: a kernel of few long
// blocks (the force walk of a small system) must not be, nor the first kernel of
// a step behind the force walk, whose last blocks it would share SMs with
// (6,007 bodies 0.136 ms with both, 0.115 without; 4M 12.98 / 12.86 ms).
#pragma once
#include <cuda_runtime.h>

namespace nbgb {

__device__ __forceinline__ void wait_for_previous() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class... Params, class... Args>
cudaError_t launch_next_shared(void (*kernel)(Params...), dim3 grid, int threads, size_t shared, cudaStream_t st,
                               Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
template <class... Params, class... Args>
cudaError_t launch_next(void (*kernel)(Params...), dim3 grid, int threads, cudaStream_t st, Args... args) {
    return launch_next_shared(kernel, grid, threads, 0, st, args...);
}

}  // namespace nbgb
