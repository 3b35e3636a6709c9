// Chains of short kernels on one stream.  Each lets the next one's blocks
// start while it runs and itself waits, before it touches memory, for the
// kernel before it to be complete; that hides most of a launch's 2 us
// (programmatic dependent launch).  A kernel that is launched plainly, or
// that follows one without chain_begin, behaves as without it.  Measured on
// whole eigensolves: 20^3 15.6 -> 14.8 ms, 46^3 18.1 -> 17.3, 64^3 74.3 ->
// 72.9, largest eigenvalues at 100^3 11.9 -> 11.1.
#pragma once

#include "common.cuh"
#include "counters.h"

namespace spx {

SPX_DEV void chain_begin() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A launch on `st`, chained or plain; what the runtime says to it.
template <class... P, class... A>
cudaError_t launch_as(bool chained, void (*kernel)(P...), dim3 grid, int threads, size_t smem,
                      cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
    note_launch();
    return e;
}
template <class... P, class... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, int threads, size_t smem,
                           cudaStream_t st, A... args) {
    return launch_as(true, kernel, grid, threads, smem, st, args...);
}
template <class... P, class... A>
cudaError_t launch_plain(void (*kernel)(P...), dim3 grid, int threads, size_t smem,
                         cudaStream_t st, A... args) {
    return launch_as(false, kernel, grid, threads, smem, st, args...);
}

}  // namespace spx
