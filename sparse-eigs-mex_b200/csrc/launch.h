// Kernel launches whose refusals are not lost.  A launch that the runtime
// refuses (too much shared memory, no cluster of that size) writes nothing and
// leaves the stream as it was, so a synchronisation reports success; the first
// such error is kept per host thread until launch_result() asks for it.
#pragma once

#include "counters.h"

#include <cuda_runtime.h>

namespace spx {

// first launch error of the calling thread since it was last cleared
inline cudaError_t &launch_error() {
    static thread_local cudaError_t e = cudaSuccess;
    return e;
}

// e, or if that is a success the calling thread's launch error; clears it
inline cudaError_t launch_result(cudaError_t e) {
    const cudaError_t l = launch_error();
    launch_error() = cudaSuccess;
    return e != cudaSuccess ? e : l;
}

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
    if (e != cudaSuccess && launch_error() == cudaSuccess) launch_error() = e;
    note_launch();
    return e;
}
// the kernel begins with chain_begin() (chain.cuh)
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
