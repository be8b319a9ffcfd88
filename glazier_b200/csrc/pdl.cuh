// Programmatic dependent launches: a kernel launched this way may start while
// the previous kernel on the stream ends, and waits before it reads anything
// that kernel writes.
#pragma once

#include <cuda_runtime.h>

namespace glz {

// Whether kernels launch programmatically (GLAZIER_SWEEP_PDL=0: plainly).
int programmatic_launch();

// The kernel's side: wait for the previous kernel and its memory, then let
// the next launch start its own prologue. Every kernel of a chain waits, so
// once one has, everything before it on the stream is complete.
__device__ __forceinline__ void grid_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... Params, class... Args>
inline cudaError_t launch_after(void (*kernel)(Params...), dim3 grid, int threads, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = programmatic_launch();
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

}  // namespace glz
