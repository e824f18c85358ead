// Programmatic launches: a kernel launched with launch_after may be set up, and after the kernel ahead of it on the
// stream has called let_next_start in every block (or ended) may start, before that one has finished.  It calls
// wait_for_previous before it touches anything that work ahead of it reads or writes.
#pragma once

#include <cuda_runtime.h>

#include "errors.h"

namespace rt {

__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), unsigned blocks, unsigned threads, size_t shared, cudaStream_t st, A... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = shared;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    check_cuda(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...), "kernel launch");
}

}  // namespace rt
