// Programmatic dependent launch: a kernel launched this way may start while the one before it in the stream is
// still running, sets itself up, and waits for it (pdl_wait) before it touches anything that earlier work reads
// or writes.  Every kernel here lets its own successor start only after that wait, so that whatever a successor
// finds complete includes everything further back.  overlap = false: the same kernels one after the other (the two
// instructions do nothing then).
#pragma once
#include <cuda_runtime.h>

namespace cbkv {

__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... Params, typename... Args>
static inline cudaError_t launch_pdl(bool overlap, void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t st, const Args&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace cbkv
