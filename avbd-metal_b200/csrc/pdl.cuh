// pdl.cuh — programmatic dependent launch for a frame, a chain
// of ~100-300 dependent kernels per frame.  Each kernel lets the next one be
// scheduled as soon as all of its own blocks are running, and waits for the
// previous grid to complete (and its writes to be visible) before touching
// solver state.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace avbd {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_prologue() {
    pdl_trigger();
    pdl_wait();
}


// `overlap`: the grid may start while the one before it still runs
template <typename... KArgs, typename... Args>
static void launch_chain(void (*kernel)(KArgs...), bool overlap, uint32_t blocks, uint32_t threads, size_t smem,
                         cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = overlap ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <typename... KArgs, typename... Args>
static void launch_pdl_smem(void (*kernel)(KArgs...), uint32_t blocks, uint32_t threads, size_t smem, cudaStream_t st,
                            Args&&... args) {
    launch_chain(kernel, true, blocks, threads, smem, st, std::forward<Args>(args)...);
}

template <typename... KArgs, typename... Args>
static void launch_pdl(void (*kernel)(KArgs...), uint32_t blocks, uint32_t threads, cudaStream_t st,
                       Args&&... args) {
    launch_pdl_smem(kernel, blocks, threads, 0, st, std::forward<Args>(args)...);
}

}  // namespace avbd
