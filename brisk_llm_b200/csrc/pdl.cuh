// Programmatic dependent launch of the batched and the single-token kernels (those of decode.cu: see pdl_mode() there). A kernel
// started with launch_dependent() becomes resident while the one before it drains; it may read constants (weights) at once,
// everything else only behind wait_for_previous(), and lets the next kernel start with release_next() some time after it
// has waited itself - so nothing runs ahead of results that are more than one kernel away. Short kernels release at once,
// long ones when their main loop is done; CTAs that wait beside a running kernel for long slow it down (prompts of 512 to
// 800 tokens: 5-18 % between the two). What it saves is the gap between two kernels, 1-2 us, of which a layer of a
// prompt has twelve, one of a few tokens eleven.
#pragma once

#include <utility>

#include "common.cuh"

namespace bk {

#ifdef __CUDACC__
// No-ops in a kernel that was launched in plain stream order.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... Params, class... Args>
void launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    BK_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}
#endif

}  // namespace bk
