// Launching the kernels of a job as a chain (programmatic dependent launch).
//
// Inside a job every kernel may be launched while the one before it is still running: it then sets itself up (barriers,
// tensor memory, and what its op declares as read early: first weights, constants, the state of a fused recurrence, which
// chain_of checks against the ops in front) and executes griddepcontrol.wait before it touches anything else that a kernel
// before it produced or still reads.  A kernel that lets its successor in early (griddepcontrol.
// launch_dependents) must have taken everything the successor could compete for (tensor memory) by then.
#pragma once

#include "kernels.h"

namespace wrk {
namespace k {

// Everything the kernels before this one wrote is visible after the wait (returns at once in a plain launch).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Launches `kernel`; as a programmatic dependent of the kernel before it while a job's launches are being issued
// (chained_launches()) and `early` is true.
template <typename... KArgs, typename... Args>
cudaError_t launch_early(bool early, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = early && chained_launches() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
cudaError_t launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
    return launch_early(true, kernel, grid, block, smem, stream, args...);
}

}  // namespace k
}  // namespace wrk
