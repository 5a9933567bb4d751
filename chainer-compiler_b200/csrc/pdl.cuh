// Programmatic dependent launch, device and host side.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace chxq {

// Programmatic dependent launch: a kernel launched with the programmatic-serialization attribute may start while the kernel
// before it in the stream is still running.  launch_dependents lets the next kernel's CTAs be scheduled as soon as this
// kernel's CTAs leave their SMs; dependency_wait blocks until the previous kernel has completed and its writes are visible.
// Everything a CTA does before dependency_wait (barrier initialisation, tensor-memory allocation) overlaps the previous
// kernel's tail; nothing before it may touch global memory that the previous kernel writes or reads.
// A kernel that never asks for launch_dependents lets the next one in when it has finished.  That is right where blocks run long and there are
// only a few per SM: blocks of the next kernel that come early take up places unevenly and its last ones finish late (global average pool of
// [41, 970, 48, 48], call after call: 139 us with an early launch, 63 us without).
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_dependency_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launch with the programmatic-serialization attribute: the kernel may begin (up to its dependency wait) while the previous
// kernel in the stream drains.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl_cluster(int cluster, void (*kernel)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = (unsigned)cluster; at[1].val.clusterDim.y = 1; at[1].val.clusterDim.z = 1;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, int block, size_t smem, cudaStream_t s, Args&&... args) {
    return launch_pdl_cluster(1, kernel, grid, block, smem, s, std::forward<Args>(args)...);
}

}  // namespace chxq
