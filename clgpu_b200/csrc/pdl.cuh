// Programmatic dependent launch for chains of kernels on one stream (split ->
// GEMM -> split -> ...): pdl_launch's kernel may have its blocks resident, and
// its barriers and TMEM set up, while the kernel before it still runs, and
// touches global memory only after pdl_wait(), which returns once everything
// before it on the stream has finished and is visible.  Every kernel launched
// so calls pdl_wait() in all its threads, so its own end still implies the
// end of all that came before: kernels, copies and events behind it are
// ordered as behind a plain launch.  pdl_trigger() lets the next such launch
// start early; it comes after pdl_wait(), so that at most two kernels of a
// chain overlap, and after the kernel's own TMEM allocation (a waiting block
// then never holds TMEM that a kernel it waits for still has to allocate).
// Without a trigger the next launch still skips the step from one grid's end
// to the next one's start.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace iclb {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... Args>
cudaError_t pdl_launch(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t stream, int cluster,
                       Args&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    const cudaError_t r = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
    return r != cudaSuccess ? r : cudaGetLastError();
}

}  // namespace iclb
