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
//
// Such a kernel starts while its inputs may still be written, so none of them
// is read as constant data (__ldg, or a const __restrict__ parameter that the
// compiler reads so): PDL_FRESH(p) after pdl_wait() gives the pointer a value
// that the compiler can't trace to the parameter.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#define PDL_FRESH(p) asm volatile("" : "+l"(p) : : "memory")

namespace iclb {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Level 1 (axpy, scal) and unaligned or small GEMV calls on up to this many
// operand elements are dependent launches. Above it a call runs for longer than
// 20 us at the memory's rate: the saved start is lost in it, and the kernels
// read faster with their inputs as constant data (SGEMV 16384^2, CGEMV 8192^2
// and Level 1 at 2^28 together: 1882 us as plain launches of plain kernels,
// 1890 with PDL_FRESH in them, 1896 dependent).
constexpr long kDependentElems = 1L << 24;
inline int dependent(long elems) { return elems <= kDependentElems ? 1 : 0; }

// cluster: 0 a plain launch (the kernel's wait returns at once), 1 a dependent
// one, above 1 a dependent one in clusters of that many blocks.
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
    cfg.numAttrs = cluster > 1 ? 2 : cluster;
    const cudaError_t r = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
    if (r != cudaSuccess) cudaGetLastError();
    return r;
}

}  // namespace iclb
