// launch.h — kernels that start while the kernel before them drains.
//
// launch_after() launches with programmatic stream serialisation: the blocks of
// the new kernel may become resident as soon as every block of the one before
// has called release_next() (or ended), and wait_previous() blocks until that
// kernel is complete and its results are visible.  A kernel releases its
// successor only after its own wait, so whatever ran two kernels earlier is
// complete when a kernel starts; before the wait it may read only what no
// kernel of the chain writes.  A kernel launched any other way is waited for in
// full, as always in a stream.
#pragma once

#include <cuda_runtime.h>

namespace {

__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void release_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

template <class... A>
cudaError_t launch_after(void (*k)(A...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args)
{
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, args...);
}

}  // namespace
