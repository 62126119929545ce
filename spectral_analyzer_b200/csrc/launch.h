// launch.h — kernels that start while the kernel before them drains.
//
// launch_after() launches with programmatic stream serialisation: the blocks of
// the new kernel may become resident as soon as every block of the one before
// has called release_next() (or ended), and wait_previous() blocks until that
// kernel is complete and its results are visible.  A kernel launched any other
// way is waited for in full, as always in a stream, and has nothing to wait for.
//
// The rule for a kernel of such a chain: it calls wait_previous() in every block
// and releases its successor only after that, so that whatever ran two kernels
// earlier is complete when a kernel starts.  Before its wait it may read only what
// neither the kernel before it nor any kernel still running beside that one writes.
//
// One kernel releases first: the velocity pass of a plate scene, which also loads
// fields before its wait.  The kernel before it is the plate update, which writes
// no field and has itself waited for the pressure pass before releasing; the one
// after it, the pressure pass, waits for it in full before it reads anything, and
// releases only then.  A kernel put on either side of it has to keep both.
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
