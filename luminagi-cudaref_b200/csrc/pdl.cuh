// pdl.cuh -- launches that start while the kernel before them in the stream still runs.
//
// A chain of short kernels pays a few microseconds between each two: the launch, and the first blocks' start.
// A kernel launched by launch_dependent has its blocks on the SMs by then.  Every such kernel calls
// begin_after_predecessors (or tc::wait_for_predecessors) in all its threads before it touches memory that
// another kernel of the stream reads or writes.
//
// One B200, plain launches -> these: a BVH build of 20,500 triangles 123 -> 95 us (13 kernels of 2 to 12 us), of
// 1,050,972 354 -> 339 us.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace lg
{
// Waits until the kernels before this one have finished and their writes can be seen, and only then lets
// the next kernel's blocks start: no more than two kernels of a chain are ever on the SMs together, and none is
// there while a kernel two before it still reads.
__device__ __forceinline__ void begin_after_predecessors()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
cudaError_t launch_dependent(void (*fn)(P...), dim3 grid, int block, int smem, cudaStream_t stream, A&&... args)
{
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3((unsigned)block);
    c.dynamicSmemBytes = (size_t)smem;
    c.stream = stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, fn, std::forward<A>(args)...);
}
}  // namespace lg
