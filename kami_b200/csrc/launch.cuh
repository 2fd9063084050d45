// launch.cuh -- launches that overlap the end of the kernel before them.
//
// Between two kernels of a stream the chip idles for a microsecond or two: the
// last CTAs leave, their writes are flushed, the next grid is sent out, its CTAs
// set up their barriers and tensor memory.  A kernel launched here may be sent
// out once the CTAs of the kernel before it have all left, and stops in
// wait_for_previous() until that kernel's writes are visible.  Every thread of
// every CTA passes it before its first access to global memory, so results are
// those of launches one after another.  (Letting the next grid in earlier, by
// griddepcontrol.launch_dependents at each kernel's start, gained nothing more:
// 592 x 128^3 FP16 10.4 us a call against 9.9 without.)
#pragma once

#include <cuda_runtime.h>

namespace kami {

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
#endif

inline cudaError_t launch_overlapped(const void *fn, dim3 grid, dim3 block, void **args, size_t smem, cudaStream_t s)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelExC(&c, fn, args);
}

} // namespace kami
