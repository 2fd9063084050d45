// launch.cuh -- launches that overlap the end of the kernel before them.
//
// Between two kernels of a stream the chip idles for a microsecond or two: the
// last CTAs leave, their writes are flushed, the next grid is sent out, its CTAs
// set up their barriers and tensor memory.  A kernel launched here may be sent
// out once every CTA of the kernel before it has left (or, where that is a
// foreign kernel that says so, has allowed it), and stops in
// wait_for_previous() until that kernel's writes are visible.  Every thread of
// every CTA passes it before its first access to global memory, so results are
// those of launches one after another.  That takes ordinary loads: a load
// through the read-only path (__ldg, a const __restrict__ parameter) tells the
// compiler that the data stays the same for as long as the kernel runs, which
// begins before the wait, so such loads have no place in a kernel launched here
// or in what it calls.  (Letting the next grid in earlier, by
// griddepcontrol.launch_dependents at each kernel's start, gained nothing more:
// 592 x 128^3 FP16 10.4 us a call against 9.9 without.)
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace kami {

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Ordinary loads of operands, which stay behind the wait (volatile) and are
// otherwise as free as those of the read-only path: plain C++ loads would have to
// keep their place among the kernel's own stores too (32^3 FP16 repeated 128 times
// 26.0 us against 22.8).
__device__ __forceinline__ uint32_t load_operand(const uint32_t *p)
{
    uint32_t v;
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint16_t load_operand(const uint16_t *p)
{
    uint16_t v;
    asm volatile("ld.global.b16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double load_operand(const double *p)
{
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint2 load_operand(const uint2 *p)
{
    uint2 v;
    asm volatile("ld.global.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double2 load_operand(const double2 *p)
{
    double2 v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 load_operand(const uint4 *p)
{
    uint4 v;
    asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
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
