// Host-side helpers shared by the C ABI translation units: error reporting and argument checks.
#pragma once
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdio.h>

#include "../../include/nestquant_b200.h"

namespace nq {

// thread-local message of the last failure (read through nq_last_error)
char* error_buffer();
int fail(int code, const char* fmt, ...);

#define NQ_REQUIRE(cond, ...)                                   \
    do {                                                        \
        if (!(cond)) return ::nq::fail(NQ_ERR_ARG, __VA_ARGS__); \
    } while (0)

// call right after a kernel launch: reports launch-configuration errors without synchronising
inline int check_launch(const char* what)
{
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(NQ_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return NQ_OK;
}
// Programmatic dependent launch: a kernel lets its successor in the stream start launching early (its CTAs take their places, set up their shared
// memory and block), and itself waits until the whole predecessor grid has completed and its writes are visible, before it touches
// anything.  Every thread of every CTA passes through it, also where there is nothing to do: a grid that ended before its predecessor would
// release the one behind it too early.  What such a kernel reads may be written while it is already there, so its parameters are not
// const __restrict__ and it reads them without __ldg: both tell the compiler that the memory does not change during the kernel, and loads of such
// memory may be non-coherent and may move in front of the wait.  (What it finds through a table row, planes and scales, is read behind
// the row and so behind the wait.)
#ifdef __CUDACC__
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// launch of a kernel that does so; check_launch follows
template <class... P, class... A>
inline void launch_dependent(void (*kernel)(P...), dim3 grid, dim3 block, size_t shared, cudaStream_t stream, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = shared; cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
#endif
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace nq
