// Programmatic dependent launch: a kernel launched with launch_pdl() may start
// while the kernel before it on the stream is still running, and reads what
// that kernel does not write (mesh, matrix) before pdl_wait(), which returns
// once that kernel has finished and its results are visible.  pdl_wait() lets
// the next kernel start in turn, and not before: so a kernel overlaps its
// predecessor alone, and everything before that one is complete and may be
// read ahead of the wait too.  Every kernel of a chain waits (a kernel that did
// not could finish before its predecessor); without the launch attribute the
// wait returns at once.
//
// What the predecessor writes is read after the wait with plain loads (ldw):
// a read-only (non-coherent) load is only for data that no kernel writes while
// this one is resident.
#pragma once

#include <cuda_runtime.h>

namespace afx {
namespace dev {

__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

__device__ __forceinline__ float4 ldw(const float4* p) {
    float4 a;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w) : "l"(p));
    return a;
}
__device__ __forceinline__ double2 ldw(const double2* p) {
    double2 a;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(a.x), "=d"(a.y) : "l"(p));
    return a;
}
__device__ __forceinline__ float ldw(const float* p) {
    float a;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(a) : "l"(p));
    return a;
}
__device__ __forceinline__ double ldw(const double* p) {
    double a;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(a) : "l"(p));
    return a;
}
__device__ __forceinline__ int ldw(const int* p) {
    int a;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(a) : "l"(p));
    return a;
}

}  // namespace dev

// on = false: an ordinary launch
template <class... P, class... A>
inline cudaError_t launch_pdl_if(const bool on, void (*kernel)(P...), const dim3 grid, const dim3 block,
                                 const size_t smem, const cudaStream_t s, A... args) {
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    c.attrs = at;
    c.numAttrs = on ? 1 : 0;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

template <class... P, class... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), const dim3 grid, const dim3 block, const size_t smem,
                              const cudaStream_t s, A... args) {
    return launch_pdl_if(true, kernel, grid, block, smem, s, args...);
}

}  // namespace afx
