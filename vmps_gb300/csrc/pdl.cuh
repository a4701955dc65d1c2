// Launches that overlap the end of the kernel before them in the stream (programmatic dependent
// launch).
//
// The paths of this library are chains of kernels of 3 to 50 us: between two of them the chip used
// to sit idle from the end of the first to the launch of the second.  The blocks of a kernel
// launched by launch_pdl may start once those of the kernel before it have exited; pdl_wait then
// holds until that kernel's writes are visible.  So every kernel launched this way calls pdl_wait in
// all of its threads before it reads or writes anything another kernel may touch; before the call
// it may set up shared and tensor memory and read work lists, which copies write when a plan is
// made.  Data of the chain is read by plain loads: the read-only path (const __restrict__, __ldg) is for
// data that does not change while the kernel runs.
//
// Before and after: one-site Heisenberg HxV at D = 64 (4 launches) 57 -> 52 us, two-site Hubbard
// HxV at D = 1024 in FP64 (6 launches) 232 -> 220, an iteration of the transfer solve at 256
// multiplets (14 launches) 140 -> 113.  Kernels that released the next one from the start
// (griddepcontrol.launch_dependents) were slower: its waiting blocks held the SMs' shared-memory
// split of the kernel before (Lanczos at D = 1024: 12.7 ms against 12.3).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace vmps {

__device__ __forceinline__ void pdl_wait() {
    asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

// a pointer to data of the chain, after pdl_wait, for ld_global
template <typename T>
__device__ __forceinline__ T* pdl_data(T* p) {
    asm volatile("" : "+l"(p));
    return p;
}
// a plain load from global memory the compiler may move past stores to shared memory, but not above
// the pdl_data its address comes from
__device__ __forceinline__ double ld_global(const double* p) {
    double v;
    asm("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

}  // namespace vmps
