// lbf_chain.cuh -- launches that overlap their start with the end of the kernel
// before them in the stream (programmatic stream serialization).
//
// A time step is one to three dependent kernels, 10-30 us each on small boxes,
// and between two of them the launch and the ramp-up of the CTAs take a few us.
// A chained kernel may be scheduled once every CTA of its predecessor has
// started; chain_begin, before its first access to global memory, waits until
// the predecessor is complete and its writes are visible, and lets the kernel's
// own successor be scheduled in the same way.  What the predecessor writes is
// read with plain loads, which stay behind the wait; __ldg is for tables that no
// kernel writes.  A step of
// D3Q19 64^3: 11.3 -> 9.6 us, of 32^3 with two components 23.0 -> 21.2 us; 256^3
// unchanged.
#pragma once
#include <cuda_runtime.h>

namespace lbf {

__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// launch a kernel that starts with chain_begin
template <typename... P, typename... A>
cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, const A&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace lbf
