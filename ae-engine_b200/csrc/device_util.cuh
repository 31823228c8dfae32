// device_util.cuh -- small device functions that several kernels share.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace aemp {

// inclusive sum over the lanes up to this one
__device__ __forceinline__ uint32_t warp_scan_incl(uint32_t x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Programmatic dependent launch: a kernel launched by launch_after may start while the kernel
// before it drains, and waits here until that one has finished and its writes are visible.  Without
// the launch attribute both are no-ops.
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

// Launches `kernel`, dependently where `early`.
template <class... P, class... A>
cudaError_t launch_after(bool early, void (*kernel)(P...), unsigned ctas, unsigned threads, size_t smem, cudaStream_t s,
                         A&&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3(ctas);
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &at;
  c.numAttrs = early ? 1 : 0;
  return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

}  // namespace aemp
