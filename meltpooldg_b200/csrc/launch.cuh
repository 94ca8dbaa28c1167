// Programmatic dependent launch for the short kernels of a Krylov iteration: a kernel launched with
// launch_dependent may start while its predecessor in the stream still runs (once every block of
// that has called dependents_may_start), sets up, and waits in wait_for_predecessor until the
// predecessor has completed and its writes are visible. Every such kernel waits before its first
// access to data that another kernel writes, also on the way to an early return. Outside such a
// launch both calls do nothing.
//
// Such a kernel reads the vectors that the iteration writes by coherent loads: load_live, or plain
// loads through pointers without __restrict__. It is resident while its predecessors still write
// them, and a non-coherent load (__ldg, or what the compiler makes of const __restrict__) is
// defined only for data that no one writes while the kernel lives; it may also be moved above
// wait_for_predecessor. What stays fixed during the solve (the diagonal, coefficients, geometry,
// indices) is read either way.
#pragma once

#include <cuda_runtime.h>

namespace mpdg {

__device__ __forceinline__ void wait_for_predecessor()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void dependents_may_start()
{
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// A load that is neither non-coherent nor moved above wait_for_predecessor (FE_Q(3) 128^3 FP64
// operator 1.39 ms, as with __ldg; a plain load in its gather was scheduled worse, 1.46 ms)
__device__ __forceinline__ double load_live(const double *p)
{
  double v;
  asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

template <typename... P, typename... A>
cudaError_t launch_dependent(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem,
                             cudaStream_t stream, const A &...args)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace mpdg
