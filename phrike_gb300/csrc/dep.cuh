// Chained launches (programmatic dependent launch).  A step is a chain of short
// kernels on one stream; launched this way the next kernel's CTAs come up, set
// up their shared-memory tables and wait while the last CTAs of the present
// kernel drain, instead of after them.
//
// Rules: a kernel launched with launch_dep calls dep_wait() before its first
// access to memory that an earlier kernel reads or writes (plan tables, which
// are written once at creation, may be read before), and reads such memory
// with plain loads (a read-only-cache load could be moved above the wait).
// dep_wait() returns when every earlier kernel of the chain has completed, so
// a chain of them orders memory as plain launches do.
//
// No kernel triggers its dependents early: the next grid comes up as the present
// one's CTAs exit.  Triggered at the start, its CTAs pile up on the SMs the
// present grid leaves idle and stay there (Orszag-Tang 512^2 step 332 us, TGV
// 64^3 149).  Per step, plain launches -> chained: KHI 128^2 112 -> 84 us, TGV 64^3
// 147 -> 100, Orszag-Tang 512^2 311 -> 269, LGL 257^2 118 -> 96, 3D MHD 128^3
// 1267 -> 1220; three steps of KHI 512^2 x 16 2460 -> 2390.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace ps {

__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
inline cudaError_t launch_dep(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &attr;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, std::forward<A>(args)...);
}

}  // namespace ps
