// Programmatic dependent launch: a kernel launched with launch_pdl may be
// scheduled while the kernel before it on the stream still runs, and waits for
// that kernel's completion (and the visibility of its results) in pdl_wait,
// which every such kernel calls before it touches memory.  pdl_trigger, after
// the wait, lets the next kernel be scheduled.  This hides a launch's latency
// (about 1.5 us) between kernels of a few microseconds.  What an earlier
// kernel writes is read through ld.global (load_link_c, __ldca): the
// non-coherent loads of __ldg ask for data that no kernel writes while this
// one is resident.
#pragma once
#include "nrq_common.cuh"

namespace nrq {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

__device__ __forceinline__ cplx ld_c(const double2 *p) {
  const double2 v = __ldca(p);
  return {v.x, v.y};
}
// link U_d(s), coherently
__device__ __forceinline__ m3 load_link_c(const double2 *U, int64_t V, int64_t s, int d) {
  m3 m;
  const double2 *p = U + (int64_t)d * 9 * V + s;
#pragma unroll
  for (int k = 0; k < 9; ++k) m.e[k] = ld_c(p + k * V);
  return m;
}

// (inside a capture an ordinary launch: graphs keep full dependencies)
template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(st, &capture);
  cfg.attrs = &attr;
  cfg.numAttrs = capture == cudaStreamCaptureStatusNone ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace nrq
