// Programmatic dependent launch (sm_90+): a kernel launched with the stream-serialisation attribute may be
// scheduled while its predecessor in the stream is still running - once every CTA of the predecessor has called
// pdl_trigger() or exited - and must call pdl_wait() before touching anything the predecessor writes (the wait
// returns when the predecessor has completed and its writes are visible). This hides the launch gap between the
// short kernels of one operation. Both instructions do nothing in a kernel that was launched normally.
// Whatever a predecessor may have written is read by plain loads: no __ldg, and no `const T* __restrict__` parameter, either of
// which lets the compiler take the read-only path (for memory that nobody writes while the kernel runs, and the predecessor may
// still run then) and move the load above the wait. Constant tables are free of this, and may be read before the wait. The
// older kernels of batchnorm, pool and norm_loss, whose first statement is the wait, keep their qualifiers: plain loads stay
// behind the stores of an unrolled loop (BatchNorm of 256 x 128 x 28 x 28, forward and backward: 101 -> 108 us).
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>

namespace gcow {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch `kernel` so that it may overlap the tail of its predecessor in the stream. Every thread of the kernel must come to
// pdl_wait() before it touches memory that another kernel reads or writes. GCOW_PDL=0 falls back to ordinary launches.
template <typename... KArgs, typename... Args>
static void launch_dependent(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
  static const bool enabled = [] { const char* e = getenv("GCOW_PDL"); return !(e && e[0] == '0'); }();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = s;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr; cfg.numAttrs = enabled ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace gcow
