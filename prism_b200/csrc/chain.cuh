// Kernels launched one after the other on a stream.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace prism_b200 {

// First statement of every kernel launched with launch_chained: lets the next
// kernel of the stream be set up beside this one, then waits until the
// previous one has completed and its writes are visible.  (The wait is a
// no-op in a plain launch.)
//
// A chained kernel's life overlaps the stores of the kernels before it, so
// what any kernel of the call writes is not read-only for that life: such
// data is read with ordinary loads, never through __ldg or a `const
// __restrict__` pointer (both let the compiler use the non-coherent path and
// move the load above the wait).  Only the caller's field may be read that
// way: the calls that read it begin with a plain launch, so the field is
// complete before any chained kernel starts.
// tests/test_chained_loads.py holds the sources to this.
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launch with programmatic stream serialisation: the kernel's CTAs may be
// resident before the previous kernel of the stream has ended (it then waits
// in chain_wait), which hides part of the 2-3 us between dependent kernels.  A
// compression's launches after the first (nine launches in all for one-plane
// fields and up to four tiles an SM; above, ten, the predictor's two plain ones
// between a fork and a join): 64x48x40 float 99.8 -> 95.5 us, 128^3 108 -> 102
// us, 384x384x256 double 602 -> 589 us.  The decompression's four gained
// nothing (128^3 64.4 -> 68.0 us) and are plain launches.
template <class... KArgs, class... Args>
inline cudaError_t launch_chained(void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem, cudaStream_t st,
                                  Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace prism_b200
