// pdl.cuh -- launches that overlap (programmatic dependent launch).
//
// The passes of a relaxation form a chain of grids of a few microseconds.
// Each is launched while the one before it drains: it calls pdl_trigger(), may
// read what no grid of the chain writes, and calls pdl_wait() before it reads
// or writes anything else.  The wait returns when the grid before it is
// complete and its writes are visible; that grid waited for the one before
// it, so by then the whole chain is complete.  A chain starts behind a plain
// launch, which waits for everything before it.  Every kernel launched early
// has to wait, also where it has nothing to do (an early return before the
// wait would let the grid after it run ahead of the grid before it).  What
// other grids of the chain write is read by plain loads: a read-only load
// (__ldg, or a const __restrict__ argument) may be moved above the wait.  Both
// calls do nothing in a plain launch.
//
// The residual and assembly kernels stay plain launches: early launches gained
// them nothing (a 24,576-cell step 0.166 ms against 0.162, 32,768 hexes REF
// 0.136 against 0.121) and their gathers need the read-only loads (663,552
// viscous tets 2.06 against 1.77).
#pragma once
#include <cuda_runtime.h>

#include "fpsi_internal.h"

namespace fpsi {
namespace dev {
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
}  // namespace dev

// early: the launch may overlap the grid before it (never while kernels are
// timed one by one)
template <class... P, class... A>
cudaError_t launch_grid(const fpsi_ctx* x, bool early, void (*kernel)(P...), int64_t grid, int block, size_t smem,
                        A... args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(unsigned(grid));
  cfg.blockDim = dim3(unsigned(block));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = x->stream;
  cfg.attrs = &at;
  cfg.numAttrs = early && !x->profiling ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}
// errors are left for the caller's cudaGetLastError
template <class... P, class... A>
void launch_chain(const fpsi_ctx* x, void (*kernel)(P...), int64_t grid, int block, size_t smem, A... args) {
  launch_grid(x, true, kernel, grid, block, smem, args...);
}
}  // namespace fpsi
