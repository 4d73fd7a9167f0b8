// Kernel launches of the stage operators.
//
// Programmatic dependent launch: a stage kernel may be scheduled once every CTA of the kernel before it on the stream
// has reached its last tile (pdl_trigger); it reads its operator's constants (matrices, tables, tile list: uploaded
// when the operator was built), then waits for that kernel to complete (pdl_wait) before it touches anything another
// kernel may have written.  This hides the launch gap and the prologue, which is most of a small problem's stage.
// The trigger comes with the last tile, not earlier: a waiting CTA holds registers and shared memory.
// The kernel's lifetime overlaps its predecessor's, so what the predecessor writes (state, residual, lists) is not read-only
// for the whole of it: such arrays are read with ordinary loads, __ldcg or __ldcs, never with __ldg / ld.global.nc, whose
// contract asks for that and which need not stay behind the wait.  Those are for the operator's constants alone.
// Alone on the GPU, two steps of small mixed problems (2 to 16 instances of 4^3 to 16^3): 112 -> 77 and 94 -> 65 us; order 2,
// 8^3 x 6 FP64 step: 40 -> 31 us; 64^3-class stages are unchanged.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <utility>

#include "kernels.hpp"
#include "runner.hpp"

namespace dgk {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A &&...args) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  cuda_check(cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...), "kernel launch");
}

// CTAs of a kernel that share an SM, and its shared-memory opt-in.  Both are asked of the driver on an operator's first
// launch and kept in its LaunchInfo (per operator, not per process: an operator never outlives its context).
template <typename K>
int resident_ctas(K kernel, int threads, size_t smem, LaunchInfo *info) {
  if (info && info->per_sm) return info->per_sm;
  cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem), "smem attribute");
  int per = 0;
  cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem), "occupancy");
  return std::max(1, per);
}

}  // namespace dgk
