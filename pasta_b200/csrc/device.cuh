// device.cuh -- small device functions shared by the kernel files.
#pragma once
#include <cuda_runtime.h>

#include "kernels.h"

namespace pb {

// Bulk prefetch of floats [lo, hi) of a row into L2 (one instruction, issued
// by one thread; a hint, nothing waits for it).  The row must start on a
// 16-byte boundary and hold hi rounded up to 4 floats.
__device__ __forceinline__ void prefetch_row_l2(const float *row, int lo, int hi) {
  lo &= ~3;
  hi = (hi + 3) & ~3;
  if (hi <= lo) return;
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(row + lo), "r"((unsigned)(hi - lo) * 4u)
               : "memory");
}

// model at the observed pixels of evaluation e
__device__ __forceinline__ const float *model_row(const EvalBatch &b, const EvalPrep &P, int e) {
  if (b.given) return b.given + (size_t)e * b.given_stride;
  return (P.mobs_in_b ? b.bufB : b.bufA) + (size_t)e * b.stride;
}

}  // namespace pb
