// noalloc_layout.h -- where the allocation-free chi2 keeps its workspace in
// the static scratch array (plain C++; the CPU tests check it at the limits).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "common.cuh"
#include "kernels.h"

namespace pb {

// 32 MiB, and what the group records have grown by since the limits on the
// label count were first set
constexpr size_t NOALLOC_SCRATCH_BYTES = (32u << 20) + 4096;

constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// bytes of scratch one label needs: prep record, rotation half spectra
// (alone and times the instrument spectrum),
// eval->star index, the two spectrum rows, the broadening block bounds and
// the partial chi2 sums
inline size_t noalloc_per_label(int64_t stride, int bnd_stride) {
  return align256(sizeof(EvalPrep)) + 2 * align256(1025 * sizeof(float2)) + align256(sizeof(int)) +
         2 * align256((size_t)stride * sizeof(float)) + align256((size_t)bnd_stride * sizeof(int)) +
         align256((size_t)MAX_CHUNKS * sizeof(double)) +
         align256(sizeof(GroupRec)) + align256(sizeof(int));
}

// the star record, and the group slots of a partly filled last segment
constexpr size_t noalloc_fixed() {
  return align256(sizeof(DevStar)) + align256((size_t)(SEG - 1) * sizeof(GroupRec)) + 256;
}

// labels the scratch holds
inline int64_t noalloc_max_labels(int64_t stride, int bnd_stride) {
  const size_t fixed = noalloc_fixed();
  return NOALLOC_SCRATCH_BYTES > fixed ? (int64_t)((NOALLOC_SCRATCH_BYTES - fixed) / noalloc_per_label(stride, bnd_stride)) : 0;
}

// offsets of the parts for L labels
struct NoallocLayout {
  size_t star, prep, H, HG, eval_star, A, B, bnd, cpart, grec, gcount, total;
};
inline NoallocLayout noalloc_layout(int64_t L, int64_t stride, int bnd_stride) {
  const size_t n = (size_t)L;
  NoallocLayout o;
  size_t at = 0;
  auto part = [&](size_t bytes) {
    const size_t p = at;
    at += align256(bytes);
    return p;
  };
  o.star = part(sizeof(DevStar));
  o.prep = part(sizeof(EvalPrep) * n);
  o.H = part(1025 * sizeof(float2) * n);
  o.HG = part(1025 * sizeof(float2) * n);
  o.eval_star = part(sizeof(int) * n);
  o.A = part((size_t)stride * sizeof(float) * n);
  o.B = part((size_t)stride * sizeof(float) * n);
  o.bnd = part((size_t)bnd_stride * sizeof(int) * n);
  o.cpart = part((size_t)MAX_CHUNKS * sizeof(double) * n);
  // SEG group slots per segment of SEG labels: L rounded up to SEG
  o.grec = part(sizeof(GroupRec) * ((n + SEG - 1) / SEG * SEG));
  o.gcount = part(sizeof(int) * ((n + SEG - 1) / SEG));
  o.total = at;
  return o;
}

}  // namespace pb
