// device.cuh -- small device functions shared by the kernel files.
#pragma once
#include <cuda_runtime.h>

#include "kernels.h"

namespace pb {

// The grid's axes and limits copied into shared memory by the CTA (the
// searches and limit scans of the label checks walk them with dependent
// reads), or the resident ones when they do not fit.  Holds a CTA barrier.
constexpr int GEOM_SMEM = 8192;
__device__ __forceinline__ GridGeom geom_shared(const GridGeom &g, double *buf) {
  const int nt = g.nt, nm = g.nm, nl = g.nl;
  if ((3 * nt + nm + nl) * 8 > GEOM_SMEM) return g;
  double *tv = buf, *mv = tv + nt, *lv = mv + nm;
  int64_t *cum = reinterpret_cast<int64_t *>(lv + nl);
  int *llo = reinterpret_cast<int *>(cum + nt), *lhi = llo + nt;
  for (int i = threadIdx.x; i < nt; i += blockDim.x) {
    tv[i] = g.tv[i];
    cum[i] = g.cum[i];
    llo[i] = g.llo[i];
    lhi[i] = g.lhi[i];
  }
  for (int i = threadIdx.x; i < nm; i += blockDim.x) mv[i] = g.mv[i];
  for (int i = threadIdx.x; i < nl; i += blockDim.x) lv[i] = g.lv[i];
  __syncthreads();
  GridGeom r = g;
  r.tv = tv;
  r.mv = mv;
  r.lv = lv;
  r.cum = cum;
  r.llo = llo;
  r.lhi = lhi;
  return r;
}

// model at the observed pixels of evaluation e
__device__ __forceinline__ const float *model_row(const EvalBatch &b, const EvalPrep &P, int e) {
  if (b.given) return b.given + (size_t)e * b.given_stride;
  return (P.mobs_in_b ? b.bufB : b.bufA) + (size_t)e * b.stride;
}

// ------------------------------------------------------------ resampling
// shift_and_resample (convolve_rv.rs:569-603): index in double, weight from
// the f32-rounded index minus the f32 floor, linear interpolation in f32.
struct ResPos {
  int j;    // left synth pixel
  float w;  // weight of pixel j + 1
};
__device__ __forceinline__ float resample_value(float w, float sj, float sj1) {
  return __fadd_rn(__fmul_rn(1.0f - w, sj), __fmul_rn(w, sj1));
}
struct Resampler {
  const float *s;
  int N, kind;
  double shift_log, shift_factor, lin_offset;
  const double *fidx, *wl_obs, *wl_vals;
  const float *given;  // model given directly at the observed pixels
  // j never decreases with i when the float indices do not
  __device__ __forceinline__ ResPos pos(int i) const {
    double idx;
    if (kind == WL_LOG) idx = fidx[i] + shift_log;
    else if (kind == WL_LIN) idx = __dadd_rn(__dmul_rn(shift_factor, fidx[i]), lin_offset);
    else {
      const double wl = __dmul_rn(wl_obs[i], shift_factor);
      bool f;
      int k = lower_bound(wl_vals, N, wl, f);
      if (f) idx = (double)k;
      else if (k == 0) idx = 0.0;
      else if (k == N) idx = (double)N - 1.0;
      else idx = __dadd_rn(__dadd_rn(__ddiv_rn(wl - wl_vals[k - 1], wl_vals[k] - wl_vals[k - 1]), (double)k), -1.0);
    }
    const double fl = floor(idx);
    int j = fl > 0 ? (int)fl : 0;
    if (j > N - 2) j = N - 2;  // the preparation kernel rejected j + 1 >= N already
    return ResPos{j, (float)idx - (float)j};
  }
  __device__ __forceinline__ float operator()(int i) const {
    if (given) return given[i];
    const ResPos q = pos(i);
    return resample_value(q.w, s[q.j], s[q.j + 1]);
  }
};

__device__ __forceinline__ Resampler make_resampler(const DevGrid &G, const DevStar &st, const EvalPrep &P,
                                                    const float *row, const float *given) {
  Resampler r;
  r.s = row;
  r.N = G.npx;
  r.kind = G.wl_kind;
  r.shift_log = P.shift_log;
  r.shift_factor = P.shift_factor;
  r.lin_offset = P.lin_offset;
  r.fidx = st.fidx;
  r.wl_obs = st.wl_obs;
  r.wl_vals = G.wl_vals;
  r.given = given;
  return r;
}

// ------------------------------------------------ instrument profile (tile)
// FixedTargetDispersionLogSpace: g[i] = sum_k gk[k] r[i + h - k], r zero
// outside the grid (convolve_rv.rs:207-210).  Per-pixel kernels
// (VariableTargetDispersion / FixedTargetDispersionNonLog):
// g[i] = kernel_i . r[i-h .. i+h], pixels within h of either end pass
// through (convolve_rv.rs:213-233, 414-430).  r(t) reads the rotation
// output for synth pixel t from wherever the caller staged it.
template <class RF>
__device__ __forceinline__ float instrument(const DevStar &st, int N, int i, int h, const RF &r) {
  const int w = 2 * h + 1;
  float acc = 0.0f;
  if (st.disp_kind == DISP_FIXED) {
    const float *g = st.gk;
    for (int k = 0; k < w; k++) acc = fmaf(__ldg(&g[k]), r(i + h - k), acc);
  } else {
    if (i < h || i >= N - h) return r(i);
    // tap-major: the lanes of a warp work neighbouring pixels and read
    // neighbouring words (k_broaden, when it had this loop too: 1.51 ms for
    // 1,000 evaluations of 80,000 pixels and 17 taps with pixel-major taps, a
    // stride of w words between the lanes, 1.27 ms with these)
    const float *kk = st.gk + i;
    for (int t = 0; t < w; t++) acc = fmaf(__ldg(&kk[(size_t)t * N]), r(i - h + t), acc);
  }
  return acc;
}

}  // namespace pb
