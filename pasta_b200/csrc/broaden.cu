// broaden.cu -- fused broadening: rotation and instrument profile by
// overlap-save FFT blocks, with the resampling to the observed pixels.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "device.cuh"
#include "fft.cuh"
#include "kernels.h"

namespace pb {

struct BroadenItem {
  int e, pair, m, hg, V, s0, s1, j0, j1;
  bool has1;
};

// the work item (evaluation e, block pair), or false when it has nothing to do
__device__ __forceinline__ bool broaden_item(const EvalBatch &b, int e, int pair, BroadenItem &w) {
  w.e = e;
  w.pair = pair;
  const EvalPrep &P = b.prep[e];
  if (P.status || !P.fused || 2 * pair >= P.nblk) return false;
  w.m = P.m;
  w.hg = P.hg;
  w.V = FFTN - (w.m - 1) - 2 * w.hg;
  w.s0 = P.o_lo + 2 * pair * (w.V - 1);
  w.s1 = w.s0 + (w.V - 1);
  w.has1 = 2 * pair + 1 < P.nblk;
  // input t of a block is synth pixel (s - hg - hw + t) for the rotation,
  // (s - hg + t) for the identity
  const int shift = w.m > 1 ? w.hg + (w.m - 1) / 2 : w.hg;
  w.j0 = w.s0 - shift;
  w.j1 = w.s1 - shift;
  return true;
}

// The items of a CTA (item = e * max_pairs + pair) come in runs of ic
// consecutive items (mostly neighbouring block pairs of one evaluation, so
// their metadata and the overlap of their inputs are still in cache): run r
// of the CTA is items [ic R, ic R + ic) with R = blockIdx.x + r gridDim.x.
struct ItemCursor {
  int e, pair, k, ic, mp, E;
  long long run;
  __device__ __forceinline__ void set_run() {
    const long long item = run * ic;
    e = (int)(item / mp);
    pair = (int)(item % mp);
    k = 0;
  }
  __device__ __forceinline__ void init(const EvalBatch &b, int run_len) {
    mp = b.max_pairs;
    E = b.E;
    ic = run_len;
    run = blockIdx.x;
    set_run();
  }
  __device__ __forceinline__ void advance() {
    if (++k < ic) {
      if (++pair >= mp) {
        pair = 0;
        e++;
      }
    } else {
      run += gridDim.x;
      set_run();
    }
  }
  __device__ __forceinline__ bool done() const { return e >= E; }
  // move to the first item with work at or after the current one
  __device__ __forceinline__ void settle(const EvalBatch &b) {
    BroadenItem w;
    while (!done() && !broaden_item(b, e, pair, w)) advance();
  }
};

// The 2 x 16 inputs of this thread for item w: block input j = 128 n1 + t
// is synth pixel j0 + j of the interpolated row (zero outside [i_lo, i_hi)).
// Interior item pairs (both blocks inside the window, the common case) load
// without per-element bounds tests.
__device__ __forceinline__ void broaden_inputs(const EvalBatch &b, const BroadenItem &w, const EvalPrep &P,
                                               float (&x0)[16], float (&x1)[16]) {
  const float *row = b.bufA + (size_t)w.e * b.stride;
  const int ilo = P.i_lo, ihi = P.i_hi;
  if (w.has1 && w.j0 >= ilo && w.j1 + FFTN <= ihi) {
    const float *r0 = row + w.j0 + (int)threadIdx.x, *r1 = row + w.j1 + (int)threadIdx.x;
#pragma unroll
    for (int n1 = 0; n1 < 16; n1++) {
      x0[n1] = __ldg(r0 + 128 * n1);
      x1[n1] = __ldg(r1 + 128 * n1);
    }
    return;
  }
#pragma unroll
  for (int n1 = 0; n1 < 16; n1++) {
    const int g0 = w.j0 + 128 * n1 + (int)threadIdx.x, g1 = w.j1 + 128 * n1 + (int)threadIdx.x;
    x0[n1] = (g0 >= ilo && g0 < ihi) ? __ldg(row + g0) : 0.0f;
    x1[n1] = (w.has1 && g1 >= ilo && g1 < ihi) ? __ldg(row + g1) : 0.0f;
  }
}

constexpr int BT = F2_T;      // threads of k_broaden
constexpr int BR_RUN = 8;     // longest run of consecutive items a CTA takes
// dynamic shared memory (bytes): exchange buffers 1 and 2 (buffer 2 also
// holds the rotation outputs, buffer 1 the outputs of the instrument taps),
// twiddles of pass 2, the fixed instrument taps
constexpr int BR_S1 = 0, BR_S2 = BR_S1 + F2_S1 * 8, BR_T2 = BR_S2 + F2_S2 * 8, BR_GK = BR_T2 + 16 * 8 * 8,
              BR_SMEM = BR_GK + 512 * 4;

// Resampling of an item's observed pixels [q0, q2) (the left synth pixel of
// [q0, q1) in block 0, of [q1, q2) in block 1) from the final outputs in
// shared memory (block 1's 2048 floats after block 0's), with the wavelength
// kind fixed at compile time.  The float indices come from the star's table
// (a star's particles share it; the item prefetched its range into L1 before
// the transforms); each thread issues the loads of EU pixels before their
// arithmetic.  The floor of an index is the low word of index + 2^52 rounded
// down: no conversion through the narrow XU pipe, and no branch in full
// rounds.  About 20 instructions a pixel (30 with floor(), per-pixel branches
// and a select of each block's arrays), a quarter of the kernel's.
template <int KIND>
__device__ __forceinline__ void resample_item(const Resampler &R, float *y, const float *ob, int q0, int q1, int q2,
                                              int s0, int V) {
  constexpr int EU = 8;
  const int off1 = 2048 - (V - 1);  // from block 0's place of a synth pixel to block 1's
  auto one = [&](int i, double fx) {
    int j;
    float w;
    if (KIND == WL_NONUNI) {
      const ResPos q = R.pos(i);
      j = q.j;
      w = q.w;
    } else {
      const double idx = KIND == WL_LOG ? fx + R.shift_log : __dadd_rn(__dmul_rn(R.shift_factor, fx), R.lin_offset);
      j = max(__double2loint(__dadd_rd(idx, 4503599627370496.0)), 0);  // negative for idx < 0
      w = (float)idx - (float)j;
    }
    // in range by construction of bnd; the minimum only keeps the read inside the buffer
    const unsigned u = min((unsigned)(j - s0 + (i >= q1 ? off1 : 0)), (unsigned)(2048 + V - 2));
    y[i] = resample_value(w, ob[u], ob[u + 1]);
  };
  int i0 = q0 + (int)threadIdx.x;
  for (int base = q0; base + EU * BT <= q2; base += EU * BT, i0 += EU * BT) {
    double fx[EU];
#pragma unroll
    for (int r = 0; r < EU; r++) fx[r] = KIND == WL_NONUNI ? 0.0 : __ldg(&R.fidx[i0 + r * BT]);
#pragma unroll
    for (int r = 0; r < EU; r++) one(i0 + r * BT, fx[r]);
  }
  double fx[EU];
#pragma unroll
  for (int r = 0; r < EU; r++) fx[r] = KIND == WL_NONUNI || i0 + r * BT >= q2 ? 0.0 : __ldg(&R.fidx[i0 + r * BT]);
#pragma unroll
  for (int r = 0; r < EU; r++)
    if (i0 + r * BT < q2) one(i0 + r * BT, fx[r]);
}

// the pass-1 twiddle W_2048^(t k1) of this thread from W^t, W^2t, W^4t and
// W^8t (table values, computed in double on the host) by at most three
// products
__device__ __forceinline__ cf tw_pass1(int k1, const cf &w1, const cf &w2, const cf &w4, const cf &w8) {
  cf r = (k1 & 1) ? w1 : cf{1.0f, 0.0f};
  if (k1 & 2) r = (k1 & 1) ? cmul(r, w2) : w2;
  if (k1 & 4) r = (k1 & 3) ? cmul(r, w4) : w4;
  if (k1 & 8) r = (k1 & 7) ? cmul(r, w8) : w8;
  return r;
}

// One work item = two overlap-save blocks of one evaluation.  Block k yields
// V = 2048 - (m - 1) - 2 hg final outputs starting at s_k = o_lo + k (V - 1):
// the rotation outputs [s - hg, s + V + hg) come from one overlap-save block
// of 2048 inputs (the reference uses overlap-add, convolve_rv.rs:121-157;
// both are the same linear convolution), and the instrument profile is then
// applied from shared memory.  Block k owns synth pixels [s_k, s_k + V - 1);
// its last output is the partner j + 1 of its last owned pixel j.  The two
// real blocks ride in the real and imaginary parts of one complex FFT (the
// kernel is real, so the two products separate after the inverse).  Rotation
// outputs outside [0, N) are zero, like the reference's cropped segment.
// With the identity rotation the FFT is skipped.  Away from the grid ends
// the instrument Gaussian acts on rotation outputs that are all inside
// [0, N), where rotation-then-Gaussian is one convolution with the combined
// kernel: the spectra are multiplied (H x G) and the taps are skipped.
//
// Epilogue: either the owned synth pixels go to row B, or (chi2 batches,
// EvalPrep::epi) the block resamples the observed pixels whose left synth
// pixel it owns (EvalBatch::bnd lists them per block) from shared memory and
// writes the model at the observed pixels to row B; the synth row never
// reaches memory.  An item's float indices are prefetched into L1 before its
// transforms; a CTA takes runs of consecutive items (ItemCursor).
//
// What bounds it: instruction issue (55% of cycles) and the latency of its
// inputs and spectra.  2,000 evaluations of 80,000 pixels with 60,000 observed
// pixels (ncu): 435 M warp instructions and 695 us with floor() and a branch
// per resampled pixel, a swizzle computed per exchange access and the 1/2048
// applied to every output; 374 M and 621 us now.
__global__ void __launch_bounds__(BT, 5) k_broaden(DevGrid G, EvalBatch b, const float2 *__restrict__ tw, int run_len) {
  extern __shared__ __align__(16) unsigned char br_smem[];
  float2 *S1 = reinterpret_cast<float2 *>(br_smem + BR_S1);
  float2 *S2 = reinterpret_cast<float2 *>(br_smem + BR_S2);
  float2 *T2 = reinterpret_cast<float2 *>(br_smem + BR_T2);
  float *gks = reinterpret_cast<float *>(br_smem + BR_GK);
  const int t = threadIdx.x, N = G.npx;
  // twiddles: T2[k2][n3] = W_128^(n3 k2) in shared memory; W_2048^(t k1)
  // from the four powers of two of W^t in registers
  for (int i = t; i < 16 * 8; i += BT) T2[i] = __ldg(&tw[(16 * (i & 7) * (i >> 3)) & (FFTN - 1)]);
  cf tw1, tw2, tw4, tw8;
  {
    const float2 a = __ldg(&tw[t]), c = __ldg(&tw[2 * t]), d = __ldg(&tw[4 * t]), f = __ldg(&tw[8 * t]);
    tw1 = cf{a.x, a.y};
    tw2 = cf{c.x, c.y};
    tw4 = cf{d.x, d.y};
    tw8 = cf{f.x, f.y};
  }
  ItemCursor cur;
  cur.init(b, run_len);
  cur.settle(b);
  const int k1p = t >> 3, n3p = t & 7;  // pass-2 role of this thread
  float2 *X2 = S2 + f2_a2(k1p, n3p);    // exchange 2 as passes 2 see it: f2_a2(k1p + 16 k2, n3p) = that + 128 k2
  const int a3 = f2_a2(t, 0);             // as pass 3 sees it: f2_a2(t + 128 h, n3) = (f2_a2(t, 0) ^ n3) + 1024 h
  int gk_star = -1;                       // star whose instrument taps are in gks
  while (!cur.done()) {
    ItemCursor nxt = cur;
    nxt.advance();
    nxt.settle(b);
    BroadenItem w;
    broaden_item(b, cur.e, cur.pair, w);
    const int e = w.e, pair = w.pair, m = w.m, hg = w.hg, V = w.V, s0 = w.s0, s1 = w.s1;
    const bool has1 = w.has1;
    const EvalPrep &P = b.prep[e];
    const int nblk = P.nblk, ohi = P.o_hi;
    const DevStar &st = b.stars[P.star];
    const bool fixedk = hg > 0 && st.disp_kind == DISP_FIXED;
    const int gw = 2 * hg + 1;
    int q0 = 0, q1 = 0, q2 = 0;
    if (P.epi) {
      const int *bd = b.bnd + (size_t)e * b.bnd_stride + 2 * pair;
      q0 = bd[0];
      q1 = bd[1];
      q2 = has1 ? bd[2] : q1;
    }
    float in0[16], in1[16];
    broaden_inputs(b, w, P, in0, in1);
    if (P.epi && G.wl_kind != WL_NONUNI) {  // the float indices the resampling reads: into L1 meanwhile
      const double *fq = st.fidx + q0;
      for (int l = t; l * 16 < q2 - q0; l += BT) asm volatile("prefetch.global.L1 [%0];" ::"l"(fq + 16 * l));
    }
    const int e_last = min((has1 ? s1 : s0) + V, ohi);
    const bool fold = fixedk && m > 1 && st.gspec != nullptr && b.HG != nullptr && s0 - hg >= 0 && e_last + hg <= N;
    __syncthreads();  // the last item's epilogue is done with the shared buffers
    if (fixedk && !fold && P.star != gk_star) {  // the taps are applied from shared memory (edge blocks)
      for (int k = t; k < gw; k += BT) gks[k] = __ldg(&st.gk[k]);
      gk_star = P.star;
    }
    float *ob0, *ob1;  // final outputs u in [0, V) of the two blocks
    if (m > 1) {
      cf v[16];
#pragma unroll
      for (int n1 = 0; n1 < 16; n1++) v[n1] = cf{in0[n1], in1[n1]};
      // pass 1: DFT-16 over n1, twiddle, exchange 1
      dft16<false>(v);
#pragma unroll
      for (int k1 = 0; k1 < 16; k1++) {
        const cf z = k1 ? cmul(v[k1], tw_pass1(k1, tw1, tw2, tw4, tw8)) : v[k1];
        S1[k1 * F2_XP + t] = make_float2(z.x, z.y);
      }
      __syncthreads();
      // pass 2: DFT-16 over n2, twiddle, exchange 2
#pragma unroll
      for (int n2 = 0; n2 < 16; n2++) {
        const float2 z = S1[k1p * F2_XP + 8 * n2 + n3p];
        v[n2] = cf{z.x, z.y};
      }
      dft16<false>(v);
#pragma unroll
      for (int k2 = 0; k2 < 16; k2++) {
        const cf z = k2 ? cmul_tw<false>(v[k2], T2[k2 * 8 + n3p]) : v[k2];
        X2[128 * k2] = make_float2(z.x, z.y);
      }
      __syncthreads();
      // pass 3 (DFT-8 over n3), the spectrum product, and the inverse DFT-8
      // over k3, for c = t and t + 128; each thread rewrites the slots it read
      const float2 *H = (fold ? b.HG : b.H) + (size_t)e * 1025;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int c = t + 128 * h;
        cf u[8];
        float2 hk[8];
        // bins k = c + 256 k3 (c < 256): k < 1024 below k3 = 4, k > 1024
        // above it (conjugate of bin 2048 - k); k3 = 4 is bin 1024 for c = 0
#pragma unroll
        for (int k3 = 0; k3 < 8; k3++) {
          const int k = c + 256 * k3;
          if (k3 < 4) {
            hk[k3] = __ldg(&H[k]);
          } else if (k3 > 4) {
            hk[k3] = __ldg(&H[FFTN - k]);
            hk[k3].y = -hk[k3].y;
          } else {
            hk[k3] = __ldg(&H[c == 0 ? 1024 : FFTN - k]);
            if (c != 0) hk[k3].y = -hk[k3].y;
          }
        }
#pragma unroll
        for (int n3 = 0; n3 < 8; n3++) {
          const float2 z = S2[(a3 ^ n3) + 1024 * h];
          u[n3] = cf{z.x, z.y};
        }
        dft8<false>(u);
#pragma unroll
        for (int k3 = 0; k3 < 8; k3++) u[k3] = cmul(u[k3], cf{hk[k3].x, hk[k3].y});
        dft8<true>(u);
#pragma unroll
        for (int n3 = 0; n3 < 8; n3++) S2[(a3 ^ n3) + 1024 * h] = make_float2(u[n3].x, u[n3].y);
      }
      __syncthreads();
      // inverse pass 2: conjugate twiddle, DFT-16 over k2, exchange 1
#pragma unroll
      for (int k2 = 0; k2 < 16; k2++) {
        const float2 z = X2[128 * k2];
        v[k2] = k2 ? cmul_tw<true>(cf{z.x, z.y}, T2[k2 * 8 + n3p]) : cf{z.x, z.y};
      }
      dft16<true>(v);
#pragma unroll
      for (int n2 = 0; n2 < 16; n2++) S1[k1p * F2_XP + 8 * n2 + n3p] = make_float2(v[n2].x, v[n2].y);
      __syncthreads();
      // inverse pass 1: conjugate twiddle, DFT-16 over k1 -> 2048 x output 128 n1 + t
#pragma unroll
      for (int k1 = 0; k1 < 16; k1++) {
        const float2 z = S1[k1 * F2_XP + t];
        v[k1] = k1 ? cmul_tw<true>(cf{z.x, z.y}, [&] {
          const cf q = tw_pass1(k1, tw1, tw2, tw4, tw8);
          return make_float2(q.x, q.y);
        }()) : cf{z.x, z.y};
      }
      dft16<true>(v);
      // FFT index i = 128 n1 + t holds rotation output (s - hg) + (i - (m - 1))
      const int base = m - 1;
      if (fold) {  // final output u = i - base - 2 hg
        ob0 = reinterpret_cast<float *>(S2);
        ob1 = ob0 + 2048;
#pragma unroll
        for (int n1 = 0; n1 < 16; n1++) {
          const int u = 128 * n1 + t - base - 2 * hg;  // at most 2047 - base - 2 hg = V - 1
          if (u >= 0) {
            ob0[u] = v[n1].x;
            ob1[u] = v[n1].y;
          }
        }
      } else {  // rotation outputs r = i - base, zero outside the grid
        const int r0 = s0 - hg, r1 = s1 - hg;
#pragma unroll
        for (int n1 = 0; n1 < 16; n1++) {
          const int r = 128 * n1 + t - base;
          if (r >= 0) {
            const int i0 = r0 + r, i1 = r1 + r;
            S2[r] = make_float2((i0 >= 0 && i0 < N) ? v[n1].x : 0.0f, (i1 >= 0 && i1 < N) ? v[n1].y : 0.0f);
          }
        }
      }
    } else {  // identity rotation: the inputs are the rotation outputs r = j
#pragma unroll
      for (int n1 = 0; n1 < 16; n1++) S2[128 * n1 + t] = make_float2(in0[n1], in1[n1]);
    }
    __syncthreads();
    if (!fold) {  // instrument taps from the rotation outputs in S2 into buffer 1
      ob0 = reinterpret_cast<float *>(S1);
      ob1 = ob0 + 2048;
      for (int u = t; u < V; u += BT) {
        const int i0 = s0 + u, i1 = s1 + u;
        float v0, v1;
        if (hg == 0) {
          const float2 x = S2[u];
          v0 = x.x;
          v1 = x.y;
        } else if (fixedk) {  // g[i] = sum_k gk[k] r[i + hg - k]; r[i] sits at i - s + hg
          float a0 = 0.0f, a1 = 0.0f;
          for (int k = 0; k < gw; k++) {
            const float g = gks[k];
            const float2 x = S2[u + 2 * hg - k];
            a0 = fmaf(g, x.x, a0);
            a1 = fmaf(g, x.y, a1);
          }
          v0 = a0;
          v1 = a1;
        } else {
          // Per-pixel kernels (tap-major; pixels within hg of the grid's ends
          // pass through, convolve_rv.rs:213-233), sums in tap order.  Bound by
          // the taps' loads from L2: the two blocks' pixels together (one value
          // pair per tap, 16 loads in flight) took the kernel from 1.26 to
          // 0.86 ms for 1,000 evaluations of 80,000 pixels and 17 taps (661 M
          // to 498 M warp instructions); unrolled by 3 or 6 1.06-1.08 ms, by 4
          // 0.94 ms.  Passed-through pixels form a sum that is not used, from
          // taps inside the table.
          const bool p0 = i0 < hg || i0 >= N - hg, p1 = !has1 || i1 < hg || i1 >= N - hg;
          const float *g0 = st.gk + (p0 ? 0 : i0);
          const int d = (p1 ? 0 : i1) - (p0 ? 0 : i0);
          float a0 = 0.0f, a1 = 0.0f;
#pragma unroll 8
          for (int k = 0; k < gw; k++) {
            const float2 x = S2[u + k];
            a0 = fmaf(__ldg(g0), x.x, a0);
            a1 = fmaf(__ldg(g0 + d), x.y, a1);
            g0 += N;
          }
          const float2 mid = S2[u + hg];
          v0 = p0 ? mid.x : a0;
          v1 = p1 ? (has1 ? mid.y : 0.0f) : a1;
        }
        ob0[u] = v0;
        ob1[u] = v1;
      }
      __syncthreads();
    }
    float *y = b.bufB + (size_t)e * b.stride;
    if (P.epi) {
      // observed pixels [q0, q2) have their left synth pixel in this item's
      // blocks; the boundary between them is q1
      const Resampler R = make_resampler(G, st, P, nullptr, nullptr);
      if (R.kind == WL_LOG) resample_item<WL_LOG>(R, y, ob0, q0, q1, q2, s0, V);
      else if (R.kind == WL_LIN) resample_item<WL_LIN>(R, y, ob0, q0, q1, q2, s0, V);
      else resample_item<WL_NONUNI>(R, y, ob0, q0, q1, q2, s0, V);
    } else {
      // owned pixels; the last block also writes its final output
      const int n0 = 2 * pair + 1 == nblk ? V : V - 1, n1 = 2 * pair + 2 == nblk ? V : V - 1;
      for (int u = t; u < V; u += BT) {
        const int i0 = s0 + u, i1 = s1 + u;
        if (u < n0 && i0 < ohi) y[i0] = ob0[u];
        if (has1 && u < n1 && i1 < ohi) y[i1] = ob1[u];
      }
    }
    cur = nxt;
  }
}

void launch_broaden(const DevGrid &G, const EvalBatch &b, const float2 *tw, cudaStream_t s) {
  if (b.E <= 0 || b.max_pairs <= 0) return;
  const size_t smem = BR_SMEM;
  static int per_sm[64] = {};  // resident CTAs per SM, per device
  int dev = 0;
  cudaGetDevice(&dev);
  int fit = 5;
  if (dev >= 0 && dev < 64) {
    if (!per_sm[dev]) {
      cudaFuncSetAttribute(k_broaden, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      int n = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_broaden, BT, smem) != cudaSuccess || n < 1) n = 1;
      per_sm[dev] = n;
    }
    fit = per_sm[dev];
  }
  const long long total = (long long)b.E * b.max_pairs;
  long long grid = (long long)num_sms() * fit;  // persistent: the CTAs that fit at once
  if (grid > total) grid = total;
  // runs of up to BR_RUN consecutive items, as long as every CTA still gets
  // 16 runs or more (small batches keep single items spread over all CTAs)
  int run_len = (int)std::min<long long>(BR_RUN, std::max<long long>(1, total / (grid * 16)));
  if (const char *rl = getenv("PASTA_BR_RUN")) run_len = std::max(1, atoi(rl));
  k_broaden<<<(unsigned)grid, BT, smem, s>>>(G, b, tw, run_len);
  count_launch();
}

}  // namespace pb
