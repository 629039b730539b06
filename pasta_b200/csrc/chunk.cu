// chunk.cu -- chunked-polynomial continuum: the fit with its chi2, and the
// continuum built from given coefficients.
#include <cuda_runtime.h>

#include "common.cuh"
#include "device.cuh"
#include "kernels.h"

namespace pb {


// Legendre P_0..P_{K-1} at x (f32, the host Gram uses the same recurrence)
template <int K>
__device__ __forceinline__ void legendre(float x, float (&P)[K]) {
  P[0] = 1.0f;
  if (K > 1) P[1] = x;
#pragma unroll
  for (int k = 1; k + 1 < K; k++) P[k + 1] = leg_step(leg_a(k), leg_c(k), x, P[k], P[k - 1]);
}

template <int K>
__device__ __forceinline__ float poly_eval(const float *coef, float x) {
  float P[K];
  legendre<K>(x, P);
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < K; k++) s = fmaf(coef[k], P[k], s);
  return s;
}

// ChunkFitter::fit_continuum + compute_chi2_from_chunks
// (continuum_fitting.rs:216-226, 280-360, 382-396), one CTA per evaluation.
// First every chunk's moments: the unweighted least-squares polynomial of
// flux/model over the chunk is the projection onto the chunk's polynomial
// space, solved here in a Legendre basis with the FP64 Cholesky factor of its
// Gram matrix (the same space as the reference's monomial SVD, far better
// conditioned).  Then every chunk section's chi2 from the polynomials in
// monomial form, reading the model row a second time while it is still in
// L2; the sections are added in chunk order in FP64 / (N - 100).
//
// Divisions are multiplications by the reciprocal (at most 2 ulp; the sums
// run over thousands of such terms).  The fast reciprocal takes a divisor
// below 2^-126 (a variance in faint absolute units) as zero, so the walks also
// come with divisions (DIV): stars with such variances take them for the
// residuals from the start (faint_star), and a piece whose sum comes out
// infinite or NaN is formed again with them if one of its divisors is that
// small (any other cause gives the same sum either way).  A chi2 call of 2,000
// evaluations of 60,000 pixels, degree 5: 0.91 ms; of a star with variances
// around 1e-40 1.01 ms and with a NaN pixel in every piece 1.11 ms (1.36 and
// 2.06 ms with every piece whose sum is not finite formed again pixel by pixel).
//
// Order of the sums: a range of pixels is cut into blocks of 32 x CU pixels;
// lane l of the warp that takes a block adds its pixels l + 32 u, u < CU, in
// f32 and that partial in FP64 (one f32 -> f64 conversion per moment and CU
// pixels: the conversions share the narrow XU pipe with the reciprocals).
//
// What bounds it: instruction issue and the latency of its loads.  Two blocks
// are worked at a time as the two halves of packed f32x2 operations (the same
// roundings as one block after the other), loads go through fixed offsets
// from one address per array, two evaluations of a star share the reads of
// its arrays and the Legendre values, and the blocks of a chunk are spread
// over CHUNK_PIECES warps, so that spectra with fewer chunks than warps keep
// all warps busy.  4,000 evaluations of 60,000 pixels, degree 5 (ncu): 654 M
// warp instructions and 914 us with one pixel per operation, 250 M and 655 us
// now; 40 evaluations of 15,000 pixels, degree 8: 53 -> 31 us.
constexpr int CHUNK_PIECES = 4;
// pixels of a lane in a block: 8 up to degree 5, 4 above
template <int K>
__host__ __device__ constexpr int chunk_cu() {
  return K <= 6 ? 8 : 4;
}
// resident CTAs the registers are sized for
__host__ __device__ constexpr int chunk_ctas(int k, int ne) { return k <= 8 ? (ne == 1 ? 3 : 2) : 2; }

__device__ __forceinline__ float2 dup2(float a) { return make_float2(a, a); }

__device__ __forceinline__ float rcp_ftz(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
// 1 / x of two pixels, with divisors below 2^-126 taken as zero
__device__ __forceinline__ float2 rcp2(float2 x) { return make_float2(rcp_ftz(x.x), rcp_ftz(x.y)); }

// a / b of two pixels, any b that is not 0
__device__ __forceinline__ float2 div2(float2 a, float2 b) { return make_float2(__fdividef(a.x, b.x), __fdividef(a.y, b.y)); }

// whether one of p[i0, i1) is not 0 and below 2^-126, by a warp
__device__ __forceinline__ bool any_subnormal(const float *__restrict__ p, int i0, int i1, int lane) {
  bool any = false;
#pragma unroll 8
  for (int i = i0 + lane; i < i1; i += 32) {
    const float a = fabsf(__ldg(p + i));
    any |= a > 0.0f && a < 1.17549435e-38f;
  }
  return __any_sync(0xffffffffu, any);
}
// whether this thread's sample of the star's variances (256 over the spectrum,
// whatever the number of threads) is near or below 2^-126
__device__ __forceinline__ bool faint_star(const DevStar &st) {
  const int t = threadIdx.x;
  if (t >= 256) return false;
  const float v = fabsf(__ldg(st.var + (long long)t * st.n_obs / 256));
  return v > 0.0f && v < 1e-35f;
}

// Two blocks' loads for one lane: (first block, second block) at the lane's
// u-th pixel.  INNER: every pixel of both blocks exists.  Otherwise pixels
// past the range's end (and the second of an odd number of blocks) read the
// last pixel and mask() replaces what comes of them.
template <bool INNER>
struct PairLoad {
  int i, i2;      // the lane's first pixel in the two blocks
  int end, end2;  // ends of the pixels that exist in them (unused when INNER)
  __device__ __forceinline__ float2 operator()(const float *__restrict__ p, int u) const {
    if constexpr (INNER) return make_float2(__ldg(p + i + 32 * u), __ldg(p + i2 + 32 * u));
    return make_float2(__ldg(p + min(i + 32 * u, end - 1)), __ldg(p + min(i2 + 32 * u, end - 1)));
  }
  __device__ __forceinline__ float2 mask(float2 x, int u) const {
    if constexpr (INNER) return x;
    return make_float2(i + 32 * u < end ? x.x : 0.0f, i2 + 32 * u < end2 ? x.y : 0.0f);
  }
};
// The blocks [j0, j1) of [a0, a1) (block j starts at a0 + 32 CU j), two at a time
template <int CU, class Body>
__device__ __forceinline__ void walk_pairs(int a0, int a1, int j0, int j1, int lane, const Body &body) {
  constexpr int B = 32 * CU;
  int j = j0;
  for (; j + 2 <= j1 && a0 + B * (j + 2) <= a1; j += 2) {
    const int i = a0 + B * j + lane;
    body(PairLoad<true>{i, i + B, 0, 0});
  }
  for (; j < j1; j += 2) {
    const int i = a0 + B * j + lane;
    body(PairLoad<false>{i, i + B, a1, j + 1 < j1 ? a1 : 0});
  }
}
__device__ __forceinline__ int blocks_of(int a0, int a1, int per) { return a1 > a0 ? (a1 - a0 + per - 1) / per : 0; }

// Adds the lane's share of sum_i P_k(x_i) flux_i / model_i over the blocks
// [j0, j1) of [a0, a1) to z, for NE models of one star.
template <int K, int NE, bool DIV>
__device__ __forceinline__ void moments_walk(const float *__restrict__ flux, const float *const (&mod)[NE],
                                             const float *__restrict__ xs, int a0, int a1, int j0, int j1, int lane,
                                             double (&z)[NE][K]) {
  constexpr int CU = chunk_cu<K>();
  walk_pairs<CU>(a0, a1, j0, j1, lane, [&](const auto &ld) {
    float2 zp[NE][K];
#pragma unroll
    for (int n = 0; n < NE; n++)
#pragma unroll
      for (int k = 0; k < K; k++) zp[n][k] = dup2(0.0f);
#pragma unroll
    for (int u0 = 0; u0 < CU; u0 += 4) {
      float2 fl[4], md[NE][4], xf[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        fl[u] = ld(flux, u0 + u);
        xf[u] = ld(xs, u0 + u);
#pragma unroll
        for (int n = 0; n < NE; n++) md[n][u] = ld(mod[n], u0 + u);
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const float2 f = ld.mask(fl[u], u0 + u);
        [[maybe_unused]] const float2 x = xf[u];
        [[maybe_unused]] float2 y[NE];
#pragma unroll
        for (int n = 0; n < NE; n++) {
          if constexpr (DIV) {
            y[n] = ld.mask(div2(f, md[n][u]), u0 + u);
            zp[n][0] = __fadd2_rn(zp[n][0], y[n]);
          } else {
            const float2 r = ld.mask(rcp2(md[n][u]), u0 + u);
            if constexpr (K == 1) {
              zp[n][0] = __ffma2_rn(f, r, zp[n][0]);
            } else {
              y[n] = __fmul2_rn(f, r);
              zp[n][0] = __fadd2_rn(zp[n][0], y[n]);
            }
          }
        }
        if constexpr (K > 1) {
          float2 p0 = dup2(1.0f), p1 = x;
#pragma unroll
          for (int k = 1; k < K; k++) {
#pragma unroll
            for (int n = 0; n < NE; n++) zp[n][k] = __ffma2_rn(p1, y[n], zp[n][k]);
            if (k + 1 < K) {  // leg_step of both pixels
              const float2 p2 = __ffma2_rn(__fmul2_rn(dup2(leg_a(k)), x), p1, __fmul2_rn(dup2(-leg_c(k)), p0));
              p0 = p1;
              p1 = p2;
            }
          }
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NE; n++)
#pragma unroll
      for (int k = 0; k < K; k++) z[n][k] += (double)zp[n][k].x + (double)zp[n][k].y;
  });
}

// Sums of K values per lane over the warp, each lane ending with the sum of
// value chunk_slot<K>(lane): the lanes exchange halves of the values first,
// so a step moves half of what the step before moved.
template <int K>
__device__ __forceinline__ int chunk_slot(int lane) {
  return K <= 8 ? ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1) : lane >> 1;
}
template <int K>
__device__ __forceinline__ double warp_sum_vec(const double (&z)[K], int lane) {
  constexpr int NV = K <= 8 ? 8 : 16;
  double v[NV];
#pragma unroll
  for (int k = 0; k < NV; k++) v[k] = k < K ? z[k] : 0.0;
  int m = 16;
#pragma unroll
  for (int n = NV / 2; n >= 1; n >>= 1) {
    const bool up = lane & m;
#pragma unroll
    for (int i = 0; i < n; i++) {
      const double send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
    }
    m >>= 1;
  }
  for (; m >= 1; m >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], m);
  return v[0];
}

// Piece p of chunk c.  The chunk's pixels below the previous chunk's stop take
// the upper-chunk coordinate xb; the pieces cut the blocks of both ranges,
// taken one after the other, at even block numbers (pairs of blocks).
template <int K>
struct MomentPiece {
  int lo, split, hi, bb, ba, nb, g0, g1;
  __device__ __forceinline__ MomentPiece(const DevStar &st, int c, int p) {
    constexpr int PER = 32 * chunk_cu<K>();
    lo = st.cstart[c];
    hi = st.cstop[c];
    const int prev = c > 0 ? st.cstop[c - 1] : -1;
    split = c > 0 ? min(max(prev, lo), hi) : lo;
    bb = blocks_of(lo, split, PER);
    ba = blocks_of(split, hi, PER);
    nb = (bb + 1) / 2;
    const int n = nb + (ba + 1) / 2;
    g0 = n * p / CHUNK_PIECES;
    g1 = n * (p + 1) / CHUNK_PIECES;
  }
  template <int NE, bool DIV>
  __device__ __forceinline__ void sums(const DevStar &st, const float *const (&mod)[NE], int lane, double (&t)[NE]) const {
    double z[NE][K];
#pragma unroll
    for (int q = 0; q < NE; q++)
#pragma unroll
      for (int k = 0; k < K; k++) z[q][k] = 0.0;
    moments_walk<K, NE, DIV>(st.flux, mod, st.xb, lo, split, 2 * min(g0, nb), min(2 * min(g1, nb), bb), lane, z);
    moments_walk<K, NE, DIV>(st.flux, mod, st.xa, split, hi, 2 * max(g0 - nb, 0), min(2 * max(g1 - nb, 0), ba), lane, z);
#pragma unroll
    for (int q = 0; q < NE; q++) t[q] = warp_sum_vec<K>(z[q], lane);
  }
};

// The lane's slot of the moments of a piece whose sums t came out infinite or
// NaN: formed with divisions if a model pixel is that small.  Not inlined, so
// that it takes no registers from the common path.
template <int K>
__device__ __noinline__ double chunk_moments_again(const DevStar &st, const float *model, int c, int p, double t) {
  constexpr int PER = 32 * chunk_cu<K>();
  const int lane = threadIdx.x & 31;
  const MomentPiece<K> P(st, c, p);
  const int i0 = P.g0 < P.nb ? P.lo + 2 * PER * P.g0 : P.split + 2 * PER * (P.g0 - P.nb);
  const int i1 = P.g1 < P.nb ? P.lo + 2 * PER * P.g1 : P.g1 == P.nb ? P.split : min(P.hi, P.split + 2 * PER * (P.g1 - P.nb));
  if (!any_subnormal(model, i0, i1, lane)) return t;
  const float *const mod[1] = {model};
  double s[1];
  P.template sums<1, true>(st, mod, lane, s);
  return s[0];
}

// Moments of piece p of chunk c by one warp, for NE models: the lane's slot
// of them (chunk_slot).
template <int K, int NE>
__device__ __forceinline__ void chunk_moments(const DevStar &st, const float *const (&mod)[NE], int c, int p, int lane,
                                              double (&t)[NE]) {
  MomentPiece<K>(st, c, p).template sums<NE, false>(st, mod, lane, t);
#pragma unroll
  for (int q = 0; q < NE; q++)
    if (!__all_sync(0xffffffffu, isfinite(t[q]))) t[q] = chunk_moments_again<K>(st, mod[q], c, p, t[q]);
}

// Monomial coefficients of the Legendre polynomials, T[k][j] = coefficient
// of x^j in P_k, from (k + 1) P_{k+1} = (2k + 1) x P_k - k P_{k-1} (dyadic
// rationals, exact in double up to degree 15).
struct LegMono {
  double c[MAX_P1][MAX_P1];
};
constexpr LegMono make_leg_mono() {
  LegMono t{};
  t.c[0][0] = 1.0;
  t.c[1][1] = 1.0;
  for (int k = 1; k + 1 < MAX_P1; k++)
    for (int j = 0; j < MAX_P1; j++)
      t.c[k + 1][j] = ((2 * k + 1) * (j > 0 ? t.c[k][j - 1] : 0.0) - k * t.c[k - 1][j]) / (k + 1);
  return t;
}
__constant__ LegMono c_leg_mono = make_leg_mono();

// FP64 Cholesky solve G a = z of chunk c, and the polynomial sum_k
// a_k P_k(x) as monomial coefficients (FP64), rounded to f32 for Horner
// evaluation; the Legendre coefficients also to b.params when requested.
template <int K>
__device__ __forceinline__ void chunk_coefs(const EvalBatch &b, const DevStar &st, int e, int c, const double *z, float *m) {
  // unrolled, so that the factor's loads do not wait for the substitution
  const double *__restrict__ L = st.chol + (size_t)c * K * K;
  double a[K];
#pragma unroll
  for (int k = 0; k < K; k++) a[k] = z[k];
#pragma unroll
  for (int k = 0; k < K; k++) {
    double t = a[k];
#pragma unroll
    for (int j = 0; j < k; j++) t -= __ldg(&L[k * K + j]) * a[j];
    a[k] = t / __ldg(&L[k * K + k]);
  }
#pragma unroll
  for (int k = K - 1; k >= 0; k--) {
    double t = a[k];
#pragma unroll
    for (int j = k + 1; j < K; j++) t -= __ldg(&L[j * K + k]) * a[j];
    a[k] = t / __ldg(&L[k * K + k]);
  }
  if (b.params) {
    double *par = b.params + (size_t)e * b.param_stride + c * K;
#pragma unroll
    for (int k = 0; k < K; k++) par[k] = a[k];
  }
#pragma unroll
  for (int j = 0; j < K; j++) {
    double s = 0.0;
#pragma unroll
    for (int k = j; k < K; k++) s = fma(a[k], c_leg_mono.c[k][j], s);
    m[j] = (float)s;
  }
}

template <int K>
__device__ __forceinline__ float2 horner2(const float (&a)[K], float2 x) {
  float2 p = dup2(a[K - 1]);
#pragma unroll
  for (int j = K - 2; j >= 0; j--) p = __ffma2_rn(p, x, dup2(a[j]));
  return p;
}

// Adds the lane's share of sum (flux - p model)^2 / var over the blocks [j0,
// j1) of [a0, a1) to acc, p = the current chunk's polynomial, or (BLEND) pv
// fac + cu (1 - fac) of the previous and the current chunk, for NE models of
// one star.  ncc, ncp: the negated coefficients.
template <int K, int NE, bool BLEND, bool DIV>
__device__ __forceinline__ void resid_walk(const DevStar &st, const float *const (&mod)[NE], int a0, int a1, int j0, int j1,
                                           int lane, const float (&ncc)[NE][K], const float (&ncp)[NE][K],
                                           double (&acc)[NE]) {
  constexpr int CU = BLEND ? 2 : chunk_cu<K>(), N = CU < 4 ? CU : 4;
  walk_pairs<CU>(a0, a1, j0, j1, lane, [&](const auto &ld) {
    float2 part[NE];
#pragma unroll
    for (int n = 0; n < NE; n++) part[n] = dup2(0.0f);
#pragma unroll
    for (int u0 = 0; u0 < CU; u0 += N) {
      float2 fl[N], md[NE][N], vr[N], xa[N];
      [[maybe_unused]] float2 xb[N], fc[N];
#pragma unroll
      for (int u = 0; u < N; u++) {
        fl[u] = ld(st.flux, u0 + u);
        vr[u] = ld(st.var, u0 + u);
        xa[u] = ld(st.xa, u0 + u);
        if constexpr (BLEND) {
          xb[u] = ld(st.xb, u0 + u);
          fc[u] = ld(st.fac, u0 + u);
        }
#pragma unroll
        for (int n = 0; n < NE; n++) md[n][u] = ld(mod[n], u0 + u);
      }
#pragma unroll
      for (int u = 0; u < N; u++) {
        [[maybe_unused]] const float2 iv = DIV ? vr[u] : ld.mask(rcp2(vr[u]), u0 + u);
#pragma unroll
        for (int n = 0; n < NE; n++) {
          float2 np;  // minus the continuum
          if constexpr (BLEND) {
            const float2 pv = horner2<K>(ncp[n], xa[u]), cu = horner2<K>(ncc[n], xb[u]);
            np = __ffma2_rn(pv, fc[u], __fmul2_rn(cu, __ffma2_rn(fc[u], dup2(-1.0f), dup2(1.0f))));
          } else {
            np = horner2<K>(ncc[n], xa[u]);
          }
          const float2 r = __ffma2_rn(np, md[n][u], fl[u]);
          if constexpr (DIV) part[n] = __fadd2_rn(ld.mask(div2(__fmul2_rn(r, r), iv), u0 + u), part[n]);
          else part[n] = __ffma2_rn(ld.mask(__fmul2_rn(r, r), u0 + u), iv, part[n]);
        }
      }
    }
#pragma unroll
    for (int n = 0; n < NE; n++) acc[n] += (double)part[n].x + (double)part[n].y;
  });
}

__device__ __forceinline__ double warp_sum_all(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Piece p of chunk section c (continuum_fitting.rs:280-360): chunk 0 alone on
// [50, start_1); chunk c >= 1 blended with chunk c - 1 (sin^2 factor) on
// [start_c, stop_{c-1}), then alone up to start_{c+1} (N - 50 for the last).
template <int K>
struct ResidPiece {
  static constexpr int PB = 64, PA = 32 * chunk_cu<K>();  // pixels per block: blended, alone
  int s0, sp, nx, bb, ba, b0, b1, g0, g1;
  __device__ __forceinline__ ResidPiece(const DevStar &st, int c, int p) {
    s0 = c == 0 ? 50 : st.cstart[c];
    sp = c == 0 ? 50 : st.cstop[c - 1];
    nx = c == st.n_chunks - 1 ? st.n_obs - 50 : st.cstart[c + 1];
    bb = blocks_of(s0, sp, PB);
    ba = blocks_of(sp, nx, PA);
    const int nb = (bb + 1) / 2, na = (ba + 1) / 2;
    b0 = nb * p / CHUNK_PIECES;
    b1 = nb * (p + 1) / CHUNK_PIECES;
    g0 = na * p / CHUNK_PIECES;
    g1 = na * (p + 1) / CHUNK_PIECES;
  }
  template <int NE, bool DIV>
  __device__ __forceinline__ void sums(const DevStar &st, const float *const (&mod)[NE], int lane,
                                       const float (&ncc)[NE][K], const float (&ncp)[NE][K], double (&t)[NE]) const {
    double acc[NE];
#pragma unroll
    for (int n = 0; n < NE; n++) acc[n] = 0.0;
    resid_walk<K, NE, true, DIV>(st, mod, s0, sp, 2 * b0, min(2 * b1, bb), lane, ncc, ncp, acc);
    resid_walk<K, NE, false, DIV>(st, mod, sp, nx, 2 * g0, min(2 * g1, ba), lane, ncc, ncp, acc);
#pragma unroll
    for (int n = 0; n < NE; n++) t[n] = warp_sum_all(acc[n]);
  }
};

// the negated coefficients of section c and of the one before, of NE evaluations
template <int K, int NE>
__device__ __forceinline__ void section_coefs(const float (*cfs)[K], int nc, int c, float (&ncc)[NE][K], float (&ncp)[NE][K]) {
#pragma unroll
  for (int n = 0; n < NE; n++)
#pragma unroll
    for (int k = 0; k < K; k++) {
      ncc[n][k] = -cfs[n * nc + c][k];
      ncp[n][k] = c > 0 ? -cfs[n * nc + c - 1][k] : 0.0f;
    }
}

// The sum of one evaluation over a piece, formed with divisions: of a faint
// star, or where the sum t came out infinite or NaN and a variance is that
// small.  Not inlined (see chunk_moments_again).
template <int K>
__device__ __noinline__ double chunk_resid_div(const DevStar &st, const float *model, int c, int p, const float (*cfs)[K],
                                               bool faint, double t) {
  const int lane = threadIdx.x & 31;
  const ResidPiece<K> P(st, c, p);
  if (!faint && !any_subnormal(st.var, P.s0 + 2 * P.PB * P.b0, min(P.sp, P.s0 + 2 * P.PB * P.b1), lane) &&
      !any_subnormal(st.var, P.sp + 2 * P.PA * P.g0, min(P.nx, P.sp + 2 * P.PA * P.g1), lane))
    return t;
  float ncc[1][K], ncp[1][K];
  section_coefs<K, 1>(cfs, 0, c, ncc, ncp);
  const float *const mod[1] = {model};
  double s[1];
  P.template sums<1, true>(st, mod, lane, ncc, ncp, s);
  return s[0];
}

// whether evaluation e is one for k_chunk_fit<K> to fit; one that failed
// earlier gets NaN and its status
template <int K>
__device__ __forceinline__ bool chunk_eval(const EvalBatch &b, const DevStar &st, int e) {
  if (st.cont_kind != CONT_CHUNK || st.p1 != K) return false;
  int status = b.prep[e].status;
  if (!status && st.cont_bad) status = S_CONTINUUM;
  if (status && threadIdx.x == 0) {
    b.cost[e] = __longlong_as_double(0x7FF8000000000000ll);
    b.status[e] = status;
  }
  return status == 0;
}

// NE evaluations e, e + 1, ... of one star by the CTA
template <int K, int NE, int NW>
__device__ __forceinline__ void chunk_fit(const EvalBatch &b, const DevStar &st, int e, double (*zs)[K], float (*cfs)[K],
                                          double *part, int *faint) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float *mod[NE];
#pragma unroll
  for (int n = 0; n < NE; n++) mod[n] = model_row(b, b.prep[e + n], e + n);
  const int nc = st.n_chunks, items = nc * CHUNK_PIECES, slot = chunk_slot<K>(lane);
  const bool sample = faint_star(st);
  for (int it = warp; it < items; it += NW) {
    double z[NE];
    chunk_moments<K, NE>(st, mod, it / CHUNK_PIECES, it % CHUNK_PIECES, lane, z);
#pragma unroll
    for (int n = 0; n < NE; n++)
      if (slot < K) zs[n * items + it][slot] = z[n];  // the lanes of a slot hold the same sum
  }
  const int f = __syncthreads_or(sample);
  if (threadIdx.x == 0) *faint = f;  // kept out of the registers of the walks
  // (evaluation, chunk) pairs spread over the warps
  for (int i = lane * NW + warp; i < NE * nc; i += 32 * NW) {
    double *a = zs[i * CHUNK_PIECES];
    for (int k = 0; k < K; k++)
      for (int p = 1; p < CHUNK_PIECES; p++) a[k] += zs[i * CHUNK_PIECES + p][k];
    chunk_coefs<K>(b, st, e + i / nc, i % nc, a, cfs[i]);
  }
  __syncthreads();
  if (*reinterpret_cast<volatile int *>(faint)) {
    for (int i = warp; i < NE * items; i += NW) {
      const int n = i / items, it = i % items;
      const double t = chunk_resid_div<K>(st, NE > 1 && n ? mod[NE - 1] : mod[0], it / CHUNK_PIECES, it % CHUNK_PIECES, cfs + n * nc, true, 0.0);
      if (lane == 0) part[i] = t;
    }
  } else {
    for (int it = warp; it < items; it += NW) {
      const int c = it / CHUNK_PIECES, p = it % CHUNK_PIECES;
      double t[NE];
      {
        float ncc[NE][K], ncp[NE][K];
        section_coefs<K, NE>(cfs, nc, c, ncc, ncp);
        ResidPiece<K>(st, c, p).template sums<NE, false>(st, mod, lane, ncc, ncp, t);
      }
#pragma unroll
      for (int n = 0; n < NE; n++) {
        if (!isfinite(t[n])) t[n] = chunk_resid_div<K>(st, mod[n], c, p, cfs + n * nc, false, t[n]);
        if (lane == 0) part[n * items + it] = t[n];
      }
    }
  }
  __syncthreads();
  if (threadIdx.x < NE) {
    double chi2 = 0.0;
    for (int c = 0; c < nc; c++) {
      const double *q = part + (threadIdx.x * nc + c) * CHUNK_PIECES;
      double acc = q[0];
      for (int p = 1; p < CHUNK_PIECES; p++) acc += q[p];
      chi2 += acc;
    }
    b.cost[e + threadIdx.x] = chi2 / (double)(st.n_obs - 100);
    b.status[e + threadIdx.x] = 0;
  }
}

// K = polynomial order + 1 (one instantiation per order present; evaluations
// of other orders are left alone).  NE = 2: two consecutive evaluations of a
// star share the reads of its arrays and the Legendre values; two that cannot
// share go one after the other.
template <int K, int NE, int NW>
__global__ void __launch_bounds__(32 * NW, NW > 8 ? 1 : chunk_ctas(K, NE)) k_chunk_fit(EvalBatch b) {
  __shared__ double zs[NE * MAX_CHUNKS * CHUNK_PIECES][K];
  __shared__ float cfs[NE * MAX_CHUNKS][K];
  __shared__ double part[NE * MAX_CHUNKS * CHUNK_PIECES];
  __shared__ int faint;
  const int e0 = blockIdx.x * NE, n = min(NE, b.E - e0);
  bool mine[NE];
#pragma unroll
  for (int q = 0; q < NE; q++) mine[q] = q < n && chunk_eval<K>(b, b.stars[b.prep[e0 + q].star], e0 + q);
  if constexpr (NE == 2) {
    if (mine[0] && mine[1] && b.prep[e0].star == b.prep[e0 + 1].star) {
      chunk_fit<K, 2, NW>(b, b.stars[b.prep[e0].star], e0, zs, cfs, part, &faint);
      return;
    }
  }
#pragma unroll 1
  for (int q = 0; q < n; q++) {
    if (!(q == 0 ? mine[0] : mine[NE - 1])) continue;
    chunk_fit<K, 1, NW>(b, b.stars[b.prep[e0 + q].star], e0 + q, zs, cfs, part, &faint);
    __syncthreads();
  }
}

template <int K>
static void launch_chunk(const EvalBatch &b, cudaStream_t s) {
  // Pairs share their star's reads once they fill the GPU (two CTAs per SM).
  // Above degree 7 their sums do not fit the registers.  4,000 evaluations of
  // 60,000 pixels, degree 5: 814 us alone, 677 us in pairs (655 us now).
  if constexpr (K <= 8) {
    if (b.seg_len != 1 && b.E >= 4 * num_sms()) {
      k_chunk_fit<K, 2, 8><<<(b.E + 1) / 2, 256, 0, s>>>(b);
      count_launch();
      return;
    }
  }
  // one evaluation per SM or fewer: 16 warps take its pieces instead of 8
  // (40 evaluations of 15,000 pixels, degree 8: 29 -> 26 us)
  if (b.E <= num_sms()) k_chunk_fit<K, 1, 16><<<b.E, 512, 0, s>>>(b);
  else k_chunk_fit<K, 1, 8><<<b.E, 256, 0, s>>>(b);
  count_launch();
}

// every polynomial order present (evaluations of another order return at once)
void launch_chunk_fit(const EvalBatch &b, cudaStream_t s) {
  const uint32_t m = b.chunk_p1_mask;
  if (m & (1u << 1)) launch_chunk<1>(b, s);
  if (m & (1u << 2)) launch_chunk<2>(b, s);
  if (m & (1u << 3)) launch_chunk<3>(b, s);
  if (m & (1u << 4)) launch_chunk<4>(b, s);
  if (m & (1u << 5)) launch_chunk<5>(b, s);
  if (m & (1u << 6)) launch_chunk<6>(b, s);
  if (m & (1u << 7)) launch_chunk<7>(b, s);
  if (m & (1u << 8)) launch_chunk<8>(b, s);
  if (m & (1u << 9)) launch_chunk<9>(b, s);
  if (m & (1u << 10)) launch_chunk<10>(b, s);
  if (m & (1u << 11)) launch_chunk<11>(b, s);
  if (m & (1u << 12)) launch_chunk<12>(b, s);
  if (m & (1u << 13)) launch_chunk<13>(b, s);
  if (m & (1u << 14)) launch_chunk<14>(b, s);
  if (m & (1u << 15)) launch_chunk<15>(b, s);
  if (m & (1u << 16)) launch_chunk<16>(b, s);
}

// ChunkFitter::build_continuum_from_chunks (continuum_fitting.rs:228-278)
// from Legendre coefficients: continuum = blend of the chunk polynomials.
template <int K>
__device__ float build_one(const DevStar &st, const double *coef, int i) {
  const int nc = st.n_chunks;
  int c = 0;
  while (c + 1 < nc && i >= st.cstart[c + 1]) c++;
  float cp[K], cc[K];
  for (int k = 0; k < K; k++) cc[k] = (float)coef[c * MAX_P1 + k];
  if (c > 0 && i < st.cstop[c - 1]) {
    for (int k = 0; k < K; k++) cp[k] = (float)coef[(c - 1) * MAX_P1 + k];
    const float pv = poly_eval<K>(cp, st.xa[i]);
    const float cu = poly_eval<K>(cc, st.xb[i]);
    const float f = st.fac[i];
    return pv * f + cu * (1.0f - f);
  }
  return poly_eval<K>(cc, st.xa[i]);
}

__global__ void k_build_chunk(const DevStar *stp, const double *coef, int n, float *out) {
  const DevStar &st = *stp;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float v;
    switch (st.p1) {
      case 1: v = build_one<1>(st, coef, i); break;
      case 2: v = build_one<2>(st, coef, i); break;
      case 3: v = build_one<3>(st, coef, i); break;
      case 4: v = build_one<4>(st, coef, i); break;
      case 5: v = build_one<5>(st, coef, i); break;
      case 6: v = build_one<6>(st, coef, i); break;
      case 7: v = build_one<7>(st, coef, i); break;
      case 8: v = build_one<8>(st, coef, i); break;
      case 9: v = build_one<9>(st, coef, i); break;
      case 10: v = build_one<10>(st, coef, i); break;
      case 11: v = build_one<11>(st, coef, i); break;
      case 12: v = build_one<12>(st, coef, i); break;
      case 13: v = build_one<13>(st, coef, i); break;
      case 14: v = build_one<14>(st, coef, i); break;
      case 15: v = build_one<15>(st, coef, i); break;
      default: v = build_one<16>(st, coef, i); break;
    }
    out[i] = v;
  }
}
void launch_build_chunk(const DevStar *star, const double *coef, int n, float *out, cudaStream_t s) {
  k_build_chunk<<<(n + 255) / 256, 256, 0, s>>>(star, coef, n, out);
  count_launch();
}

}  // namespace pb
