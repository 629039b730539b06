// kernels.cu -- the bandwidth, FFT and reduction kernels of the hot path.
//
// Buffer protocol per evaluation e (rows of `stride` floats):
//   k_interp writes the interpolated spectrum to A.
//   k_broaden (rotation FFT + instrument profile, fused) reads A and writes
//   the broadened synth row to B, or in chi2 batches the model resampled
//   to the observed pixels (EvalPrep::epi).
//   Very wide kernels (m - 1 + 2 hg > 2048 - 128) take the unfused pair
//   k_rot (A -> B) and k_gauss (B -> A, or A -> B when the rotation is the
//   identity).  EvalPrep::final_in_b says where the synth row is.
//   k_resample_obs resamples the synth rows k_broaden did not, into the
//   other buffer (EvalPrep::mobs_in_b); the chi2 kernels read that model.
//   k_resample_out / k_copy_broadened serve the model entry points.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "device.cuh"
#include "fft.cuh"
#include "kernels.h"

namespace pb {

__device__ __forceinline__ const float *final_row(const EvalBatch &b, const EvalPrep &P, int e) {
  return (P.final_in_b ? b.bufB : b.bufA) + (size_t)e * b.stride;
}

static int g_num_sms = 0;
int num_sms() {
  if (!g_num_sms) {
    int dev;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
    if (g_num_sms <= 0) g_num_sms = 148;
  }
  return g_num_sms;
}

// Asynchronous 16-byte global -> shared copies (cp.async): the next tile's
// input streams in while the current one is worked.  A copy with ok ==
// false reads nothing and fills zeros.
__device__ __forceinline__ void cp_async16(float *smem, const float *gmem, bool ok) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  const int n = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(sa), "l"(gmem), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// ---------------------------------------------------------------- interp
// flux[px] = sum_n w_n * u16_n[px] * factor_n over the 64 neighbours
// (interpolate.rs:954-981).  Particles of one star soon sit in the same grid
// cube and then read the same 64 rows, so evaluations are grouped first:
// k_group finds, among SEG consecutive evaluations, those with identical
// neighbour columns and records each group's rows once.  k_interp then
// converts every row tile once per group and applies each member's weights
// to it: the reads and the u16 -> f32 conversions are shared, each member
// keeps its own accumulators, and each member's sum runs over its rows in
// reference order (rows another member needs add exactly 0), so the result
// is the same as interpolating every evaluation alone.

// whether evaluations e and u have the same neighbour columns (keys a, c)
__device__ __forceinline__ bool same_cols(const DevGrid &G, const EvalBatch &b, int e, unsigned long long a, int u,
                                          unsigned long long c) {
  if (a != c) return false;
  if (max(G.g.nt, max(G.g.nm, G.g.nl)) <= AXIS_KEY) return true;
  for (int n = 0; n < 64; n++)
    if (b.prep[e].cols[n] != b.prep[u].cols[n]) return false;
  return true;
}

// Segment s of a batch: [start, start + len), a chunk of at most SEG
// evaluations of one star (EvalBatch::seg_len), len <= 0 when empty.
__device__ __forceinline__ void seg_range(const EvalBatch &b, int s, int &start, int &len) {
  const int L = b.seg_len > 0 ? b.seg_len : b.E;
  const int spb = (L + SEG - 1) / SEG;
  const int j = s / spb, q = s - j * spb;
  start = j * L + q * SEG;
  len = min(min(SEG, L - q * SEG), b.E - start);
}
int num_segments(const EvalBatch &b) {
  if (b.E <= 0) return 0;
  const int L = b.seg_len > 0 ? b.seg_len : b.E;
  return (b.E + L - 1) / L * ((L + SEG - 1) / SEG);
}

// The record of a group by one warp: the rows any member (evaluations
// mem[0 .. GROUP_MAX), -1: unused) weighs, in reference order, with every
// member's weight, padded to a multiple of 8 rows with zero weights.
__device__ __forceinline__ void write_group(const DevGrid &G, const EvalBatch &b, GroupRec &R, const int *mem, int lane) {
  int c[2], nm = 0;
  float f[2], w[2][GROUP_MAX], wf[2][GROUP_MAX];
  unsigned bal[2];
#pragma unroll
  for (int m = 0; m < GROUP_MAX; m++) nm += mem[m] >= 0;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int i = lane + 32 * h;
    c[h] = b.prep[mem[0]].cols[i];
    f[h] = c[h] >= 0 ? G.factor[c[h]] : 0.0f;
    bool keep = false;
#pragma unroll
    for (int m = 0; m < GROUP_MAX; m++) {
      w[h][m] = (m < nm && c[h] >= 0) ? b.prep[mem[m]].w[i] : 0.0f;
      wf[h][m] = w[h][m] * f[h];
      keep |= wf[h][m] != 0.0f;
    }
    bal[h] = __ballot_sync(0xffffffffu, keep);
  }
  const unsigned below = (1u << lane) - 1u;
  const int kept = __popc(bal[0]) + __popc(bal[1]), padded = (kept + 7) & ~7;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const int pos = (h ? __popc(bal[0]) : 0) + __popc(bal[h] & below);
    if (bal[h] >> lane & 1u) {
      R.wf[pos][0] = make_float4(wf[h][0], wf[h][1], wf[h][2], wf[h][3]);
      R.wf[pos][1] = make_float4(wf[h][4], wf[h][5], wf[h][6], wf[h][7]);
      R.w[pos][0] = make_float4(w[h][0], w[h][1], w[h][2], w[h][3]);
      R.w[pos][1] = make_float4(w[h][4], w[h][5], w[h][6], w[h][7]);
      R.col[pos] = c[h];
      R.f[pos] = f[h];
    }
  }
  if (lane < padded - kept) {  // zero-weight padding rows (add exactly 0)
    const float4 z4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int pos = kept + lane;
    R.wf[pos][0] = R.wf[pos][1] = R.w[pos][0] = R.w[pos][1] = z4;
    R.col[pos] = 0;
    R.f[pos] = 0.0f;
  }
  if (lane < GROUP_MAX) {
    const int m = mem[lane];
    R.member[lane] = m;
    R.lo[lane] = m >= 0 ? b.prep[m].i_lo : 0;
    R.hi[lane] = m >= 0 ? b.prep[m].i_hi : 0;
  }
  if (lane == 0) {
    R.nmem = nm;
    R.nn = padded;
  }
}

// One CTA per segment: SEG threads find the groups, then every warp writes
// group records (a lane per neighbour row and its 32nd next).  Columns shared
// by TC_MIN_MEMBERS or more evaluations form tensor-core groups (with the
// tensor-core path on); the others form groups of up to GROUP_MAX, numbered
// in evaluation order.  All of it is latency: with the columns compared one
// by one, the groups numbered by one thread and 4 records written at a time
// between CTA barriers a segment took 41-60 us, 15-22 us now (cold, under ncu).
constexpr int GROUP_T = 512, GROUP_W = GROUP_T / 32;
__global__ void __launch_bounds__(GROUP_T) k_group(DevGrid G, EvalBatch b) {
  __shared__ unsigned long long key[SEG];
  __shared__ int ok[SEG], lead[SEG], cnt[SEG], tcg[SEG], tclead[TC_MAX_GROUPS];
  __shared__ int opened[SEG][SEG / GROUP_MAX], mem[SEG][GROUP_MAX];
  __shared__ unsigned bal[2][2];
  const int s = blockIdx.x, t = threadIdx.x, lane = t & 31, warp = t >> 5;
  int start, len;
  seg_range(b, s, start, len);
  if (len <= 0) {
    if (t == 0) {
      b.gcount[s] = 0;
      if (b.tccount) b.tccount[s] = 0;
    }
    return;
  }
  const int e = start + t;
  int L = -1, rank = 0, n = 0;
  if (t < SEG) {
    ok[t] = t < len && b.prep[e].status == 0;
    key[t] = ok[t] ? b.prep[e].key : 0ull;
  }
  for (int i = t; i < SEG * GROUP_MAX; i += GROUP_T) mem[i / GROUP_MAX][i % GROUP_MAX] = -1;
  __syncthreads();
  if (t < SEG) {  // leader: the first evaluation with the same columns; rank among them, their number
    if (ok[t])
      for (int u = 0; u < SEG; u++)
        if (ok[u] && same_cols(G, b, e, key[t], start + u, key[u])) {
          if (L < 0) L = u;
          rank += u < t;
          n++;
        }
    lead[t] = L;
    cnt[t] = n;
    const bool tc = L == t && b.tcrec && n >= max(b.tc_min, TC_MIN_MEMBERS);
    const unsigned m = __ballot_sync(0xffffffffu, tc);
    if (lane == 0) bal[0][warp] = m;
    tcg[t] = tc ? __popc(m & ((1u << lane) - 1u)) : -1;  // within the warp
  }
  __syncthreads();
  if (t < SEG && warp == 1 && tcg[t] >= 0) tcg[t] += __popc(bal[0][0]);
  if (t < SEG && tcg[t] >= 0) tclead[tcg[t]] = t;  // at most SEG / TC_MIN_MEMBERS groups
  const int ntc = __popc(bal[0][0]) + __popc(bal[0][1]);
  __syncthreads();
  bool open = false;
  if (t < SEG) {  // a group opens at every GROUP_MAX-th evaluation of a leader
    open = ok[t] && tcg[L] < 0 && rank % GROUP_MAX == 0;
    const unsigned m = __ballot_sync(0xffffffffu, open);
    if (lane == 0) bal[1][warp] = m;
    if (open) opened[L][rank / GROUP_MAX] = __popc(m & ((1u << lane) - 1u));
  }
  __syncthreads();
  const int ng = __popc(bal[1][0]) + __popc(bal[1][1]);
  if (open && warp == 1) opened[L][rank / GROUP_MAX] += __popc(bal[1][0]);
  __syncthreads();
  if (t < SEG && ok[t] && tcg[L] < 0) {
    const int g = opened[L][rank / GROUP_MAX];
    mem[g][rank % GROUP_MAX] = e;
    if (b.mkey && n == 1) {  // alone in its segment: offer it to the batch-wide table of column sets
      const unsigned long long k = key[t];
      unsigned slot = (unsigned)((k * 0x9E3779B97F4A7C15ull) >> 32) & (unsigned)(b.mtab - 1);
      for (int probe = 0; probe < b.mtab; probe++) {  // the table is at most half full
        const unsigned long long old = atomicCAS(&b.mkey[slot], 0ull, k);
        if (old == 0ull || old == k) break;
        slot = (slot + 1) & (unsigned)(b.mtab - 1);
      }
      const int r = atomicAdd(&b.mcnt[slot], 1);
      if (r < MERGE_CAP) b.mmem[(size_t)slot * MERGE_CAP + r] = e;
      if (r == 1) b.mslot[atomicAdd(b.mslot_count, 1)] = (int)slot;
      b.erec[e] = start + g;
    }
  }
  if (t == 0) {
    b.gcount[s] = ng;
    if (b.tccount) b.tccount[s] = ntc;
    if (ntc > 0) {
      const int at = atomicAdd(b.tclist_count, ntc);
      for (int k = 0; k < ntc; k++) b.tclist[at + k] = start + k;
    }
  }
  __syncthreads();
  // tensor-core group records, a warp per group
  for (int g = warp; g < ntc; g += GROUP_W) {
    TcGroup &T = b.tcrec[start + g];
    const int l = tclead[g];
    int lo = 1 << 30, hi = 0;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int i = lane + 32 * h, c = b.prep[start + l].cols[i];
      T.col[i] = c;
      T.f[i] = c >= 0 ? G.factor[c] : 0.0f;
      if (ok[i] && lead[i] == l) {
        lo = min(lo, b.prep[start + i].i_lo);
        hi = max(hi, b.prep[start + i].i_hi);
      }
    }
    const unsigned m0 = __ballot_sync(0xffffffffu, ok[lane] && lead[lane] == l);
    const unsigned m1 = __ballot_sync(0xffffffffu, ok[lane + 32] && lead[lane + 32] == l);
    const unsigned below = (1u << lane) - 1u;  // members in evaluation order
    if (m0 >> lane & 1u) T.member[__popc(m0 & below)] = start + lane;
    if (m1 >> lane & 1u) T.member[__popc(m0) + __popc(m1 & below)] = start + lane + 32;
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
      T.nmem = cnt[l];
      T.lo = lo;
      T.hi = hi;
    }
  }
  for (int g = warp; g < ng; g += GROUP_W) write_group(G, b, b.grec[(size_t)start + g], mem[g], lane);
}

// One warp per listed table slot (two or more evaluations alone in their
// segments chose it): the evaluations with the first one's columns become
// group records of up to GROUP_MAX members, and their own single-member
// records are switched off (nmem 0).
constexpr int MERGE_W = 4;
__global__ void __launch_bounds__(32 * MERGE_W) k_merge(DevGrid G, EvalBatch b) {
  __shared__ int mem[MERGE_W][MERGE_CAP + GROUP_MAX];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nlist = *b.mslot_count;
  for (int j = blockIdx.x * MERGE_W + warp; j < nlist; j += gridDim.x * MERGE_W) {
    const int slot = b.mslot[j], nc = min(b.mcnt[slot], MERGE_CAP);
    const int *list = b.mmem + (size_t)slot * MERGE_CAP;
    const int e0 = list[0];
    int nt = 0;  // the matching evaluations, in list order
    for (int i = lane; i < MERGE_CAP; i += 32) {
      const int e = i < nc ? list[i] : -1;
      const bool same = e >= 0 && same_cols(G, b, e0, b.prep[e0].key, e, b.prep[e].key);
      const unsigned bal = __ballot_sync(0xffffffffu, same);
      if (same) mem[warp][nt + __popc(bal & ((1u << lane) - 1u))] = e;
      nt += __popc(bal);
    }
    if (lane < GROUP_MAX) mem[warp][nt + lane] = -1;
    __syncwarp();
    if (nt >= 2)
      for (int g0 = 0; g0 < nt; g0 += GROUP_MAX) {
        int rec = 0;
        if (lane == 0) rec = atomicAdd(b.mrcount, 1);
        rec = __shfl_sync(0xffffffffu, rec, 0);
        write_group(G, b, b.mrec[rec], mem[warp] + g0, lane);
        if (lane < GROUP_MAX && g0 + lane < nt) b.grec[b.erec[mem[warp][g0 + lane]]].nmem = 0;  // interpolated here instead
      }
    __syncwarp();
  }
}

void launch_group(const DevGrid &G, const EvalBatch &b, cudaStream_t s) {
  if (b.E <= 0) return;
  if (b.mkey) cudaMemsetAsync(b.mkey, 0, (size_t)b.mtab * (sizeof(unsigned long long) + sizeof(int)), s);  // and mcnt
  k_group<<<num_segments(b), GROUP_T, 0, s>>>(G, b);
  count_launch();
  if (b.mkey) {
    k_merge<<<num_sms() * 4, 32 * MERGE_W, 0, s>>>(G, b);
    count_launch();
  }
}

constexpr int IT_T = 256, IT_PX = 4, IT_TILE = IT_T * IT_PX;

// member m's weight (x factor when wf) of compacted row n
__device__ __forceinline__ float grp_w(const float4 (&v)[2], int m) {
  const float4 q = v[m >> 2];
  const int k = m & 3;
  return k == 0 ? q.x : k == 1 ? q.y : k == 2 ? q.z : q.w;
}

// the NM members of a group on this thread's 4 pixels (one 64-bit load per row)
template <int NM>
__device__ __forceinline__ void interp_members(const DevGrid &G, const EvalBatch &b, const GroupRec &R, int px) {
  // member m's window holds px (read again at the stores, so that the windows
  // need no registers across the row loop)
  auto inside = [&](int m) { return px >= R.lo[m] && px < R.hi[m]; };
  bool any = false;
#pragma unroll
  for (int m = 0; m < NM; m++) any |= inside(m);
  if (!any) return;
  const int nn = R.nn;
  if (px + IT_PX <= G.tail_start) {
    float2 acc[NM][2];
#pragma unroll
    for (int m = 0; m < NM; m++) acc[m][0] = acc[m][1] = make_float2(0.0f, 0.0f);
    const float2 bias = make_float2(-8388608.0f, -8388608.0f);
    constexpr int UNR = NM > 4 ? 4 : 8;  // row loads in flight per thread (with their weights in registers)
#pragma unroll UNR
    for (int n = 0; n < nn; n++) {
      const uint2 q = __ldg(reinterpret_cast<const uint2 *>(G.spectra + (size_t)R.col[n] * G.stride + px));
      float ws[8];
      const float4 w0 = R.wf[n][0];
      ws[0] = w0.x; ws[1] = w0.y; ws[2] = w0.z; ws[3] = w0.w;
      if (NM > 4) {
        const float4 w1 = R.wf[n][1];
        ws[4] = w1.x; ws[5] = w1.y; ws[6] = w1.z; ws[7] = w1.w;
      }
      const uint32_t u[2] = {q.x, q.y};
#pragma unroll
      for (int k = 0; k < 2; k++) {
        float2 v = make_float2(__int_as_float(__byte_perm(u[k], 0x4B000000u, 0x7410)),
                               __int_as_float(__byte_perm(u[k], 0x4B000000u, 0x7432)));
        v = __fadd2_rn(v, bias);  // exact u16 -> f32
#pragma unroll
        for (int m = 0; m < NM; m++) acc[m][k] = __ffma2_rn(make_float2(ws[m], ws[m]), v, acc[m][k]);
      }
    }
#pragma unroll
    for (int m = 0; m < NM; m++) {
      if (!inside(m)) continue;
      *reinterpret_cast<float4 *>(b.bufA + (size_t)R.member[m] * b.stride + px) =
          make_float4(acc[m][0].x, acc[m][0].y, acc[m][1].x, acc[m][1].y);
    }
    return;
  }
  // last tile: the final npx % 128 pixels carry an extra 1/65535 (interpolate.rs:978)
#pragma unroll
  for (int m = 0; m < NM; m++) {
    if (!inside(m)) continue;
    float acc[IT_PX];
#pragma unroll
    for (int k = 0; k < IT_PX; k++) acc[k] = 0.0f;
    for (int n = 0; n < nn; n++) {
      const uint2 q = __ldg(reinterpret_cast<const uint2 *>(G.spectra + (size_t)R.col[n] * G.stride + px));
      const float wn = grp_w(R.w[n], m), fn = R.f[n];
      const uint32_t u[2] = {q.x, q.y};
#pragma unroll
      for (int k = 0; k < IT_PX; k++) {
        const float x = (float)((u[k >> 1] >> (16 * (k & 1))) & 0xFFFFu);
        const float v = px + k >= G.tail_start ? __fmul_rn(__fdiv_rn(x, 65535.0f), fn) : __fmul_rn(x, fn);
        acc[k] = fmaf(wn, v, acc[k]);
      }
    }
    *reinterpret_cast<float4 *>(b.bufA + (size_t)R.member[m] * b.stride + px) =
        make_float4(acc[0], acc[1], acc[2], acc[3]);
  }
}

// one group record on this thread's pixels (nmem 0: a record switched off)
__device__ __forceinline__ void interp_group(const DevGrid &G, const EvalBatch &b, const GroupRec &R, int px) {
  switch (R.nmem) {
    case 0: break;
    case 1: interp_members<1>(G, b, R, px); break;
    case 2: interp_members<2>(G, b, R, px); break;
    case 3: interp_members<3>(G, b, R, px); break;
    case 4: interp_members<4>(G, b, R, px); break;
    case 5: interp_members<5>(G, b, R, px); break;
    case 6: interp_members<6>(G, b, R, px); break;
    case 7: interp_members<7>(G, b, R, px); break;
    default: interp_members<8>(G, b, R, px); break;
  }
}

// group record -> shared memory, 16 bytes per copy, not waited for
__device__ __forceinline__ void rec_load(GroupRec *dst, const GroupRec *src) {
  static_assert(sizeof(GroupRec) % 16 == 0, "16-byte copies");
  const float *s = reinterpret_cast<const float *>(src);
  float *d = reinterpret_cast<float *>(dst);
  for (int i = threadIdx.x; i < (int)(sizeof(GroupRec) / 16); i += IT_T) cp_async16(d + 4 * i, s + 4 * i, true);
}

// Grid: x = segment, y = tile of IT_TILE pixels, so CTAs that run together read
// the same tile slab of the resident grid (28 MB for 13,860 models), which
// stays in L2; z = slice of the segment's groups (groups z, z + Z, ...), more
// than one only for batches too small to fill the GPU otherwise.  Groups have
// disjoint members, so the slicing does not change any result.  The next
// record is copied in while the rows of one are read (one barrier a group);
// its members' windows come with it.  Bound by instruction issue (67%: the
// u16 -> f32 conversions) and the rows' L2 latency: 2,500 evaluations spread
// over 13,860 x 80,000 models, alone and merged: 599 + 795 us with the record
// and the windows read between two barriers at 3 CTAs per SM (80 registers),
// 503 + 822 us with the copy ahead, 490 + 714 us at 4 CTAs (64 registers, 24
// bytes spilled by the largest groups); 2 rows in flight for those instead
// of 4: 478 + 947.
__global__ void __launch_bounds__(IT_T, 4) k_interp(DevGrid G, EvalBatch b) {
  __shared__ GroupRec R[2];
  const int s = blockIdx.x;
  const int px = blockIdx.y * IT_TILE + threadIdx.x * IT_PX;
  const int ng = b.gcount[s];
  int start, len;
  seg_range(b, s, start, len);
  const GroupRec *rec = b.grec + start;
  int k = 0;
  if ((int)blockIdx.z < ng) rec_load(&R[0], rec + blockIdx.z);
  for (int g = blockIdx.z; g < ng; g += gridDim.z, k ^= 1) {
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();  // this record is here, and the other buffer is no longer read
    if (g + (int)gridDim.z < ng) rec_load(&R[k ^ 1], rec + g + gridDim.z);
    interp_group(G, b, R[k], px);
  }
}

// Groups merged across segments (k_merge), in work items (record, tile)
// taken tile by tile, so that CTAs that run together read the same tile
// slab of the grid; their number is known on the device only.
__global__ void __launch_bounds__(IT_T, 4) k_interp_merged(DevGrid G, EvalBatch b) {
  __shared__ GroupRec R[2];
  const int nrec = *b.mrcount;
  const long long work = (long long)nrec * ((G.npx + IT_TILE - 1) / IT_TILE);
  int k = 0;
  if (blockIdx.x < work) rec_load(&R[0], b.mrec + blockIdx.x % nrec);
  for (long long w = blockIdx.x; w < work; w += gridDim.x, k ^= 1) {
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    if (w + gridDim.x < work) rec_load(&R[k ^ 1], b.mrec + (w + gridDim.x) % nrec);
    interp_group(G, b, R[k], (int)(w / nrec) * IT_TILE + threadIdx.x * IT_PX);
  }
}

void launch_interp(const DevGrid &G, const EvalBatch &b, cudaStream_t s) {
  if (b.E <= 0) return;
  const int segs = num_segments(b), tiles = (G.npx + IT_TILE - 1) / IT_TILE;
  const int want = num_sms() * 8;  // two waves of the 4 CTAs an SM holds
  const int z = segs * tiles >= want ? 1 : std::min(SEG, (want + segs * tiles - 1) / (segs * tiles));
  dim3 grid(segs, tiles, z);
  k_interp<<<grid, IT_T, 0, s>>>(G, b);
  count_launch();
  if (b.mkey) {
    k_interp_merged<<<num_sms() * 8, IT_T, 0, s>>>(G, b);
    count_launch();
  }
}

// ----------------------------------------------- direct broadening (narrow)
// Evaluations whose combined kernel (m rotation taps + 2 hg instrument taps)
// is narrow are convolved directly: per tile of DIRECT_TILE - 2 hg final
// outputs [t0, t0 + n) the DIRECT_TILE rotation outputs [t0 - hg, t0 + n + hg) (zero outside the
// grid, like the reference's cropped segment) and then the instrument
// profile, both from shared memory, into B.  The result is the same linear
// convolution the FFT path computes (convolve_rv.rs:121-157, 207-210,
// 414-430, 484-529), to f32 roundoff.
constexpr int DT_T = 256;
constexpr int DT_X = DIRECT_TILE + DIRECT_MAX_TAPS + 32;  // staged input / rotation output (floats)
constexpr int DT_HALF = DT_X / 2;                          // 1296 = 16 mod 32 (see dchunk)
constexpr int DT_K = DIRECT_MAX_TAPS + 32;                // zero-padded taps
static_assert(DT_X % 8 == 0 && DT_HALF % 32 == 16, "direct tile layout");

// Rows of the direct path sit in shared memory chunk-interleaved: float4
// chunk c (elements 4c..4c+3) at (c & 1) * DT_HALF + (c >> 1) * 4.  The
// chunks 2t + q that the threads t of a warp read together are then
// consecutive 16-byte words (no bank conflicts), and so are the chunks 2t,
// 2t + 1 each thread writes.
__device__ __forceinline__ int dchunk(int c) { return ((c & 1) ? DT_HALF : 0) + ((c >> 1) << 2); }
__device__ __forceinline__ int dperm(int i) { return dchunk(i >> 2) + (i & 3); }

// out(v) = sum_{j=-h..h} k[h + j] x(D + v - j), v in [0, n), n <= 8 DT_T: the
// eight consecutive outputs v0 = 8t.. of thread t.  x (chunk-interleaved) is
// readable (finite) over [0, n + 2h + 16); D - h is 0..3; kp holds k[0..2h]
// at offset zp = 12 + the amount that makes 2h + (D - h) + zp a multiple of
// 4, zeros around it, so every window of 12 taps is three aligned float4
// reads and taps outside the kernel are exact zeros.  Each chunk of 4 inputs
// costs 2 shared-memory reads (the input, one new tap float4) for 32 FMAs.
__device__ __forceinline__ int direct_zp(int h, int pl) { return 12 + ((4 - ((2 * h + pl) & 3)) & 3); }

__device__ __forceinline__ void conv_step(const float4 a, const float4 lo, float4 &mid, float4 &hi, float (&acc)[8]) {
  const float T[12] = {lo.x, lo.y, lo.z, lo.w, mid.x, mid.y, mid.z, mid.w, hi.x, hi.y, hi.z, hi.w};
  const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
  for (int c = 0; c < 8; c++)
#pragma unroll
    for (int r = 0; r < 4; r++) acc[c] = fmaf(T[4 + c - r], av[r], acc[c]);
  hi = mid;
  mid = lo;
}

template <class Store>
__device__ __forceinline__ void conv_blocked(const float *__restrict__ x, int D, int h, const float *__restrict__ kp,
                                             int n, const Store &st) {
  const int v0 = 8 * threadIdx.x;
  if (v0 >= n) return;
  const int pl = D - h;
  const int z0 = 2 * h + pl + direct_zp(h, pl);  // multiple of 4
  const int Q = (pl + 7 + 2 * h) / 4 + 1;
  const float4 *xe = reinterpret_cast<const float4 *>(x) + threadIdx.x;            // chunks 2t, 2t + 2, ...
  const float4 *xo = reinterpret_cast<const float4 *>(x + DT_HALF) + threadIdx.x;  // chunks 2t + 1, ...
  const float4 *k4 = reinterpret_cast<const float4 *>(kp) + z0 / 4;
  float acc[8];
#pragma unroll
  for (int c = 0; c < 8; c++) acc[c] = 0.0f;
  // chunk q: inputs x(v0 + 4q + r), taps kp[z0 - 4q - 4 + i], i = 4 + c - r in 1..10
  float4 hi = k4[1], mid = k4[0];
  int q = 0;
  for (; q + 1 < Q; q += 2) {
    conv_step(xe[q >> 1], k4[-q - 1], mid, hi, acc);
    conv_step(xo[q >> 1], k4[-q - 2], mid, hi, acc);
  }
  if (q < Q) conv_step(xe[q >> 1], k4[-q - 1], mid, hi, acc);
  st(v0, acc);
}

// taps k[0..2h] (or the single tap 1 when taps == null) into kp with the
// padding of conv_blocked for this D - h
__device__ __forceinline__ void direct_taps(float *kp, const float *taps, int h, int pl) {
  const int zp = direct_zp(h, pl);
  for (int t = threadIdx.x; t < DT_K; t += DT_T) {
    const int u = t - zp;
    kp[t] = (u >= 0 && u <= 2 * h) ? (taps ? taps[u] : 1.0f) : 0.0f;
  }
}

// final outputs per direct tile of an evaluation: a multiple of 4, so the
// input alignment (and with it the padding of the rotation taps) is the same
// for every tile of the evaluation; tiles start at o_lo rounded down to 4,
// so the outputs are 16-byte aligned in the row
__device__ __forceinline__ int direct_td(int hg) { return (DIRECT_TILE - 2 * hg) & ~3; }

struct DirectTile {
  int e, tile, m, hw, hg, t0, n, p0, nr, pl, x0;
};
__device__ __forceinline__ bool direct_tile(const EvalBatch &b, int e, int tile, DirectTile &d) {
  const EvalPrep &P = b.prep[e];
  if (P.status || !P.direct || tile >= P.ndt) return false;
  d.e = e;
  d.tile = tile;
  d.m = P.m;
  d.hw = (d.m - 1) / 2;
  d.hg = P.hg;
  const int td = direct_td(d.hg);
  d.t0 = (P.o_lo & ~3) + tile * td;
  d.n = min(td, P.o_hi - d.t0);
  d.p0 = d.t0 - d.hg;  // rotation outputs [p0, p0 + nr)
  d.nr = d.n + 2 * d.hg;
  d.pl = (((d.p0 - d.hw) % 4) + 4) % 4;
  d.x0 = d.p0 - d.hw - d.pl;  // inputs staged from x0, a multiple of 4
  return true;
}
__device__ __forceinline__ void direct_stage(const EvalBatch &b, const DirectTile &d, float *xs) {
  const EvalPrep &P = b.prep[d.e];
  const float *row = b.bufA + (size_t)d.e * b.stride;
  const int nx = (d.nr + 2 * d.hw + 16 + 3) & ~3;
  for (int c = threadIdx.x; c < nx / 4; c += DT_T) {
    const int g = d.x0 + 4 * c;
    const bool ok = g >= P.i_lo && g + 4 <= P.i_hi;
    cp_async16(xs + dchunk(c), ok ? row + g : row + P.i_lo, ok);
  }
}
// the next item with work at or after i in steps of gridDim.x, or false;
// item i is tile i % max_dtiles of the listed evaluation i / max_dtiles
__device__ __forceinline__ bool direct_next(const EvalBatch &b, long long &i, long long total, DirectTile &d) {
  for (; i < total; i += gridDim.x)
    if (direct_tile(b, b.direct_list[i / b.max_dtiles], (int)(i % b.max_dtiles), d)) return true;
  return false;
}

// CTAs take the tiles of the evaluations k_prep listed in grid strides, so
// those tiles (often all particles of a few stars) spread over the whole GPU;
// the next item's input is copied in (cp.async) while the current one is
// convolved.
__global__ void __launch_bounds__(DT_T) k_direct(DevGrid G, EvalBatch b) {
  __shared__ __align__(16) float xs[2][DT_X];
  __shared__ __align__(16) float rs[DT_X];
  __shared__ __align__(16) float kr[DT_K];
  __shared__ __align__(16) float kg[DT_K];
  const int N = G.npx;
  const long long total = (long long)*b.direct_count * b.max_dtiles;
  long long ic = blockIdx.x;
  DirectTile cur, nxt;
  bool have = direct_next(b, ic, total, cur);
  if (have) direct_stage(b, cur, xs[0]);
  cp_async_commit();
  int buf = 0, taps_e = -1;
  while (have) {
    long long in = ic + gridDim.x;
    const bool more = direct_next(b, in, total, nxt);
    if (more) direct_stage(b, nxt, xs[buf ^ 1]);
    cp_async_commit();
    const EvalPrep &P = b.prep[cur.e];
    const DevStar &st = b.stars[P.star];
    const bool fixedk = st.disp_kind == DISP_FIXED && cur.hg > 0;
    if (cur.e != taps_e) {
      direct_taps(kr, cur.m > 1 ? reinterpret_cast<const float *>(b.H + (size_t)cur.e * 1025) : nullptr,
                  cur.m > 1 ? cur.hw : 0, cur.pl);
      direct_taps(kg, fixedk ? st.gk : nullptr, fixedk ? cur.hg : 0, 0);
      taps_e = cur.e;
    }
    const int p0 = cur.p0, nr = cur.nr, n = cur.n, hg = cur.hg;
    for (int t = nr + threadIdx.x; t < nr + 16; t += DT_T) rs[dperm(t)] = 0.0f;
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // this item's input (the next may be in flight)
    __syncthreads();
    const float *x = xs[buf];
    if (cur.m > 1) {
      conv_blocked(x, cur.hw + cur.pl, cur.hw, kr, nr, [&](int v0, float (&acc)[8]) {
#pragma unroll
        for (int c = 0; c < 8; c++) {  // zero outside the grid and past the tile
          const int v = v0 + c, p = p0 + v;
          if (!(v < nr && p >= 0 && p < N)) acc[c] = 0.0f;
        }
        float4 *r4 = reinterpret_cast<float4 *>(rs);
        r4[dchunk(v0 >> 2) >> 2] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        r4[dchunk((v0 >> 2) + 1) >> 2] = make_float4(acc[4], acc[5], acc[6], acc[7]);
      });
    } else {  // identity rotation: the staged input itself (zero outside the grid)
      for (int v = threadIdx.x; v < nr; v += DT_T) {
        const int p = p0 + v;
        rs[dperm(v)] = (p >= 0 && p < N) ? x[dperm(v + cur.pl)] : 0.0f;
      }
    }
    __syncthreads();
    float *y = b.bufB + (size_t)cur.e * b.stride + cur.t0;  // 16-byte aligned
    if (hg == 0 || fixedk) {
      conv_blocked(rs, fixedk ? hg : 0, fixedk ? hg : 0, kg, n, [&](int v0, float (&acc)[8]) {
        if (v0 + 8 <= n) {
          reinterpret_cast<float4 *>(y + v0)[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
          reinterpret_cast<float4 *>(y + v0)[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
        } else {
#pragma unroll
          for (int c = 0; c < 8; c++)
            if (v0 + c < n) y[v0 + c] = acc[c];
        }
      });
    } else {  // per-pixel instrument kernels (edge pixels pass through)
      for (int v = threadIdx.x; v < n; v += DT_T)
        y[v] = instrument(st, N, cur.t0 + v, hg, [&](int i) { return rs[dperm(i - p0)]; });
    }
    __syncthreads();  // rs and this buffer are rewritten for the item after next
    buf ^= 1;
    have = more;
    ic = in;
    cur = nxt;
  }
  cp_async_wait_all();
}

void launch_direct(const DevGrid &G, const EvalBatch &b, cudaStream_t s) {
  if (b.E <= 0 || b.direct_max <= 0 || b.max_dtiles <= 0 || !b.direct_list) return;
  static int per_sm[64] = {};  // resident CTAs per SM, per device
  int dev = 0;
  cudaGetDevice(&dev);
  int fit = 4;
  if (dev >= 0 && dev < 64) {
    if (!per_sm[dev]) {
      int n = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_direct, DT_T, 0) != cudaSuccess || n < 1) n = 1;
      per_sm[dev] = n;
    }
    fit = per_sm[dev];
  }
  const long long total = (long long)b.E * b.max_dtiles;
  long long grid = (long long)num_sms() * fit;
  if (grid > total) grid = total;
  k_direct<<<(unsigned)grid, DT_T, 0, s>>>(G, b);
  count_launch();
}

// First observed pixel of every fused broadening block: bnd[k] = the
// smallest i whose left synth pixel is >= s_k (binary search on the
// monotone resampling index); bnd[0] = 0, bnd[nblk] = n_obs.
__global__ void k_obs_bounds(DevGrid G, EvalBatch b) {
  const int e = blockIdx.x;
  const EvalPrep &P = b.prep[e];
  if (P.status || !P.epi) return;
  const int k = blockIdx.y * blockDim.x + threadIdx.x, nblk = P.nblk;
  if (k > nblk) return;
  const DevStar &st = b.stars[P.star];
  int *bd = b.bnd + (size_t)e * b.bnd_stride;
  if (k == 0 || k == nblk) {
    bd[k] = k == 0 ? 0 : st.n_obs;
    return;
  }
  const int target = P.o_lo + k * (FFTN - (P.m - 1) - 2 * P.hg - 1);
  const Resampler R = make_resampler(G, st, P, nullptr, nullptr);
  int lo = 0, hi = st.n_obs;
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (R.pos(mid).j < target) lo = mid + 1;
    else hi = mid;
  }
  bd[k] = lo;
}

void launch_obs_bounds(const DevGrid &G, const EvalBatch &b, cudaStream_t s) {
  if (b.E <= 0 || b.max_pairs <= 0 || !b.obs_epi) return;
  dim3 grid(b.E, (2 * b.max_pairs + 1 + 63) / 64);
  k_obs_bounds<<<grid, 64, 0, s>>>(G, b);
  count_launch();
}

// ------------------------------------------- unfused rotation (wide kernels)
// Overlap-save with the rotation kernel alone: block b produces rotation
// outputs [g_lo + b V, g_lo + (b+1) V), V = 2048 - (m - 1), into B.
__global__ void __launch_bounds__(FFT_T, 3) k_rot(DevGrid G, EvalBatch b, const float2 *__restrict__ tw) {
  __shared__ float2 c[FFT_SM];
  const long long total = (long long)b.E * b.max_pairs_unfused;
  for (long long item = blockIdx.x; item < total; item += gridDim.x) {
    const int e = (int)(item / b.max_pairs_unfused), pair = (int)(item % b.max_pairs_unfused);
    const EvalPrep &P = b.prep[e];
    const int m = P.m, nblk = P.nblk;
    if (P.status || P.fused || m <= 1 || 2 * pair >= nblk) continue;
    const int V = FFTN - (m - 1), hw = (m - 1) / 2;
    const int s0 = P.g_lo + 2 * pair * V, s1 = s0 + V;
    const bool has1 = 2 * pair + 1 < nblk;
    const int ilo = P.i_lo, ihi = P.i_hi, ghi = P.g_hi;
    const float *x = b.bufA + (size_t)e * b.stride;
    for (int t = threadIdx.x; t < FFTN; t += FFT_T) {
      const int j0 = s0 - hw + t, j1 = s1 - hw + t;
      c[pidx(t)] = make_float2((j0 >= ilo && j0 < ihi) ? x[j0] : 0.0f, (has1 && j1 >= ilo && j1 < ihi) ? x[j1] : 0.0f);
    }
    __syncthreads();
    fft2048<false>(c, tw);
    const float2 *H = b.H + (size_t)e * 1025;
    for (int k = threadIdx.x; k < FFTN; k += FFT_T) {
      float2 h = k <= 1024 ? H[k] : H[FFTN - k];
      if (k > 1024) h.y = -h.y;
      const int a = pidx(k);
      const float2 v = c[a];
      const cf z = cmul(cf{v.x, v.y}, cf{h.x, h.y});
      c[a] = make_float2(z.x, z.y);
    }
    __syncthreads();
    fft2048<true>(c, tw);
    float *y = b.bufB + (size_t)e * b.stride;
    const float sc = 1.0f / 2048.0f;
    for (int t = m - 1 + threadIdx.x; t < FFTN; t += FFT_T) {
      const int i0 = s0 + t - (m - 1);
      if (i0 < ghi) y[i0] = c[pidx(t)].x * sc;
      if (has1) {
        const int i1 = s1 + t - (m - 1);
        if (i1 < ghi) y[i1] = c[pidx(t)].y * sc;
      }
    }
    __syncthreads();
  }
}

void launch_rot(const DevGrid &G, const EvalBatch &b, const float2 *tw, cudaStream_t s) {
  if (b.E <= 0 || b.max_pairs_unfused <= 0) return;
  const long long total = (long long)b.E * b.max_pairs_unfused;
  long long grid = (long long)num_sms() * 6;
  if (grid > total) grid = total;
  k_rot<<<(unsigned)grid, FFT_T, 0, s>>>(G, b, tw);
  count_launch();
}

// unfused instrument profile: src = rotation output, dst = the other buffer
constexpr int GT = 256, G_TILE = 4096, G_HMAX = 256;

__global__ void __launch_bounds__(GT) k_gauss(DevGrid G, EvalBatch b) {
  __shared__ float sbuf[G_TILE + 2 * G_HMAX];
  const int e = blockIdx.x;
  const EvalPrep &P = b.prep[e];
  if (P.status || P.fused || P.hg == 0) return;
  const DevStar &st = b.stars[P.star];
  const int t0 = max((int)blockIdx.y * G_TILE, P.o_lo), t1 = min((int)(blockIdx.y + 1) * G_TILE, P.o_hi);
  if (t0 >= t1) return;
  const bool rot_in_b = P.m > 1;
  const float *src = (rot_in_b ? b.bufB : b.bufA) + (size_t)e * b.stride;
  float *dst = (rot_in_b ? b.bufA : b.bufB) + (size_t)e * b.stride;
  const int h = P.hg, base = t0 - h;
  for (int j = threadIdx.x; j < (t1 - t0) + 2 * h; j += blockDim.x) {
    const int g = base + j;
    sbuf[j] = (g >= P.g_lo && g < P.g_hi) ? src[g] : 0.0f;
  }
  __syncthreads();
  for (int i = t0 + threadIdx.x; i < t1; i += blockDim.x)
    dst[i] = instrument(st, G.npx, i, h, [&](int t) { return sbuf[t - base]; });
}

void launch_gauss(const DevGrid &G, const EvalBatch &b, cudaStream_t s) {
  if (b.E <= 0) return;
  dim3 grid(b.E, (G.npx + G_TILE - 1) / G_TILE);
  k_gauss<<<grid, GT, 0, s>>>(G, b);
  count_launch();
}

// standalone PyWavelengthDispersion.convolve (lib.rs:671-680): in -> out, all pixels
// tile blockIdx.x of one spectrum: in -> out, all pixels
__device__ __forceinline__ void k_gauss_alone_body(int N, const DevStar &st, const float *in, float *out) {
  __shared__ float sbuf[G_TILE + 2 * G_HMAX];
  const int t0 = blockIdx.x * G_TILE, t1 = min(t0 + G_TILE, N);
  if (st.disp_kind == DISP_NONE) {
    for (int i = t0 + threadIdx.x; i < t1; i += blockDim.x) out[i] = in[i];
    return;
  }
  const int h = (st.gw - 1) / 2, base = t0 - h;
  for (int j = threadIdx.x; j < (t1 - t0) + 2 * h; j += blockDim.x) {
    const int g = base + j;
    sbuf[j] = (g >= 0 && g < N) ? in[g] : 0.0f;
  }
  __syncthreads();
  for (int i = t0 + threadIdx.x; i < t1; i += blockDim.x)
    out[i] = instrument(st, N, i, h, [&](int t) { return sbuf[t - base]; });
}
__global__ void __launch_bounds__(GT) k_gauss_alone(int N, const DevStar *stp, const float *in, float *out) {
  k_gauss_alone_body(N, *stp, in, out);
}
// M spectra of N pixels at once: grid y = spectrum
__global__ void __launch_bounds__(GT) k_gauss_batch(int N, const DevStar *stp, const float *in, float *out) {
  const size_t off = (size_t)blockIdx.y * N;
  k_gauss_alone_body(N, *stp, in + off, out + off);
}
void launch_gauss_batch(int N, const DevStar *star, const float *in, float *out, int M, cudaStream_t s) {
  if (M <= 0 || N <= 0) return;
  k_gauss_batch<<<dim3((N + G_TILE - 1) / G_TILE, M), GT, 0, s>>>(N, star, in, out);
  count_launch();
}

// shift_and_resample at RV 0 (convolve_rv.rs:532-604) of M rows of N synth
// pixels to the star's observed pixels: out [M][n_obs]
__global__ void k_resample_rows(int N, int kind, const DevStar *stp, const float *in, float *out) {
  const DevStar &st = *stp;
  Resampler R;
  R.s = in + (size_t)blockIdx.y * N;
  R.N = N;
  R.kind = kind;
  R.shift_log = 0.0;
  R.shift_factor = 1.0;
  R.lin_offset = 0.0;
  R.fidx = st.fidx;
  R.wl_obs = st.wl_obs;
  R.wl_vals = nullptr;
  R.given = nullptr;
  float *o = out + (size_t)blockIdx.y * st.n_obs;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < st.n_obs; i += gridDim.x * blockDim.x) o[i] = R(i);
}
void launch_resample_rows(int N, int kind, const DevStar *star, int n_obs, const float *in, float *out, int M,
                          cudaStream_t s) {
  if (M <= 0 || n_obs <= 0) return;
  k_resample_rows<<<dim3((n_obs + 255) / 256, M), 256, 0, s>>>(N, kind, star, in, out);
  count_launch();
}

void launch_gauss_standalone(const DevGrid &G, const DevStar *star, const float *in, float *out, cudaStream_t s) {
  k_gauss_alone<<<(G.npx + G_TILE - 1) / G_TILE, GT, 0, s>>>(G.npx, star, in, out);
  count_launch();
}

__global__ void k_resample_out(DevGrid G, EvalBatch b, float *out, int64_t out_stride) {
  const int e = blockIdx.x;
  const EvalPrep &P = b.prep[e];
  if (P.status) return;
  const DevStar &st = b.stars[P.star];
  const Resampler R = make_resampler(G, st, P, final_row(b, P, e), nullptr);
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < st.n_obs; i += gridDim.y * blockDim.x)
    out[(size_t)e * out_stride + i] = R(i);
}
void launch_resample_out(const DevGrid &G, const EvalBatch &b, float *out, int64_t out_stride, cudaStream_t s) {
  if (b.E <= 0) return;
  dim3 grid(b.E, 16);
  k_resample_out<<<grid, 256, 0, s>>>(G, b, out, out_stride);
  count_launch();
}

__global__ void k_copy_broadened(DevGrid G, EvalBatch b, float *out) {
  const int e = blockIdx.x;
  const EvalPrep &P = b.prep[e];
  if (P.status) return;
  const float *row = final_row(b, P, e);
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < G.npx; i += gridDim.y * blockDim.x)
    out[(size_t)e * G.npx + i] = row[i];
}
void launch_copy_broadened(const DevGrid &G, const EvalBatch &b, float *out, cudaStream_t s) {
  if (b.E <= 0) return;
  dim3 grid(b.E, 16);
  k_copy_broadened<<<grid, 256, 0, s>>>(G, b, out);
  count_launch();
}

// ------------------------------------------------------------------ chi2
constexpr int CT = 256, CW = CT / 32;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}

// Dot product of each row with x (InMemInterpolator.ccf, lib.rs:1340-1371):
// one CTA per row, FP64 sums, rounded to f32 once; NaN for a failed row.
__global__ void __launch_bounds__(256) k_dot_rows(const float *rows, int64_t stride, int n, const float *x,
                                                   const int *status, float *out) {
  __shared__ double ws[8];
  const int r = blockIdx.x, t = threadIdx.x;
  const bool ok = status[r] == 0;
  double acc = 0.0;
  if (ok) {
    const float *row = rows + (size_t)r * stride;
    for (int i = t; i < n; i += 256) acc = fma((double)row[i], (double)x[i], acc);
  }
  acc = warp_sum(acc);
  if ((t & 31) == 0) ws[t >> 5] = acc;
  __syncthreads();
  if (t == 0) {
    double tot = 0.0;
    for (int k = 0; k < 8; k++) tot += ws[k];
    out[r] = ok ? (float)tot : __int_as_float(0x7fc00000);
  }
}
void launch_dot_rows(const float *rows, int64_t stride, int n, const float *x, const int *status, float *out, int L,
                     cudaStream_t s) {
  if (L <= 0) return;
  k_dot_rows<<<L, 256, 0, s>>>(rows, stride, n, x, status, out);
  count_launch();
}

// block sum of K per-thread doubles into out[0..K)
template <int K>
__device__ __forceinline__ void block_sum_vec(const double (&v)[K], double (*ws)[MAX_P1], double *out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const double s = warp_sum(v[k]);
    if (lane == 0) ws[warp][k] = s;
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      double s = lane < CW ? ws[lane][k] : 0.0;
      s = warp_sum(s);
      if (lane == 0) out[k] = s;
    }
  }
  __syncthreads();
}

__device__ __forceinline__ double block_sum(double v, double (*ws)[MAX_P1]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) ws[warp][0] = v;
  __syncthreads();
  double r = 0.0;
  if (warp == 0) {
    r = lane < CW ? ws[lane][0] : 0.0;
    r = warp_sum(r);
    if (lane == 0) ws[0][1] = r;
  }
  __syncthreads();
  r = ws[0][1];
  __syncthreads();
  return r;
}

__device__ __forceinline__ void write_result(const EvalBatch &b, int e, double chi2, int status) {
  if (threadIdx.x == 0) {
    b.cost[e] = status ? __longlong_as_double(0x7FF8000000000000ll) : chi2;
    b.status[e] = status;
  }
}

// Evaluations that k_broaden did not resample: the model at the observed
// pixels from the final synth row, into the buffer the synth row is not in.
__global__ void k_resample_obs(DevGrid G, EvalBatch b) {
  const int e = blockIdx.x;
  const EvalPrep &P = b.prep[e];
  if (P.status || P.epi) return;
  const DevStar &st = b.stars[P.star];
  const Resampler R = make_resampler(G, st, P, final_row(b, P, e), nullptr);
  float *out = (P.mobs_in_b ? b.bufB : b.bufA) + (size_t)e * b.stride;
  for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < st.n_obs; i += gridDim.y * blockDim.x) out[i] = R(i);
}
void launch_resample_obs(const DevGrid &G, const EvalBatch &b, cudaStream_t s) {
  if (b.E <= 0) return;
  dim3 grid(b.E, 8);
  k_resample_obs<<<grid, 256, 0, s>>>(G, b);
  count_launch();
}

// LinearModelFitter (continuum_fitting.rs:68-95): projection onto the design
// matrix's column space through its orthonormal basis Q; chi2 of the
// ratio-space residual over [50, N-50) divided by N.  FixedContinuum
// (441-474) and ConstantContinuum (484-500) too.  One CTA per evaluation.
__global__ void __launch_bounds__(CT) k_chi2_other(DevGrid G, EvalBatch b) {
  __shared__ double ws[CW][MAX_P1];
  __shared__ double zs[MAX_LIN_K];
  const int e = blockIdx.x;
  const EvalPrep &P = b.prep[e];
  const DevStar &st = b.stars[P.star];
  if (st.cont_kind == CONT_CHUNK) return;
  if (st.cont_kind == CONT_LINEAR && st.kp > 0 && b.lin_group > 0) return;  // k_linear_tc
  if (P.status) {
    write_result(b, e, 0.0, P.status);
    return;
  }
  if (st.cont_bad) {
    write_result(b, e, 0.0, S_CONTINUUM);
    return;
  }
  const int N = st.n_obs;
  const float *mod = model_row(b, P, e);
  const float *flux = st.flux, *var = st.var;
  double chi2 = 0.0;
  double *par = b.params ? b.params + (size_t)e * b.param_stride : nullptr;
  if (st.cont_kind == CONT_LINEAR) {
    const int K = st.k_lin;
    for (int g0 = 0; g0 < K; g0 += MAX_P1) {
      const int nk = min(MAX_P1, K - g0);
      double z[MAX_P1];
#pragma unroll
      for (int k = 0; k < MAX_P1; k++) z[k] = 0.0;
      for (int i = threadIdx.x; i < N; i += CT) {
        const double bd = (double)(flux[i] / mod[i]);
#pragma unroll
        for (int k = 0; k < MAX_P1; k++)
          if (k < nk) z[k] = fma((double)__ldg(&st.q[(size_t)(g0 + k) * N + i]), bd, z[k]);
      }
      block_sum_vec<MAX_P1>(z, ws, zs + g0);
    }
    if (par)
      for (int k = threadIdx.x; k < K; k += CT) par[k] = zs[k];
    double acc = 0.0;
    for (int i = 50 + threadIdx.x; i < N - 50; i += CT) {
      const float bb = flux[i] / mod[i];
      double fit = 0.0;
      for (int k = 0; k < K; k++) fit = fma((double)__ldg(&st.q[(size_t)k * N + i]), zs[k], fit);
      const float r = (float)fit - bb;
      acc += (double)(r / var[i] * r);
    }
    chi2 = block_sum(acc, ws) / (double)N;
  } else if (st.cont_kind == CONT_FIXED) {
    const int ig = st.ignore;
    double acc = 0.0;
    for (int i = ig + threadIdx.x; i < N - ig; i += CT) {
      const float r = flux[i] - mod[i] * st.cont[i];
      acc += (double)(r / var[i] * r);
    }
    chi2 = block_sum(acc, ws) / (double)(N - 2 * ig);
    if (par && threadIdx.x == 0) par[0] = 0.0;
  } else {
    double sum = 0.0;
    for (int i = threadIdx.x; i < N; i += CT) sum += (double)(flux[i] / mod[i]);
    const float mean = (float)(block_sum(sum, ws) / (double)N);
    double acc = 0.0;
    for (int i = threadIdx.x; i < N; i += CT) {
      const float r = flux[i] - mod[i] * mean;
      acc += (double)(r / var[i] * r);
    }
    chi2 = block_sum(acc, ws) / (double)N;
    if (par && threadIdx.x == 0) par[0] = (double)mean;
  }
  write_result(b, e, chi2, 0);
}

// chi2 of every evaluation from the model at its observed pixels
// (model_row: resampled by k_broaden / k_resample_obs, or given)
void launch_chi2(const DevGrid &G, const EvalBatch &b, cudaStream_t s) {
  if (b.E <= 0) return;
  if (b.chunk_p1_mask && b.max_chunks > 0) launch_chunk_fit(b, s);
  if (b.other_cont) {
    if (b.lin_group > 0) launch_linear_tc(b, s);
    k_chi2_other<<<b.E, CT, 0, s>>>(G, b);
    count_launch();
  }
}

// per-evaluation status when no chi2 is computed (model / spectrum outputs)
__global__ void k_prep_status(EvalBatch b) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < b.E) b.status[e] = b.prep[e].status;
}
void launch_prep_status(const EvalBatch &b, cudaStream_t s) {
  k_prep_status<<<(b.E + 255) / 256, 256, 0, s>>>(b);
  count_launch();
}

void pipeline_pairs(int npx, int max_m, int max_hg, int *max_pairs, int *max_pairs_unfused, int *may_unfuse) {
  const int wide = (max_m - 1) + 2 * max_hg;
  *may_unfuse = wide > FFTN - MIN_FUSED_OUTPUTS ? 1 : 0;
  if (max_m <= 1 && max_hg == 0) {
    *max_pairs = 0;
  } else {
    const int V = (*may_unfuse ? MIN_FUSED_OUTPUTS : FFTN - wide) - 1;  // block advance
    const int nblk = (npx + V - 1) / V;
    *max_pairs = (nblk + 1) / 2;
  }
  if (*may_unfuse && max_m > 1) {
    const int V = FFTN - (max_m - 1);
    const int nblk = (npx + V - 1) / V;
    *max_pairs_unfused = (nblk + 1) / 2;
  } else {
    *max_pairs_unfused = 0;
  }
}

void launch_pipeline(const DevGrid &G, const EvalBatch &b, const float2 *tw, const PipelineOpts &o, cudaStream_t s) {
  if (o.full_window) launch_prep_full(G, b, s);
  else launch_prep(G, b, s);
  // The rotation spectra and the block bounds need the preparation only; the
  // broadening is the first to read them.  On a stream of their own they take
  // 18 us off a batch of 40 evaluations (and are a branch of a captured graph).
  // What they write is read by kernels on s alone, after the join, so the next
  // batch's fork is behind every reader.
  const bool fork = o.side && (o.rot || (b.obs_epi && b.max_pairs > 0));
  cudaStream_t q = fork ? o.side : s;
  if (fork) {
    cudaEventRecord(o.fork, s);
    cudaStreamWaitEvent(q, o.fork, 0);
  }
  if (o.rot) launch_rotker(G, b, tw, q);
  launch_obs_bounds(G, b, q);
  if (fork) cudaEventRecord(o.join, q);
  launch_group(G, b, s);
  launch_interp_tc(G, b, s);
  launch_interp(G, b, s);
  if (fork) cudaStreamWaitEvent(s, o.join, 0);
  launch_broaden(G, b, tw, s);
  launch_direct(G, b, s);
  if (o.may_unfuse) {
    launch_rot(G, b, tw, s);
    launch_gauss(G, b, s);
  }
  if (b.need_chi2) {
    // k_broaden resamples every evaluation with an instrument profile and
    // sorted pixels, unless another kernel broadens it
    if (b.late_resample || b.direct_max > 0 || o.may_unfuse || !b.obs_epi) launch_resample_obs(G, b, s);
    launch_chi2(G, b, s);
  } else if (b.status) {
    launch_prep_status(b, s);
  }
}

}  // namespace pb
