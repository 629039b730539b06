// hostmem.h -- device and host memory of the engine: errors, per-device
// contexts, the scratch pool, staged host copies.  Plain C++ on the CUDA
// runtime API (no kernels), part of engine.cu; the CPU tests compile it on its
// own against a stand-in runtime whose calls can be made to fail.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <thread>
#include <vector>

#include "../../include/pasta_b200.h"
#include "common.cuh"

using namespace pb;

namespace {

struct PErr : std::runtime_error {
  int code;
  PErr(int c, const std::string &m) : std::runtime_error(m), code(c) {}
};
[[noreturn]] void fail(int code, const char *fmt, ...) {
  char buf[1024];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  throw PErr(code, buf);
}
#define CK(call)                                                                                 \
  do {                                                                                           \
    cudaError_t e_ = (call);                                                                     \
    if (e_ != cudaSuccess) fail(PASTA_E_CUDA, "%s failed: %s", #call, cudaGetErrorString(e_)); \
  } while (0)

// ---------------------------------------------------------------- memory
// Scratch memory of the entry points, kept per device between calls: a call
// allocated and freed 8 to 30 buffers, and each cudaFree waits for the device
// (with the staging below: one model of 15,000 pixels 161 -> 125 us, chi2 of 40
// labels 239 -> 182 us, of 160 binary labels 1.30 -> 0.59 ms end to end, and a
// batch of fits no longer varies between 28 and 158 ms).
// Bounded (SCRATCH_BLOCK per block, SCRATCH_TOTAL in all; anything larger goes
// straight to cudaMalloc and cudaFree), given back when a grid is destroyed or
// an allocation fails.  A block may still be read by work in flight when it is
// put back (that work is on the device's one stream): the first block taken
// after any was put back waits for the stream.
constexpr size_t SCRATCH_BLOCK = 64ull << 20, SCRATCH_TOTAL = 256ull << 20;
void *scratch_take(size_t bytes, size_t *got);
void scratch_put(void *p, size_t bytes, int dev);
int scratch_device();
cudaStream_t scratch_stream();
void scratch_flush(int dev);

// Waits for the DBuf uploads made so far.  cudaMemcpy returns when a pageable
// source has been staged, and what it still has under way is on the legacy
// stream, which the library's non-blocking streams do not wait for: whoever
// makes an object waits once, before it hands it out or enqueues work on it
// (a wait after every upload keeps the next one from being staged meanwhile: a
// chunk continuum of 60,000 pixels 2.45 ms instead of 2.0).
inline void wait_uploads() { CK(cudaStreamSynchronize(cudaStreamLegacy)); }

// POOL: scratch of one call or fit (see scratch_take); its uploads are ordered
// on the device's stream
template <class T, bool POOL = false>
struct DBuf {
  T *p = nullptr;
  size_t n = 0;
  size_t bytes = 0;  // of the scratch block
  int dev = -1;
  DBuf() = default;
  DBuf(const DBuf &) = delete;
  DBuf &operator=(const DBuf &) = delete;
  ~DBuf() { release(); }
  void release() {
    if (p) {
      if (POOL) scratch_put(p, bytes, dev);
      else cudaFree(p);
    }
    p = nullptr;
    n = 0;
  }
  // flush: give the scratch pools back and try again when there is no memory
  // (not under g_ctx_mu, which the flush takes)
  void alloc(size_t count, bool flush = true) {
    release();
    if (count == 0) return;
    if (POOL) {
      dev = scratch_device();
      p = (T *)scratch_take(count * sizeof(T), &bytes);
    } else {
      cudaError_t e = cudaMalloc(&p, count * sizeof(T));
      if (e != cudaSuccess) {
        p = nullptr;
        cudaGetLastError();
        if (flush) {
          scratch_flush(-1);
          e = cudaMalloc(&p, count * sizeof(T));
        }
      }
      if (e != cudaSuccess) {
        p = nullptr;
        cudaGetLastError();
        fail(PASTA_E_NOMEM, "cudaMalloc of %zu bytes failed: %s", count * sizeof(T), cudaGetErrorString(e));
      }
    }
    n = count;
  }
  void upload(const T *h, size_t count) {
    alloc(count);
    if (!count) return;
    if (POOL) CK(cudaMemcpyAsync(p, h, count * sizeof(T), cudaMemcpyHostToDevice, scratch_stream()));
    else CK(cudaMemcpy(p, h, count * sizeof(T), cudaMemcpyHostToDevice));  // see wait_uploads
  }
  void upload(const std::vector<T> &v) { upload(v.data(), v.size()); }
};
template <class T>
using SBuf = DBuf<T, true>;

// page-locked host buffer: copies from and to it are asynchronous and can
// be captured in a CUDA graph
template <class T>
struct HostBuf {
  T *p = nullptr;
  HostBuf() = default;
  HostBuf(const HostBuf &) = delete;
  HostBuf &operator=(const HostBuf &) = delete;
  ~HostBuf() {
    if (p) cudaFreeHost(p);
  }
  void alloc(size_t count) {
    if (p) cudaFreeHost(p);
    p = nullptr;
    if (count == 0) return;
    cudaError_t e = cudaMallocHost(&p, count * sizeof(T));
    if (e != cudaSuccess) {
      p = nullptr;
      cudaGetLastError();
      fail(PASTA_E_NOMEM, "cudaMallocHost of %zu bytes failed: %s", count * sizeof(T), cudaGetErrorString(e));
    }
  }
};

// an instantiated CUDA graph, destroyed with its owner
struct GraphHold {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  GraphHold() = default;
  GraphHold(const GraphHold &) = delete;
  GraphHold &operator=(const GraphHold &) = delete;
  ~GraphHold() {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
  }
};

// Page-locked staging for the copies of host arrays: pageable copies run at
// 6-8 GB/s and wait (61 models of 37,501 pixels, 9 MB: 1.5 -> 1.1 ms).  Two
// halves in turn; a half is written again once the copy that used it is done
// (its event).
constexpr size_t STAGE_HALF = 4ull << 20, STAGE_MIN = 64ull << 10;
struct Stage {
  std::mutex mu;
  HostBuf<unsigned char> buf;
  cudaEvent_t ev[2] = {};
  int at = 0;       // half in use
  size_t fill = 0;  // bytes used of it
  // the buffer with both events, or nothing
  bool ready() {
    if (buf.p) return true;
    HostBuf<unsigned char> b;
    cudaEvent_t e[2] = {};
    bool made = cudaMallocHost(&b.p, 2 * STAGE_HALF) == cudaSuccess;
    if (!made) b.p = nullptr;
    for (int k = 0; k < 2 && made; k++) made = cudaEventCreateWithFlags(&e[k], cudaEventDisableTiming) == cudaSuccess;
    if (!made) {
      cudaGetLastError();
      for (cudaEvent_t x : e)
        if (x) cudaEventDestroy(x);
      return false;
    }
    std::swap(buf.p, b.p);
    std::copy(e, e + 2, ev);
    return true;
  }
};
// A stream with its side stream (see PipelineOpts::side)
struct Lane {
  cudaStream_t stream = nullptr, side = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  void make() {
    CK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
    CK(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
    CK(cudaEventCreateWithFlags(&fork, cudaEventDisableTiming));
    CK(cudaEventCreateWithFlags(&join, cudaEventDisableTiming));
  }
};
// A device's context.  Calls are serialised per grid, so two grids' calls
// enqueue on the lane at the same time; graphs are captured on a lane of their
// own (Capture), or what another thread enqueues, copies or waits for
// meanwhile would become part of the graph or end the capture.
struct Ctx : Lane {
  int dev = 0;
  Lane cap;
  std::mutex cap_mu;
  DBuf<float2> tw;  // W_2048^k
  Stage stage;
  std::mutex scratch_mu;
  std::multimap<size_t, void *> scratch;  // free blocks by size
  size_t scratch_total = 0;
  bool scratch_dirty = false;  // blocks were put back since the last wait for the stream
};
std::mutex g_ctx_mu;
std::map<int, std::unique_ptr<Ctx>> g_ctx;
thread_local int g_dev = -1;

Ctx &ctx() {
  if (g_dev < 0) {
    int d;
    CK(cudaGetDevice(&d));
    g_dev = d;
  }
  std::lock_guard<std::mutex> lk(g_ctx_mu);
  std::unique_ptr<Ctx> &slot = g_ctx[g_dev];
  if (!slot) {
    std::unique_ptr<Ctx> c(new Ctx());  // kept once it is whole
    c->dev = g_dev;
    CK(cudaSetDevice(g_dev));
    c->make();
    c->cap.make();
    std::vector<float2> t(FFTN);
    for (int k = 0; k < FFTN; k++) {
      double a = -2.0 * M_PI * (double)k / (double)FFTN;
      t[k] = make_float2((float)std::cos(a), (float)std::sin(a));
    }
    c->tw.alloc(t.size(), false);
    CK(cudaMemcpy(c->tw.p, t.data(), t.size() * sizeof(float2), cudaMemcpyHostToDevice));
    wait_uploads();
    slot = std::move(c);
  }
  CK(cudaSetDevice(slot->dev));
  return *slot;
}

// One graph capture on the device's capture lane (one at a time); ends the
// capture when the scope is left without finish().
class Capture {
  Ctx &C;
  std::lock_guard<std::mutex> lk;
  bool open = false;

 public:
  explicit Capture(Ctx &c) : C(c), lk(c.cap_mu) {
    CK(cudaStreamBeginCapture(C.cap.stream, cudaStreamCaptureModeThreadLocal));
    open = true;
  }
  Capture(const Capture &) = delete;
  Capture &operator=(const Capture &) = delete;
  ~Capture() {
    if (!open) return;
    cudaGraph_t dead = nullptr;
    cudaStreamEndCapture(C.cap.stream, &dead);
    if (dead) cudaGraphDestroy(dead);
    cudaGetLastError();
  }
  cudaStream_t stream() const { return C.cap.stream; }
  void finish(cudaGraph_t *graph) {
    open = false;
    CK(cudaStreamEndCapture(C.cap.stream, graph));
  }
};

// ------------------------------------------------------------ scratch pool
int scratch_device() { return ctx().dev; }
cudaStream_t scratch_stream() { return ctx().stream; }
size_t scratch_round(size_t b) {  // 512 bytes, or an eighth of the power of two below
  size_t step = 512;
  while (step * 16 <= b) step *= 2;
  return (b + step - 1) / step * step;
}
void scratch_flush(int dev) {
  std::lock_guard<std::mutex> lk(g_ctx_mu);
  for (auto &kv : g_ctx) {
    if (dev >= 0 && kv.first != dev) continue;
    Ctx &C = *kv.second;
    std::lock_guard<std::mutex> l2(C.scratch_mu);
    for (auto &b : C.scratch) cudaFree(b.second);  // waits for the device
    C.scratch.clear();
    C.scratch_total = 0;
    C.scratch_dirty = false;
  }
}
void *scratch_take(size_t bytes, size_t *got) {
  Ctx &C = ctx();
  const size_t want = bytes <= SCRATCH_BLOCK ? scratch_round(bytes) : bytes;  // no slack for blocks that are not kept
  *got = want;
  if (want <= SCRATCH_BLOCK) {
    std::lock_guard<std::mutex> lk(C.scratch_mu);
    auto it = C.scratch.lower_bound(want);
    if (it != C.scratch.end() && it->first <= 2 * want + (64u << 10)) {
      if (C.scratch_dirty) {
        CK(cudaStreamSynchronize(C.stream));
        C.scratch_dirty = false;
      }
      void *p = it->second;
      *got = it->first;
      C.scratch_total -= it->first;
      C.scratch.erase(it);
      return p;
    }
  }
  void *p = nullptr;
  cudaError_t e = cudaMalloc(&p, want);
  if (e != cudaSuccess) {
    cudaGetLastError();
    scratch_flush(-1);
    *got = bytes;  // no slack either when memory is short
    e = cudaMalloc(&p, bytes);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    fail(PASTA_E_NOMEM, "cudaMalloc of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
  }
  return p;
}
void scratch_put(void *p, size_t bytes, int dev) {
  Ctx *C = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_ctx_mu);
    auto it = g_ctx.find(dev);
    if (it != g_ctx.end()) C = it->second.get();
  }
  if (C && bytes <= SCRATCH_BLOCK) {
    std::lock_guard<std::mutex> lk(C->scratch_mu);
    if (C->scratch_total + bytes <= SCRATCH_TOTAL) {
      C->scratch.emplace(bytes, p);
      C->scratch_total += bytes;
      C->scratch_dirty = true;
      return;
    }
  }
  cudaFree(p);
}

// ------------------------------------------------------------- host copies
// memcpy of large arrays by a few threads (one core moves 8-10 GB/s, less
// into pages touched for the first time)
void copy_threads(void *dst, const void *src, size_t n) {
  constexpr size_t MOST = 4;
  const size_t parts = std::min(MOST, n >> 20);
  if (parts < 2) {
    std::memcpy(dst, src, n);
    return;
  }
  std::thread th[MOST];  // no allocation while threads run: nothing but a thread's start can fail
  const size_t per = (n / parts + 4095) & ~(size_t)4095;
  for (size_t k = 1; k < parts; k++) {
    const size_t o = k * per, m = k + 1 == parts ? n - o : per;
    try {
      th[k] = std::thread([=] { std::memcpy((char *)dst + o, (const char *)src + o, m); });
    } catch (const std::exception &) {  // no thread, or no memory for one
      std::memcpy((char *)dst + o, (const char *)src + o, m);
    }
  }
  std::memcpy(dst, src, per);
  for (auto &t : th)
    if (t.joinable()) t.join();
}

// Copies between host arrays and the device through the staging buffer, in
// order on the device's stream; pageable copies while another thread holds it
// or when no page-locked memory is to be had.
struct HostCopy {
  Ctx &C;
  std::unique_lock<std::mutex> lk;
  bool ok;
  explicit HostCopy(Ctx &c) : C(c), lk(c.stage.mu, std::try_to_lock), ok(lk.owns_lock() && c.stage.ready()) {}
  // room for n bytes (at most STAGE_HALF) in the current half, or the next one
  unsigned char *room(size_t n) {
    Stage &S = C.stage;
    if (S.fill + n > STAGE_HALF) {
      CK(cudaEventRecord(S.ev[S.at], C.stream));
      S.at ^= 1;
      S.fill = 0;
      CK(cudaEventSynchronize(S.ev[S.at]));
    }
    unsigned char *p = S.buf.p + (size_t)S.at * STAGE_HALF + S.fill;
    S.fill += (n + 255) & ~(size_t)255;
    return p;
  }
  void up(void *dst, const void *src, size_t n) {
    if (!ok) {
      CK(cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, C.stream));
      return;
    }
    for (size_t o = 0; o < n;) {
      const size_t m = std::min(n - o, STAGE_HALF);
      unsigned char *p = room(m);
      copy_threads(p, (const char *)src + o, m);
      CK(cudaMemcpyAsync((char *)dst + o, p, m, cudaMemcpyHostToDevice, C.stream));
      o += m;
    }
  }
  // waits for the copy; the next part is on its way while one is copied out
  void down(void *dst, const void *src, size_t n) {
    if (!ok || n < STAGE_MIN) {
      CK(cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, C.stream));
      CK(cudaStreamSynchronize(C.stream));
      return;
    }
    Stage &S = C.stage;
    CK(cudaStreamSynchronize(C.stream));  // both halves free
    S.at = 0;
    S.fill = STAGE_HALF;  // the next upload starts on the other half
    const size_t parts = (n + STAGE_HALF - 1) / STAGE_HALF;
    auto issue = [&](size_t k) {
      const size_t o = k * STAGE_HALF, m = std::min(n - o, STAGE_HALF);
      CK(cudaMemcpyAsync(S.buf.p + (k & 1) * STAGE_HALF, (const char *)src + o, m, cudaMemcpyDeviceToHost, C.stream));
      CK(cudaEventRecord(S.ev[k & 1], C.stream));
    };
    issue(0);
    for (size_t k = 0; k < parts; k++) {
      if (k + 1 < parts) issue(k + 1);
      CK(cudaEventSynchronize(S.ev[k & 1]));
      const size_t o = k * STAGE_HALF, m = std::min(n - o, STAGE_HALF);
      copy_threads((char *)dst + o, S.buf.p + (k & 1) * STAGE_HALF, m);
    }
  }
};

}  // namespace
