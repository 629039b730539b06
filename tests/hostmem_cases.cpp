// Failure paths of pasta_b200/csrc/hostmem.h on the CPU: the CUDA runtime is
// replaced by the stand-ins below, whose calls can be made to fail.
//   hostmem_cases <case>     exit code 0: passed
#include <atomic>
#include <chrono>
#include <cstdlib>
#include <cstring>
#include <new>
#include <set>

#include "../pasta_b200/csrc/hostmem.h"

// ------------------------------------------------- a runtime that can fail
namespace fake {
std::mutex mu;
size_t capacity = 1ull << 40, used = 0;  // "device memory" (nothing that large is touched)
std::map<void *, size_t> blocks;
std::vector<size_t> asked;               // sizes of all device allocations, in order
std::atomic<bool> pinned_fails{false}, events_fail{false}, streams_fail{false};
std::atomic<uintptr_t> next_handle{16};
std::set<cudaEvent_t> events;
std::set<cudaStream_t> capturing;
std::atomic<int> legacy_pending{0};      // copies on the legacy stream nothing has waited for
std::atomic<int> into_capture{0};        // calls that landed in a capture, or that end one
cudaError_t last = cudaSuccess;
cudaError_t set(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
bool in_capture(cudaStream_t s) {
  std::lock_guard<std::mutex> lk(mu);
  const bool c = capturing.count(s);
  into_capture += c;
  return c;
}
}  // namespace fake

extern "C" {
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  std::lock_guard<std::mutex> lk(fake::mu);
  return fake::capturing.insert(s).second ? cudaSuccess : fake::set(cudaErrorIllegalState);
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t *g) {
  std::lock_guard<std::mutex> lk(fake::mu);
  *g = (cudaGraph_t)(fake::next_handle += 16);
  return fake::capturing.erase(s) ? cudaSuccess : fake::set(cudaErrorIllegalState);
}
cudaError_t cudaMalloc(void **p, size_t n) {
  std::lock_guard<std::mutex> lk(fake::mu);
  fake::asked.push_back(n);
  if (fake::used + n > fake::capacity) {
    *p = nullptr;
    return fake::set(cudaErrorMemoryAllocation);
  }
  *p = std::malloc(std::min<size_t>(n, 64u << 20));
  fake::blocks[*p] = n;
  fake::used += n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  std::lock_guard<std::mutex> lk(fake::mu);
  auto it = fake::blocks.find(p);
  if (it == fake::blocks.end()) return fake::set(cudaErrorInvalidValue);
  fake::used -= it->second;
  fake::blocks.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
  if (fake::pinned_fails) return fake::set(cudaErrorMemoryAllocation);
  *p = std::malloc(n);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = fake::last;
  fake::last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
  std::memcpy(d, s, n);
  fake::legacy_pending++;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  if (!st || fake::in_capture(st)) return fake::set(cudaErrorInvalidResourceHandle);
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (!s || s == cudaStreamLegacy) fake::legacy_pending = 0;
  return fake::in_capture(s) ? fake::set(cudaErrorStreamCaptureUnsupported) : cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
  if (fake::streams_fail) return fake::set(cudaErrorMemoryAllocation);
  *s = (cudaStream_t)(fake::next_handle += 16);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) {
  if (fake::events_fail) return fake::set(cudaErrorMemoryAllocation);
  *e = (cudaEvent_t)(fake::next_handle += 16);
  std::lock_guard<std::mutex> lk(fake::mu);
  fake::events.insert(*e);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  std::lock_guard<std::mutex> lk(fake::mu);
  return fake::events.erase(e) ? cudaSuccess : fake::set(cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  fake::in_capture(s);
  std::lock_guard<std::mutex> lk(fake::mu);
  return fake::events.count(e) ? cudaSuccess : fake::set(cudaErrorInvalidResourceHandle);
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) { return cudaEventRecord(e, nullptr); }
cudaError_t cudaGetDevice(int *d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
}

// the n-th host allocation of this thread from now on fails (0: none)
static thread_local int new_countdown = 0;
void *operator new(size_t n) {
  if (new_countdown > 0 && --new_countdown == 0) throw std::bad_alloc();
  if (void *p = std::malloc(n)) return p;
  throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

#define EXPECT(cond)                                                     \
  do {                                                                   \
    if (!(cond)) {                                                       \
      std::fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #cond);    \
      std::_Exit(1);                                                     \
    }                                                                    \
  } while (0)

// ------------------------------------------------------------------- cases
// An allocation that only fits once the pool's free blocks are given back
// succeeds, also while another thread is inside ctx() or a release.
static void flush_while_contexts_are_looked_up() {
  ctx();
  {
    SBuf<char> a, b, c;
    a.alloc(60u << 20);
    b.alloc(60u << 20);
    c.alloc(60u << 20);
  }
  EXPECT(ctx().scratch_total >= (180u << 20));
  fake::capacity = 300ull << 20;
  std::atomic<bool> held{false};
  std::thread other([&] {
    std::lock_guard<std::mutex> lk(g_ctx_mu);
    held = true;
    std::this_thread::sleep_for(std::chrono::milliseconds(200));
  });
  while (!held) std::this_thread::yield();
  DBuf<char> big;
  int code = 0;
  try {
    // past the context lookup a scratch buffer makes: straight to the allocation
    big.alloc(200u << 20);
  } catch (const PErr &e) {
    code = e.code;
  }
  other.join();
  EXPECT(code == 0 && big.p);
  EXPECT(ctx().scratch.empty());
}

// No memory for a context's own table: an error, without a wait for a lock the
// thread itself holds.
static void context_without_memory() {
  fake::capacity = 0;
  int code = 0;
  try {
    ctx();
  } catch (const PErr &e) {
    code = e.code;
  }
  EXPECT(code == PASTA_E_NOMEM);
}

// A context that could not be made is made by the next call, whole.
static void context_made_again() {
  for (int what = 0; what < 3; what++) {
    fake::streams_fail = what == 0;
    fake::events_fail = what == 1;
    if (what == 2) fake::capacity = 0;
    int code = 0;
    try {
      ctx();
    } catch (const PErr &e) {
      code = e.code;
    }
    EXPECT(code != 0);
    fake::streams_fail = fake::events_fail = false;
    fake::capacity = 1ull << 40;
  }
  Ctx &C = ctx();
  EXPECT(C.stream && C.side && C.fork && C.join && C.tw.p);
  EXPECT(C.tw.p[0].x == 1.0f && C.tw.p[FFTN / 2].x == -1.0f);
}

// n bytes there and back through HostCopy, in one piece and in small pieces
static void copies_agree(size_t n) {
  std::vector<unsigned char> in(n), out(n, 0);
  for (size_t i = 0; i < n; i++) in[i] = (unsigned char)(i * 131 + (i >> 9));
  SBuf<unsigned char> d;
  d.alloc(n);
  HostCopy hc(ctx());
  hc.up(d.p, in.data(), n / 3);
  hc.up(d.p + n / 3, in.data() + n / 3, n - n / 3);
  hc.down(out.data(), d.p, n);
  EXPECT(in == out);
}

// Without page-locked memory, or without an event for it, copies go on
// unstaged; staged again once both can be had.
static void copies_without_staging() {
  for (int what = 0; what < 2; what++) {
    fake::pinned_fails = what == 0;
    ctx();
    fake::events_fail = what == 1;
    for (size_t n : {(size_t)1000, (size_t)200000, (size_t)9 << 20}) copies_agree(n);
    EXPECT(!ctx().stage.buf.p && !ctx().stage.ev[0] && !ctx().stage.ev[1]);
    fake::pinned_fails = fake::events_fail = false;
  }
  for (size_t n : {(size_t)1000, (size_t)200000, (size_t)9 << 20}) copies_agree(n);
  EXPECT(ctx().stage.buf.p && ctx().stage.ev[0] && ctx().stage.ev[1]);
}

// A copy by several threads is whole whichever of its host allocations fails.
static void threads_without_host_memory() {
  const size_t n = (4u << 20) + 4097;
  std::vector<unsigned char> in(n), out(n);
  for (size_t i = 0; i < n; i++) in[i] = (unsigned char)(i * 131 + (i >> 9));
  for (int k = 0; k < 10; k++) {
    std::fill(out.begin(), out.end(), 0);
    new_countdown = k;
    copy_threads(out.data(), in.data(), n);
    new_countdown = 0;
    EXPECT(in == out);
  }
}

// A buffer that fits the device's free memory exactly is had, small or large.
static void exact_fits() {
  ctx();
  for (size_t n : {(size_t)1000, (size_t)9 << 20, ((size_t)60 << 20) + 1, (size_t)64 << 20, ((size_t)64 << 20) + 1,
                   (size_t)1000 << 20, ((size_t)9 << 30) + 12}) {
    fake::capacity = fake::used + n;
    int code = 0;
    try {
      SBuf<char> b;
      b.alloc(n);
    } catch (const PErr &e) {
      code = e.code;
    }
    EXPECT(code == 0);
    scratch_flush(-1);
  }
}

// Another thread's copies and pool waits while a graph is captured stay out of
// the capture; captures come one at a time; one left by an exception is ended.
static void captures_are_alone() {
  Ctx &C = ctx();
  for (size_t n : {(size_t)1000, (size_t)5 << 20}) copies_agree(n);
  std::thread rival;
  std::atomic<bool> second{false};
  {
    Capture cap(C);
    EXPECT(cap.stream() != C.stream && cap.stream() != C.side);
    std::thread([] {
      for (int k = 0; k < 3; k++)
        for (size_t n : {(size_t)1000, (size_t)200000, (size_t)9 << 20}) copies_agree(n);
    }).join();
    rival = std::thread([&] {
      Capture again(ctx());
      second = true;
      cudaGraph_t g = nullptr;
      again.finish(&g);
    });
    std::this_thread::sleep_for(std::chrono::milliseconds(50));
    EXPECT(!second);
    cudaGraph_t g = nullptr;
    cap.finish(&g);
    EXPECT(g);
  }
  rival.join();
  EXPECT(second);
  try {
    Capture cap(C);
    fail(PASTA_E_INTERNAL, "a launch that failed");
  } catch (const PErr &) {
  }
  EXPECT(fake::capturing.empty() && fake::into_capture == 0);
  Capture cap(C);
  cudaGraph_t g = nullptr;
  cap.finish(&g);
}

// A context's own table is complete when it is handed out, other uploads after
// wait_uploads(): nothing orders the library's streams behind the legacy stream.
static void uploads_are_waited_for() {
  ctx();
  EXPECT(fake::legacy_pending == 0);
  DBuf<int> a;
  a.upload(std::vector<int>(1000, 3));
  wait_uploads();
  EXPECT(fake::legacy_pending == 0 && a.p[999] == 3);
}

int main(int argc, char **argv) {
  const std::string which = argc > 1 ? argv[1] : "";
  if (which == "flush_while_contexts_are_looked_up") flush_while_contexts_are_looked_up();
  else if (which == "context_without_memory") context_without_memory();
  else if (which == "context_made_again") context_made_again();
  else if (which == "copies_without_staging") copies_without_staging();
  else if (which == "threads_without_host_memory") threads_without_host_memory();
  else if (which == "exact_fits") exact_fits();
  else if (which == "captures_are_alone") captures_are_alone();
  else if (which == "uploads_are_waited_for") uploads_are_waited_for();
  else return 2;
  std::_Exit(0);
}
