// host_copy.cu — copies between ordinary (pageable) host memory and the device.
//
// cudaMemcpy stages such memory through the driver's own page-locked buffers on the calling thread: 10 to 18 GB/s on the 16-core
// hosts measured, of the 50 GB/s that the link takes from page-locked memory.  Here a few helper threads and the caller move
// pieces of 64 KB between the caller's memory and a page-locked ring, while the caller issues the DMA of whole segments of up
// to 2 MB (a copy command costs about 8 us on these hosts whatever its size, so small segments from several threads gave
// 15 GB/s, and 2 MB to the host in four of them took 95 us where one takes 46).  To the device the first segments are small, so that the
// link starts early; to the host the last one is, so that little is left to move when the link is done.  The helpers make no CUDA calls.  Used from COPY_MIN bytes up, with helpers
// from HELP_MIN up (waking them costs more than a piece), and for pageable memory only; page-locked memory goes straight to cudaMemcpyAsync.
//   9.4 MB to the device 0.51 -> 0.25 ms, 6.3 MB to the host 0.31 -> 0.20 ms, 64 MB 4.4 -> 1.6 and 1.8 ms (42 and 38 GB/s)
#include <immintrin.h>

#include <chrono>
#include <condition_variable>
#include <cstring>
#include <new>
#include <system_error>
#include <thread>

#include "ops.h"

namespace mb {
namespace {

constexpr size_t COPY_MIN = size_t(64) << 10;
constexpr size_t PIECE = size_t(64) << 10;
constexpr size_t HELP_MIN = size_t(88) << 10;  // in and out of an element-wise layer: 72 KB 45 us with helpers, 43 without; 88 KB 46 and 47; 128 KB 50 and 66
constexpr size_t SEGMENT = size_t(2) << 20;
constexpr int RING = 8;  // segments: 16 MB of page-locked memory per device
constexpr int MAX_HELPERS = 5;

void cpu_relax() { __builtin_ia32_pause(); }

// Into the ring with streaming stores: lines left dirty in the helpers' caches made the copy engine's reads slow (9.4 MB to the
// device 0.61 ms with plain stores).
__attribute__((target("avx2"))) void copy_streaming(uint8_t* dst, const uint8_t* src, size_t n) {
  size_t i = 0;
  for (; i + 128 <= n; i += 128) {
    const __m256i a = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(src + i)), b = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(src + i + 32));
    const __m256i c = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(src + i + 64)), d = _mm256_loadu_si256(reinterpret_cast<const __m256i*>(src + i + 96));
    _mm256_stream_si256(reinterpret_cast<__m256i*>(dst + i), a);
    _mm256_stream_si256(reinterpret_cast<__m256i*>(dst + i + 32), b);
    _mm256_stream_si256(reinterpret_cast<__m256i*>(dst + i + 64), c);
    _mm256_stream_si256(reinterpret_cast<__m256i*>(dst + i + 96), d);
  }
  if (i < n) memcpy(dst + i, src + i, n - i);
  _mm_sfence();
}
void copy_into_ring(uint8_t* dst, const uint8_t* src, size_t n) {
  static const bool avx2 = __builtin_cpu_supports("avx2");
  if (avx2) copy_streaming(dst, src, n); else memcpy(dst, src, n);
}

struct Job {
  bool to_device = false;
  uint8_t* dev = nullptr;
  uint8_t* host = nullptr;
  size_t bytes = 0, pieces = 0, segments = 0;
  size_t lead = 0, last = 0;  // to the host: segments of SEGMENT bytes, bytes of the one behind them (all but the last)
  std::atomic<size_t> next{0};   // next piece to move
  std::atomic<size_t> open{0};   // segments whose ring slot may be filled (to the device) / has landed (to the host)
  std::atomic<uint32_t> moved[RING];
  std::atomic<bool> cancel{false};

  void cut() {
    pieces = (bytes + PIECE - 1) / PIECE;
    if (to_device) {  // 512 KB, 1 MB, then SEGMENT each
      segments = seg_of(pieces - 1) + 1;
      return;
    }
    size_t rest = bytes;
    while (rest > SEGMENT + SEGMENT / 2) { rest -= SEGMENT; ++lead; }
    // (a rest of 512 KB and less goes as one)
    last = rest <= SEGMENT / 4 ? rest : (rest * 5 / 8 + PIECE - 1) / PIECE * PIECE;
    if (last > SEGMENT) last = SEGMENT;
    segments = lead + (rest > last ? 2 : 1);
  }
  size_t seg_off(size_t s) const {
    if (to_device) return s == 0 ? 0 : s == 1 ? SEGMENT / 4 : SEGMENT / 4 * 3 + (s - 2) * SEGMENT;
    return s <= lead ? s * SEGMENT : lead * SEGMENT + last;
  }
  size_t seg_of(size_t piece) const {
    const size_t off = piece * PIECE;
    if (to_device) return off < SEGMENT / 4 ? 0 : off < SEGMENT / 4 * 3 ? 1 : 2 + (off - SEGMENT / 4 * 3) / SEGMENT;
    return off < lead * SEGMENT ? off / SEGMENT : off < lead * SEGMENT + last ? lead : lead + 1;
  }
  size_t pieces_of(size_t s) const { return (seg_bytes(s) + PIECE - 1) / PIECE; }
  size_t seg_bytes(size_t s) const { return (s + 1 == segments ? bytes : seg_off(s + 1)) - seg_off(s); }
  void move(size_t piece, uint8_t* ring) {
    const size_t off = piece * PIECE, s = seg_of(piece), n = bytes - off < PIECE ? bytes - off : PIECE;
    uint8_t* slot = ring + (s % RING) * SEGMENT + (off - seg_off(s));
    if (to_device) copy_into_ring(slot, host + off, n); else memcpy(host + off, slot, n);
    moved[s % RING].fetch_add(1, std::memory_order_release);
  }
};

}  // namespace

// The helpers and the ring of one device.  One job at a time (`call` is held for the whole copy, waits for the caller's own stream
// included, so nobody queues for it); a helper that wakes late finds no piece left.  `active` counts the helpers that may still touch the current job.
struct HostCopier {
  std::mutex call, mu;
  std::condition_variable cv;
  std::vector<std::thread> threads;
  Job* job = nullptr;
  std::atomic<uint64_t> epoch{0};
  int active = 0;
  bool stop = false, no_ring = false;
  int inject = 0;  // host_copy_selftest: 1 no page-locked memory, 2 no second thread
  uint8_t* ring = nullptr;
  cudaEvent_t ev[RING] = {};
  bool in_flight[RING] = {};
  std::thread::id by[RING] = {};  // whose copy is in flight in a slot

  // The ring, and as many helpers as the machine starts; false: no ring to be had (asked for once), copies go without
  bool init() {
    if (ring) return true;
    if (no_ring) return false;
    void* p = nullptr;
    cudaError_t e = inject & 1 ? cudaErrorMemoryAllocation : cudaHostAlloc(&p, RING * SEGMENT, cudaHostAllocPortable);
    for (auto& v : ev)
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming);
    if (e != cudaSuccess) {
      cudaGetLastError();  // (not an error of the copy's)
      for (auto& v : ev) {
        if (v) cudaEventDestroy(v);
        v = nullptr;
      }
      if (p) cudaFreeHost(p);
      no_ring = true;
      return false;
    }
    ring = static_cast<uint8_t*>(p);
    const unsigned cores = std::thread::hardware_concurrency();
    const int helpers = cores >= 4 ? static_cast<int>(cores / 2 < MAX_HELPERS ? cores / 2 : MAX_HELPERS) : 0;
    try {
      for (int i = 0; i < helpers; ++i) {
        if ((inject & 2) && i > 0) throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
        threads.emplace_back([this] { loop(); });
      }
    } catch (...) {
      // no more threads, or no memory: the caller moves what the ones that run do not
    }
    return true;
  }

  void loop() {
    uint64_t seen = 0;
    for (;;) {
      // The copies of one call, and the calls of a loop, follow each other closely: stay awake for a moment before sleeping.  An element-
      // wise layer of 1 MB 145 us with 100 us, 151 with 75, 153 with 50; a decode step of 16 samples 818 us with 100, 820 with 40, 826
      // with 20.  A call burns up to 0.5 ms of CPU time for it, on all helpers together.
      const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(100);
      while (epoch.load(std::memory_order_acquire) == seen && std::chrono::steady_clock::now() < until) cpu_relax();
      Job* j;
      {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return stop || epoch.load() != seen; });
        if (stop) return;
        seen = epoch.load();
        j = job;
        if (!j) continue;
        ++active;
      }
      for (;;) {
        const size_t i = j->next.fetch_add(1, std::memory_order_relaxed);
        if (i >= j->pieces) break;
        while (j->seg_of(i) >= j->open.load(std::memory_order_acquire) && !j->cancel.load()) cpu_relax();
        if (j->cancel.load()) break;
        j->move(i, ring);
      }
      std::lock_guard<std::mutex> lk(mu);
      if (--active == 0) cv.notify_all();
    }
  }

  // the caller's share: one piece of an open segment; false when there is none to take
  bool help(Job& j) {
    size_t i = j.next.load(std::memory_order_relaxed);
    while (i < j.pieces && j.seg_of(i) < j.open.load(std::memory_order_relaxed)) {
      if (j.next.compare_exchange_weak(i, i + 1, std::memory_order_relaxed)) {
        j.move(i, ring);
        return true;
      }
    }
    return false;
  }
  void wait_moved(Job& j, size_t s) {
    while (j.moved[s % RING].load(std::memory_order_acquire) < j.pieces_of(s))
      if (!help(j)) cpu_relax();
  }

  cudaError_t drive(Job& j, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    if (j.to_device) {
      auto free_slot = [&](size_t s) {  // the DMA that last read this slot (of this job or an earlier one)
        if (in_flight[s % RING] && e == cudaSuccess) e = cudaEventSynchronize(ev[s % RING]);
        in_flight[s % RING] = false;
        j.moved[s % RING].store(0);
        j.open.store(s + 1, std::memory_order_release);
      };
      for (size_t s = 0; s < j.segments && s < RING && e == cudaSuccess; ++s) free_slot(s);
      for (size_t s = 0; s < j.segments && e == cudaSuccess; ++s) {
        wait_moved(j, s);
        e = cudaMemcpyAsync(j.dev + j.seg_off(s), ring + (s % RING) * SEGMENT, j.seg_bytes(s), cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(ev[s % RING], st);
        in_flight[s % RING] = true;
        by[s % RING] = std::this_thread::get_id();
        if (s + RING < j.segments && e == cudaSuccess) free_slot(s + RING);
      }
      return e;
    }
    auto fetch = [&](size_t s) {
      if (in_flight[s % RING] && e == cudaSuccess) e = cudaEventSynchronize(ev[s % RING]);  // an earlier job's
      in_flight[s % RING] = false;
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(ring + (s % RING) * SEGMENT, j.dev + j.seg_off(s), j.seg_bytes(s), cudaMemcpyDeviceToHost, st);
      if (e == cudaSuccess) e = cudaEventRecord(ev[s % RING], st);
    };
    for (size_t s = 0; s < j.segments && s < RING && e == cudaSuccess; ++s) fetch(s);
    for (size_t s = 0; s < j.segments && e == cudaSuccess; ++s) {
      e = cudaEventSynchronize(ev[s % RING]);
      if (e != cudaSuccess) break;
      j.moved[s % RING].store(0);
      j.open.store(s + 1, std::memory_order_release);
      if (s + RING < j.segments) {
        wait_moved(j, s);
        fetch(s + RING);
      }
    }
    if (e == cudaSuccess)
      for (size_t s = j.segments > RING ? j.segments - RING : 0; s < j.segments; ++s) wait_moved(j, s);
    return e;
  }

  // Does another thread's copy, which may stand behind its kernels, hold one of the first slots?  (A thread's own earlier copies are done, or
  // copies in of the same call.  Waiting for one of these before a slot is used again waits for nothing that this copy does not stand
  // behind itself: on one stream it is ahead of it, and a copy out on a stream of its own follows the kernels that read what came in.)
  bool held_by_others(const Job& j) {
    for (size_t s = 0; s < j.segments && s < RING; ++s)
      if (in_flight[s] && by[s] != std::this_thread::get_id()) {
        if (cudaEventQuery(ev[s]) != cudaSuccess) return true;
        in_flight[s] = false;
      }
    return false;
  }

  // *taken = false: there is no ring, or it is another call's at the moment; nothing was done.  Its copies may stand behind
  // kernels, for which a call of another thread must not wait; the caller copies without the ring.
  int copy(Job& j, cudaStream_t st, bool* taken) {
    std::unique_lock<std::mutex> one(call, std::try_to_lock);
    *taken = one.owns_lock() && init();
    if (!*taken) return MIMIR_B200_OK;
    j.cut();
    if (held_by_others(j)) {
      *taken = false;
      return MIMIR_B200_OK;
    }
    if (j.bytes >= HELP_MIN) {  // (the caller moves less by itself)
      {
        std::lock_guard<std::mutex> lk(mu);
        job = &j;
        epoch.fetch_add(1, std::memory_order_release);
      }
      cv.notify_all();
    }
    const cudaError_t e = drive(j, st);
    if (e != cudaSuccess) j.cancel.store(true);
    {
      std::unique_lock<std::mutex> lk(mu);
      job = nullptr;  // nobody joins any more
      cv.wait(lk, [&] { return active == 0; });
    }
    if (e != cudaSuccess) return fail(MIMIR_B200_E_CUDA, "host copy failed: %s", cudaGetErrorString(e));
    return MIMIR_B200_OK;
  }

  ~HostCopier() {
    {
      std::lock_guard<std::mutex> lk(mu);
      stop = true;
      epoch.fetch_add(1);
    }
    cv.notify_all();
    for (auto& t : threads) t.join();
    if (ring) cudaFreeHost(ring);
    for (auto e : ev) if (e) cudaEventDestroy(e);
  }
};

namespace {
bool pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}
}  // namespace
bool host_memory(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered || a.type == cudaMemoryTypeHost;
}
namespace {
HostCopier* copier() {
  static std::mutex mu;
  std::lock_guard<std::mutex> lk(mu);
  if (!ctx().copier) ctx().copier = new (std::nothrow) HostCopier();  // (never destroyed at exit: a helper may be waiting in it)
  return ctx().copier;
}
int copy(HostCopier* c, bool to_device, void* dev, void* host, size_t bytes, cudaStream_t st, bool* taken) {
  *taken = false;
  if (bytes >= COPY_MIN && pageable(host)) {
    Job j;
    j.to_device = to_device;
    j.dev = static_cast<uint8_t*>(dev);
    j.host = static_cast<uint8_t*>(host);
    j.bytes = bytes;
    if (c) MB_TRY(c->copy(j, st, taken));
    if (*taken) return MIMIR_B200_OK;
    // (the driver has locks of its own: while one thread's copy of pageable memory stands behind a kernel the others' wait)
    MB_CUDA(cudaStreamSynchronize(st));
  }
  MB_CUDA(cudaMemcpyAsync(to_device ? dev : host, to_device ? host : dev, bytes, to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, st));
  return MIMIR_B200_OK;
}
}  // namespace

int copy_to_device(void* dev, const void* host, size_t bytes, cudaStream_t st) {
  bool taken;
  return copy(bytes >= COPY_MIN ? copier() : nullptr, true, dev, const_cast<void*>(host), bytes, st, &taken);
}
int copy_to_host(void* host, const void* dev, size_t bytes, cudaStream_t st) {
  bool taken;
  return copy(bytes >= COPY_MIN ? copier() : nullptr, false, const_cast<void*>(dev), host, bytes, st, &taken);
}
int host_copy_selftest(int inject, const float* src, float* dst, size_t n, int* ring_copies) {
  HostCopier* c = new (std::nothrow) HostCopier();
  if (!c) return fail(MIMIR_B200_E_INVALID, "selftest: no memory");
  c->inject = inject;
  void* dev = nullptr;
  int s = dev_alloc(&dev, n * sizeof(float), "host copy selftest");
  bool in = false, out = false;
  cudaStream_t st[2] = {};  // in and out on streams of their own, as a model copies
  cudaEvent_t done = nullptr;
  if (s == MIMIR_B200_OK && (cudaStreamCreateWithFlags(&st[0], cudaStreamNonBlocking) != cudaSuccess || cudaStreamCreateWithFlags(&st[1], cudaStreamNonBlocking) != cudaSuccess ||
                             cudaEventCreateWithFlags(&done, cudaEventDisableTiming) != cudaSuccess))
    s = fail(MIMIR_B200_E_CUDA, "selftest: no streams");
  if (s == MIMIR_B200_OK) s = copy(c, true, dev, const_cast<float*>(src), n * sizeof(float), st[0], &in);
  if (s == MIMIR_B200_OK && (cudaEventRecord(done, st[0]) != cudaSuccess || cudaStreamWaitEvent(st[1], done, 0) != cudaSuccess)) s = fail(MIMIR_B200_E_CUDA, "selftest: ordering failed");
  if (s == MIMIR_B200_OK) s = copy(c, false, dev, dst, n * sizeof(float), st[1], &out);
  for (auto v : st) {
    if (v && cudaStreamSynchronize(v) != cudaSuccess && s == MIMIR_B200_OK) s = fail(MIMIR_B200_E_CUDA, "selftest: synchronisation failed");
    if (v) cudaStreamDestroy(v);
  }
  if (done) cudaEventDestroy(done);
  dev_free(dev, n * sizeof(float));
  delete c;
  if (ring_copies) *ring_copies = static_cast<int>(in) + static_cast<int>(out);
  return s;
}
void release_host_copier() {
  delete ctx().copier;
  ctx().copier = nullptr;
}

}  // namespace mb
