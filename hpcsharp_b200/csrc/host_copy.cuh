// Host <-> device copies of the host-array entry points.
//
// A caller array in page-locked (pinned) memory is moved by one cudaMemcpyAsync.  A pageable
// array -- a .NET array fixed for P/Invoke is pageable memory -- would otherwise be staged by
// the CUDA driver through its own small pinned buffers, copied on the calling thread alone, and
// its transfer then runs well below the host link's bandwidth.  Instead it is cut into chunks:
// a few host worker threads copy each chunk into a slot of a pinned ring that the context owns,
// and one cudaMemcpyAsync per chunk moves it, so the host copies of later chunks overlap the
// DMA of earlier ones.  Device-to-host runs the same ring backwards.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <fstream>
#include <functional>
#include <mutex>
#include <string>
#include <system_error>
#include <thread>
#include <vector>
#if defined(__x86_64__)
#include <emmintrin.h>
#endif

#include "sort_host.cuh"

namespace hpcs {

// memcpy with streaming (non-temporal) stores on x86-64: the destination's cache lines are
// written without being read first, so a copy moves two bytes of host memory traffic per byte
// instead of three, and it does not evict the caches.  The stores are fenced before return
// (the DMA engine reads the destination after the copying thread signals completion).
inline void stream_copy(void* dst_v, const void* src_v, size_t bytes) {
#if defined(__x86_64__)
  auto* dst = static_cast<unsigned char*>(dst_v);
  const auto* src = static_cast<const unsigned char*>(src_v);
  size_t head = (16u - (reinterpret_cast<uintptr_t>(dst) & 15u)) & 15u;
  if (head > bytes) head = bytes;
  std::memcpy(dst, src, head);
  dst += head;
  src += head;
  bytes -= head;
  const size_t blocks = bytes / 64;
  for (size_t i = 0; i < blocks; i++, dst += 64, src += 64) {
    const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src));
    const __m128i b = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + 16));
    const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + 32));
    const __m128i d = _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + 48));
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst), a);
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + 16), b);
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + 32), c);
    _mm_stream_si128(reinterpret_cast<__m128i*>(dst + 48), d);
  }
  std::memcpy(dst, src, bytes - blocks * 64);
  _mm_sfence();
#else
  std::memcpy(dst_v, src_v, bytes);
#endif
}

// A fixed set of worker threads that run one memcpy split into equal pieces; the calling thread
// copies the first piece itself and returns when every piece is done.  A worker looks for the next
// copy for SPIN before it goes to sleep, and the caller for the last piece: the chunks of one call
// follow each other within that time, and a wake-up through the kernel costs as much as a 1 MiB chunk.
class CopyPool {
 public:
  explicit CopyPool(int workers) {
    threads_.reserve(size_t(workers));
    try {
      for (int i = 0; i < workers; i++) threads_.emplace_back([this, i] { loop(i + 1); });
    } catch (const std::system_error&) {  // no more threads here: copy with those that started
    }
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : threads_) t.join();
  }
  int parts() const { return int(threads_.size()) + 1; }
  void copy(void* dst, const void* src, size_t bytes) {
    if (threads_.empty()) {
      stream_copy(dst, src, bytes);
      return;
    }
    {
      std::lock_guard<std::mutex> lk(mu_);
      dst_ = static_cast<unsigned char*>(dst);
      src_ = static_cast<const unsigned char*>(src);
      bytes_ = bytes;
      pending_.store(int(threads_.size()), std::memory_order_relaxed);
      gen_.fetch_add(1, std::memory_order_release);
    }
    cv_.notify_all();
    piece(0);
    if (spin([this] { return pending_.load(std::memory_order_acquire) == 0; })) return;
    std::unique_lock<std::mutex> lk(mu_);
    done_cv_.wait(lk, [this] { return pending_.load(std::memory_order_acquire) == 0; });
  }

 private:
  // Looks at `ready` for up to SPIN before the caller blocks.
  static constexpr std::chrono::microseconds SPIN{100};
  template <class F>
  static bool spin(F&& ready) {
    const auto until = std::chrono::steady_clock::now() + SPIN;
    do {
      for (int i = 0; i < 64; i++) {
        if (ready()) return true;
#if defined(__x86_64__)
        _mm_pause();
#endif
      }
      std::this_thread::yield();  // where threads outnumber CPUs the one looked for may need this one
    } while (std::chrono::steady_clock::now() < until);
    return false;
  }
  void piece(int idx) {
    const size_t per = ((bytes_ + size_t(parts()) - 1) / size_t(parts()) + 63) & ~size_t(63);  // covers bytes_
    const size_t lo = std::min(bytes_, per * size_t(idx));
    const size_t hi = std::min(bytes_, lo + per);
    if (hi > lo) stream_copy(dst_ + lo, src_ + lo, hi - lo);
  }
  void loop(int idx) {
    uint64_t seen = 0;
    for (;;) {
      if (seen == 0 || !spin([&] { return gen_.load(std::memory_order_acquire) != seen; })) {
        std::unique_lock<std::mutex> lk(mu_);
        cv_.wait(lk, [&] { return stop_ || gen_.load(std::memory_order_relaxed) != seen; });
        if (stop_) return;
      }
      // (a new generation starts only after every worker finished the last one)
      seen = gen_.load(std::memory_order_acquire);
      piece(idx);
      if (pending_.fetch_sub(1, std::memory_order_acq_rel) == 1) {
        std::lock_guard<std::mutex> lk(mu_);  // the caller is either before its wait or in it
        done_cv_.notify_one();
      }
    }
  }
  std::vector<std::thread> threads_;
  std::mutex mu_;
  std::condition_variable cv_, done_cv_;
  bool stop_ = false;
  std::atomic<uint64_t> gen_{0};
  std::atomic<int> pending_{0};
  unsigned char* dst_ = nullptr;
  const unsigned char* src_ = nullptr;
  size_t bytes_ = 0;
};

// CPUs that the process may use at a time by its control group's quota (cgroup v2, its group and every group
// above; else v1), at least 1; no quota: 0.  `root` and `self` stand for /sys/fs/cgroup and /proc/self/cgroup.
inline int quota_cpus(const std::string& root, const std::string& self) {
  int least = 0;
  auto note = [&](double quota, double period) {
    if (quota <= 0 || period <= 0) return;
    const int cpus = std::max(1, int(quota / period + 0.5));
    least = least ? std::min(least, cpus) : cpus;
  };
  auto number = [](const std::string& path) {
    double v = 0;
    std::ifstream(path) >> v;
    return v;
  };
  std::string line, group;
  for (std::ifstream f(self); std::getline(f, line);)
    if (line.compare(0, 3, "0::") == 0) group = line.substr(3);
  for (;;) {
    while (!group.empty() && group.back() == '/') group.pop_back();
    std::ifstream f(root + group + "/cpu.max");  // "quota period", or "max period"
    double quota = 0, period = 0;
    if (f >> quota >> period) note(quota, period);
    if (group.empty()) break;
    group.erase(group.rfind('/') == std::string::npos ? 0 : group.rfind('/'));
  }
  note(number(root + "/cpu/cpu.cfs_quota_us"), number(root + "/cpu/cpu.cfs_period_us"));
  return least;
}

// Copy threads: the host's hardware threads, at most 8, and no more than a CPU quota allows (the threads look
// for work between chunks: more of them than CPUs wait for one another, and spend the quota).  Measured on a 16-core host of a B200
// node (1 GiB through 16 MiB chunks): pageable -> pinned 10 GB/s on one thread, 46-48 GB/s on
// 8, 44-45 GB/s on 16; pinned -> pageable with streaming stores 61 GB/s on 8 and 51 GB/s on
// 16.  The DMA engine moves about 56 GB/s each way over the host link.
inline int stager_threads() {
  static const int threads = [] {
    const unsigned hw = std::thread::hardware_concurrency();
    const int quota = quota_cpus("/sys/fs/cgroup", "/proc/self/cgroup");
    const int cpus = std::min(8, int(hw ? hw : 1u));
    return std::max(1, quota ? std::min(cpus, quota) : cpus);
  }();
  return threads;
}

// Two rings, each allocated when first needed.  Arrays of 32 MiB and more run in 16 MiB chunks, where
// the chunk's DMA (0.3 ms) is long beside its hand-over.  Shorter ones run in quarters of 512 KiB to
// 2 MiB, so that a 2 MB array still has its host copies and its DMA overlapped, and the chunk's pieces
// are worth a thread each.  What bounds such a call is the host's side of the copy, not the link: the
// driver's own staging of pageable memory moves 7-8 GB/s on the calling thread.  Sorting n u32 keys of
// a pageable array, driver's staging -> this one, microseconds per call (16 host threads):
//   10,000: 82 -> 64    65,536: 127 -> 91    262,144: 296 -> 186    1,000,003: 715 -> 350
//   2,000,000: 1290 -> 610    4,000,000: 2440 -> 930    8,000,000: 4810 -> 1690
// and with 16 contexts sorting at once from 16 threads, 20,000: 1206 -> 484, 1,000,003: 9490 -> 7450.
struct HostStager {
  static constexpr int SLOTS = 4;
  static constexpr size_t CHUNK = size_t(16) << 20;
  static constexpr size_t SMALL_CHUNK = size_t(2) << 20;
  static constexpr size_t MIN_CHUNK = size_t(512) << 10;
  static constexpr size_t SHARE_BYTES = size_t(256) << 10;
  // A ring of SLOTS chunks of pinned host memory, allocated when first needed.
  struct Ring {
    unsigned char* mem = nullptr;
    size_t slot_bytes = 0;
    cudaEvent_t slot_done[SLOTS] = {};
    unsigned char* slot(int i) const { return mem + size_t(i) * slot_bytes; }
  };
  Ring rings[2];  // for short and long arrays
  CopyPool* pool = nullptr;  // started by the first chunk that is shared out
  void copy(void* dst, const void* src, size_t bytes);
  ~HostStager() {
    delete pool;
    for (Ring& r : rings) {
      for (auto& e : r.slot_done)
        if (e) cudaEventDestroy(e);
      if (r.mem) cudaFreeHost(r.mem);
    }
  }
};

// One chunk of the host's side of a copy: by the pool from SHARE_BYTES on, else on this thread.
inline void HostStager::copy(void* dst, const void* src, size_t bytes) {
  if (bytes < SHARE_BYTES) {
    std::memcpy(dst, src, bytes);
    return;
  }
  if (!pool) pool = new CopyPool(stager_threads() - 1);
  pool->copy(dst, src, bytes);
}

// The ring and the chunk size for an array of `bytes`.  *ring stays null where the pinned memory of the
// short arrays' ring cannot be had: such an array is then copied by the driver.
inline int get_stager(hpcs_ctx* ctx, size_t bytes, HostStager::Ring** ring, size_t* chunk) {
  *ring = nullptr;
  if (!ctx->stager) ctx->stager = new HostStager();
  const bool large = bytes >= 2 * HostStager::CHUNK;
  HostStager::Ring& r = ctx->stager->rings[large ? 1 : 0];
  if (!r.mem) {
    r.slot_bytes = large ? HostStager::CHUNK : HostStager::SMALL_CHUNK;
    cudaError_t e = cudaSuccess;
    for (int i = 0; e == cudaSuccess && i < HostStager::SLOTS; i++)
      if (!r.slot_done[i]) e = cudaEventCreateWithFlags(&r.slot_done[i], cudaEventDisableTiming);
    if (e == cudaSuccess)
      e = cudaHostAlloc(reinterpret_cast<void**>(&r.mem), HostStager::SLOTS * r.slot_bytes, cudaHostAllocDefault);
    if (e != cudaSuccess) {
      r.mem = nullptr;
      if (large) return cuda_fail(e, "pinned staging ring");
      cudaGetLastError();
      return HPCS_OK;
    }
  }
  // a quarter of a short array in whole 64 KiB, so that its chunks are equal
  const size_t quarter = (bytes / 4 + 65535) & ~size_t(65535);
  *chunk = large ? r.slot_bytes : std::min(r.slot_bytes, std::max(HostStager::MIN_CHUNK, quarter));
  *ring = &r;
  return HPCS_OK;
}

// True when the copy should be staged: a pageable host range of at least STAGE_MIN_BYTES, and the
// context allows staging.  Shorter ones are left to the driver, which puts them into the command itself.
constexpr size_t STAGE_MIN_BYTES = size_t(32) << 10;
inline bool stage_copy(hpcs_ctx* ctx, const void* host, size_t bytes) {
  if (!ctx->cfg.staged_host_copies || bytes < STAGE_MIN_BYTES) return false;
  cudaPointerAttributes attr{};
  if (cudaPointerGetAttributes(&attr, host) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return attr.type == cudaMemoryTypeUnregistered;
}

// Host -> device on stream s.  Returns when the last chunk is enqueued (the host array may be
// reused once the stream has passed that point: the caller synchronises before returning).
inline int copy_to_device(hpcs_ctx* ctx, void* dev, const void* host, size_t bytes, cudaStream_t s) {
  HostStager::Ring* ring = nullptr;
  size_t chunk = 0;
  if (stage_copy(ctx, host, bytes)) {
    int rc = get_stager(ctx, bytes, &ring, &chunk);
    if (rc != HPCS_OK) return rc;
  }
  if (!ring) {
    HPCS_CUDA(cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, s));
    return HPCS_OK;
  }
  HostStager* st = ctx->stager;
  const auto* src = static_cast<const unsigned char*>(host);
  auto* dst = static_cast<unsigned char*>(dev);
  size_t off = 0;
  for (int c = 0; off < bytes; c++) {
    const int slot = c % HostStager::SLOTS;
    const size_t sz = std::min(chunk, bytes - off);
    unsigned char* buf = ring->slot(slot);
    HPCS_CUDA(cudaEventSynchronize(ring->slot_done[slot]));  // the slot's previous DMA is done
    st->copy(buf, src + off, sz);
    HPCS_CUDA(cudaMemcpyAsync(dst + off, buf, sz, cudaMemcpyHostToDevice, s));
    HPCS_CUDA(cudaEventRecord(ring->slot_done[slot], s));
    off += sz;
  }
  return HPCS_OK;
}

// Device -> host after the work already on stream s; returns with the data in the host array.
inline int copy_to_host(hpcs_ctx* ctx, void* host, const void* dev, size_t bytes, cudaStream_t s) {
  HostStager::Ring* ring = nullptr;
  size_t chunk = 0;
  if (stage_copy(ctx, host, bytes)) {
    int rc = get_stager(ctx, bytes, &ring, &chunk);
    if (rc != HPCS_OK) return rc;
  }
  if (!ring) {
    HPCS_CUDA(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, s));
    HPCS_CUDA(cudaStreamSynchronize(s));
    return HPCS_OK;
  }
  HostStager* st = ctx->stager;
  auto* dst = static_cast<unsigned char*>(host);
  const auto* src = static_cast<const unsigned char*>(dev);
  const int64_t chunks = int64_t((bytes + chunk - 1) / chunk);
  auto chunk_size = [&](int64_t c) { return std::min(chunk, bytes - size_t(c) * chunk); };
  // keep SLOTS chunks in flight: issue chunk c, then drain chunk c - SLOTS + 1 ... in order
  int64_t drained = 0;
  for (int64_t c = 0; c < chunks; c++) {
    const int slot = int(c % HostStager::SLOTS);
    if (c >= HostStager::SLOTS) {  // the slot's previous chunk must be copied out first
      const int64_t d = c - HostStager::SLOTS;
      HPCS_CUDA(cudaEventSynchronize(ring->slot_done[slot]));
      st->copy(dst + size_t(d) * chunk, ring->slot(slot), chunk_size(d));
      drained = d + 1;
    }
    HPCS_CUDA(cudaMemcpyAsync(ring->slot(slot), src + size_t(c) * chunk,
                              chunk_size(c), cudaMemcpyDeviceToHost, s));
    HPCS_CUDA(cudaEventRecord(ring->slot_done[slot], s));
  }
  for (int64_t d = drained; d < chunks; d++) {
    const int slot = int(d % HostStager::SLOTS);
    HPCS_CUDA(cudaEventSynchronize(ring->slot_done[slot]));
    st->copy(dst + size_t(d) * chunk, ring->slot(slot), chunk_size(d));
  }
  return HPCS_OK;
}

}  // namespace hpcs
