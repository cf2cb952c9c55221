// Copies between a caller's pageable host memory and the device, through a
// small ring of pinned slots that worker threads fill (or drain) while earlier
// slots cross the bus.
//
// A pageable cudaMemcpyAsync stages with one host thread (18 GB/s up; down
// into fresh pages 5 GB/s, most of it page faults) and costs 5 to 10 us
// however small it is.  Eight threads keep the bus busy (256 MB up in 6.0 ms
// against 24.6), and scattered pieces that lie back to back on the device (the
// graphs of a batch) cross as one copy per slot.  But a thread that was asleep
// copies its first megabytes at a fifth of the caller's rate, so small copies
// gain nothing from it, parts are small, and nobody waits for a thread that
// has not joined (upload, begin_call).
//
// The ring and the threads belong to one context, are made on the first use
// that is worth them, and go with it (or with stc_ctx_trim).  Where they cannot
// be had (no more pinned memory, a limit on threads) the copies go on without.
#pragma once
#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace stc {

void cuda_check(cudaError_t e, const char* what);

// True when p is plain host memory the driver would have to stage.
inline bool is_pageable(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

// malloc whose large blocks ask for huge pages (release with free): first
// touches then fault once per 2 MB.
inline void* host_alloc(size_t bytes) {
  constexpr size_t kHuge = 2u << 20;
  if (bytes < 2 * kHuge) return malloc(bytes ? bytes : 1);
  const size_t n = (bytes + kHuge - 1) / kHuge * kHuge;
  void* p = aligned_alloc(kHuge, n);
  if (p) (void)madvise(p, n, MADV_HUGEPAGE);
  return p;
}

class HostCopier {
 public:
  struct Piece {
    char* device;
    char* host;  // only read by upload
    size_t bytes;
  };

  HostCopier() = default;
  HostCopier(const HostCopier&) = delete;
  HostCopier& operator=(const HostCopier&) = delete;
  ~HostCopier() { release(); }

  // Host pieces to the device, in stream order; the host memory may be reused
  // on return.  Pieces that follow each other on the device share copies.
  void upload(const std::vector<Piece>& pieces, cudaStream_t st) {
    const size_t total = bytes_of(pieces);
    // On a host of 16 virtual CPUs, three pieces of 3 / 8 / 12 / 32 / 256 MB in
    // all took 189 / 420 / 646 / 1,750 / 24,600 us as plain copies, 228 / 561 /
    // 846 / 2,370 / 27,000 through the ring by the caller alone, 247 / 410 /
    // 512 / 1,070 / 9,220 with three helpers and 254 / 553 / 738 / 1,180 /
    // 6,010 with seven (64 MB: 2,140 with three, 1,850 with seven).  2 MB in
    // pieces of 8 / 16 / 32 / 64 / 128 KB took 540 / 320 / 207 / 185 / 147 as
    // plain copies and 215 / 184 / 175 / 170 / 170 through the ring.
    if (total < kUploadRing && total >= pieces.size() * kUploadPiece) plain(pieces, st, true);
    else run(pieces, st, true, total < kUploadRing ? 0u : total < kUploadAll ? 3u : kHelpers);
  }
  // Device to host pieces; done on return.  Page faults are most of the work,
  // so helpers pay from 2 MB on (with them 80 us, without 170, a plain copy
  // 130; at 1 MB all three within 15 us; 32 MB 2.3 / 4.6 / 6.8 ms): they are
  // awake by the time the kernels ahead of the copy are done.
  void download(const std::vector<Piece>& pieces, cudaStream_t st) {
    run(pieces, st, false, bytes_of(pieces) < kDownloadThreads ? 0u : kHelpers);
  }

  void release() {
    if (!threads_.empty()) {
      {
        std::lock_guard<std::mutex> l(mu_);
        quit_ = true;
      }
      cv_.notify_all();
      for (auto& t : threads_) t.join();
      threads_.clear();
      quit_ = false;
    }
    free_ring();
  }

 private:
  static constexpr int kSlots = 8;
  static constexpr size_t kSlotBytes = 2u << 20;
  // What a thread copies at a time; with 256 KB the call waited for the last
  // part of a slow helper (8 MB up with seven: 1,000 us, with 32 KB 553).
  static constexpr size_t kPart = 32u << 10;
  static constexpr unsigned kHelpers = 7;
  static constexpr size_t kUploadRing = 8u << 20;       // less goes up as plain copies,
  static constexpr size_t kUploadPiece = 64u << 10;     // unless in pieces smaller than this
  static constexpr size_t kUploadAll = 48u << 20;       // all helpers from here on
  static constexpr size_t kDownloadThreads = 2u << 20;
  // How long a helper waits for a part (a count may run before a download)
  // before it sleeps again.
  static constexpr std::chrono::milliseconds kIdle{2};
  // A part of one slot's contents, between `ring` and `host`.
  struct Part {
    char* ring;
    char* host;
    size_t bytes;
  };
  struct Chunk {  // one slot's contents: a run of device memory
    char* device;
    size_t bytes;
    uint32_t part0, part1;
    std::atomic<uint32_t> left{0};  // parts not copied yet
    Chunk(char* d, uint32_t p) : device(d), bytes(0), part0(p), part1(p) {}
    Chunk(const Chunk& o) : device(o.device), bytes(o.bytes), part0(o.part0), part1(o.part1) {}
  };

  static size_t bytes_of(const std::vector<Piece>& pieces) {
    size_t total = 0;
    for (const Piece& p : pieces) total += p.bytes;
    return total;
  }

  // The driver's own copies.
  static void plain(const std::vector<Piece>& pieces, cudaStream_t st, bool up) {
    for (const Piece& p : pieces)
      cuda_check(up ? cudaMemcpyAsync(p.device, p.host, p.bytes, cudaMemcpyHostToDevice, st)
                    : cudaMemcpyAsync(p.host, p.device, p.bytes, cudaMemcpyDeviceToHost, st),
                 "cudaMemcpyAsync(pageable)");
    if (!up) cuda_check(cudaStreamSynchronize(st), "cudaStreamSynchronize");
  }

  // The ring and its events, or neither.
  bool make_ring() {
    if (ring_) return true;
    bool ok = cudaMallocHost(reinterpret_cast<void**>(&ring_), kSlots * kSlotBytes) == cudaSuccess;
    if (!ok) ring_ = nullptr;
    for (auto& e : event_)
      if (ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        e = nullptr;
        ok = false;
      }
    if (!ok) {
      (void)cudaGetLastError();
      free_ring();
    }
    return ok;
  }
  void free_ring() {
    for (auto& e : event_) {
      if (!e) continue;
      (void)cudaEventSynchronize(e);
      (void)cudaEventDestroy(e);
      e = nullptr;
    }
    if (ring_) (void)cudaFreeHost(ring_);
    ring_ = nullptr;
  }

  void run(const std::vector<Piece>& pieces, cudaStream_t st, bool up, unsigned helpers) {
    if (bytes_of(pieces) == 0) return;
    if (!make_ring()) return plain(pieces, st, up);
    // Cut the pieces into slots and parts.
    std::vector<Chunk> chunks;
    parts_.clear();
    part_chunk_.clear();
    for (const Piece& p : pieces) {
      size_t at = 0;
      while (at < p.bytes) {
        if (chunks.empty() || chunks.back().device + chunks.back().bytes != p.device + at ||
            chunks.back().bytes == kSlotBytes)
          chunks.emplace_back(p.device + at, (uint32_t)parts_.size());
        Chunk& c = chunks.back();
        const size_t n = std::min({p.bytes - at, kSlotBytes - c.bytes, kPart});
        parts_.push_back(Part{ring_ + ((chunks.size() - 1) % kSlots) * kSlotBytes + c.bytes,
                              p.host + at, n});
        part_chunk_.push_back((uint32_t)chunks.size() - 1);
        c.part1 = (uint32_t)parts_.size();
        c.bytes += n;
        at += n;
      }
    }
    for (Chunk& c : chunks) c.left.store(c.part1 - c.part0, std::memory_order_relaxed);
    chunks_ = &chunks;
    up_ = up;
    next_.store(0);
    open_.store(0);  // parts below it may be copied
    cancel_.store(false);
    struct Guard {  // whatever happens, no thread touches this call's memory after it
      HostCopier* c;
      ~Guard() { c->end_call(); }
    } guard{this};
    if (helpers) begin_call(helpers);
    const uint32_t nc = (uint32_t)chunks.size();
    auto event_done = [&](uint32_t c) {  // the slot's last transfer
      cuda_check(cudaEventSynchronize(event_[c % kSlots]), "cudaEventSynchronize(staging)");
    };
    auto finish = [&](uint32_t c) {  // the chunk's parts are copied
      while (chunks[c].left.load(std::memory_order_acquire) != 0)
        if (!copy_part()) std::this_thread::yield();
    };
    if (up) {
      uint32_t opened = 0;
      for (uint32_t c = 0; c < nc; c++) {
        for (; opened < nc && opened < c + kSlots - 1; opened++) {
          event_done(opened);  // recorded by the chunk kSlots before, or an earlier call
          open_.store(chunks[opened].part1, std::memory_order_release);
        }
        finish(c);
        cuda_check(cudaMemcpyAsync(chunks[c].device, ring_ + (c % kSlots) * kSlotBytes,
                                   chunks[c].bytes, cudaMemcpyHostToDevice, st),
                   "cudaMemcpyAsync(staging)");
        cuda_check(cudaEventRecord(event_[c % kSlots], st), "cudaEventRecord(staging)");
      }
    } else {
      uint32_t issued = 0;
      for (uint32_t c = 0; c < nc; c++) {
        for (; issued < nc && issued < c + kSlots; issued++) {
          if (issued >= kSlots) finish(issued - kSlots);  // the slot is drained
          else event_done(issued);                        // an earlier call's transfer
          cuda_check(cudaMemcpyAsync(ring_ + (issued % kSlots) * kSlotBytes, chunks[issued].device,
                                     chunks[issued].bytes, cudaMemcpyDeviceToHost, st),
                     "cudaMemcpyAsync(staging)");
          cuda_check(cudaEventRecord(event_[issued % kSlots], st), "cudaEventRecord(staging)");
        }
        event_done(c);
        open_.store(chunks[c].part1, std::memory_order_release);
        if (helpers) wake_again();
      }
      for (uint32_t c = 0; c < nc; c++) finish(c);
    }
  }

  // Copies the next part if one is open.
  bool copy_part() {
    uint32_t i = next_.load(std::memory_order_relaxed);
    do {
      if (i >= open_.load(std::memory_order_acquire)) return false;
    } while (!next_.compare_exchange_weak(i, i + 1, std::memory_order_relaxed));
    const Part& p = parts_[i];
    if (up_) memcpy(p.ring, p.host, p.bytes);
    else memcpy(p.host, p.ring, p.bytes);
    (*chunks_)[part_chunk_[i]].left.fetch_sub(1, std::memory_order_release);
    return true;
  }

  // Lets up to `helpers` threads join the call and wakes the first; each wakes
  // the next while parts are left, so that the caller pays for one wake-up only.
  // They join under the mutex and end_call waits only for those that did: a
  // thread that wakes late finds the call over, and delays nobody.
  void begin_call(unsigned helpers) {
    if (threads_.empty()) {
      const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
      const unsigned n = std::min(kHelpers, hw > 2 ? hw / 2 : 1u);  // the caller is one more
      try {
        for (unsigned i = 0; i < n; i++) threads_.emplace_back([this] { work(); });
      } catch (const std::system_error&) {  // with those there are, if any
      }
    }
    {
      std::lock_guard<std::mutex> l(mu_);
      seats_ = (int)std::min<size_t>(helpers, threads_.size());
      wakes_ = 1;
    }
    cv_.notify_one();
  }
  // Wakes a helper if all have left (kIdle without a part).
  void wake_again() {
    {
      std::lock_guard<std::mutex> l(mu_);
      if (joined_ > 0 || wakes_ > 0) return;
      wakes_ = 1;
    }
    cv_.notify_one();
  }

  void end_call() {
    cancel_.store(true);
    std::unique_lock<std::mutex> l(mu_);
    seats_ = wakes_ = 0;
    idle_.wait(l, [this] { return joined_ == 0; });
  }

  void work() {
    std::unique_lock<std::mutex> l(mu_);
    while (true) {
      cv_.wait(l, [this] { return quit_ || (wakes_ > 0 && seats_ > 0); });
      if (quit_) return;
      wakes_--;
      seats_--;
      joined_++;
      const uint32_t n = (uint32_t)parts_.size();
      const bool more = seats_ > 0 && wakes_ == 0 && next_.load(std::memory_order_relaxed) < n;
      if (more) wakes_ = 1;
      l.unlock();
      if (more) cv_.notify_one();
      auto since = std::chrono::steady_clock::now();
      bool idle = false;  // since then
      while (!cancel_.load(std::memory_order_relaxed) && next_.load(std::memory_order_relaxed) < n) {
        if (copy_part()) {
          idle = false;
          continue;
        }
        const auto t = std::chrono::steady_clock::now();
        if (!idle) since = t;
        idle = true;
        if (t - since > kIdle) break;
        std::this_thread::yield();
      }
      l.lock();
      seats_ += cancel_.load(std::memory_order_relaxed) ? 0 : 1;
      if (--joined_ == 0) idle_.notify_one();
    }
  }

  char* ring_ = nullptr;
  cudaEvent_t event_[kSlots] = {};
  std::vector<Part> parts_;
  std::vector<uint32_t> part_chunk_;
  std::vector<Chunk>* chunks_ = nullptr;
  bool up_ = true;
  std::atomic<uint32_t> next_{0}, open_{0};
  std::atomic<bool> cancel_{false};
  std::vector<std::thread> threads_;
  std::mutex mu_;
  std::condition_variable cv_, idle_;
  int seats_ = 0;   // threads that may still join the call
  int wakes_ = 0;   // wake-ups on their way to one
  int joined_ = 0;  // threads that touch the call's memory
  bool quit_ = false;
};

}  // namespace stc
