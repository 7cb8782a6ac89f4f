// Host-to-device copies of pageable memory by way of pinned slots.
//
// A cudaMemcpyAsync from pageable memory is staged by the driver in the calling
// thread: one core's copy rate (14 GB/s), and no launch is issued meanwhile. Here a
// team of threads, started for the call and joined before it returns, copies
// chunks of the input into a ring of pinned slots and the calling thread sends each
// slot on as its turn comes. The order of the chunks is fixed, so the calling
// thread can issue a slab's kernels between them.
//
// numpy volume in, host volume out, 96x96x48x48 / 11^3 / stride 3 (85 MB each way),
// B200 and 16 host cores: 9.4 -> 4.5 ms; 128x128x64x48 (201 MB) 20.4 -> 8.8. 8 threads and
// half the chunk 5.8 and 11.6.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstring>
#include <memory>
#include <thread>
#include <utility>
#include <vector>

namespace lrd {

constexpr size_t kStageChunk = size_t(1) << 20;
constexpr int kStageSlots = 16;    // 16 MiB pinned per plan that has staged
constexpr int kStageThreads = 6;   // at most; and at most half of the host's cores
// Smaller volumes are left to the driver (ms, driver / team: 10.6 MB 1.3 / 1.8, 18.9 MB
// 1.7 / 2.0, 37.7 MB 3.5 / 2.7): starting and joining the team costs some 0.3 ms.
constexpr long long kStageMinBytes = 32ll << 20;

// The pinned slots; a plan's, made at its first staged call and freed with it.
struct StageRing {
  char* slots = nullptr;
  cudaEvent_t sent[kStageSlots] = {};  // a slot's last copy
  bool make() {
    if (slots) return true;
    for (auto& e : sent)
      if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
        e = nullptr;
        cudaGetLastError();
        return false;
      }
    if (cudaHostAlloc(reinterpret_cast<void**>(&slots), kStageChunk * kStageSlots, cudaHostAllocDefault) != cudaSuccess) {
      slots = nullptr;
      cudaGetLastError();
      return false;
    }
    return true;
  }
  ~StageRing() {
    for (auto& e : sent)
      if (e) cudaEventDestroy(e);
    if (slots) cudaFreeHost(slots);
  }
};

// One call's copy. The caller holds the ring for as long as this lives.
class StagedCopy {
 public:
  // [ends[i - 1], ends[i]) bytes of ``src`` are sent by the i-th send(). Throws what
  // the allocations and the first thread's start throw.
  StagedCopy(StageRing& ring, const void* src, const std::vector<size_t>& ends, int device)
      : ring_(ring), src_(static_cast<const char*>(src)), device_(device) {
    size_t at = 0;
    for (const size_t end : ends)
      for (; at < end; at = chunks_.back().second) chunks_.emplace_back(at, at + kStageChunk < end ? at + kStageChunk : end);
    staged_ = std::make_unique<std::atomic<bool>[]>(chunks_.size());
    for (size_t i = 0; i < chunks_.size(); ++i) staged_[i].store(false, std::memory_order_relaxed);
    const unsigned half = std::thread::hardware_concurrency() / 2;
    const int want = half < 1 ? 1 : (half < (unsigned)kStageThreads ? (int)half : kStageThreads);
    team_.reserve(want);
    for (int i = 0; i < want; ++i) {
      try {
        team_.emplace_back([this] { work(); });
      } catch (...) {
        if (team_.empty()) throw;
        break;
      }
    }
  }
  StagedCopy(const StagedCopy&) = delete;
  StagedCopy& operator=(const StagedCopy&) = delete;
  ~StagedCopy() {
    stop_.store(true);
    for (auto& t : team_) t.join();
  }

  // Enqueues the copies of the bytes up to ``end`` on ``st``.
  cudaError_t send(void* dst, size_t end, cudaStream_t st) {
    for (; next_ < chunks_.size() && chunks_[next_].second <= end; ++next_) {
      while (!staged_[next_].load(std::memory_order_acquire)) {
        const int err = error_.load();
        if (err != cudaSuccess) return (cudaError_t)err;
        std::this_thread::yield();
      }
      const int slot = (int)(next_ % kStageSlots);
      const size_t at = chunks_[next_].first, n = chunks_[next_].second - at;
      cudaError_t e = cudaMemcpyAsync(static_cast<char*>(dst) + at, ring_.slots + slot * kStageChunk, n,
                                      cudaMemcpyHostToDevice, st);
      if (e == cudaSuccess) e = cudaEventRecord(ring_.sent[slot], st);
      if (e != cudaSuccess) return e;
      issued_.store(next_ + 1, std::memory_order_release);
    }
    return cudaSuccess;
  }

 private:
  // Chunks in order; a slot is written again once its previous chunk was sent and
  // that copy has ended (an earlier call's too: it may have returned on an error).
  void work() {
    cudaError_t e = cudaSetDevice(device_);
    for (;;) {
      const size_t i = taken_.fetch_add(1);
      if (i >= chunks_.size()) return;
      while (e == cudaSuccess && issued_.load(std::memory_order_acquire) + kStageSlots <= i) {
        if (stop_.load()) return;
        std::this_thread::yield();
      }
      const int slot = (int)(i % kStageSlots);
      if (e == cudaSuccess) e = cudaEventSynchronize(ring_.sent[slot]);
      if (e != cudaSuccess) {
        error_.store((int)e);
        return;
      }
      if (stop_.load()) return;
      memcpy(ring_.slots + slot * kStageChunk, src_ + chunks_[i].first, chunks_[i].second - chunks_[i].first);
      staged_[i].store(true, std::memory_order_release);
    }
  }

  StageRing& ring_;
  const char* src_;
  int device_;
  std::vector<std::pair<size_t, size_t>> chunks_;
  std::unique_ptr<std::atomic<bool>[]> staged_;
  std::atomic<size_t> taken_{0}, issued_{0};
  std::atomic<int> error_{(int)cudaSuccess};
  std::atomic<bool> stop_{false};
  size_t next_ = 0;
  std::vector<std::thread> team_;
};

}  // namespace lrd
