// Pageable host memory to and from pinned staging slots with several threads.
//
// cudaMemcpy of pageable memory goes through one driver thread (7-10 GB/s, less
// where the destination's pages are touched for the first time); the seam
// calls on ordinary arrays spent most of their time there.  Here the calling
// thread and a few workers copy a chunk between the caller's array and a
// pinned slot while the previous chunk is on the bus.
//
// One set of slots and workers serves the process, leased to one call at a time (a
// call that finds it taken uses plain copies) and given back when the last
// context is destroyed.  Making it takes 4 to 13 ms (pinning the slots), which it
// earns back at about 0.13 ms per MB moved: it is made once kStagingPays bytes have
// gone by plain copies since the first context, so a program that moves less never
// pays for it.
// Workers only copy host memory; every CUDA call is the calling thread's.
#pragma once

#include <cstddef>
#include <functional>

namespace ofb {

constexpr int kStagingSlots = 4;
constexpr size_t kStagingBytes = size_t(2) << 20;  // per slot
constexpr size_t kStagingPays = size_t(64) << 20;

// Maps the pages of [p, p + bytes) for writing without changing them (what the
// first write to fresh memory would do one page at a time); best effort.
void populate(void* p, size_t bytes);

// A context exists / is gone.
void staging_retain();
void staging_release();

class StagingLease {
 public:
  // For a transfer of `bytes`.
  explicit StagingLease(size_t bytes);
  ~StagingLease();
  StagingLease(const StagingLease&) = delete;
  StagingLease& operator=(const StagingLease&) = delete;
  explicit operator bool() const { return held_; }
  char* slot(int i) const;
  // Runs fn(0) .. fn(parts - 1), on the workers and the calling thread.
  void parallel(int parts, const std::function<void(int)>& fn) const;

 private:
  bool held_ = false;
};

}  // namespace ofb
