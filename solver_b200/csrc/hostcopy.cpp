#include "hostcopy.hpp"

#include <cuda_runtime.h>
#include <sched.h>
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <memory>
#include <mutex>
#include <thread>
#include <vector>

namespace ofb {

namespace {

// Workers wait for the next job actively for a short while (the chunks of one
// transfer follow each other within it), then asleep.
constexpr auto kSpin = std::chrono::microseconds(200);

class Workers {
 public:
  explicit Workers(int n) {
    for(int i = 0; i < n; ++i) {
      try {
        threads_.emplace_back([this] { loop(); });
      } catch(...) {
        break;  // the calling thread does the work alone
      }
    }
  }
  ~Workers() {
    {
      std::lock_guard<std::mutex> lock(mutex_);
      quit_ = true;
    }
    wake_.notify_all();
    for(std::thread& t : threads_) t.join();
  }

  // In a child of fork() the threads do not exist: it must neither join them nor
  // take a lock that one of them may have held.
  bool forked() const { return getpid() != pid_; }

  void run(int parts, const std::function<void(int)>& fn) {
    if(forked()) {
      for(int i = 0; i < parts; ++i) fn(i);
      return;
    }
    auto job = std::make_shared<Job>();
    job->fn = &fn;
    job->parts = parts;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      job_ = job;
      epoch_.fetch_add(1, std::memory_order_release);
    }
    if(asleep_.load(std::memory_order_acquire) > 0) wake_.notify_all();
    job->work();
    while(job->done.load(std::memory_order_acquire) < parts) std::this_thread::yield();
  }

 private:
  // Parts are taken from a counter, so a worker that comes late finds none and
  // never touches fn after run() has returned.
  struct Job {
    const std::function<void(int)>* fn;
    int parts;
    std::atomic<int> next{0}, done{0};
    void work() {
      for(int i; (i = next.fetch_add(1)) < parts;) {
        (*fn)(i);
        done.fetch_add(1, std::memory_order_release);
      }
    }
  };

  void loop() {
    unsigned seen = 0;
    for(;;) {
      const auto until = std::chrono::steady_clock::now() + kSpin;
      while(epoch_.load(std::memory_order_acquire) == seen && std::chrono::steady_clock::now() < until)
        std::this_thread::yield();
      std::shared_ptr<Job> job;
      {
        std::unique_lock<std::mutex> lock(mutex_);
        asleep_.fetch_add(1);
        wake_.wait(lock, [&] { return quit_ || epoch_.load() != seen; });
        asleep_.fetch_sub(1);
        if(quit_) return;
        seen = epoch_.load();
        job = job_;
      }
      job->work();
    }
  }

  const pid_t pid_ = getpid();
  std::vector<std::thread> threads_;
  std::mutex mutex_;
  std::condition_variable wake_;
  std::shared_ptr<Job> job_;
  std::atomic<unsigned> epoch_{0};
  std::atomic<int> asleep_{0};
  bool quit_ = false;
};

// CPUs that this process may use.
int usable_cpus() {
  cpu_set_t set;
  if(sched_getaffinity(0, sizeof(set), &set) == 0) return CPU_COUNT(&set);
  return static_cast<int>(std::thread::hardware_concurrency());
}

std::mutex g_mutex;  // guards the variables below
int g_contexts = 0;
size_t g_plain = 0;  // bytes moved without slots since the first context
bool g_leased = false;
char* g_slots = nullptr;
Workers* g_workers = nullptr;  // not destroyed at exit: the threads end with the process

}  // namespace

void populate(void* p, size_t bytes) {
#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23  // Linux 5.14; older kernels refuse it
#endif
  static const uintptr_t page = static_cast<uintptr_t>(sysconf(_SC_PAGESIZE));
  const uintptr_t lo = reinterpret_cast<uintptr_t>(p) / page * page;
  const uintptr_t hi = (reinterpret_cast<uintptr_t>(p) + bytes + page - 1) / page * page;
  madvise(reinterpret_cast<void*>(lo), hi - lo, MADV_POPULATE_WRITE);
}

void staging_retain() {
  std::lock_guard<std::mutex> lock(g_mutex);
  ++g_contexts;
}

void staging_release() {
  std::unique_ptr<Workers> workers;  // joined after the lock is gone
  std::lock_guard<std::mutex> lock(g_mutex);
  if(--g_contexts > 0 || g_leased) return;
  g_plain = 0;
  if(g_workers != nullptr && !g_workers->forked()) workers.reset(g_workers);
  g_workers = nullptr;
  if(g_slots != nullptr) cudaFreeHost(g_slots);
  g_slots = nullptr;
}

StagingLease::StagingLease(size_t bytes) {
  std::lock_guard<std::mutex> lock(g_mutex);
  if(g_leased) return;
  if(g_slots == nullptr) {
    if(g_plain < kStagingPays) {
      g_plain += bytes;
      return;
    }
    void* p = nullptr;
    if(cudaHostAlloc(&p, kStagingSlots * kStagingBytes, cudaHostAllocPortable) != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    g_slots = static_cast<char*>(p);
  }
  if(g_workers == nullptr) {
    g_workers = new Workers(std::min(7, std::max(0, usable_cpus() - 1)));
  }
  g_leased = held_ = true;
}

StagingLease::~StagingLease() {
  if(!held_) return;
  std::lock_guard<std::mutex> lock(g_mutex);
  g_leased = false;
}

char* StagingLease::slot(int i) const { return g_slots + i * kStagingBytes; }

void StagingLease::parallel(int parts, const std::function<void(int)>& fn) const { g_workers->run(parts, fn); }

}  // namespace ofb
