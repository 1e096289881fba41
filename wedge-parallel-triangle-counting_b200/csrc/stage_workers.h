// stage_workers.h -- host threads that copy staged pieces of pageable columns.
#pragma once
#include <stddef.h>
#include <string.h>

#include <atomic>
#include <chrono>
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

namespace wetric {

// Threads that share the copying of staged pieces for the length of one
// call, in place of OpenMP: its teams spin on after their work, and the two
// that the driver's callback threads made could spin against each other's
// copies (R-MAT scale 20 from pageable arrays on 16 cores: 50 ms a call, 45 of
// them the device waiting for 64 MB of copies). These look for the next piece
// for kLook, longer than a piece's DMA takes, and then sleep: threads that
// slept at once were woken too late for much of a piece. tc_GPU on 16 cores,
// columns: OpenMP undisturbed / sleeping at once / this, ms: 8M 3.4 / 5.0 /
// 2.8, 16M 6.0 / 5.8 / 4.1, 64M 19 / 17 / 14.5 (3, 5 and 11 threads: 16M 4.5,
// 5.4, 6.9).
class StageWorkers {
 public:
  static constexpr size_t kBlock = 1ull << 20;
  static constexpr std::chrono::milliseconds kLook{4};
  ~StageWorkers() {
    {
      std::lock_guard<std::mutex> lk(mu_);
      stop_ = true;
      posted_.fetch_add(1, std::memory_order_relaxed);
    }
    work_.notify_all();
    for (std::thread &t : threads_) t.join();
  }
  void start() {
    const unsigned cores = std::thread::hardware_concurrency();
    const unsigned want = cores > 15 ? 7 : cores / 2;
    try {
      for (unsigned i = 0; i < want; ++i) threads_.emplace_back([this] { loop(); });
    } catch (...) {  // fewer threads: the caller of copy() copies too
    }
  }
  // Copies a piece; returns when it is done.
  void copy(const void *src, void *dst, size_t bytes) {
    Job job;
    job.src = static_cast<const char *>(src);
    job.dst = static_cast<char *>(dst);
    job.bytes = bytes;
    job.blocks = (bytes + kBlock - 1) / kBlock;
    Job **slot = nullptr;
    {
      std::lock_guard<std::mutex> lk(mu_);
      for (Job *&j : jobs_)
        if (!j) slot = &j;
      if (slot) {  // else both slots are taken: copied here alone
        *slot = &job;
        posted_.fetch_add(1, std::memory_order_relaxed);
      }
    }
    if (slot) work_.notify_all();
    run(&job);
    if (!slot) return;
    std::unique_lock<std::mutex> lk(mu_);
    *slot = nullptr;  // no thread joins it any more; those in it are waited for
    lk.unlock();
    const auto left = [&] { return job.users.load(std::memory_order_acquire) == 0; };
    if (look(left)) return;
    lk.lock();
    left_.wait(lk, left);
  }

 private:
  struct Job {
    const char *src = nullptr;
    char *dst = nullptr;
    size_t bytes = 0, blocks = 0;
    std::atomic<size_t> next{0};
    std::atomic<unsigned> users{0};  // threads in run(); changed under mu_
  };
  // Whether `there` comes true within kLook.
  template <class There>
  static bool look(const There &there) {
    const auto end = std::chrono::steady_clock::now() + kLook;
    do {
      for (int i = 0; i < 64; ++i) {
        if (there()) return true;
        __builtin_ia32_pause();
      }
    } while (std::chrono::steady_clock::now() < end);
    return false;
  }
  static void run(Job *job) {
    for (size_t b; (b = job->next.fetch_add(1, std::memory_order_relaxed)) < job->blocks;) {
      const size_t o = b * kBlock;
      memcpy(job->dst + o, job->src + o, o + kBlock <= job->bytes ? kBlock : job->bytes - o);
    }
  }
  void loop() {
    std::unique_lock<std::mutex> lk(mu_);
    for (;;) {
      Job *job = nullptr;
      for (Job *j : jobs_)
        if (j && j->next.load(std::memory_order_relaxed) < j->blocks) job = j;
      if (job) {
        job->users.fetch_add(1, std::memory_order_relaxed);
        lk.unlock();
        run(job);
        lk.lock();
        if (job->users.fetch_sub(1, std::memory_order_release) == 1) left_.notify_all();
      } else if (stop_) {
        return;
      } else {
        const unsigned seen = posted_.load(std::memory_order_relaxed);
        const auto more = [&] { return posted_.load(std::memory_order_relaxed) != seen; };
        lk.unlock();
        const bool found = look(more);
        lk.lock();
        if (!found) work_.wait(lk, more);
      }
    }
  }
  std::mutex mu_;
  std::condition_variable work_, left_;
  Job *jobs_[2] = {};
  std::atomic<unsigned> posted_{0};  // jobs so far; changed under mu_
  bool stop_ = false;
  std::vector<std::thread> threads_;
};

}  // namespace wetric
