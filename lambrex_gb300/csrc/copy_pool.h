// copy_pool.h -- the process's copy threads (plain C++, so that the tests run
// it without the library).
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>
#include <vector>

namespace lbx {

// Persistent copy threads: copy() splits one memcpy over all of them (the
// caller takes part 0) and returns when every part is done.  The threads
// sleep on a condition variable between copies.  There is one job at a time:
// a second caller waits for the first one's (copy) or is told so (try_copy).
class CopyPool {
 public:
  // with as many of the threads as the system gives: at worst the caller's alone
  explicit CopyPool(unsigned threads) {
    try {
      ts_.reserve(threads);
      for (unsigned i = 1; i < threads; ++i) {
        ts_.emplace_back([this, i] { worker(i); });
        T_ = i + 1;  // no worker reads it before the first job
      }
    } catch (const std::exception&) {
    }
  }
  ~CopyPool() {
    {
      std::lock_guard<std::mutex> l(mu_);
      stop_ = true;
    }
    cv_.notify_all();
    for (auto& t : ts_) t.join();
  }
  void copy(char* dst, const char* src, size_t len) {
    std::lock_guard<std::mutex> job(job_);
    run(dst, src, len);
  }
  // false, nothing copied, while another caller's copy runs
  bool try_copy(char* dst, const char* src, size_t len) {
    std::unique_lock<std::mutex> job(job_, std::try_to_lock);
    if (!job) return false;
    run(dst, src, len);
    return true;
  }

 private:
  void run(char* dst, const char* src, size_t len) {
    {
      std::lock_guard<std::mutex> l(mu_);
      dst_ = dst;
      src_ = src;
      len_ = len;
      left_.store(T_ - 1);
      ++gen_;
    }
    cv_.notify_all();
    part(0);
    while (left_.load() > 0) std::this_thread::yield();
  }
  void part(unsigned i) {
    const size_t p = (len_ + T_ - 1) / T_, o = (size_t)i * p;
    if (o < len_) std::memcpy(dst_ + o, src_ + o, std::min(p, len_ - o));
  }
  void worker(unsigned i) {
    long seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> l(mu_);
        cv_.wait(l, [&] { return stop_ || gen_ != seen; });
        if (stop_) return;
        seen = gen_;
      }
      part(i);
      left_.fetch_sub(1);
    }
  }
  unsigned T_ = 1;  // the caller and the threads
  std::vector<std::thread> ts_;
  std::mutex job_;  // held for the whole of a copy
  std::mutex mu_;
  std::condition_variable cv_;
  long gen_ = 0;
  bool stop_ = false;
  char* dst_ = nullptr;
  const char* src_ = nullptr;
  size_t len_ = 0;
  std::atomic<unsigned> left_{0};
};

}  // namespace lbx
