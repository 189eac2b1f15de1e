// Threads that add the forces of a host-pointer evaluation into the caller's array, or copy the state
// of an MD run into it, while the device->host copies land piece by piece: worker k (the calling
// thread is worker 0) waits for each piece and adds or copies its share of it.  Between calls the
// workers sleep on a condition variable (spinning would take cores from the caller's own threads).
// Host code only: what a piece is waited for with is the caller's (CUDA events, in the library).
#pragma once
#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace pmb {

struct AddPool {
  typedef int (*Wait)(const void *events, int c);  // waits until piece c has landed; 0 or an error
  typedef void (*Init)(int device);                // run once by each worker

  // threads in all; fewer where the system gives no more
  void start(int threads, Init init, int device) {
    try {
      for (int k = 1; k < threads; k++) {
        th.emplace_back([this, k, init, device] {
          init(device);
          worker(k);
        });
        nthreads = k + 1;
      }
    } catch (const std::system_error &) {
    }
  }

  // dst[0..n) += src[0..n) (or =), piece c of `chunk` elements once wait(events, c) has returned 0.
  // Returns 0, or the error of a wait: its piece and those after it are left as they were.
  int run(double *d, const double *s, long long n_, long long chunk_, int nchunks_, Wait wait_, const void *events_,
          bool copy_ = false) {
    copy = copy_;
    dst = d;
    src = s;
    n = n_;
    chunk = chunk_;
    nchunks = nchunks_;
    wait = wait_;
    events = events_;
    error.store(0, std::memory_order_relaxed);
    pending.store(nthreads - 1, std::memory_order_release);
    {
      std::lock_guard<std::mutex> lk(mu);
      gen.fetch_add(1, std::memory_order_acq_rel);
    }
    cv.notify_all();
    part(0);
    while (pending.load(std::memory_order_acquire) > 0) std::this_thread::yield();
    return error.load(std::memory_order_relaxed);
  }

  ~AddPool() {
    {
      std::lock_guard<std::mutex> lk(mu);
      stop = true;
    }
    cv.notify_all();
    for (std::thread &t : th) t.join();
  }

 private:
  int nthreads = 1;
  std::vector<std::thread> th;
  std::mutex mu;
  std::condition_variable cv;
  std::atomic<long long> gen{0};
  std::atomic<int> pending{0}, error{0};
  std::atomic<bool> stop{false};
  // the job
  double *dst = nullptr;
  const double *src = nullptr;
  long long n = 0, chunk = 0;
  int nchunks = 0;
  Wait wait = nullptr;
  const void *events = nullptr;
  bool copy = false;  // dst = src instead of dst += src

  void part(int k) {
    for (int c = 0; c < nchunks; c++) {
      if (const int e = wait(events, c)) {
        error.store(e, std::memory_order_relaxed);
        return;
      }
      const long long b0 = c * chunk, b1 = std::min(n, b0 + chunk), len = b1 - b0;
      const long long q0 = b0 + len * k / nthreads, q1 = b0 + len * (k + 1) / nthreads;
      double *__restrict__ d = dst;
      const double *__restrict__ s = src;
      if (copy) std::memcpy(d + q0, s + q0, sizeof(double) * (size_t)(q1 - q0));
      else
        for (long long i = q0; i < q1; i++) d[i] += s[i];
    }
  }
  void worker(int k) {
    long long seen = 0;
    for (;;) {
      {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return stop.load() || gen.load(std::memory_order_acquire) != seen; });
        if (stop) return;
        seen = gen.load(std::memory_order_acquire);
      }
      part(k);
      pending.fetch_sub(1, std::memory_order_acq_rel);
    }
  }
};

}  // namespace pmb
