// Host loops on up to 16 threads: the field conversions between the caller's
// doubles and the staging buffer.  Host code only.
#pragma once
#include <algorithm>
#include <array>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstddef>
#include <mutex>
#include <thread>
#include <vector>

namespace quasi {

constexpr int kHostThreads = 16;
constexpr std::chrono::microseconds kHostSpin{100};
inline int host_threads(size_t most) {
  const unsigned hw = std::thread::hardware_concurrency();
  return int(std::min<size_t>({size_t(hw ? hw : 1), size_t(kHostThreads), most}));
}

// f(lo, hi) over [0, n) split into contiguous chunks.
template <class F>
inline void host_parallel(size_t n, F&& f) {
  const int nt = host_threads(kHostThreads);
  if (nt <= 1 || n < (size_t(1) << 20)) {
    f(size_t(0), n);
    return;
  }
  std::vector<std::thread> pool;
  const size_t chunk = (n + nt - 1) / nt;
  for (int t = 1; t < nt; ++t) {
    const size_t lo = std::min(n, t * chunk), hi = std::min(n, lo + chunk);
    pool.emplace_back([&f, lo, hi] { f(lo, hi); });
  }
  f(size_t(0), std::min(n, chunk));
  for (auto& th : pool) th.join();
}

// work(c) for every chunk on several threads, this one among them, each chunk
// after arrived(c) has returned true on this thread (called in order).  A chunk
// that does not arrive ends the loop and those after it are not worked on.  The
// others sleep until a chunk arrives, however long that takes (threads that looked
// out for it took 22 s of CPU time while 400 steps at 256^3 ran before the copy).  A
// thread that has worked looks out for the next chunk for kHostSpin before it sleeps
// again: chunks of a running copy follow each other in 10 to 80 us (a field of
// 96x96x192 doubles: 1.07 ms, 1.2 without, 0.78 with 15 threads that never sleep).
template <class A, class W>
inline void host_chunks(int chunks, A&& arrived, W&& work) {
  const int nt = host_threads(size_t(std::max(chunks, 1)));
  std::mutex mu;
  std::condition_variable more;
  std::atomic<int> ready{0}, next{0};   // written under the mutex
  std::atomic<bool> end{false};         // no further chunk will arrive
  auto drain = [&](bool wait) {
    auto any = [&] { return next < ready || end; };
    std::unique_lock<std::mutex> lk(mu);
    for (;;) {
      if (wait) more.wait(lk, any);
      if (next >= ready) return;
      const int c = next++;
      lk.unlock();
      work(c);
      if (wait)
        for (const auto until = std::chrono::steady_clock::now() + kHostSpin;
             !any() && std::chrono::steady_clock::now() < until;)
          std::this_thread::yield();
      lk.lock();
    }
  };
  std::array<std::thread, kHostThreads> pool;
  int started = 0;
  for (; started < nt - 1; ++started) {
    try {
      pool[started] = std::thread(drain, true);
    } catch (...) {   // no more threads: the others do the work
      break;
    }
  }
  bool all = true;
  for (int c = 0; c < chunks && all; ++c) {
    all = arrived(c);
    std::lock_guard<std::mutex> lk(mu);
    if (all) ++ready;
    if (!all || c + 1 == chunks) end = true;
    if (end) more.notify_all();
    else more.notify_one();
  }
  drain(false);
  for (int t = 0; t < started; ++t) pool[t].join();
}

}  // namespace quasi
