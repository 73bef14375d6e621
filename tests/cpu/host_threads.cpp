// csrc/host_threads.cuh: what a download's conversion threads do while nothing has
// arrived, and that every chunk that arrives is worked on once.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <ctime>

#include "../../smaiso_quasi_b200/csrc/host_threads.cuh"

static double cpu_seconds() { return double(std::clock()) / CLOCKS_PER_SEC; }

int main() {
  // CPU time of all threads over half a second in which the first chunk has not arrived
  std::atomic<int> seen[32] = {};
  const double t0 = cpu_seconds();
  quasi::host_chunks(
      32,
      [](int c) {
        if (c == 0) std::this_thread::sleep_for(std::chrono::milliseconds(500));
        return true;
      },
      [&](int c) { ++seen[c]; });
  std::printf("cpu %.3f\n", cpu_seconds() - t0);
  bool once = true;
  for (auto& s : seen) once = once && s == 1;
  // chunks of any number; from the one that does not arrive on, none is worked on
  for (int chunks : {0, 1, 2, 5, 32, 100})
    for (int stop : {-1, 0, 3, 99}) {
      std::atomic<int> done[100] = {};
      std::atomic<int> ready{0};
      std::atomic<bool> early{false};
      quasi::host_chunks(
          chunks,
          [&](int c) {
            if (c == stop) return false;
            ready = c + 1;
            return true;
          },
          [&](int c) {
            if (c >= ready) early = true;
            ++done[c];
          });
      for (int c = 0; c < 100; ++c) once = once && done[c] == (c < chunks && (stop < 0 || c < stop));
      once = once && !early;
    }
  std::printf("once %d\n", int(once));
}
