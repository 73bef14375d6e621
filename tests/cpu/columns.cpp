// The lane map of the x and y passes (ColTile) with host threads as the threads of
// a tile, against the defining sums.  Prints the worst error of the four kinds over
// the largest output, one line per tile: <type> <n> <pencils> <split> <error>.
#include <barrier>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <memory>
#include <random>
#include <thread>
#include <vector>

#include "../../smaiso_quasi_b200/csrc/pencil_core.cuh"
using namespace quasi;

struct Warp {
  std::barrier<> bar{32};
  double x[32], y[32];
};
template <class C>
struct HostCol {
  template <class T> static constexpr bool split() { return C::template split<T>(); }
  C c;
  Warp* wp;
  std::barrier<>* tile;
  int lane;
  int l() const { return c.l(); }
  int partner() const { return c.partner(); }
  int at(int place) const {
    const int e = c.at(place);
    if (place < 0 || e < 0 || e >= C::XCH) std::exit(1);
    return e;
  }
  void sync() const { tile->arrive_and_wait(); }
  template <typename T>
  Cx<T> shfl(Cx<T> v, int src) const {
    if (src < 0 || src > 31) std::exit(1);
    wp->x[lane] = v.x, wp->y[lane] = v.y;
    wp->bar.arrive_and_wait();
    const Cx<T> r{T(wp->x[src]), T(wp->y[src])};
    wp->bar.arrive_and_wait();
    return r;
  }
};

template <class T, int N, int G, bool SPLIT>
double worst_error(int kind) {
  using C = ColTile<N, G, false, SPLIT>;
  using F = PencilFFT<T, N>;
  constexpr int P = 2 * G;
  const long double pi = std::acos(-1.0L);
  std::vector<Cx<T>> root(N), quarter(N), tables(F::kTables), xch(C::XCH);
  for (int t = 0; t < N; ++t) {
    root[t] = {T(std::cos(-2 * pi * t / N)), T(std::sin(-2 * pi * t / N))};
    quarter[t] = {T(std::cos(-pi * t / 2 / N)), T(std::sin(-pi * t / 2 / N))};
  }
  const auto tb = F::fill_tables(tables.data(), Tables<T>{root.data(), quarter.data()}, 0, 1);
  std::mt19937_64 gen(N * 7 + kind);
  std::uniform_real_distribution<double> uni(-1, 1);
  std::vector<T> x(N * P), y(N * P);   // [n][2 G]
  for (auto& v : x) v = T(uni(gen));
  const bool fwd = is_forward(kind), sine = is_sine(kind);
  std::barrier<> tile(C::THREADS);
  std::vector<std::unique_ptr<Warp>> warps;
  for (int w = 0; w < C::THREADS / 32; ++w) warps.push_back(std::make_unique<Warp>());
  std::vector<std::thread> threads;
  for (int r = 0; r < C::THREADS; ++r)
    threads.emplace_back([&, r] {
      const HostCol<C> w{C(r, 1), warps[r / 32].get(), &tile, r % 32};
      Cx<T> v[F::E];
      const int l = w.l(), g = 2 * w.c.g;
      const T s = sine ? T(-1) : T(1);
      for (int t = 0; t < F::E; ++t) {
        const int k = l + F::L * t, n = fwd ? F::pos(k) : F::spec(k, sine);
        const T f = fwd && t >= F::H ? s : T(1);
        v[t] = {f * x[n * P + g], f * x[n * P + g + 1]};
      }
      if (fwd) F::forward(w, v, xch.data(), tb);
      else F::inverse(w, v, xch.data(), tb);
      for (int t = 0; t < F::E; ++t) {
        const int k = l + F::L * t, n = fwd ? F::spec(k, sine) : F::pos(k);
        const T f = !fwd && t >= F::H ? s : T(1);
        y[n * P + g] = f * (fwd ? v[t].x : v[t].y);
        y[n * P + g + 1] = f * (fwd ? v[t].y : v[t].x);
      }
    });
  for (auto& t : threads) t.join();
  std::vector<long double> cs(4 * N), sn(4 * N);   // angles are multiples of pi / 2N
  for (int u = 0; u < 4 * N; ++u) cs[u] = std::cos(pi * u / (2 * N)), sn[u] = std::sin(pi * u / (2 * N));
  double err = 0, top = 0;
  for (int p = 0; p < P; ++p)
    for (int k = 0; k < N; ++k) {
      long double sum = 0;
      for (int n = 0; n < N; ++n) {
        long double c;
        if (fwd) c = 2 * (sine ? sn[(k + 1) * (2 * n + 1) % (4 * N)] : cs[k * (2 * n + 1) % (4 * N)]);
        else if (!sine) c = n ? 2 * cs[n * (2 * k + 1) % (4 * N)] : 1;
        else c = n == N - 1 ? (k % 2 ? -1 : 1) : 2 * sn[(n + 1) * (2 * k + 1) % (4 * N)];
        sum += c * x[n * P + p];
      }
      err = std::max(err, double(std::fabs(sum - y[k * P + p])));
      top = std::max(top, double(std::fabs(sum)));
    }
  return err / top;
}

template <class T, int N, int G, bool SPLIT>
void tile() {
  if constexpr (G * row_plan(N).lanes % 32 == 0) {
    double e = 0;
    for (int kind = 0; kind < 4; ++kind) e = std::max(e, worst_error<T, N, G, SPLIT>(kind));
    std::printf("%s %d %d %d %.3g\n", sizeof(T) == 8 ? "fp64" : "fp32", N, G, int(SPLIT), e);
  }
}
template <int N>
void all() {
  tile<double, N, 8, false>(), tile<double, N, 8, true>(), tile<float, N, 8, false>();
  tile<double, N, 4, false>(), tile<double, N, 4, true>(), tile<float, N, 4, false>();
}
int main() { all<8>(), all<16>(), all<32>(), all<64>(), all<96>(), all<128>(), all<192>(), all<256>(), all<512>(); }
