// Register transforms of csrc/pencil_core.cuh with 32 host threads as the lanes of
// a warp, against the defining sums.  Prints the worst error of the four kinds over
// the largest output, one line per plan: <type> <n> <wide> <error>.
#include <barrier>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <thread>
#include <vector>

#include "../../smaiso_quasi_b200/csrc/pencil_core.cuh"
using namespace quasi;

struct Shared {
  std::barrier<> bar{32};
  double x[32], y[32];
};
template <class F>
struct HostWarp {
  template <class> static constexpr bool split() { return F::kSplit; }
  Shared* s;
  int lane;
  int l() const { return lane % F::L; }
  int pencil() const { return lane / F::L; }
  int partner() const { return lane - l() + ((F::L - l()) & (F::L - 1)); }
  int mirror() const { return lane + F::L - 1 - 2 * l(); }
  int at(int place) const {
    if (place < 0 || place >= F::kPadded) std::exit(1);
    return pencil() * F::XS + place;
  }
  void sync() const { s->bar.arrive_and_wait(); }
  template <typename T>
  Cx<T> shfl(Cx<T> v, int src) const {
    if (src < 0 || src > 31) std::exit(1);
    s->x[lane] = v.x, s->y[lane] = v.y;
    sync();
    const Cx<T> r{T(s->x[src]), T(s->y[src])};
    sync();
    return r;
  }
};

template <class T, int N, bool W>
double worst_error(int kind) {
  using F = RowFFT<T, N, W>;
  const double pi = std::acos(-1.0);
  std::vector<Cx<T>> root(N), quarter(N), tables(F::kTables), xch(F::xch_bytes() / sizeof(Cx<T>) + 1);
  for (int t = 0; t < N; ++t) {
    root[t] = {T(std::cos(-2 * pi * t / N)), T(std::sin(-2 * pi * t / N))};
    quarter[t] = {T(std::cos(-pi * t / 2 / N)), T(std::sin(-pi * t / 2 / N))};
  }
  const auto tb = F::fill_tables(tables.data(), Tables<T>{root.data(), quarter.data()}, 0, 1);
  std::mt19937_64 gen(N * 7 + kind);
  std::uniform_real_distribution<double> uni(-1, 1);
  std::vector<T> x(F::ROWS * N), y(F::ROWS * N);
  for (auto& v : x) v = T(uni(gen));
  Shared sh;
  const bool fwd = is_forward(kind), sine = is_sine(kind);
  std::vector<std::thread> lanes;
  for (int lane = 0; lane < 32; ++lane)
    lanes.emplace_back([&, lane] {
      const HostWarp<F> w{&sh, lane};
      Cx<T> v[F::E];
      const int l = w.l();
      const T* in = &x[2 * w.pencil() * N];
      T* out = &y[2 * w.pencil() * N];
      if (fwd) {
        for (int t = 0; t < F::H; ++t) {
          const int n = 2 * l + 2 * F::L * t;
          v[t] = {in[n], in[n + 1]};
          v[F::E - 1 - t] = {in[N + n], in[N + n + 1]};
        }
        F::from_pairs(w, v, sine);
        F::forward(w, v, xch.data(), tb);
        for (int t = 0; t < F::E; ++t) {
          const int k = F::spec(l + F::L * t, sine);
          out[k] = v[t].x, out[N + k] = v[t].y;
        }
      } else {
        for (int t = 0; t < F::E; ++t) {
          const int k = F::spec(l + F::L * t, sine);
          v[t] = {in[k], in[N + k]};
        }
        F::inverse(w, v, xch.data(), tb);
        F::to_pairs(w, v, sine);
        for (int t = 0; t < F::H; ++t) {
          const int n = 2 * l + 2 * F::L * t;
          out[n] = v[t].x, out[n + 1] = v[t].y;
          out[N + n] = v[F::E - 1 - t].x, out[N + n + 1] = v[F::E - 1 - t].y;
        }
      }
    });
  for (auto& t : lanes) t.join();
  // the sums in long double: the angles reach N pi, whose rounding in double is above the transform's own
  const long double pl = std::acos(-1.0L);
  double err = 0, top = 0;
  for (int r = 0; r < F::ROWS; ++r)
    for (int k = 0; k < N; ++k) {
      long double s = 0;
      for (int n = 0; n < N; ++n) {
        long double c;
        if (fwd) c = 2 * (sine ? std::sin(pl * (k + 1) * (2 * n + 1) / (2 * N)) : std::cos(pl * k * (2 * n + 1) / (2 * N)));
        else if (!sine) c = n ? 2 * std::cos(pl * n * (2 * k + 1) / (2 * N)) : 1;
        else c = n == N - 1 ? (k % 2 ? -1 : 1) : 2 * std::sin(pl * (n + 1) * (2 * k + 1) / (2 * N));
        s += c * x[r * N + n];
      }
      err = std::max(err, double(std::fabs(s - y[r * N + k])));
      top = std::max(top, double(std::fabs(s)));
    }
  return err / top;
}

template <class T, int N, bool W = false>
void all() {
  double e = 0;
  for (int kind = 0; kind < 4; ++kind) e = std::max(e, worst_error<T, N, W>(kind));
  std::printf("%s %d %d %.3g\n", sizeof(T) == 8 ? "fp64" : "fp32", N, int(W), e);
}
template <class T>
void lengths() {
  all<T, 16>(), all<T, 32>(), all<T, 64>(), all<T, 96>(), all<T, 128>(), all<T, 192>(), all<T, 256>(), all<T, 512>();
  all<T, 128, true>(), all<T, 256, true>();
}
int main() {
  lengths<double>();
  lengths<float>();
}
