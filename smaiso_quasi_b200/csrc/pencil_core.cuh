// Transforms of pencils held in registers: the building block of the z passes
// (rows, row_pass.cuh), the x / y passes (columns, col_pass.cuh) and of the
// stages fused between them.
//
// L lanes share one complex pencil (two adjacent real pencils of the field, the
// real and the imaginary part).  Lane l holds the elements k = l + L t,
// t < E = N / L, before and after every radix stage: a Stockham stage of radix R
// reads e = b + t N/R with b = l + L c, which is that set, and the last stage
// writes it.  Only the writes in between are scattered; they go through an
// exchange buffer in shared memory and are read back in order, so a transform
// costs (stages - 1) shared-memory round trips and nothing else (the tile
// transforms of r2r_core.cuh stage their input and output as well and read the
// input twice).
//
// The pairing (k, N - k) of the inverse pre-twiddle and of the forward unpack is
// lane l against lane (L - l) mod L: shuffles.  Kinds and Makhoul's permutation
// are those of r2r_core.cuh.
//
// `W` places a pencil's lanes: l(), partner() (the lane of the warp that holds
// l' = (L - l) mod L of the same pencil), at(place) (a padded place of this pencil
// in the exchange buffer), shfl(value, lane) and sync() (all lanes of the exchange
// buffer).  A test runs the same code with host threads as lanes.
#pragma once
#include "r2r_core.cuh"

namespace quasi {

// 12 = 3 x 4 without twiddles (Good's prime factor mapping): with n = 4 n1 + 3 n2 and
// k = 4 k1 + 9 k2 (mod 12), W_12^{n k} = W_3^{n1 k1} W_4^{n2 k2}.
template <typename T> struct Dft<T, 12> {
  QHD static void run(Cx<T>* a) {
    Cx<T> t[3][4];
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) {
#pragma unroll
      for (int n2 = 0; n2 < 4; ++n2) t[n1][n2] = a[(4 * n1 + 3 * n2) % 12];
      Dft<T, 4>::run(t[n1]);
    }
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
      Cx<T> u[3] = {t[0][k2], t[1][k2], t[2][k2]};
      Dft<T, 3>::run(u);
#pragma unroll
      for (int k1 = 0; k1 < 3; ++k1) a[(4 * k1 + 9 * k2) % 12] = u[k1];
    }
  }
};

// Lanes per pencil and radices: the first radix is E = N / L, and every stage's
// N / R butterflies are a multiple of L.  The plain plans have the fewest
// exchanges (a float row pass at N = 256: 23 us with 16 lanes, 29 with 32).  The
// wide ones have half the elements per lane, for double stages that would have
// too few warps otherwise (a double row pass: 48.5 us and 49.5, the second at
// half the registers and exchange buffer per warp).
struct RowPlan {
  int lanes, n_stages, r[3];
};
QHD constexpr RowPlan row_plan(int n, bool wide = false) {
  if (wide && n == 256) return {32, 3, {8, 8, 4}};
  if (wide && n == 128) return {16, 3, {8, 4, 4}};
  switch (n) {
    case 8: return {4, 3, {2, 2, 2}};
    case 16: return {4, 2, {4, 4, 0}};
    case 32: return {4, 2, {8, 4, 0}};
    case 64: return {8, 2, {8, 8, 0}};
    case 96: return {8, 3, {12, 4, 2}};
    case 128: return {8, 2, {16, 8, 0}};
    case 192: return {16, 3, {12, 4, 4}};
    case 256: return {16, 2, {16, 16, 0}};
    case 512: return {32, 3, {16, 8, 4}};
    default: return {0, 0, {0, 0, 0}};
  }
}

template <typename T, int N, bool WIDE = false>
struct PencilFFT {
  static constexpr RowPlan plan = row_plan(N, WIDE);
  static_assert(plan.lanes > 0, "unsupported transform length");
  static constexpr int L = plan.lanes, E = N / L, H = E / 2;
  static constexpr int R1 = plan.r[0];
  static_assert(R1 == E && E % 2 == 0, "the first radix is a lane's share");
  // Padded place of element e of the exchange buffer, e + e / R1 (the first stage
  // writes with stride R1).  In the forms the stages use, as a lane's base plus a
  // constant, which the accesses take as immediates:
  QHD static constexpr int phi(int e) { return e + e / R1; }
  static constexpr int kPadded = N - 1 + (N - 1) / R1 + 1;
  // element l + L t
  QHD static int phi_read(int l, int t) {
    if constexpr (L % R1 == 0) return l + l / R1 + t * (L + L / R1);
    else if constexpr (R1 % L == 0) return l + (L * t + L * t / R1);
    else return int(unsigned(l + L * t) + unsigned(l + L * t) / unsigned(R1));
  }
  // output u of butterfly b = l + L c of stage ST (radix R, stride s)
  template <int ST>
  QHD static int phi_write(int l, int c, int u) {
    if constexpr (ST == 0) {
      return (R1 + 1) * l + (R1 + 1) * L * c + u;
    } else {   // s = R1: e = q + R1 (R2 p + u), p = b / R1, q = b % R1
      constexpr int R = plan.r[1];
      if constexpr (L % R1 == 0) return l % R1 + (R1 + 1) * R * (l / R1) + (R1 + 1) * (R * (L / R1) * c + u);
      const unsigned b = unsigned(l + L * c), p = b / unsigned(R1);
      return int(b - p * R1 + (R1 + 1) * R * p) + (R1 + 1) * u;
    }
  }
  // Tables in shared memory, per CTA: the first stage's twiddles W_N^{l u} as
  // [u][l], i times the quarter-wave table, and the second stage's W_N^{s p u} (s = R1)
  // as [u][p] when there is a third.
  static constexpr int R2 = plan.r[1], P2 = N / (R1 * R2);
  static constexpr int kTables = 2 * N + (plan.n_stages > 2 ? R2 * P2 : 0);   // complex entries
  struct Tab {
    const Cx<T>*tw1, *iquarter, *tw2;
  };
  static constexpr size_t table_bytes() { return (size_t(kTables) * sizeof(Cx<T>) + 15) / 16 * 16; }
  // fills the tables at `t`; the caller synchronises
  QHD static Tab fill_tables(Cx<T>* t, Tables<T> tb, int tid, int nt) {
    for (int e = tid; e < N; e += nt) {
      t[e] = tb.root[(e / L) * (e % L)];
      t[N + e] = Cx<T>{-tb.quarter[e].y, tb.quarter[e].x};
      if (plan.n_stages > 2 && e < R2 * P2) t[2 * N + e] = tb.root[R1 * (e / P2) * (e % P2)];
    }
    return Tab{t, t + N, t + 2 * N};
  }

  // One stage and (unless it is the last) the exchange after it.
  template <int ST, class W>
  QHD static void stage(const W& w, Cx<T>* v, Cx<T>* xb, const Tab& tb) {
    constexpr int R = plan.r[ST], B = E / R;
    constexpr int s = ST == 0 ? 1 : ST == 1 ? plan.r[0] : plan.r[0] * plan.r[1];
    constexpr bool last = ST == plan.n_stages - 1;
    const int l = w.l();
#pragma unroll
    for (int c = 0; c < B; ++c) {
      Cx<T> a[R];
#pragma unroll
      for (int u = 0; u < R; ++u) a[u] = v[c + B * u];
      Dft<T, R>::run(a);
      if constexpr (last) {
#pragma unroll
        for (int u = 0; u < R; ++u) v[c + B * u] = a[u];
      } else {
        const int p = ST == 0 ? 0 : int(unsigned(l + L * c) / unsigned(s));
#pragma unroll
        for (int u = 0; u < R; ++u) {
          Cx<T> f = a[u];
          if (u) f = cmul(f, ST == 0 ? tb.tw1[u * L + l] : tb.tw2[u * P2 + p]);
          if constexpr (W::template split<T>()) v[c + B * u] = f;
          else xb[w.at(phi_write<ST>(l, c, u))] = f;
        }
      }
    }
    if constexpr (!last && W::template split<T>()) {   // the real parts, then the imaginary ones
      T* xr = reinterpret_cast<T*>(xb);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int c = 0; c < B; ++c)
#pragma unroll
          for (int u = 0; u < R; ++u) xr[w.at(phi_write<ST>(l, c, u))] = h ? v[c + B * u].y : v[c + B * u].x;
        w.sync();
#pragma unroll
        for (int t = 0; t < E; ++t) {
          const T x = xr[w.at(phi_read(l, t))];
          if (h) v[t].y = x;
          else v[t].x = x;
        }
        w.sync();
      }
    } else if constexpr (!last) {
      w.sync();
#pragma unroll
      for (int t = 0; t < E; ++t) v[t] = xb[w.at(phi_read(l, t))];
      w.sync();
    }
  }
  template <class W>
  QHD static void dft(const W& w, Cx<T>* v, Cx<T>* xb, const Tab& tb) {
    stage<0>(w, v, xb, tb);
    stage<1>(w, v, xb, tb);
    if constexpr (plan.n_stages > 2) stage<2>(w, v, xb, tb);
  }

  // Inverse kinds (REDFT01; RODFT01 with its input reversed by the caller):
  // v[t] = (y_k of row a, y_k of row b) -> v[t] = (b, a) of the permuted outputs.
  // The inverse DFT of z is the forward DFT with real and imaginary parts swapped
  // on both sides; the swapped input is i quarter_k ((a_k + b_{N-k}) + i (a_{N-k} - b_k)).
  template <class W>
  QHD static void inverse(const W& w, Cx<T>* v, Cx<T>* xb, const Tab& tb) {
    const int l = w.l(), src = w.partner();
    Cx<T> prev = {T(0), T(0)};   // lane 0: y_N = 0, then its element E - t
#pragma unroll
    for (int t = 0; t < H; ++t) {
      const int u = E - 1 - t;
      const Cx<T> lo = v[t], hi = v[u], up = v[t + 1];
      const Cx<T> plo = w.shfl(l ? hi : prev, src), phi_ = w.shfl(l ? lo : up, src);
      prev = hi;
      v[t] = cmul(tb.iquarter[l + L * t], Cx<T>{lo.x + plo.y, plo.x - lo.y});
      v[u] = cmul(tb.iquarter[l + L * u], Cx<T>{hi.x + phi_.y, phi_.x - hi.y});
    }
    dft(w, v, xb, tb);
  }

  // Forward kinds (REDFT10; RODFT10 with odd positions negated and its output
  // reversed by the caller): v[t] = the permuted input -> v[t] = (y_k of row a,
  // y_k of row b).
  template <class W>
  QHD static void forward(const W& w, Cx<T>* v, Cx<T>* xb, const Tab& tb) {
    dft(w, v, xb, tb);
    const int l = w.l(), src = w.partner();
    Cx<T> prev = v[0];   // lane 0: Z_N = Z_0
#pragma unroll
    for (int t = 0; t < H; ++t) {
      const int u = E - 1 - t;
      const Cx<T> lo = v[t], hi = v[u], up = v[t + 1];
      const Cx<T> plo = w.shfl(l ? hi : prev, src), phi_ = w.shfl(l ? lo : up, src);
      prev = hi;
      v[t] = unpack(lo, plo, tb.iquarter[l + L * t]);
      v[u] = unpack(hi, phi_, tb.iquarter[l + L * u]);
    }
  }
  // y_k of both rows from Z_k and Z_{N-k}; q = i quarter_k
  QHD static Cx<T> unpack(Cx<T> z, Cx<T> n, Cx<T> q) {
    return Cx<T>{q.y * (z.x + n.x) + q.x * (z.y - n.y), q.y * (z.y + n.y) - q.x * (z.x - n.x)};
  }

  // Position of y_k along the axis.  sine: the kind's own order (k reversed);
  // mode (sine only): by mode number N - k, where the top mode N (k = 0) has no
  // place and the caller takes it as zero.
  QHD static int spec(int k, bool sine, bool mode = false) { return !sine ? k : mode ? (k ? N - k : 0) : N - 1 - k; }
  // Position of the permuted element k: even positions first, then the odd ones
  // from the top (sine kinds: odd positions negated).
  QHD static int pos(int k) { return k < N / 2 ? 2 * k : 2 * (N - 1 - k) + 1; }
};

// Rows: pencils of 2 rows, 32 / L pencils per warp.  Makhoul's permutation maps
// k < N/2 to position 2k and k >= N/2 to 2 (N - 1 - k) + 1, so the pair of
// adjacent positions (n, n + 1), n = 2 l + 2 L t, is this lane's element t and
// lane L - 1 - l's element E - 1 - t: one shuffle gives each lane adjacent pairs
// of both rows, and every real-space access is a 2-element vector.
template <typename T, int N, bool WIDE = false>
struct RowFFT : PencilFFT<T, N, WIDE> {
  using P = PencilFFT<T, N, WIDE>;
  using P::E;
  using P::H;
  using P::L;
  static constexpr int PPW = 32 / L, ROWS = 2 * PPW;   // pencils and rows of a warp
  // Double rows of more than 8 elements per lane exchange real and imaginary
  // parts one after the other: half the buffer at the same time (48.5 us at
  // N = 256 either way; in float 23 -> 27 us).
  static constexpr bool kSplit = sizeof(T) == 8 && E > 8;
  // elements between the pencils of a warp: the lanes of one access phase (16 of
  // 8 bytes, 8 of 16) that span several pencils hit distinct banks
  static constexpr int pencil_stride() {
    constexpr int ph = sizeof(T) == 8 && !kSplit ? 8 : 16;
    int x = P::kPadded;
    if (L < ph)
      while (x % ph != L) ++x;
    return x;
  }
  static constexpr int XS = pencil_stride();
  static constexpr size_t xch_bytes() {   // of a warp's exchange buffer
    return (size_t(PPW) * XS * (kSplit ? sizeof(T) : sizeof(Cx<T>)) + 15) / 16 * 16;
  }
  // Permuted outputs (b, a) -> adjacent positions: v[t] = row a at (n, n + 1), v[E - 1 - t]
  // = row b, n = 2 l + 2 L t.  sine: odd positions negated.
  template <class W>
  QHD static void to_pairs(const W& w, Cx<T>* v, bool sine) {
    const int src = w.mirror();
    const T s = sine ? T(-1) : T(1);
#pragma unroll
    for (int t = 0; t < H; ++t) {
      const Cx<T> o = w.shfl(v[E - 1 - t], src), e = v[t];
      v[t] = Cx<T>{e.y, s * o.y};
      v[E - 1 - t] = Cx<T>{e.x, s * o.x};
    }
  }
  // pairs -> (a, b) of the permuted positions, a forward kind's input
  template <class W>
  QHD static void from_pairs(const W& w, Cx<T>* v, bool sine) {
    const int src = w.mirror();
    const T s = sine ? T(-1) : T(1);
#pragma unroll
    for (int t = 0; t < H; ++t) {
      const Cx<T> a = v[t], b = v[E - 1 - t];
      v[t] = Cx<T>{a.x, b.x};
      v[E - 1 - t] = w.shfl(Cx<T>{s * a.y, s * b.y}, src);
    }
  }

};

#ifdef __CUDACC__
// The lanes of a warp as RowFFT places them.
template <typename T, int N, bool WIDE = false>
struct RowWarp {
  using F = RowFFT<T, N, WIDE>;
  template <typename> static constexpr bool split() { return F::kSplit; }
  int lane;
  __device__ __forceinline__ int l() const { return lane % F::L; }
  __device__ __forceinline__ int pencil() const { return lane / F::L; }
  __device__ __forceinline__ int partner() const { return lane - l() + ((F::L - l()) & (F::L - 1)); }
  __device__ __forceinline__ int mirror() const { return lane + F::L - 1 - 2 * l(); }
  __device__ __forceinline__ int at(int place) const { return pencil() * F::XS + place; }
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  __device__ __forceinline__ Cx<T> shfl(Cx<T> v, int src) const {
    return Cx<T>{__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
  }
};
#endif

// Columns: a tile of G pencils (2 G adjacent k) along the x or y axis on
// THREADS = G L threads (whole warps).  A warp holds S = 32 / G values of l for
// all G pencils, chosen so that l and L - l share it (the partner stays a
// shuffle): l and L - l for l in [w S / 2, (w + 1) S / 2), with L / 2 beside 0.
// Neighbouring l differ in parity, which puts a half-warp's float accesses to
// the exchange rows [e][g] on distinct banks.  Tiles of one warp synchronise the
// warp, wider ones a named barrier.
template <int N, int G, bool WIDE = false, bool SPLIT = false>
struct ColTile {
  // double real and imaginary parts exchanged one after the other
  template <typename T> static constexpr bool split() { return SPLIT && sizeof(T) == 8; }
  static constexpr int L = row_plan(N, WIDE).lanes, R1 = N / L, S = 32 / G;
  static constexpr int THREADS = G * L;
  static_assert(THREADS % 32 == 0 && S >= 2, "a tile is whole warps");
  static constexpr int ROWS = N - 1 + (N - 1) / R1 + 1;   // padded rows of G of the exchange buffer
  static constexpr int XCH = ROWS * G;                    // its complex elements
  int ll, part, g, bar;
  // r: thread of the tile; bar: its named barrier
  QHD ColTile(int r, int barrier) : bar(barrier) {
    const int lane = r & 31, sub = lane / G, h = sub % (S / 2), lo = (r / 32) * (S / 2) + h;
    g = lane % G;
    ll = sub < S / 2 ? lo : (lo == 0 ? L / 2 : L - lo);
    part = (lo == 0 ? sub : sub ^ (S / 2)) * G + g;
  }
  QHD int l() const { return ll; }
  QHD int partner() const { return part; }
  QHD int at(int place) const { return place * G + g; }
#ifdef __CUDACC__
  __device__ __forceinline__ void sync() const {
    if constexpr (THREADS == 32) __syncwarp();
    else asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(THREADS) : "memory");
  }
  // sync(), and whether `ok` held for every thread of the tile
  __device__ __forceinline__ bool sync_all(bool ok) const {
    if constexpr (THREADS == 32) {
      return __all_sync(0xffffffffu, ok);
    } else {
      uint32_t r;
      asm volatile(
          "{\n .reg .pred p, q;\n setp.ne.u32 q, %3, 0;\n barrier.cta.red.and.pred p, %1, %2, q;\n"
          " selp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(r)
          : "r"(bar), "n"(THREADS), "r"(uint32_t(ok))
          : "memory");
      return r != 0;
    }
  }
  template <typename T>
  __device__ __forceinline__ Cx<T> shfl(Cx<T> v, int src) const {
    return Cx<T>{__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src)};
  }
#endif
};

}  // namespace quasi
