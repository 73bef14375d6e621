// Element-fastest tile transform of P = 2G dense rows [p][n]: the first stage
// reads the dense rows, later stages a padded complex tile, and the output rows
// are staged densely over it.  The z passes transform their rows in registers
// (row_pass.cuh: fewer shared-memory round trips); this form, whose index
// arithmetic runs on the host, is their counterpart in tests/cpu/tiles.cpp.
//
// Element-fastest: the work items of a stage are numbered butterfly-fastest
// within a pencil (g = w / (N/R)), so a warp reads and writes runs of one
// row.  Where two pencils share a warp, odd pencils take the partner half of
// each (even n, odd n) or (e, e + N/R) pair first, which puts the two
// half-warps on disjoint banks.  The padded tile keeps complex e of pencil g
// at g * LDC + e + e / R1 (R1 = first radix), conflict-free for the stage-1
// writes (stride R1) and every later stage.
//
// Kinds, Makhoul reordering and the pairing of two real pencils into one
// complex DFT are those of r2r_core.cuh (FFTW's REDFT10/01, RODFT10/01).
#pragma once
#include <cstddef>

#include "r2r_core.cuh"

namespace quasi {

// SUB: the dense rows are held as SUB blocks [SUB][2G][N/SUB] (a TMA box side
// is at most 256 elements, so N = 512 moves as two boxes per row).
template <typename T, int N, int G, int NT, int SUB = 1>
struct ZTile {
  static constexpr RadixPlan plan = radix_plan(N, max_radix<T>());
  static constexpr int BN = N / SUB;
  static_assert(BN * SUB == N, "SUB divides N");
  // element n of dense row r
  QHD static constexpr int ri(int r, int n) {
    return SUB == 1 ? r * N + n : (n / BN) * (2 * G * BN) + r * BN + (n - (n / BN) * BN);
  }
  static_assert(plan.n_stages > 0, "unsupported transform length");
  static constexpr int R1 = plan.r[0];
  QHD static constexpr int phi(int e) { return e + e / R1; }
  // padded pencil stride (complex).  FP32: rounded to 8 mod 16 so that two
  // pencils sharing a warp start on different bank halves; FP64 (a warp
  // never spans two pencils of the sizes that matter) just even
  static constexpr int LDC =
      sizeof(T) == 8 ? ((phi(N - 1) + 2) / 2) * 2 : ((phi(N - 1) + 1 + 7) / 16) * 16 + 8;
  static constexpr size_t cb_bytes() { return size_t(G) * LDC * sizeof(Cx<T>); }
  static_assert(LDC >= N, "the staging rows overlay the padded tile");

  template <int R> static constexpr int per_thread() { return (G * (N / R) + NT - 1) / NT; }
  template <int R> struct Regs { Cx<T> v[per_thread<R>()][R]; };

  // stage-1 input e of pencil g from the dense rows (row[n + ks], zero past
  // the end): forward kinds with the Makhoul reorder, inverse kinds with the
  // pre-twiddle of r2r_core's first_input
  struct Rows {
    const T* raw;
    int ks;
    QHD T at(int r, int n) const { return n + ks < N ? raw[ri(r, n + ks)] : T(0); }
  };
  // the same with the shift fixed at compile time (the kernel's form); KS = 2:
  // row[n + 1] times -mk[n] (a z gradient's shift and wavenumber, zero at the top)
  template <int KS> struct RowsK {
    const T* raw;
    const T* mk = nullptr;
    QHD T at(int r, int n) const {
      if constexpr (KS == 0) return raw[ri(r, n)];
      else if constexpr (KS == 1) return n + 1 < N ? raw[ri(r, n + 1)] : T(0);
      else return n + 1 < N ? -mk[n] * raw[ri(r, n + 1)] : T(0);
    }
  };
  template <class Src>
  QHD static Cx<T> fwd_in(const Src& src, int kind, int g, int e) {
    int n;
    T sgn = T(1);
    if (e < N / 2) n = 2 * e;
    else { n = 2 * (N - 1 - e) + 1; if (kind == O10) sgn = T(-1); }
    return Cx<T>{sgn * src.at(2 * g, n), sgn * src.at(2 * g + 1, n)};
  }
  template <class Src>
  QHD static Cx<T> inv_in(const Src& src, int kind, int g, int k, Tables<T> tb) {
    const bool rev = kind == O01;
    const int n0 = rev ? N - 1 - k : k;
    const T ak = src.at(2 * g, n0), bk = src.at(2 * g + 1, n0);
    T an = T(0), bn = T(0);
    if (k) {
      const int n1 = rev ? k - 1 : N - k;
      an = src.at(2 * g, n1);
      bn = src.at(2 * g + 1, n1);
    }
    const Cx<T> q = tb.quarter[k];
    const Cx<T> ec = {q.x, -q.y};
    const Cx<T> va = cmul(ec, Cx<T>{ak, -an});
    const Cx<T> vb = cmul(ec, Cx<T>{bk, -bn});
    return Cx<T>{va.x - vb.y, -(va.y + vb.x)};
  }

  // first stage read (s = 1): butterfly b of pencil g takes e = b + t N/R
  // tw1 (optional): the first stage's twiddles W_N^{b u} as tw1[u * (N/R1) + b]
  // (a warp reads consecutive entries); otherwise tb.root[b u]
  template <class Src>
  QHD static void first_read(int tid, const Src& src, int kind, Tables<T> tb, Regs<R1>& r,
                             const Cx<T>* tw1 = nullptr) {
    constexpr int R = R1, M = N / R;
#pragma unroll
    for (int c = 0; c < per_thread<R>(); ++c) {
      const int w = tid + c * NT;
      if (w >= G * M) break;
      const int g = w / M, b = w - g * M;
      const bool x = g & 1;
      if (is_forward(kind)) {
        // pairs (t, t + R/2): even and odd Makhoul positions
#pragma unroll
        for (int t = 0; t < R / 2; ++t) {
          const Cx<T> A = fwd_in(src, kind, g, b + M * (x ? t + R / 2 : t));
          const Cx<T> B = fwd_in(src, kind, g, b + M * (x ? t : t + R / 2));
          r.v[c][t] = x ? B : A;
          r.v[c][t + R / 2] = x ? A : B;
        }
      } else {
        // pairs (t, t ^ 1): elements M apart
#pragma unroll
        for (int t = 0; t < R; t += 2) {
          const Cx<T> A = inv_in(src, kind, g, b + M * (x ? t + 1 : t), tb);
          const Cx<T> B = inv_in(src, kind, g, b + M * (x ? t : t + 1), tb);
          r.v[c][t] = x ? B : A;
          r.v[c][t + 1] = x ? A : B;
        }
      }
      Dft<T, R>::run(r.v[c]);
#pragma unroll
      for (int u = 1; u < R; ++u)
        if (b) r.v[c][u] = cmul(r.v[c][u], tw1 ? tw1[u * M + b] : tb.root[b * u]);
    }
  }

  // stage ST > 0 read from the padded tile (stride s, sub-length n = N / s)
  template <int R, int n, int s>
  QHD static void stage_read(int tid, const Cx<T>* cb, Tables<T> tb, Regs<R>& r) {
    constexpr int m = n / R, NB = N / R;
#pragma unroll
    for (int c = 0; c < per_thread<R>(); ++c) {
      const int w = tid + c * NT;
      if (w >= G * NB) break;
      const int g = w / NB, bfl = w - g * NB;
      const int p = bfl / s, q = bfl - p * s;
#pragma unroll
      for (int t = 0; t < R; ++t) r.v[c][t] = cb[g * LDC + phi(q + s * (p + t * m))];
      Dft<T, R>::run(r.v[c]);
      const int step = (N / n) * p;
#pragma unroll
      for (int u = 1; u < R; ++u)
        if (p) r.v[c][u] = cmul(r.v[c][u], tb.root[step * u]);
    }
  }

  // stage write into the padded tile
  template <int R, int s>
  QHD static void stage_write(int tid, Cx<T>* cb, const Regs<R>& r) {
    constexpr int NB = N / R;
#pragma unroll
    for (int c = 0; c < per_thread<R>(); ++c) {
      const int w = tid + c * NT;
      if (w >= G * NB) break;
      const int g = w / NB, bfl = w - g * NB;
      const int p = bfl / s, q = bfl - p * s;
#pragma unroll
      for (int u = 0; u < R; ++u) cb[g * LDC + phi(q + s * (R * p + u))] = r.v[c][u];
    }
  }

  // last stage of an inverse kind: u_k = conj(F_k) -> x_{2k} (k < N/2) or
  // x_{2(N-1-k)+1}, into the dense staging rows (real pencil 2g, 2g + 1)
  QHD static void put_inv(T* stg, int kind, int g, int k, Cx<T> f) {
    int n;
    T sgn = T(1);
    if (k < N / 2) n = 2 * k;
    else { n = 2 * (N - 1 - k) + 1; if (kind == O01) sgn = T(-1); }
    stg[ri(2 * g, n)] = sgn * f.x;
    stg[ri(2 * g + 1, n)] = -sgn * f.y;
  }
  template <int R, int s>
  QHD static void last_write_inv(int tid, T* stg, int kind, const Regs<R>& r) {
    constexpr int NB = N / R;   // = s: the last stage has p = 0
#pragma unroll
    for (int c = 0; c < per_thread<R>(); ++c) {
      const int w = tid + c * NT;
      if (w >= G * NB) break;
      const int g = w / NB, q = w - g * NB;
      const bool x = g & 1;
      if constexpr (R % 2 == 0) {
        // pairs (u, u + R/2): even and odd output positions
#pragma unroll
        for (int u = 0; u < R / 2; ++u) {
          const int ua = x ? u + R / 2 : u, ub = x ? u : u + R / 2;
          put_inv(stg, kind, g, q + s * ua, x ? r.v[c][u + R / 2] : r.v[c][u]);
          put_inv(stg, kind, g, q + s * ub, x ? r.v[c][u] : r.v[c][u + R / 2]);
        }
      } else {
#pragma unroll
        for (int u = 0; u < R; ++u) put_inv(stg, kind, g, q + s * u, r.v[c][u]);
      }
    }
  }

  // forward kinds: y(k), y(N-k) from (Z_k, Z_{N-k}); item k = 0 also makes
  // the self-paired y(N/2)
  static constexpr int kUnpack = (G * (N / 2) + NT - 1) / NT;
  struct UnpackRegs {
    T ya[kUnpack][2], yb[kUnpack][2];   // [1]: y(N-k), or y(N/2) for k = 0
  };
  QHD static void unpack_one(Cx<T> zk, Cx<T> zr_conj_src, Cx<T> qk, T& ya, T& yb) {
    const Cx<T> zr = conj(zr_conj_src);
    const Cx<T> va = zk + zr;
    const Cx<T> d = zk - zr;
    const Cx<T> vb = {d.y, -d.x};
    ya = qk.x * va.x - qk.y * va.y;
    yb = qk.x * vb.x - qk.y * vb.y;
  }
  QHD static void unpack_read(int tid, const Cx<T>* cb, Tables<T> tb, UnpackRegs& r) {
    constexpr int H = N / 2;
#pragma unroll
    for (int c = 0; c < kUnpack; ++c) {
      const int w = tid + c * NT;
      if (w >= G * H) break;
      const int g = w / H, k = w - g * H;
      const Cx<T>* pc = cb + g * LDC;
      const Cx<T> z0 = pc[phi(k)];
      const Cx<T> z1 = pc[phi(k ? N - k : H)];
      if (k) {
        unpack_one(z0, z1, tb.quarter[k], r.ya[c][0], r.yb[c][0]);
        unpack_one(z1, z0, tb.quarter[N - k], r.ya[c][1], r.yb[c][1]);
      } else {
        unpack_one(z0, z0, tb.quarter[0], r.ya[c][0], r.yb[c][0]);
        unpack_one(z1, z1, tb.quarter[H], r.ya[c][1], r.yb[c][1]);   // z1 = Z_{N/2}
      }
    }
  }
  QHD static void unpack_write(int tid, T* stg, int kind, const UnpackRegs& r) {
    constexpr int H = N / 2;
#pragma unroll
    for (int c = 0; c < kUnpack; ++c) {
      const int w = tid + c * NT;
      if (w >= G * H) break;
      const int g = w / H, k = w - g * H;
      auto idx = [&](int kk) { return kind == O10 ? N - 1 - kk : kk; };
      stg[ri(2 * g, idx(k))] = r.ya[c][0];
      stg[ri(2 * g + 1, idx(k))] = r.yb[c][0];
      const int k1 = k ? N - k : H;
      stg[ri(2 * g, idx(k1))] = r.ya[c][1];
      stg[ri(2 * g + 1, idx(k1))] = r.yb[c][1];
    }
  }
};

// Stages 1 .. last of the tile after the first stage's writes, then (forward)
// the unpack: `ex.phase(rd, wr, ...)` as in r2r_core.cuh.  Leaves the dense
// output rows in `stg` (which overlays `cb`) without a closing barrier: the
// caller fences them for the TMA store and synchronises.
template <typename T, int N, int G, int NT, int ST, int SUB = 1, class Exec>
QHD void ztile_rest(Exec& ex, int tid, int kind, Cx<T>* cb, T* stg, Tables<T> tb) {
  using Z = ZTile<T, N, G, NT, SUB>;
  if constexpr (ST < Z::plan.n_stages) {
    constexpr int R = Z::plan.r[ST];
    constexpr int s = stage_stride(N, ST, max_radix<T>()), n = N / s;
    constexpr bool last = ST == Z::plan.n_stages - 1;
    using Regs = typename Z::template Regs<R>;
    Regs regs;
    if (last && !is_forward(kind)) {
      ex.phase([&](int t, Regs& rg) { Z::template stage_read<R, n, s>(t, cb, tb, rg); },
               [&](int t, Regs& rg) { Z::template last_write_inv<R, s>(t, stg, kind, rg); }, tid, regs, true, false);
      return;
    }
    ex.phase([&](int t, Regs& rg) { Z::template stage_read<R, n, s>(t, cb, tb, rg); },
             [&](int t, Regs& rg) { Z::template stage_write<R, s>(t, cb, rg); }, tid, regs, true, true);
    if constexpr (last) {
      typename Z::UnpackRegs ur;
      ex.phase([&](int t, typename Z::UnpackRegs& rg) { Z::unpack_read(t, cb, tb, rg); },
               [&](int t, typename Z::UnpackRegs& rg) { Z::unpack_write(t, stg, kind, rg); }, tid, ur, true, false);
    } else {
      ztile_rest<T, N, G, NT, ST + 1, SUB>(ex, tid, kind, cb, stg, tb);
    }
  }
}

// Single-stage plans (N = R1) end in the first stage: its output goes through
// the padded tile so that the write above stays uniform.
template <typename T, int N, int G, int NT, int SUB = 1, class Exec>
QHD void ztile_after_first(Exec& ex, int tid, int kind, Cx<T>* cb, T* stg, Tables<T> tb) {
  using Z = ZTile<T, N, G, NT, SUB>;
  if constexpr (Z::plan.n_stages > 1) {
    ztile_rest<T, N, G, NT, 1, SUB>(ex, tid, kind, cb, stg, tb);
  } else {
    // the first stage wrote Z (or F) in natural order: finish like a last stage
    if (is_forward(kind)) {
      typename Z::UnpackRegs ur;
      ex.phase([&](int t, typename Z::UnpackRegs& rg) { Z::unpack_read(t, cb, tb, rg); },
               [&](int t, typename Z::UnpackRegs& rg) { Z::unpack_write(t, stg, kind, rg); }, tid, ur, true, false);
    } else {
      struct One {
        T x[(G * N + NT - 1) / NT], y[(G * N + NT - 1) / NT];
      } one;
      ex.phase(
          [&](int t, One& o) {
            for (int c = 0; c < (G * N + NT - 1) / NT; ++c) {
              const int w = t + c * NT;
              if (w >= G * N) break;
              const int g = w / N, k = w - g * N;
              const Cx<T> f = cb[g * Z::LDC + Z::phi(k)];
              o.x[c] = f.x;
              o.y[c] = f.y;
            }
          },
          [&](int t, One& o) {
            for (int c = 0; c < (G * N + NT - 1) / NT; ++c) {
              const int w = t + c * NT;
              if (w >= G * N) break;
              const int g = w / N, k = w - g * N;
              Z::put_inv(stg, kind, g, k, Cx<T>{o.x[c], o.y[c]});
            }
          },
          tid, one, true, false);
    }
  }
}

}  // namespace quasi
