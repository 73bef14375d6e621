// The real-space stages of the step, each between the z passes around it, on
// rows held in a warp's registers (pencil_core.cuh): a stage's inverse z passes,
// its pointwise work and its forward z passes are one kernel, and a field that
// only the stage itself needs in real space is never written.
//   gradient_stage     psi, grad psi from their spectra; the density law -> its z pass
//   density_stage      rho, grad rho -> divv -> its z pass
//   stress_stage       df, lap, grad lap psi -> the stress -> its z passes
//   nonlinear_stage    v, p -> N -> its z pass
// The inverse's output and the forward's input place positions alike, so the
// pointwise work needs no exchange; fields in memory are read and written as
// adjacent pairs of two rows (RowFFT::to_pairs).
//
// Bound: HBM, one read or write of each field named above.  Values that a later
// transform of the same rows needs stay in a warp's private shared memory
// (8-byte slots in float, 16-byte in double, no synchronisation), since they and
// a transform's registers together would spill.
#pragma once
#include <cuda_runtime.h>

#include "col_pass.cuh"

namespace quasi {

// The double stages use the wide plans: a warp then holds half the rows, in half
// the registers and shared memory, and an SM 16 warps or more (with the plain
// plans 8: the FP64 stages ran at 0.4 of the HBM rate, waiting for memory).
template <typename T> constexpr bool kWide = sizeof(T) == 8;

// CTAs of 4 warps per SM that a stage's registers must allow: 16 warps, 12 where
// a lane's double rows alone take 48 registers or more.
template <typename T, int N>
constexpr int stage_ctas() { return sizeof(T) == 8 && RowFFT<T, N, kWide<T>>::E > 8 ? 3 : 4; }

// Float stages that spill at 16 warps (128 registers) run on 12 (168 registers),
// faster per round of groups (256^3: stress 10 rounds in 317 us against 7 in 434, 2.0
// times per round; nonlinear 232 and 247 us, 1.5 times), unless that takes 8/5 as many
// rounds: 96x96x192 has 1.3 rounds of 12 warps and one of 16 (stress 57 and 46 us,
// nonlinear 39 and 34), 128^3 two and one (64 and 67, 45 and 38).  Sixteen have to
// fit: at N = 512 only three CTAs of four warps do (stress of 64x64x512 70 us with
// their registers, 95 without).
template <class S>
constexpr bool kSixteenFit = 4 * (S::bytes() + 1024) <= 228 * 1024;   // an SM's shared memory, 1 KB per CTA reserved
inline bool sixteen_warps(int groups, int sms) {
  const int r12 = (groups + 12 * sms - 1) / (12 * sms), r16 = (groups + 16 * sms - 1) / (16 * sms);
  return 8 * r16 < 5 * r12;
}

// A lane's pairs: pair i (< E) of its two rows, element offset from row a.
template <class F, int N>
__device__ __forceinline__ int pair_off(int i, int l) {
  return (i < F::H ? 0 : N) + 2 * (l + F::L * (i < F::H ? i : F::E - 1 - i));
}

// Spectral rows whose direction is known at run time only.  sine: by mode number
// (element k is mode N - k, element 0 nothing); grad: a cosine spectrum read as
// the sine spectrum of its derivative, -q_m c_m.
template <class F, int N, typename T>
__device__ __forceinline__ void load_rows(const T* a, int l, Cx<T>* v, bool sine, const double* grad = nullptr) {
  const int n0 = sine ? N - l : l, dn = sine ? -F::L : F::L;
#pragma unroll
  for (int t = 0; t < F::E; ++t) {
    const bool none = t == 0 && sine && l == 0;
    const int n = none ? 0 : n0 + dn * t;
    v[t] = Cx<T>{a[n], a[N + n]};
    if (grad && sine) v[t] = cscale(v[t], T(-grad[n]));
    if (none) v[t] = Cx<T>{T(0), T(0)};
  }
}
template <class F, int N, typename T>
__device__ __forceinline__ void store_rows(T* a, int l, const Cx<T>* v, bool sine) {
  const int n0 = sine ? N - l : l, dn = sine ? -F::L : F::L;
#pragma unroll
  for (int t = 0; t < F::E; ++t) {
    const bool none = t == 0 && sine && l == 0;
    const int n = none ? 0 : n0 + dn * t;
    a[n] = none ? T(0) : v[t].x;
    a[N + n] = none ? T(0) : v[t].y;
  }
}

// Shared memory of a row stage on W warps: twiddles in T (and in double when
// DBL), the z wavenumbers, and per warp an exchange buffer and SLOTS private
// arrays of E complex values of T per lane.
template <typename T, int N, int W, bool DBL, int SLOTS>
struct RowStage {
  using F = RowFFT<T, N, kWide<T>>;
  using FD = RowFFT<double, N, kWide<T>>;
  static constexpr int kWarps = W;
  static constexpr bool kTwo = DBL && sizeof(T) == 4;
  static constexpr int NT = 32 * W;
  static constexpr size_t xch_bytes() {
    return kTwo && FD::xch_bytes() > F::xch_bytes() ? FD::xch_bytes() : F::xch_bytes();
  }
  static constexpr size_t warp_bytes() { return xch_bytes() + size_t(SLOTS) * F::E * 32 * sizeof(Cx<T>); }
  static constexpr size_t bytes() {
    return F::table_bytes() + (kTwo ? FD::table_bytes() : 0) + N * sizeof(double) + W * warp_bytes();
  }
  typename F::Tab t;
  typename FD::Tab td;
  const double* qz;
  Cx<T>* xb;
  Cx<double>* xd;
  Cx<T>* slots;
  __device__ __forceinline__ RowStage(unsigned char* sm, Tables<T> tb, Tables<double> tb64, const double* vqz) {
    if constexpr (kTwo) {
      td = FD::fill_tables(reinterpret_cast<Cx<double>*>(sm), tb64, threadIdx.x, NT);
      sm += FD::table_bytes();
    }
    t = F::fill_tables(reinterpret_cast<Cx<T>*>(sm), tb, threadIdx.x, NT);
    sm += F::table_bytes();
    double* q = reinterpret_cast<double*>(sm);
    for (int e = threadIdx.x; e < N; e += NT) q[e] = vqz[e];
    qz = q;
    sm += N * sizeof(double) + (threadIdx.x >> 5) * warp_bytes();
    xb = reinterpret_cast<Cx<T>*>(sm);
    xd = reinterpret_cast<Cx<double>*>(sm);
    slots = reinterpret_cast<Cx<T>*>(sm + xch_bytes()) + (threadIdx.x & 31);
    __syncthreads();
    pdl_begin();
  }
  // this lane's slot s of array a
  __device__ __forceinline__ Cx<T>& slot(int a, int s) const { return slots[(a * F::E + s) * 32]; }
  // slot array 0 in double; FP32: 16-byte slots over two arrays
  __device__ __forceinline__ Cx<double>& wide(int s) const {
    if constexpr (sizeof(T) == 8) {
      return slot(0, s);
    } else {
      static_assert(SLOTS >= 2, "two arrays");
      return reinterpret_cast<Cx<double>*>(slots - (threadIdx.x & 31))[s * 32 + (threadIdx.x & 31)];
    }
  }
  // an 8-byte slot as a double
  __device__ __forceinline__ double& dslot(int a, int s) const {
    static_assert(sizeof(T) == 4, "an 8-byte slot");
    return *reinterpret_cast<double*>(&slots[(a * F::E + s) * 32]);
  }
};

// A warp's rows of a field are one block of memory: lane 0 starts fetching it
// into L2 while the fields before it are worked on, since a stage's registers and
// shared memory leave 8 to 16 warps per SM, too few to hide HBM latency.
template <class F, int N, typename P>
__device__ __forceinline__ void prefetch_rows(const P* f, int grp, int lane) {
  if (lane == 0) prefetch_l2(f + size_t(grp) * F::ROWS * N, F::ROWS * N * sizeof(P));
}

// psi and grad psi (all double) from the x- and y-transformed spectra: psi and
// grad_z from `both` (quasi.cpp:1120-1186, 1963-1965), then with `law` the z pass
// of rho = kp sqrt(q0^2 psi^2 + |grad psi|^2) + rho_0 (quasi.cpp:1243-1247).
// count: the step counter, bumped once when the stage ends a step.
struct GradientStage {
  const double *both, *sy, *sx;   // spectra of psi (cosine), grad_y, grad_x
  double *psi, *gx, *gy, *gz;
  double* law;                    // nullptr: quasi-stb (rho == 1)
  const double* vqz;
  double kp, q0, rho0;
  int* count;
};
template <int N>
using GradientSmem = RowStage<double, N, 4, true, 1>;
template <int N>
__global__ void __launch_bounds__(GradientSmem<N>::NT, N >= 512 ? 3 : 4)
    gradient_stage_kernel(const __grid_constant__ GradientStage a, int groups, Tables<double> tb) {
  using S = GradientSmem<N>;
  using F = typename S::F;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const S sh(smem_raw, tb, tb, a.vqz);
  if (a.count && blockIdx.x == 0 && threadIdx.x == 0) *a.count += 1;
  const RowWarp<double, N, true> w{int(threadIdx.x & 31)};
  const int l = w.l(), stride = gridDim.x * S::kWarps;
  const double q02 = a.q0 * a.q0;
  for (int grp = blockIdx.x * S::kWarps + (threadIdx.x >> 5); grp < groups; grp += stride) {
    const int rg = groups - 1 - grp;
    const size_t row = (size_t(rg) * F::ROWS + 2 * w.pencil()) * N;
    Cx<double> v[F::E];
#pragma unroll 1
    for (int f = 0; f < 4; ++f) {   // grad_x, grad_y, grad_z, psi
      const bool sine = f == 2;
      if (f < 2) prefetch_rows<F, N>(f == 0 ? a.sy : a.both, rg, w.lane);
      if (f == 3 && grp + stride < groups) prefetch_rows<F, N>(a.sx, rg - stride, w.lane);
      load_rows<F, N>((f == 0 ? a.sx : f == 1 ? a.sy : a.both) + row, l, v, sine, sh.qz);
      F::inverse(w, v, sh.xb, sh.t);
      F::to_pairs(w, v, sine);
      double* out = (f == 0 ? a.gx : f == 1 ? a.gy : f == 2 ? a.gz : a.psi) + row;
      const double c = f == 3 ? q02 : 1.0;
#pragma unroll
      for (int i = 0; i < F::E; ++i) {
        st2(out + pair_off<F, N>(i, l), v[i]);
        Cx<double> r{c * v[i].x * v[i].x, c * v[i].y * v[i].y};
        if (f) r = r + sh.slot(0, i);
        sh.slot(0, i) = r;
      }
    }
    if (a.law) {
#pragma unroll
      for (int i = 0; i < F::E; ++i) {
        const Cx<double> r = sh.slot(0, i);
        v[i] = Cx<double>{a.kp * sqrt(r.x) + a.rho0, a.kp * sqrt(r.y) + a.rho0};
      }
      F::from_pairs(w, v, false);
      F::forward(w, v, sh.xb, sh.t);
      store_rows<F, N>(a.law + row, l, v, false);
    }
  }
}

// rho and divv of the density-varying model: from the x- and y-transformed spectra
//   grad rho of the previous step's rho^ (quasi.cpp:1188-1232) -> |grad rho| times the pressure factor
//   rho (quasi.cpp:1266-1268); divv after the switch (quasi.cpp:1273-1289) -> its z pass
// The difference quotient and the advection sum are taken in double.  (One stage
// with the stress below saved a read of rho, but left 8 warps per SM: 610 us at
// 256^3 in the FP32 form, against 198 and 266 apart; now, with the stress's sums in
// double, 203 and 320.)
template <typename T>
struct DensityStage {
  const T *rdx, *rdy, *rdz;         // grad rho's spectra; FP64: rdz is the cosine spectrum of that rho
  const double *rho_s, *rho_old;    // rho's spectrum, the previous step's rho
  const T* v[3];
  double* rho;
  T *grad, *divv, *divv_s;
  const double* vqz;
  double dt, cp;
  int divv_switch;
  const int* nloop;
};
// FP32: the advection sum takes two 8-byte slot arrays and rho a double exchange
// buffer, 12.6 KB per warp.  Two CTAs of 6 warps per SM: 7 fit, but with 128
// registers per thread the kernel spills (256^3: 230 us against 194, 5 warps 217).
template <typename T> constexpr int density_warps() { return sizeof(T) == 4 ? 6 : 4; }
template <typename T, int N>
using DensitySmem = RowStage<T, N, density_warps<T>(), true, sizeof(T) == 4 ? 2 : 1>;
template <typename T, int N>
__global__ void __launch_bounds__(32 * density_warps<T>(), sizeof(T) == 4 ? 2 : stage_ctas<T, N>() - 1)
    density_stage_kernel(const __grid_constant__ DensityStage<T> a, int groups, Tables<T> tb, Tables<double> tb64) {
  using S = DensitySmem<T, N>;
  using F = typename S::F;
  using FD = typename S::FD;
  constexpr bool kDbl = sizeof(T) == 8;
  constexpr int W = density_warps<T>();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const S sh(smem_raw, tb, tb64, a.vqz);
  const RowWarp<T, N, kWide<T>> w{int(threadIdx.x & 31)};
  const RowWarp<double, N, kWide<T>> wd{int(threadIdx.x & 31)};
  const int l = w.l(), stride = gridDim.x * W;
  const bool on = *a.nloop + 1 > a.divv_switch;
  const double idt = 1.0 / a.dt;
  const T cp = T(a.cp);
  for (int grp = blockIdx.x * W + (threadIdx.x >> 5); grp < groups; grp += stride) {
    const int rg = groups - 1 - grp;
    const size_t row = (size_t(rg) * F::ROWS + 2 * w.pencil()) * N;
    Cx<T> v[F::E], sq[F::E];
    // rho's rows and divv from them; d: the pairs of divv
    auto density = [&](const Cx<double>* r, Cx<T>* d) {
#pragma unroll
      for (int i = 0; i < F::E; ++i) {
        const size_t at = row + pair_off<F, N>(i, l);
        const Cx<double> x = r[i];
        st2(a.rho + at, x);
        Cx<double> adv;
        if constexpr (kDbl) adv = sh.slot(0, i);
        else adv = Cx<double>{sh.dslot(0, i), sh.dslot(1, i)};
        if (on) {
          const Cx<double> o = ld2(a.rho_old + at);
          d[i] = Cx<T>{T(-((x.x - o.x) * idt + adv.x) / (0.5 * (x.x + o.x))),
                       T(-((x.y - o.y) * idt + adv.y) / (0.5 * (x.y + o.y)))};
          st2(a.divv + at, d[i]);
        } else {
          d[i] = ld2(a.divv + at);
        }
      }
    };
#pragma unroll 1
    for (int c = 0; c < (kDbl ? 4 : 3); ++c) {   // grad rho; FP64: rho
      if (c < 2) {
        prefetch_rows<F, N>(c == 0 ? a.rdy : a.rdz, rg, w.lane);
        prefetch_rows<F, N>(a.v[c + 1], rg, w.lane);
      } else if (c == 2) {
        prefetch_rows<F, N>(a.rho_s, rg, w.lane);
        prefetch_rows<F, N>(a.rho_old, rg, w.lane);
      }
      const T* src = c == 0 ? a.rdx : c == 1 ? a.rdy : a.rdz;
      if constexpr (kDbl) src = c == 3 ? a.rho_s : src;
      load_rows<F, N>(src + row, l, v, c == 2, kDbl ? sh.qz : nullptr);
      F::inverse(w, v, sh.xb, sh.t);
      F::to_pairs(w, v, c == 2);
      if (c < 3) {
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
          const Cx<T> u = ld2(a.v[c] + row + pair_off<F, N>(i, l));
          const double ax = double(u.x) * double(v[i].x), ay = double(u.y) * double(v[i].y);
          const Cx<T> r{v[i].x * v[i].x, v[i].y * v[i].y};
          sq[i] = c ? sq[i] + r : r;
          if constexpr (kDbl) {
            sh.slot(0, i) = c ? sh.slot(0, i) + Cx<double>{ax, ay} : Cx<double>{ax, ay};
          } else {
            sh.dslot(0, i) = c ? sh.dslot(0, i) + ax : ax;
            sh.dslot(1, i) = c ? sh.dslot(1, i) + ay : ay;
          }
        }
      }
      if (c == 2) {
#pragma unroll
        for (int i = 0; i < F::E; ++i)
          st2(a.grad + row + pair_off<F, N>(i, l), Cx<T>{cp * sqrt(sq[i].x), cp * sqrt(sq[i].y)});
      }
    }
    if (grp + stride < groups) {
      prefetch_rows<F, N>(a.rdx, rg - stride, w.lane);
      prefetch_rows<F, N>(a.v[0], rg - stride, w.lane);
    }
    if constexpr (kDbl) {
      density(v, v);
    } else {
      Cx<double> r[FD::E];
      load_rows<FD, N>(a.rho_s + row, l, r, false);
      FD::inverse(wd, r, sh.xd, sh.td);
      FD::to_pairs(wd, r, false);
      density(r, v);
    }
    F::from_pairs(w, v, false);
    F::forward(w, v, sh.xb, sh.t);
    store_rows<F, N>(a.divv_s + row, l, v, false);
  }
}

// The stress: from the x- and y-transformed spectra of lap, df and grad lap psi,
// and rho, psi, grad psi
//   df, and the part of N that needs neither velocity nor pressure (quasi.cpp:1905-1929)
//   S = rho (lap grad psi - df grad lap psi) (quasi.cpp:1305-1317) -> their z passes
// quasi-stb: mu = sh - beta psi^3 + gamma psi^5 in df's place, S = mu grad psi
// (quasi-stb.cpp:1295-1305); in the FP32 form a kernel of its own (StressStb).
template <typename T>
struct StressStage {
  const T *lap_s, *df_s;   // quasi-stb: df_s is sh's spectrum
  const T* ld[3];
  const double *rho, *psi, *g[3];
  T *df, *base, *s[3];     // quasi-stb: df is mu
  const double* vqz;
  double ep, beta, gamma;
  int variant;
};
template <typename T, int N>
using StressSmem = RowStage<T, N, 4, false, sizeof(T) == 4 ? 2 : 1>;
template <typename T, int N, int CTAS>
__global__ void __launch_bounds__(128, CTAS)
    stress_stage_kernel(const __grid_constant__ StressStage<T> a, int groups, Tables<T> tb) {
  using S = StressSmem<T, N>;
  using F = typename S::F;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const S sh(smem_raw, tb, Tables<double>{}, a.vqz);
  const RowWarp<T, N, kWide<T>> w{int(threadIdx.x & 31)};
  const int l = w.l(), stride = gridDim.x * 4;
  const bool quasi = a.variant == 0;
  const T beta = T(a.beta), gamma = T(a.gamma);
  for (int grp = blockIdx.x * 4 + (threadIdx.x >> 5); grp < groups; grp += stride) {
    const int rg = groups - 1 - grp;
    const size_t row = (size_t(rg) * F::ROWS + 2 * w.pencil()) * N;
    // FP32: lap and df, and rho in the slots (double); FP64: rho lap, and rho df in
    // the slots.  quasi-stb: mu in the slots.
    constexpr bool kDbl = sizeof(T) == 8;
    Cx<T> v[F::E], lap[F::E], df[kDbl ? 1 : F::E];
#pragma unroll 1
    for (int f = quasi ? 0 : 1; f < 5; ++f) {   // lap, df, then the three components
      if (quasi) {
        if (f == 0) {
          prefetch_rows<F, N>(a.df_s, rg, w.lane);
          prefetch_rows<F, N>(a.psi, rg, w.lane);
          prefetch_rows<F, N>(a.rho, rg, w.lane);
        } else if (f < 4) {
          prefetch_rows<F, N>(a.ld[f - 1], rg, w.lane);
        } else if (grp + stride < groups) {
          prefetch_rows<F, N>(a.lap_s, rg - stride, w.lane);
        }
      } else if (f == 4 && grp + stride < groups) {
        prefetch_rows<F, N>(a.df_s, rg - stride, w.lane);
        prefetch_rows<F, N>(a.psi, rg - stride, w.lane);
      }
      if (f >= 1 && f < 4) prefetch_rows<F, N>(a.g[f - 1], rg, w.lane);
      if (quasi || f == 1) {
        load_rows<F, N>((f == 0 ? a.lap_s : f == 1 ? a.df_s : a.ld[f - 2]) + row, l, v, f == 4);
        F::inverse(w, v, sh.xb, sh.t);
        F::to_pairs(w, v, f == 4);
      }
      if (f == 0) {
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
          lap[i] = v[i];
        }
      } else if (f == 1) {
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
          const size_t at = row + pair_off<F, N>(i, l);
          const Cx<double> ps = ld2(a.psi + at);
          if (quasi) {
            // in double: near equilibrium the terms cancel, and what is left drives
            // the density whose time derivative is divv
            const Cx<double> r = ld2(a.rho + at);
            auto part = [&](double p, double rr, double d, double lp) {
              const double p2 = p * p;
              return T(rr * (p * (a.ep + p2 * (a.beta - a.gamma * p2)) - d - lp));
            };
            st2(a.df + at, v[i]);
            st2(a.base + at, Cx<T>{part(ps.x, r.x, v[i].x, lap[i].x), part(ps.y, r.y, v[i].y, lap[i].y)});
            if constexpr (kDbl) {
              sh.slot(0, i) = Cx<T>{r.x * v[i].x, r.y * v[i].y};
              lap[i] = Cx<T>{r.x * lap[i].x, r.y * lap[i].y};
            } else {
              sh.wide(i) = r;
              df[i] = v[i];
            }
          } else if constexpr (kDbl) {
            auto pot = [&](T x) { return beta * x * x * x - gamma * x * x * x * x * x; };
            const Cx<T> p{pot(ps.x), pot(ps.y)}, m{v[i].x - p.x, v[i].y - p.y};
            st2(a.df + at, m);
            st2(a.base + at, p);
            sh.slot(0, i) = m;
          }
        }
      } else {
        const int c = f - 2;
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
          const Cx<double> g = ld2(a.g[c] + row + pair_off<F, N>(i, l));
          if (quasi && kDbl) {
            const Cx<T> rd = sh.slot(0, i);
            v[i] = Cx<T>{T(lap[i].x * g.x - rd.x * v[i].x), T(lap[i].y * g.y - rd.y * v[i].y)};
          } else if (quasi) {   // in double: the two products nearly cancel
            const Cx<double> r = sh.wide(i);
            v[i] = Cx<T>{T(r.x * (double(lap[i].x) * g.x - double(df[kDbl ? 0 : i].x) * v[i].x)),
                         T(r.y * (double(lap[i].y) * g.y - double(df[kDbl ? 0 : i].y) * v[i].y))};
          } else if constexpr (kDbl) {
            const Cx<T> m = sh.slot(0, i);
            v[i] = Cx<T>{m.x * g.x, m.y * g.y};
          }
        }
        F::from_pairs(w, v, c == 2);
        F::forward(w, v, sh.xb, sh.t);
        store_rows<F, N>(a.s[c] + row, l, v, c == 2);
      }
    }
  }
}

// The stress of quasi-stb in the FP32 form: sh, mu and its products with grad psi
// in double, each result rounded once.  (mu in float would do; sh is what has to
// be in double, see update_x_kernel.)
struct StressStb {
  const double *sh_s, *psi, *g[3];   // sh_s: sh's spectrum
  float *mu, *base, *s[3];
  const double* vqz;
  double beta, gamma;
};
template <int N>
using StressStbSmem = RowStage<float, N, 4, true, 2>;
template <int N, int CTAS>
__global__ void __launch_bounds__(128, CTAS)
    stress_stb_kernel(const __grid_constant__ StressStb a, int groups, Tables<float> tb, Tables<double> tb64) {
  using S = StressStbSmem<N>;
  using F = typename S::F;
  using FD = typename S::FD;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const S sh(smem_raw, tb, tb64, a.vqz);
  const RowWarp<float, N> w{int(threadIdx.x & 31)};
  const RowWarp<double, N> wd{w.lane};
  const int l = w.l(), stride = gridDim.x * 4;
  for (int grp = blockIdx.x * 4 + (threadIdx.x >> 5); grp < groups; grp += stride) {
    const int rg = groups - 1 - grp;
    const size_t row = (size_t(rg) * F::ROWS + 2 * w.pencil()) * N;
    prefetch_rows<F, N>(a.psi, rg, w.lane);
    prefetch_rows<F, N>(a.g[0], rg, w.lane);
    Cx<double> x[FD::E];
    load_rows<FD, N>(a.sh_s + row, l, x, false);
    FD::inverse(wd, x, sh.xd, sh.td);
    FD::to_pairs(wd, x, false);
#pragma unroll
    for (int i = 0; i < FD::E; ++i) {
      const size_t at = row + pair_off<F, N>(i, l);
      const Cx<double> p = ld2(a.psi + at);
      auto pot = [&](double y) { return a.beta * y * y * y - a.gamma * y * y * y * y * y; };
      const Cx<double> n{pot(p.x), pot(p.y)}, m{x[i].x - n.x, x[i].y - n.y};
      st2(a.mu + at, as<float>(m));
      st2(a.base + at, as<float>(n));
      sh.wide(i) = m;
    }
#pragma unroll 1
    for (int c = 0; c < 3; ++c) {
      if (c < 2) prefetch_rows<F, N>(a.g[c + 1], rg, w.lane);
      else if (grp + stride < groups) prefetch_rows<F, N>(a.sh_s, rg - stride, w.lane);
      Cx<float> v[F::E];
#pragma unroll
      for (int i = 0; i < F::E; ++i) {
        const Cx<double> g = ld2(a.g[c] + row + pair_off<F, N>(i, l)), m = sh.wide(i);
        v[i] = Cx<float>{float(m.x * g.x), float(m.y * g.y)};
      }
      F::from_pairs(w, v, c == 2);
      F::forward(w, v, sh.xb, sh.t);
      store_rows<F, N>(a.s[c] + row, l, v, c == 2);
    }
  }
}

// v and p from their spectra, then N (quasi.cpp:1905-1929, quasi-stb.cpp:1900-1924)
// -> its z pass.  quasi: N = base - v . grad psi [+ p |grad rho|-term after the
// switch]; quasi-stb: N = base - v . grad psi, dtpsi = -mu - v . grad psi.
template <typename T>
struct NonlinearStage {
  T *v[3], *p;             // spectra in, real out (quasi-stb leaves p as it is)
  const double* g[3];
  const T *base, *grad, *mu;
  T *dtpsi, *out;
  const double* vqz;
  int variant, divv_switch;
  const int* nloop;
};
template <typename T, int N>
using NonlinearSmem = RowStage<T, N, 4, false, sizeof(T) == 4 ? 2 : 1>;   // v . grad psi in double
template <typename T, int N, int CTAS>
__global__ void __launch_bounds__(NonlinearSmem<T, N>::NT, CTAS)
    nonlinear_stage_kernel(const __grid_constant__ NonlinearStage<T> a, int groups, Tables<T> tb) {
  using S = NonlinearSmem<T, N>;
  using F = typename S::F;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const S sh(smem_raw, tb, Tables<double>{}, a.vqz);
  const RowWarp<T, N, kWide<T>> w{int(threadIdx.x & 31)};
  const int l = w.l(), stride = gridDim.x * S::kWarps;
  const bool quasi = a.variant == 0, pcoup = quasi && *a.nloop + 1 > a.divv_switch + 1;
  Cx<T> next[F::E];   // the field after the one at work, loaded while that is transformed
  auto fetch = [&](int c, int g) {
    const size_t at = (size_t(groups - 1 - g) * F::ROWS + 2 * w.pencil()) * N;
    load_rows<F, N>((c < 3 ? a.v[c] : a.p) + at, l, next, c == 2);
  };
  int grp = blockIdx.x * S::kWarps + (threadIdx.x >> 5);
  if (grp < groups) fetch(0, grp);
  for (; grp < groups; grp += stride) {
    const int rg = groups - 1 - grp;
    const size_t row = (size_t(rg) * F::ROWS + 2 * w.pencil()) * N;
    Cx<T> v[F::E];
#pragma unroll 1
    for (int c = 0; c < (quasi ? 4 : 3); ++c) {   // v, then p
      if (c < 2) {
        prefetch_rows<F, N>(a.v[c + 1], rg, w.lane);
        prefetch_rows<F, N>(a.g[c + 1], rg, w.lane);
      } else if (c == 2) {
        if (quasi) prefetch_rows<F, N>(a.p, rg, w.lane);
        prefetch_rows<F, N>(a.base, rg, w.lane);
        if (pcoup) prefetch_rows<F, N>(a.grad, rg, w.lane);
      }
      if (c == (quasi ? 3 : 2) && grp + stride < groups) {
        prefetch_rows<F, N>(a.v[0], rg - stride, w.lane);
        prefetch_rows<F, N>(a.g[0], rg - stride, w.lane);
      }
      T* f = (c < 3 ? a.v[c] : a.p) + row;
#pragma unroll
      for (int i = 0; i < F::E; ++i) v[i] = next[i];
      if (c < (quasi ? 3 : 2)) fetch(c + 1, grp);
      else if (grp + stride < groups) fetch(0, grp + stride);
      F::inverse(w, v, sh.xb, sh.t);
      F::to_pairs(w, v, c == 2);
      if (c < 3) {
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
          const int o = pair_off<F, N>(i, l);
          st2(f + o, v[i]);
          const Cx<double> g = ld2(a.g[c] + row + o), x{double(v[i].x) * g.x, double(v[i].y) * g.y};
          sh.wide(i) = c ? sh.wide(i) + x : x;
        }
      } else {
#pragma unroll
        for (int i = 0; i < F::E; ++i) st2(f + pair_off<F, N>(i, l), v[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < F::E; ++i) {
      const size_t at = row + pair_off<F, N>(i, l);
      const Cx<T> b = ld2(a.base + at), p = v[i];
      const Cx<double> adv = sh.wide(i);
      Cx<double> n{b.x - adv.x, b.y - adv.y};
      if (pcoup) {
        const Cx<T> g = ld2(a.grad + at);
        n = n + Cx<double>{double(p.x) * g.x, double(p.y) * g.y};
      }
      if (!quasi) {
        const Cx<T> m = ld2(a.mu + at);
        st2(a.dtpsi + at, Cx<T>{T(-m.x - adv.x), T(-m.y - adv.y)});
      }
      v[i] = as<T>(n);
    }
    F::from_pairs(w, v, false);
    F::forward(w, v, sh.xb, sh.t);
    store_rows<F, N>(a.out + row, l, v, false);
  }
}

// Launchers, instantiated per type in row_stage_f32.cu and row_stage_f64.cu.
cudaError_t launch_gradient_stage(const Geom& g, const GradientStage& a, Tables<double> tb, int sms, cudaStream_t s);
template <typename T>
cudaError_t launch_density_stage(const Geom& g, const DensityStage<T>& a, Tables<T> tb, Tables<double> tb64, int sms,
                                 cudaStream_t s);
template <typename T>
cudaError_t launch_stress_stage(const Geom& g, const StressStage<T>& a, Tables<T> tb, int sms, cudaStream_t s);
cudaError_t launch_stress_stb(const Geom& g, const StressStb& a, Tables<float> tb, Tables<double> tb64, int sms,
                              cudaStream_t s);
template <typename T>
cudaError_t launch_nonlinear_stage(const Geom& g, const NonlinearStage<T>& a, Tables<T> tb, int sms, cudaStream_t s);

#define QUASI_ROW_LENGTHS(n, call)           \
  switch (n) {                               \
    case 16: return call(16);                \
    case 32: return call(32);                \
    case 64: return call(64);                \
    case 96: return call(96);                \
    case 128: return call(128);              \
    case 192: return call(192);              \
    case 256: return call(256);              \
    case 512: return call(512);              \
    default: return cudaErrorInvalidValue;   \
  }
template <class S>
inline int stage_groups(const Geom& g) { return g.nx * g.ny / S::F::ROWS; }
// Launch of a stage on the shared memory layout S: the resident CTAs, at most one
// per S::NT / 32 groups of rows.
template <class S, int VARIANT = 0, class K, class A, class... Args>
cudaError_t launch_rows(K kern, const Geom& g, int sms, cudaStream_t s, const A& a, Args... args) {
  static std::atomic<int> cache[kMaxDevices];   // per instantiation: S, A and VARIANT name the kernel
  int per_sm = 1;
  static_assert(S::bytes() <= kSmemPerCta);
  const cudaError_t e = resident_ctas(kern, S::NT, S::bytes(), cache, &per_sm);
  if (e != cudaSuccess) return e;
  constexpr int W = S::NT / 32;
  const int groups = stage_groups<S>(g);
  return launch_dependent(kern, std::min(per_sm * sms, (groups + W - 1) / W), S::NT, S::bytes(), s, a, groups, args...);
}

}  // namespace quasi
