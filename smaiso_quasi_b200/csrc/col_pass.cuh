// Passes along the x and y axes on tiles of G pencils x all N rows, the pencils
// in registers (pencil_core.cuh, ColTile): rows of 2 G adjacent k (64 to 128 bytes)
// move by tensor copies in the batches and directly in the x stages, with one
// exchange through shared memory in between.  Everything that a field goes through between two y passes runs in
// one kernel:
//   col_batch_kernel   the passes of several fields along one axis in one launch
//   density_x_kernel   rho: forward x, the density filter, every inverse x pass
//                      taken from rho^
//   update_x_kernel    N: forward x, the semi-implicit update, every inverse x
//                      pass taken from the new psi^
//   project_x_kernel   the stress and divv: forward x, pressure and velocity
//                      projection, inverse x
//
// Sine spectra between passes are stored by mode number: place m holds mode m
// (place 0 is zero, the top mode N, which nothing reads, has no place).  The
// reference keeps mode m at index m - 1 (quasi.cpp:397-431), so that every term
// that couples a sine and a cosine spectrum reads a neighbour; by mode number it
// is local, and the projection needs no neighbouring tile.
#pragma once
#include <cuda_runtime.h>

#include "row_pass.cuh"
#include "tma.cuh"

namespace quasi {

__device__ __forceinline__ double rcp(double x) { return __drcp_rn(x); }
// FP32: the hardware reciprocal (within 2 ulp, below the FP32 storage rounding)
__device__ __forceinline__ float rcp(float x) { return __fdividef(1.0f, x); }

// Keeps the compiler from hoisting the E row offsets of a tile (64 bits each)
// out of the tile loop, where they spill.
__device__ __forceinline__ int opaque(int x) {
  asm volatile("" : "+r"(x));
  return x;
}

// The tiles of an x stage in a field.
struct ColGeom {
  int stride;      // elements between rows along x
  int kt;          // tiles per j
  size_t outer;    // elements between j
};
template <int G>
__device__ __forceinline__ ColGeom x_geom(const Geom& g) { return {g.ny * g.nz, g.nz / (2 * G), size_t(g.nz)}; }
inline int x_tiles(const Geom& g, int G) { return g.ny * (g.nz / (2 * G)); }

// How a spectral position is read or written along the axis.
//   cosine: place k.  sine by mode: element k is mode N - k, element 0 nothing.
template <typename T, int N>
struct ColIO {
  using F = PencilFFT<T, N>;
  __device__ __forceinline__ static int place(int k, bool sine) { return F::spec(k, sine, true); }
  // real positions
  __device__ __forceinline__ static void load_pos(const T* a, int stride0, int l, Cx<T>* v, bool sine) {
    const int stride = opaque(stride0);
    const T s = sine ? T(-1) : T(1);
#pragma unroll
    for (int t = 0; t < F::E; ++t) {
      v[t] = ld2(a + unsigned(F::pos(l + F::L * t) * stride));
      if (t >= F::H) v[t] = cscale(v[t], s);
    }
  }
  // an inverse's output (b, a), odd positions negated for sine kinds
  __device__ __forceinline__ static void store_pos(T* a, int stride0, int l, const Cx<T>* v, bool sine) {
    const int stride = opaque(stride0);
    const T s = sine ? T(-1) : T(1);
#pragma unroll
    for (int t = 0; t < F::E; ++t) {
      const Cx<T> u = t < F::H ? v[t] : cscale(v[t], s);
      st2(a + unsigned(F::pos(l + F::L * t) * stride), Cx<T>{u.y, u.x});
    }
  }
  // (a branch outside the loop: the positions of either order are then multiples
  // of the stride from one base)
  __device__ __forceinline__ static void load_spec(const T* a, int stride0, int l, Cx<T>* v, bool sine) {
    const int stride = opaque(stride0);
    if (!sine) {
#pragma unroll
      for (int t = 0; t < F::E; ++t) v[t] = ld2(a + unsigned((l + F::L * t) * stride));
    } else {
#pragma unroll
      for (int t = 0; t < F::E; ++t) {
        const int k = l + F::L * t, n = t || k ? N - k : 0;
        v[t] = ld2(a + unsigned(n * stride));
        if (t == 0 && k == 0) v[t] = Cx<T>{T(0), T(0)};
      }
    }
  }
  // sine spectra in FFTW's order: element k at N - 1 - k
  __device__ __forceinline__ static void load_index(const T* a, int stride0, int l, Cx<T>* v) {
    const int stride = opaque(stride0);
#pragma unroll
    for (int t = 0; t < F::E; ++t) v[t] = ld2(a + unsigned((N - 1 - l - F::L * t) * stride));
  }
  __device__ __forceinline__ static void store_index(T* a, int stride0, int l, const Cx<T>* v) {
    const int stride = opaque(stride0);
#pragma unroll
    for (int t = 0; t < F::E; ++t) st2(a + unsigned((N - 1 - l - F::L * t) * stride), v[t]);
  }
  __device__ __forceinline__ static void store_spec(T* a, int stride0, int l, const Cx<T>* v, bool sine) {
    const int stride = opaque(stride0);
    if (!sine) {
#pragma unroll
      for (int t = 0; t < F::E; ++t) st2(a + unsigned((l + F::L * t) * stride), v[t]);
    } else {
#pragma unroll
      for (int t = 0; t < F::E; ++t) {
        const int k = l + F::L * t, n = t || k ? N - k : 0;
        st2(a + unsigned(n * stride), t == 0 && k == 0 ? Cx<T>{T(0), T(0)} : v[t]);
      }
    }
  }
};

// ---------------------------------------------------------------------------
// Passes of several fields
// ---------------------------------------------------------------------------
enum ColOp : int {
  kColCos = 0,    // cosine kind
  kColSine = 1,   // sine kind, its spectrum by mode number
  kColBoth = 2,   // (inverse) dst = the cosine transform, dst2 = RODFT01 of the modes -q_m c_m (the derivative
                  // along the axis), one tile load
  kColIndex = 3   // sine kind, its spectrum in FFTW's order (mode m at m - 1)
};
template <typename T>
struct ColJob {
  const T* src;
  T *dst, *dst2;
  int op;
};
constexpr int kMaxJobs = 8;
template <typename T>
struct ColJobs {
  ColJob<T> job[kMaxJobs];
};
struct ColMaps {   // a job's fields as tensor maps (the tile's box)
  CUtensorMap src[kMaxJobs], dst[kMaxJobs], dst2[kMaxJobs];
  int op[kMaxJobs];
};
// Waits of the passes: the flag that a timed-out wait sets, its limit in polls, and
// (failure tests) a tile whose copy is never issued.
constexpr uint32_t kPollLimit = 1u << 24;
struct ColWait {
  int* err = nullptr;
  uint32_t polls = kPollLimit;
  int skip = -1;
};

// Pencils of a tile (G): 8, as nz is a multiple of 16; 4 as "warp tiles", which
// make tiles of the lengths with 8 lanes one warp's own (no barrier).
// threads of a CTA: at least four warps, one tile per THREADS
template <int N, int G> constexpr int col_cta() { return ColTile<N, G>::THREADS >= 128 ? ColTile<N, G>::THREADS : 128; }

// Shared memory of a pass: per tile the landing buffers and the exchange buffer
// (also the staging rows of the tile's store), then tables and barriers.
template <typename T, int N, int G>
struct ColSmem {
  using C = ColTile<N, G>;
  static constexpr int NT = col_cta<N, G>(), SETS = NT / C::THREADS;
  // tiles in flight beyond the one worked on: a register's worth of time is enough
  // for float (22.7 us a pass at 256^3 with one or two buffers), double takes two
  // (51 -> 48 us)
  static constexpr int BUFS = sizeof(T) == 8 ? 2 : 1;
  static constexpr int TILE = 2 * G * N;   // elements
  static constexpr size_t xch_bytes() { return (size_t(C::XCH) * sizeof(Cx<T>) + 127) / 128 * 128; }
  static constexpr size_t set_bytes() { return size_t(BUFS) * TILE * sizeof(T) + xch_bytes(); }
  static constexpr size_t bytes() {
    return SETS * set_bytes() + PencilFFT<T, N>::table_bytes() + N * sizeof(T) + SETS * BUFS * sizeof(uint64_t);
  }
  static_assert(TILE * sizeof(T) <= size_t(C::XCH) * sizeof(Cx<T>), "the staging rows overlay the exchange buffer");
  static_assert(TILE * sizeof(T) % 128 == 0, "tensor copies land on 128-byte boundaries");
};

// Tiles arrive by TMA, land as rows [n][2G] and are read into registers once; the
// next tile's copy is issued as soon as every thread has read.  The output rows are
// staged over the exchange buffer and leave by a TMA store.  Bound: HBM; with the
// threads loading and storing global rows themselves the address arithmetic took a
// third of the instructions (float 28.6 us a pass at 256^3, 22.7 now; double 50 -> 48).
template <typename T, int N, int G, bool FWD>
__global__ void __launch_bounds__(col_cta<N, G>(), (sizeof(T) == 8 ? 384 : 512) / col_cta<N, G>())
    col_batch_kernel(const __grid_constant__ ColMaps maps, int axis, int kt, int tiles, int njobs, Tables<T> tb,
                     const double* vq, T scale, ColWait wait) {
  using S = ColSmem<T, N, G>;
  using C = typename S::C;
  using F = PencilFFT<T, N>;
  constexpr int SETS = S::SETS, BUFS = S::BUFS, P = 2 * G, SUB = (N + 255) / 256, BN = N / SUB;   // box sides <= 256
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int set = threadIdx.x / C::THREADS, r = threadIdx.x % C::THREADS;
  T* raw = reinterpret_cast<T*>(smem_raw + set * S::set_bytes());
  Cx<T>* xb = reinterpret_cast<Cx<T>*>(raw + BUFS * S::TILE);
  T* stage = reinterpret_cast<T*>(xb);
  unsigned char* sm = smem_raw + SETS * S::set_bytes();
  const typename F::Tab t = F::fill_tables(reinterpret_cast<Cx<T>*>(sm), tb, threadIdx.x, S::NT);
  sm += F::table_bytes();
  T* q = reinterpret_cast<T*>(sm);
  for (int e = threadIdx.x; e < N; e += S::NT) q[e] = vq ? T(-vq[e]) : T(0);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + N * sizeof(T)) + set * BUFS;
  if (r == 0) {
#pragma unroll
    for (int b = 0; b < BUFS; ++b) mbar_init(&bar[b], 1);
    mbar_fence_init();
    const int j = min(int(blockIdx.x * SETS + set) / tiles, njobs - 1);
    prefetch_map(&maps.src[j]);
    prefetch_map(&maps.dst[j]);
  }
  __syncthreads();
  pdl_begin();
  const C w(r, 1 + set);
  const int l = w.l(), all = tiles * njobs, stride = gridDim.x * SETS;
  auto issue = [&](int x, int b) {
    if (x == wait.skip) return;
    const int j = x / tiles, tile = x - j * tiles, o = tile / kt, k0 = (tile - o * kt) * P;
    mbar_expect_tx(&bar[b], S::TILE * sizeof(T));
#pragma unroll
    for (int sb = 0; sb < SUB; ++sb)
      tma_load_3d(raw + b * S::TILE + sb * BN * P, &maps.src[j], &bar[b], k0, axis == 1 ? sb * BN : o,
                  axis == 1 ? o : sb * BN);
  };
  int x = blockIdx.x * SETS + set;
  if (r == 0) {
#pragma unroll
    for (int b = 0; b < BUFS; ++b)
      if (x + b * stride < all) issue(x + b * stride, b);
  }
  for (int it = 0; x < all; x += stride, ++it) {
    const int b = it % BUFS, j = x / tiles, tile = x - j * tiles, op = maps.op[j];
    const T* tl = raw + b * S::TILE + 2 * w.g;
    bool ok = mbar_wait_bounded(&bar[b], (it / BUFS) & 1, wait.polls);
    // kColBoth: the derivative first
#pragma unroll 1
    for (int pass = !FWD && op == kColBoth ? 0 : 1; pass < 2; ++pass) {
      const bool grad = !FWD && pass == 0, sine = grad || op == kColSine || op == kColIndex;
      const int order = sine && op != kColIndex ? N - l : N - 1 - l;   // place of a sine spectrum's element l
      Cx<T> v[F::E];
      if constexpr (FWD) {
        const T s = sine ? T(-1) : T(1);
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
          v[i] = ld2(tl + F::pos(l + F::L * i) * P);
          if (i >= F::H) v[i] = cscale(v[i], s);
        }
      } else if (!sine) {
#pragma unroll
        for (int i = 0; i < F::E; ++i) v[i] = ld2(tl + (l + F::L * i) * P);
      } else {
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
          const int n = i == 0 && order == N ? 0 : order - F::L * i;
          v[i] = ld2(tl + n * P);
          if (grad) v[i] = cscale(v[i], q[n]);
          if (i == 0 && order == N) v[i] = Cx<T>{T(0), T(0)};   // the top mode has no place
        }
      }
      if (r == 0) bulk_wait_read0();   // the previous store has read the staging rows
      ok = w.sync_all(ok);
      if (!ok) break;
      if (pass == 1 && r == 0 && x + BUFS * stride < all) {   // this landing buffer has been read
        fence_proxy_async_smem();
        issue(x + BUFS * stride, b);
      }
      if constexpr (FWD) {
        F::forward(w, v, xb, t);
        if (scale != T(1)) {
#pragma unroll
          for (int i = 0; i < F::E; ++i) v[i] = cscale(v[i], scale);
        }
        if (!sine) {
#pragma unroll
          for (int i = 0; i < F::E; ++i) st2(stage + 2 * w.g + (l + F::L * i) * P, v[i]);
        } else {
#pragma unroll
          for (int i = 0; i < F::E; ++i) {
            const bool none = i == 0 && order == N;
            st2(stage + 2 * w.g + (none ? 0 : order - F::L * i) * P, none ? Cx<T>{T(0), T(0)} : v[i]);
          }
        }
      } else {
        F::inverse(w, v, xb, t);
        const T s = sine ? T(-1) : T(1);
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
          const Cx<T> u = i < F::H ? v[i] : cscale(v[i], s);
          st2(stage + 2 * w.g + F::pos(l + F::L * i) * P, Cx<T>{u.y, u.x});
        }
      }
      fence_proxy_async_smem();
      w.sync();
      if (r == 0) {
        const int o = tile / kt, k0 = (tile - o * kt) * P;
#pragma unroll
        for (int sb = 0; sb < SUB; ++sb)
          tma_store_3d(pass == 0 ? &maps.dst2[j] : &maps.dst[j], stage + sb * BN * P, k0, axis == 1 ? sb * BN : o,
                       axis == 1 ? o : sb * BN);
        bulk_commit();
      }
    }
    if (!ok) {   // a copy never arrived: flag it, wait for the others in flight, leave
      if (r == 0) {
        atomicExch(wait.err, 1);
        for (int d = 1; d < BUFS; ++d) {
          const int xo = x + d * stride;
          if (xo < all && xo != wait.skip) mbar_wait_bounded(&bar[(it + d) % BUFS], ((it + d) / BUFS) & 1, wait.polls);
        }
      }
      break;
    }
  }
  if (r == 0) bulk_wait0();
}

template <typename T, int N, int G, bool FWD>
cudaError_t launch_col_batch_g(const Geom& g, int axis, const ColJobs<T>& jobs, int njobs, Tables<T> tb,
                               const double* vq, T scale, const ColWait& wait, int sms, cudaStream_t s) {
  using S = ColSmem<T, N, G>;
  auto kern = col_batch_kernel<T, N, G, FWD>;
  static std::atomic<int> cache[kMaxDevices];
  int per_sm = 1;
  static_assert(S::bytes() <= kSmemPerCta);
  const cudaError_t e = resident_ctas(kern, S::NT, S::bytes(), cache, &per_sm);
  if (e != cudaSuccess) return e;
  constexpr uint32_t BN = N > 256 ? N / ((N + 255) / 256) : N;
  const uint32_t box[3] = {uint32_t(2 * G), axis == 1 ? BN : 1, axis == 1 ? 1 : BN};
  ColMaps maps{};
  for (int j = 0; j < njobs; ++j) {
    const ColJob<T>& jb = jobs.job[j];
    maps.op[j] = jb.op;
    if (!make_field_map(&maps.src[j], jb.src, int(sizeof(T)), g.nx, g.ny, g.nz, box)) return cudaErrorInvalidValue;
    if (jb.dst == jb.src) maps.dst[j] = maps.src[j];
    else if (!make_field_map(&maps.dst[j], jb.dst, int(sizeof(T)), g.nx, g.ny, g.nz, box)) return cudaErrorInvalidValue;
    if (jb.dst2 && !make_field_map(&maps.dst2[j], jb.dst2, int(sizeof(T)), g.nx, g.ny, g.nz, box))
      return cudaErrorInvalidValue;
  }
  const int kt = g.nz / (2 * G), tiles = (axis == 1 ? g.nx : g.ny) * kt, work = (tiles * njobs + S::SETS - 1) / S::SETS;
  return launch_dependent(kern, std::min(per_sm * sms, work), S::NT, S::bytes(), s, maps, axis, kt, tiles, njobs, tb,
                          vq, scale, wait);
}
template <typename T, int N>
cudaError_t launch_col_batch_n(const Geom& g, int axis, bool forward, const ColJobs<T>& jobs, int njobs, Tables<T> tb,
                               const double* vq, T scale, const ColWait& wait, bool narrow, int sms, cudaStream_t s) {
  if constexpr (row_plan(N).lanes == 8) {
    if (narrow)
      return forward ? launch_col_batch_g<T, N, 4, true>(g, axis, jobs, njobs, tb, vq, scale, wait, sms, s)
                     : launch_col_batch_g<T, N, 4, false>(g, axis, jobs, njobs, tb, vq, scale, wait, sms, s);
  }
  return forward ? launch_col_batch_g<T, N, 8, true>(g, axis, jobs, njobs, tb, vq, scale, wait, sms, s)
                 : launch_col_batch_g<T, N, 8, false>(g, axis, jobs, njobs, tb, vq, scale, wait, sms, s);
}

// ---------------------------------------------------------------------------
// x stages.  Per-axis double tables: wavenumbers and density filter factors.
// ---------------------------------------------------------------------------
struct XTables {
  const double *vqx, *vqy, *vqz, *fx, *fy, *fz;
};

// rho (double, z and y transformed) -> rho^ = scale CT(rho) exp(-1.57^2 q^2 8)
// (quasi.cpp:1260-1261) -> the x-inverse of rho^ and of its gradient's spectra.
//   DBL: out0 = x(rho^), out1 = x'(rho^) in double (grad_y, grad_z follow from out0)
//   else out0 = x(rho^) in double and the three gradient spectra's x passes in
//   float, each with its own multiplier (in double, rounded once before the
//   transform, so that float rounding is not multiplied by the wavenumber)
// from_spec: take rho^ from memory and leave `in` alone (a loaded state).
template <typename T>
struct DensityX {
  const double* in;
  double *rhoq, *out0, *out1;
  T *gx, *gy, *gz;   // float form
  XTables x;
  double scale;
  int from_spec;
};

// psi^: N -> N^, the semi-implicit update (quasi.cpp:1944-1962,
// quasi-stb.cpp:1946-1958), then from psi^ the x-inverse passes of the next
// step: psi and d_x psi in double (grad_y, grad_z share the first), and each with
// its multiplier, in T, df, lap and the three of grad lap psi (quasi) or, in
// double, sh = -aLin psi^ (stb).
template <typename T>
struct UpdateX {
  const T* in;
  T *Nq;
  const T* Nq_old;
  const double *psiq, *psiq_old;
  double* psiq_new;
  double *out0, *out1;
  T* out[5];      // quasi
  double* sh;     // quasi-stb
  XTables x;
  double ep, alpha, q0, rho_m, dt, scale;
  const int* nloop;   // steps completed
  int variant, from_spec;
};

// Tiles of an x stage: 8 pencils (4 at N = 512), doubles exchanged in halves: a
// tile then takes 49 KB at N = 256 and four of 4 warps fill an SM (whole exchanges
// leave room for three: density_x 200 us at 256^3 in the FP32 form against 174;
// three tiles of 8 warps on 32 lanes per pencil: 217 us, bound by shared memory).
template <int N> constexpr int x_pencils() { return N >= 512 ? 4 : 8; }
template <int N, int G> using XTile = ColTile<N, G, false, true>;
// At N = 512 the FP32 form's second set of tables leaves room for three.
template <typename T, int N> constexpr int x_sets() { return N >= 512 && sizeof(T) == 4 ? 3 : 4; }
// CTAs per SM that the registers must allow
template <int N>
constexpr int x_ctas() {
  return N >= 192 ? 1 : N >= 96 ? 2 : N >= 64 ? 2 : 4;
}
template <typename T, int N, int G> constexpr int x_cta() { return x_sets<T, N>() * XTile<N, G>::THREADS; }
// exchange buffer (double complex, or split: double; and float complex), then the spectrum
template <int N, int G>
constexpr size_t x_xch_bytes() { return (size_t(XTile<N, G>::XCH) * (XTile<N, G>::template split<double>() ? 8 : 16) + 15) / 16 * 16; }
template <int N, int G>
constexpr size_t x_tile_bytes() { return x_xch_bytes<N, G>() + size_t(N) * G * sizeof(Cx<double>); }
template <typename T, int N, int G>
constexpr size_t x_stage_smem() {   // tables of both types, wavenumbers and filter, exchange and spectrum in double
  return PencilFFT<double, N>::table_bytes() + (sizeof(T) == 4 ? PencilFFT<float, N>::table_bytes() : 0) +
         2 * N * sizeof(double) + size_t(x_sets<T, N>()) * x_tile_bytes<N, G>();
}

// Shared memory of an x stage, as one tile's threads see it.
template <typename T, int N, int G>
struct XStage {
  using C = XTile<N, G>;
  using F = PencilFFT<T, N>;
  using FD = PencilFFT<double, N>;
  static constexpr int NT = x_cta<T, N, G>();
  typename FD::Tab td;
  typename F::Tab tt;
  double *q, *f;      // wavenumbers and filter factors along x
  Cx<double>* xd;     // exchange
  Cx<T>* xt;          // the same bytes for T
  Cx<double>* spec;   // the tile's spectrum [k][g]
  __device__ __forceinline__ XStage(unsigned char* sm, int set, Tables<double> tb64, Tables<T> tb, const double* vq,
                                    const double* fl) {
    td = FD::fill_tables(reinterpret_cast<Cx<double>*>(sm), tb64, threadIdx.x, NT);
    sm += FD::table_bytes();
    if constexpr (sizeof(T) == 4) {
      tt = F::fill_tables(reinterpret_cast<Cx<T>*>(sm), tb, threadIdx.x, NT);
      sm += F::table_bytes();
    } else {
      tt = td;
    }
    q = reinterpret_cast<double*>(sm);
    f = q + N;
    for (int e = threadIdx.x; e < N; e += NT) {
      q[e] = vq[e];
      f[e] = fl[e];
    }
    sm = reinterpret_cast<unsigned char*>(f + N) + set * x_tile_bytes<N, G>();
    xd = reinterpret_cast<Cx<double>*>(sm);
    xt = reinterpret_cast<Cx<T>*>(sm);
    spec = reinterpret_cast<Cx<double>*>(sm + x_xch_bytes<N, G>());
    __syncthreads();
    pdl_begin();
  }
};

template <typename T, int N, int G>
__global__ void __launch_bounds__(x_cta<T, N, G>(), x_ctas<N>())
    density_x_kernel(const __grid_constant__ DensityX<T> a, Geom geom, int tiles, Tables<double> tb64, Tables<T> tb) {
  using X = XStage<T, N, G>;
  using C = typename X::C;
  using F = typename X::F;
  using FD = typename X::FD;
  using IO = ColIO<T, N>;
  using IOD = ColIO<double, N>;
  constexpr bool kDbl = sizeof(T) == 8;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int set = threadIdx.x / C::THREADS;
  const X sh(smem_raw, set, tb64, tb, a.x.vqx, a.x.fx);
  const C w(threadIdx.x % C::THREADS, 1 + set);
  const int l = w.l();
  const ColGeom cg = x_geom<G>(geom);
  for (int tile = blockIdx.x * x_sets<T, N>() + set; tile < tiles; tile += gridDim.x * x_sets<T, N>()) {
    const int j = tile / cg.kt, k0 = (tile - j * cg.kt) * 2 * G + 2 * w.g;
    const size_t base = j * cg.outer + k0;
    const double qy = a.x.vqy[j], qz0 = a.x.vqz[k0], qz1 = a.x.vqz[k0 + 1];
    Cx<double> v[FD::E];
    if (!a.from_spec) {
      IOD::load_pos(a.in + base, cg.stride, l, v, false);
      FD::forward(w, v, sh.xd, sh.td);
      const double fy = a.x.fy[j], fz0 = a.x.fz[k0], fz1 = a.x.fz[k0 + 1];
#pragma unroll
      for (int t = 0; t < FD::E; ++t) {
        const double fx = sh.f[l + FD::L * t];
        v[t] = Cx<double>{a.scale * v[t].x * (fx * fy * fz0), a.scale * v[t].y * (fx * fy * fz1)};
      }
      IOD::store_spec(a.rhoq + base, cg.stride, l, v, false);
    } else {
      IOD::load_spec(a.rhoq + base, cg.stride, l, v, false);
    }
#pragma unroll
    for (int t = 0; t < FD::E; ++t) sh.spec[(l + FD::L * t) * G + w.g] = v[t];
    w.sync();
#pragma unroll 1
    for (int o = 0; o < (kDbl ? 2 : 1); ++o) {
#pragma unroll
      for (int t = 0; t < FD::E; ++t) {
        const int k = l + FD::L * t, n = IOD::place(k, o == 1);
        v[t] = sh.spec[n * G + w.g];
        if (o == 1) v[t] = cscale(v[t], -sh.q[n]);   // (mode 0: q = 0)
      }
      FD::inverse(w, v, sh.xd, sh.td);
      IOD::store_pos((o ? a.out1 : a.out0) + base, cg.stride, l, v, o == 1);
    }
    if constexpr (!kDbl) {
#pragma unroll 1
      for (int o = 0; o < 3; ++o) {
        Cx<T> u[F::E];
#pragma unroll
        for (int t = 0; t < F::E; ++t) {
          const int n = IO::place(l + F::L * t, o == 0);
          const Cx<double> y = sh.spec[n * G + w.g];
          const double m0 = o == 0 ? -sh.q[n] : o == 1 ? -qy : -qz0, m1 = o == 2 ? -qz1 : m0;
          u[t] = Cx<T>{T(y.x * m0), T(y.y * m1)};
        }
        F::inverse(w, u, sh.xt, sh.tt);
        IO::store_pos((o == 0 ? a.gx : o == 1 ? a.gy : a.gz) + base, cg.stride, l, u, o == 0);
      }
    }
    w.sync();   // the next tile rewrites the spectrum
  }
}

template <typename T, int N, int G>
__global__ void __launch_bounds__(x_cta<T, N, G>(), x_ctas<N>())
    update_x_kernel(const __grid_constant__ UpdateX<T> a, Geom geom, int tiles, Tables<double> tb64, Tables<T> tb) {
  using X = XStage<T, N, G>;
  using C = typename X::C;
  using F = typename X::F;
  using FD = typename X::FD;
  using IO = ColIO<T, N>;
  using IOD = ColIO<double, N>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int set = threadIdx.x / C::THREADS;
  const X sh(smem_raw, set, tb64, tb, a.x.vqx, a.x.vqx);
  const C w(threadIdx.x % C::THREADS, 1 + set);
  const int l = w.l();
  const bool quasi = a.variant == 0, first = *a.nloop == 0;
  const ColGeom cg = x_geom<G>(geom);
  const double dtd2 = a.dt / 2, dsc = dtd2 * a.scale, q02 = a.q0 * a.q0;
  for (int tile = blockIdx.x * x_sets<T, N>() + set; tile < tiles; tile += gridDim.x * x_sets<T, N>()) {
    const int j = tile / cg.kt, k0 = (tile - j * cg.kt) * 2 * G + 2 * w.g;
    const size_t base = j * cg.outer + k0;
    const double qy = a.x.vqy[j], qz0 = a.x.vqz[k0], qz1 = a.x.vqz[k0 + 1];
    const double s0 = qy * qy + qz0 * qz0, s1 = qy * qy + qz1 * qz1;
    if (!a.from_spec) {
      // in double in both forms: N^ is differenced with what it nearly balances
      Cx<T> in[F::E];
      IO::load_pos(a.in + base, cg.stride, l, in, false);
      Cx<double> u[FD::E];
#pragma unroll
      for (int t = 0; t < FD::E; ++t) u[t] = as<double>(in[t]);
      FD::forward(w, u, sh.xd, sh.td);
#pragma unroll
      for (int t = 0; t < F::E; ++t) in[t] = as<T>(u[t]);
      IO::store_spec(a.Nq + base, cg.stride, l, in, false);
      const int stride = opaque(cg.stride);
#pragma unroll
      for (int t = 0; t < F::E; ++t) {
        const int k = l + F::L * t;
        const size_t at = base + unsigned(k * stride);
        const Cx<double> pq = ld2(a.psiq + at);
        const Cx<double> po = quasi ? ld2(a.psiq_old + at) : Cx<double>{0.0, 0.0};
        const Cx<double> no = first ? u[t] : as<double>(ld2(a.Nq_old + at));   // quasi.cpp:1936-1938
        auto advance = [&](double s, double n, double n_old, double p, double p_old) {
          const double d = q02 - (sh.q[k] * sh.q[k] + s);
          const double alin = a.ep - a.alpha * (d * d);
          const double forcing = dsc * (3.0 * n - n_old);
          if (quasi) {
            const double c1 = 2.0 - a.dt * a.rho_m * alin, c2 = 1.5 - a.dt * a.rho_m * alin;   // quasi.cpp:886-887
            return (c1 * p - 0.5 * p_old + forcing) / c2;
          }
          const double c1 = 1.0 + dtd2 * alin, c2 = 1.0 - dtd2 * alin;   // quasi-stb.cpp:855-856
          return (c1 * p + forcing) / c2;
        };
        const Cx<double> v{advance(s0, u[t].x, no.x, pq.x, po.x), advance(s1, u[t].y, no.y, pq.y, po.y)};
        st2(a.psiq_new + at, v);
        sh.spec[k * G + w.g] = v;
      }
    } else {
      const int stride = opaque(cg.stride);
#pragma unroll
      for (int t = 0; t < FD::E; ++t) {
        const int k = l + FD::L * t;
        sh.spec[k * G + w.g] = ld2(a.psiq_new + base + unsigned(k * stride));
      }
    }
    w.sync();
    // psi, d_x psi; quasi-stb: sh.  aLin grows like q^4 and psi^ concentrates on
    // |q| = q0, so a transform of -aLin psi^ rounds relative to high modes that it
    // has amplified, and the growth rate divides that by dt: in float sh alone was
    // nearly all of the rates' error (2e-6 over a stability ensemble).
#pragma unroll 1
    for (int o = 0; o < (quasi ? 2 : 3); ++o) {
      Cx<double> v[FD::E];
#pragma unroll
      for (int t = 0; t < FD::E; ++t) {
        const int n = IOD::place(l + FD::L * t, o == 1);
        v[t] = sh.spec[n * G + w.g];
        if (o == 1) v[t] = cscale(v[t], -sh.q[n]);
        if (o == 2) {   // quasi-stb.cpp:1019
          auto mul = [&](double s) {
            const double d = q02 - (sh.q[n] * sh.q[n] + s);
            return a.alpha * (d * d) - a.ep;
          };
          v[t] = Cx<double>{v[t].x * mul(s0), v[t].y * mul(s1)};
        }
      }
      FD::inverse(w, v, sh.xd, sh.td);
      IOD::store_pos((o == 0 ? a.out0 : o == 1 ? a.out1 : a.sh) + base, cg.stride, l, v, o == 1);
    }
    // quasi's T fields: the multiplier of quasi.cpp:1044-1047, 1120-1186 in double,
    // rounded once; grad lap psi is |q|^2 q_A psi^ in each mode, the derivative -q_A
    // of lap psi = -|q|^2 psi.  All of them are
    //   (a0 + a1 q2) (b2 q2 + bx x + bc),  q2 = |q|^2, x = q_x,
    // so one copy of the code serves every output (a branch per output made the
    // kernel outgrow the instruction cache).
#pragma unroll 1
    for (int o = 0; o < (quasi ? 5 : 0); ++o) {
      const bool ring = o < 2, x_axis = o == 2;
      const double a0 = ring ? a.alpha * q02 : 0.0, a1 = ring ? -a.alpha : 1.0;
      const double b2 = o == 1 ? -1.0 : 0.0, bx = x_axis ? 1.0 : 0.0;
      const double bc0 = o == 0 ? 1.0 : o == 3 ? qy : o == 4 ? qz0 : 0.0, bc1 = o == 4 ? qz1 : bc0;
      Cx<T> u[F::E];
      const int n0 = x_axis ? N - l : l, dn = x_axis ? -F::L : F::L;
#pragma unroll
      for (int t = 0; t < F::E; ++t) {
        const int n = t == 0 && l == 0 ? 0 : n0 + dn * t;   // (mode 0: x = 0)
        const Cx<double> y = sh.spec[n * G + w.g];
        const double x = sh.q[n], xx = x * x, bxx = bx * x;
        auto mul = [&](double s, double bc) {
          const double q2 = xx + s;
          return (a0 + a1 * q2) * (b2 * q2 + (bxx + bc));
        };
        u[t] = Cx<T>{T(y.x * mul(s0, bc0)), T(y.y * mul(s1, bc1))};
      }
      F::inverse(w, u, sh.xt, sh.tt);
      IO::store_pos(a.out[o] + base, cg.stride, l, u, x_axis);
    }
    w.sync();   // the next tile rewrites the spectrum
  }
}

// Pressure, staggered Stokes projection (quasi.cpp:1336-1884) between the x
// passes of the stress (and divv) and those of p and v.  Four groups of threads,
// one per field: each transforms its input and leaves its spectrum in its exchange
// buffer; after a CTA barrier all threads share the modes (a, b, c), replacing the
// four inputs by the four outputs
//   p = scale (-(q . S) / q^2 [+ nu D in stb]),  v = scale / (nu q^2) (S - q (q . S) / q^2 + nu q D)
// and after another each group transforms one of those back.
template <typename T>
struct ProjectX {
  const T* in[4];   // Sx (x sine), Sy, Sz by mode; divv
  T* out[4];        // p, vx, vy, vz by mode
  XTables x;
  double nu, scale;
  int variant, n0;   // n0: planes per emulated MPI rank (quasi.cpp:1641-1690)
};
// Tiles: 8 pencils in float (at N = 256 two CTAs of 512 threads per SM, 202 us at
// 256^3; one of 1024 on 32 lanes per pencil: 268 us), 4 in double for N >= 64 and
// at N = 512.
template <typename T, int N> constexpr int project_pencils() {
  return N >= 512 || (sizeof(T) == 8 && N >= 64) ? 4 : 8;
}
template <typename T, int N, int G>
constexpr size_t project_smem() {
  return PencilFFT<T, N>::table_bytes() +
         size_t(4) * ColTile<N, G>::XCH * sizeof(Cx<T>) + N * sizeof(T);
}
template <typename T, int N, int G> constexpr int project_cta() { return 4 * ColTile<N, G>::THREADS; }
// CTAs per SM that the registers must allow: 1024 threads in float with 8
// elements per lane, else 512
template <typename T, int N, int G>
constexpr int project_ctas() {
  constexpr int want = sizeof(T) == 4 ? 1024 : 512, nt = project_cta<T, N, G>();
  return want > nt ? want / nt : 1;
}
template <typename T, int N, int G>
__global__ void __launch_bounds__(project_cta<T, N, G>(), project_ctas<T, N, G>())
    project_x_kernel(const __grid_constant__ ProjectX<T> a, Geom geom, int tiles, Tables<T> tb) {
  using C = ColTile<N, G>;
  using F = PencilFFT<T, N>;
  using IO = ColIO<T, N>;
  constexpr int NT = project_cta<T, N, G>();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int field = threadIdx.x / C::THREADS;
  Cx<T>* buf = reinterpret_cast<Cx<T>*>(smem_raw + F::table_bytes());
  Cx<T>* xb = buf + field * C::XCH;
  T* q = reinterpret_cast<T*>(buf + 4 * C::XCH);
  const typename F::Tab t = F::fill_tables(reinterpret_cast<Cx<T>*>(smem_raw), tb, threadIdx.x, NT);
  for (int e = threadIdx.x; e < N; e += NT) q[e] = T(a.x.vqx[e]);
  __syncthreads();
  pdl_begin();
  const C w(threadIdx.x % C::THREADS, 1 + field);
  const int l = w.l();
  // padded place of mode N - (l + L i)
  auto phi_mirror = [](int l1, int i) {
    if constexpr (F::L % F::R1 == 0) return F::phi_read(F::L - l1, F::E - 1 - i);
    else return int(F::phi(N - l1 - F::L * i));
  };
  const bool stb = a.variant != 0;
  const T scale = T(a.scale), nu = T(a.nu), inu = T(1.0 / a.nu);
  const ColGeom cg = x_geom<G>(geom);
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int b = tile / cg.kt, c00 = (tile - b * cg.kt) * 2 * G;
    const size_t base = b * cg.outer + c00 + 2 * w.g;
    const T qy = T(a.x.vqy[b]);
    Cx<T> v[F::E];
    if (field < 3 || !stb) {
      IO::load_pos(a.in[field] + base, cg.stride, l, v, field == 0);
      F::forward(w, v, xb, t);
      if (field) {
#pragma unroll
        for (int i = 0; i < F::E; ++i) xb[w.at(F::phi_read(l, i))] = v[i];
      } else {   // by mode: element k is mode N - k, element 0 nothing
#pragma unroll
        for (int i = 0; i < F::E; ++i) {
          const bool none = i == 0 && l == 0;
          xb[w.at(none ? 0 : phi_mirror(l, i))] = none ? Cx<T>{T(0), T(0)} : v[i];
        }
      }
    } else {   // quasi-stb never transforms divv: its spectrum stays 0
#pragma unroll
      for (int i = 0; i < F::E; ++i) xb[w.at(F::phi_read(l, i))] = Cx<T>{T(0), T(0)};
    }
    __syncthreads();
    // every mode once: all four spectra in, p and v out, in place.  halo: plane
    // "i - 1" of S_x as halo #4 delivers it to vy and vz (quasi.cpp:1649)
    constexpr int ITER = (N * G + NT - 1) / NT, MS = NT / G;   // modes between a thread's
    const int m0 = threadIdx.x / G, pg = threadIdx.x % G, c0 = c00 + 2 * pg;
    const T qz0 = T(a.x.vqz[c0]), qz1 = T(a.x.vqz[c0 + 1]);
    auto place = [&](int i) {   // of mode m0 + i MS
      if constexpr (MS % C::R1 == 0) return (m0 + m0 / C::R1) * G + pg + i * (MS + MS / C::R1) * G;
      else return int(unsigned(m0 + i * MS) + unsigned(m0 + i * MS) / unsigned(C::R1)) * G + pg;
    };
    Cx<T> halo[ITER];
    if (a.n0 < N) {
#pragma unroll
      for (int i = 0; i < ITER; ++i) {
        const int m = m0 + i * MS, m1 = m > 0 && m % a.n0 == 0 ? m - a.n0 + 1 : m;
        if (N * G % NT == 0 || m < N) halo[i] = buf[F::phi(m1) * G + pg];
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < ITER; ++i) {
      const int m = m0 + i * MS, at = place(i);
      if (N * G % NT && m >= N) break;
      const Cx<T> sx = buf[at], sy = buf[C::XCH + at], sz = buf[2 * C::XCH + at], dv = buf[3 * C::XCH + at];
      const Cx<T> sh = a.n0 < N ? halo[i] : sx;
      const T qx = q[m];
      Cx<T> p, vx, vy, vz;
      auto one = [&](T x, T xh, T y, T z, T d, T qz, int c, T& po, T& vxo, T& vyo, T& vzo) {
        const T q2 = qx * qx + qy * qy + qz * qz;
        const T inv = m + b + c ? rcp(q2) : T(0);
        const T yz = qy * y + qz * z, dot = (qx * x + yz) * inv, doth = (qx * xh + yz) * inv, nd = nu * d;
        const T cv = scale * inv * inu;
        po = stb ? (m * b * c ? scale * (nd - dot) : T(0)) : -scale * dot;
        // no mode 0 of a sine axis; vy, vz: zero on the last y and z planes of
        // the reference's index (quasi.cpp:1683-1872)
        vxo = m > 0 ? cv * (x - qx * dot + qx * nd) : T(0);
        vyo = b > 0 && c < geom.nz - 1 ? cv * (y - qy * doth + qy * nd) : T(0);
        vzo = c > 0 && b < geom.ny - 1 ? cv * (z - qz * doth + qz * nd) : T(0);
      };
      one(sx.x, sh.x, sy.x, sz.x, dv.x, qz0, c0, p.x, vx.x, vy.x, vz.x);
      one(sx.y, sh.y, sy.y, sz.y, dv.y, qz1, c0 + 1, p.y, vx.y, vy.y, vz.y);
      buf[at] = p;
      buf[C::XCH + at] = vx;
      buf[2 * C::XCH + at] = vy;
      buf[3 * C::XCH + at] = vz;
    }
    __syncthreads();
    const bool sine = field == 1;   // vx
    if (!sine) {
#pragma unroll
      for (int i = 0; i < F::E; ++i) v[i] = xb[w.at(F::phi_read(l, i))];
    } else {   // (mode 0 of vx is zero)
#pragma unroll
      for (int i = 0; i < F::E; ++i) v[i] = xb[w.at(i == 0 && l == 0 ? 0 : phi_mirror(l, i))];
    }
    w.sync();   // read before the exchanges of the inverse overwrite it
    if (stb && field == 0) {   // quasi-stb's pressure is not transformed back
      IO::store_spec(a.out[0] + base, cg.stride, l, v, false);
    } else {
      F::inverse(w, v, xb, t);
      IO::store_pos(a.out[field] + base, cg.stride, l, v, sine);
    }
    w.sync();   // the next tile rewrites this group's buffer
  }
}

// ---------------------------------------------------------------------------
// Launchers, instantiated per type in col_pass_f32.cu and col_pass_f64.cu.
// ---------------------------------------------------------------------------
// Passes of njobs fields along axis 0 or 1, all forward (REDFT10 / RODFT10, the
// result times scale) or all inverse.  vq: the axis's wavenumbers (kColBoth).
// narrow: tiles of 4 pencils where that makes them one warp's.
template <typename T>
cudaError_t launch_col_batch(const Geom& g, int axis, bool forward, const ColJobs<T>& jobs, int njobs, Tables<T> tb,
                             const double* vq, T scale, const ColWait& wait, bool narrow, int sms, cudaStream_t s);
template <typename T>
cudaError_t launch_density_x(const Geom& g, const DensityX<T>& a, Tables<double> tb64, Tables<T> tb, int sms,
                             cudaStream_t s);
template <typename T>
cudaError_t launch_update_x(const Geom& g, const UpdateX<T>& a, Tables<double> tb64, Tables<T> tb, int sms,
                            cudaStream_t s);
template <typename T>
cudaError_t launch_project_x(const Geom& g, const ProjectX<T>& a, Tables<T> tb, int sms, cudaStream_t s);

template <typename T, int N>
cudaError_t launch_density_x_n(const Geom& g, const DensityX<T>& a, Tables<double> tb64, Tables<T> tb, int sms,
                               cudaStream_t s) {
  constexpr int G = x_pencils<N>(), NT = x_cta<T, N, G>(), SETS = x_sets<T, N>();
  constexpr size_t smem = x_stage_smem<T, N, G>();
  static_assert(smem <= kSmemPerCta);
  auto kern = density_x_kernel<T, N, G>;
  static std::atomic<int> cache[kMaxDevices];
  int per_sm = 1;
  const cudaError_t e = resident_ctas(kern, NT, smem, cache, &per_sm);
  if (e != cudaSuccess) return e;
  const int tiles = x_tiles(g, G);
  return launch_dependent(kern, std::min(per_sm * sms, (tiles + SETS - 1) / SETS), NT, smem, s, a, g, tiles, tb64, tb);
}
template <typename T, int N>
cudaError_t launch_update_x_n(const Geom& g, const UpdateX<T>& a, Tables<double> tb64, Tables<T> tb, int sms,
                              cudaStream_t s) {
  constexpr int G = x_pencils<N>(), NT = x_cta<T, N, G>(), SETS = x_sets<T, N>();
  constexpr size_t smem = x_stage_smem<T, N, G>();
  static_assert(smem <= kSmemPerCta);
  auto kern = update_x_kernel<T, N, G>;
  static std::atomic<int> cache[kMaxDevices];
  int per_sm = 1;
  const cudaError_t e = resident_ctas(kern, NT, smem, cache, &per_sm);
  if (e != cudaSuccess) return e;
  const int tiles = x_tiles(g, G);
  return launch_dependent(kern, std::min(per_sm * sms, (tiles + SETS - 1) / SETS), NT, smem, s, a, g, tiles, tb64, tb);
}
template <typename T, int N>
cudaError_t launch_project_x_n(const Geom& g, const ProjectX<T>& a, Tables<T> tb, int sms, cudaStream_t s) {
  constexpr int G = project_pencils<T, N>(), NT = project_cta<T, N, G>();
  constexpr size_t smem = project_smem<T, N, G>();
  static_assert(smem <= kSmemPerCta);
  auto kern = project_x_kernel<T, N, G>;
  static std::atomic<int> cache[kMaxDevices];
  int per_sm = 1;
  const cudaError_t e = resident_ctas(kern, NT, smem, cache, &per_sm);
  if (e != cudaSuccess) return e;
  const int tiles = x_tiles(g, G);
  return launch_dependent(kern, std::min(per_sm * sms, tiles), NT, smem, s, a, g, tiles, tb);
}

#define QUASI_COL_LENGTHS(n, call)           \
  switch (n) {                               \
    case 8: return call(8);                  \
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
#define QUASI_COL_BATCH(N) launch_col_batch_n<QT, N>(g, axis, forward, jobs, njobs, tb, vq, scale, wait, narrow, sms, s)
#define QUASI_DENSITY_X(N) launch_density_x_n<QT, N>(g, a, tb64, tb, sms, s)
#define QUASI_UPDATE_X(N) launch_update_x_n<QT, N>(g, a, tb64, tb, sms, s)
#define QUASI_PROJECT_X(N) launch_project_x_n<QT, N>(g, a, tb, sms, s)

}  // namespace quasi
