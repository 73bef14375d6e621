// The z pass (transform along the contiguous axis): every warp transforms its
// own groups of rows in registers (pencil_core.cuh, RowFFT), loading and storing
// them directly, so the kernel has no CTA barrier after its tables are in place
// and no staging of its input or output.
//
// Bound: HBM.  At 256^3 the floor of a pass is 20.5 us (float) and 41 us
// (double) at the measured copy bandwidth.  Tiles staged through shared memory
// (one TMA landing buffer read twice, three padded round trips, staged output
// rows) took 28.7 / 60.3 us: the double pass moved 94 bytes of shared memory per
// element, near the 128 bytes per clock of an SM.  In registers it moves 36 (one
// exchange, the twiddles, and shuffles): 22.9 / 48.9 us.  Sixteen lanes with 16
// elements each (one exchange) rather than 32 with 8 (two) for that reason.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>

#include "pencil_core.cuh"

namespace quasi {

struct Geom {
  int nx, ny, nz;
};

template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };

template <typename T>
__device__ __forceinline__ Cx<T> ld2(const T* p) {
  const typename Vec2<T>::type v = *reinterpret_cast<const typename Vec2<T>::type*>(p);
  return Cx<T>{v.x, v.y};
}
template <typename T>
__device__ __forceinline__ void st2(T* p, Cx<T> v) {
  typename Vec2<T>::type w;
  w.x = v.x;
  w.y = v.y;
  *reinterpret_cast<typename Vec2<T>::type*>(p) = w;
}

// A pair in another type.
template <typename T, typename U>
__device__ __forceinline__ Cx<T> as(Cx<U> v) { return Cx<T>{T(v.x), T(v.y)}; }
// Starts fetching `bytes` (a multiple of 16) at p (16-byte aligned) into L2.
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Programmatic dependent launch.  A kernel launched through launch_dependent may
// start while the kernel before it in its stream still runs; everything up to
// pdl_begin() (twiddle tables, which nothing writes, barriers) overlaps that
// kernel's end, and pdl_begin() returns when it has completed and its memory is
// visible.  Every such kernel calls it, so completion stays transitive along a
// stream.  A kernel of few CTAs also lets the next one start before it ends: the
// idle SMs take it (16x16x32: 71 -> 67 us per step).  A kernel that fills the GPU
// does not: the waiting CTAs would take room from its own (256^3: 2667 -> 2989 us
// per FP32 step, 64x64x128: 153 -> 177 us).
constexpr unsigned kPdlEarly = 74;   // half the SMs
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (gridDim.x <= kPdlEarly) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... P, class... A>
inline cudaError_t launch_dependent(void (*kern)(P...), int grid, int block, size_t smem, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, P(args)...);
}

// Resident CTAs per SM of a kernel, its dynamic shared memory allowed; found
// once per device and instantiation.
constexpr int kMaxDevices = 64;
constexpr size_t kSmemPerCta = 227 * 1024;   // the most a CTA may take
template <class K>
inline cudaError_t resident_ctas(K kern, int threads, size_t smem, std::atomic<int>* cache, int* out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const bool cached = dev < kMaxDevices;
  if (cached && (*out = cache[dev].load(std::memory_order_relaxed)) > 0) return cudaSuccess;
  e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  int n = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, threads, smem);
  if (e != cudaSuccess) return e;
  *out = std::max(n, 1);
  if (cached) cache[dev].store(*out, std::memory_order_relaxed);
  return cudaSuccess;
}

// Loads of a group's rows into a lane's elements, and stores.  `a` is the lane's
// first row (row 2 pencil of the group), the second follows it.
template <typename T, int N>
struct RowIO {
  using F = RowFFT<T, N>;
  // real rows: adjacent pairs (row a in v[t], row b in v[E - 1 - t])
  __device__ __forceinline__ static void load_pairs(const T* a, int l, Cx<T>* v) {
#pragma unroll
    for (int t = 0; t < F::H; ++t) {
      v[t] = ld2(a + 2 * (l + F::L * t));
      v[F::E - 1 - t] = ld2(a + N + 2 * (l + F::L * t));
    }
  }
  __device__ __forceinline__ static void store_pairs(T* a, int l, const Cx<T>* v) {
#pragma unroll
    for (int t = 0; t < F::H; ++t) {
      st2(a + 2 * (l + F::L * t), v[t]);
      st2(a + N + 2 * (l + F::L * t), v[F::E - 1 - t]);
    }
  }
  // spectral rows: v[t] = (row a, row b) at k = l + L t.  GRAD (sine kinds): -mk[k]
  // row[k + 1], the reversed input reads position N - k, nothing for k = 0
  template <bool SINE, bool GRAD = false>
  __device__ __forceinline__ static void load_spec(const T* a, int l, Cx<T>* v, const T* mk = nullptr) {
    static_assert(!GRAD || SINE, "shifted rows are sine rows");
#pragma unroll
    for (int t = 0; t < F::E; ++t) {
      const int k = l + F::L * t, n = F::spec(k, SINE, GRAD);
      v[t] = Cx<T>{a[n], a[N + n]};
      if constexpr (GRAD) {
        v[t] = cscale(v[t], -mk[k ? N - k - 1 : 0]);
        if (t == 0 && k == 0) v[t] = Cx<T>{T(0), T(0)};
      }
    }
  }
  template <bool SINE>
  __device__ __forceinline__ static void store_spec(T* a, int l, const Cx<T>* v) {
#pragma unroll
    for (int t = 0; t < F::E; ++t) {
      const int n = F::spec(l + F::L * t, SINE);
      a[n] = v[t].x;
      a[N + n] = v[t].y;
    }
  }
};

constexpr int kRowWarps = 8;   // warps per CTA of the row kernels
template <typename T, int N>
constexpr size_t row_smem(int warps = kRowWarps) {
  return RowFFT<T, N>::table_bytes() + size_t(warps) * RowFFT<T, N>::xch_bytes();
}

// Groups are walked from the last x plane to the first when rev: the pass before
// a z pass ends on the last planes, which are still in L2.  Float kernels load
// the next group's rows before they transform the current ones (32 more
// registers: 23.3 -> 22.7 us at 256^3); in double the registers are the rows.
template <typename T, int N, int KIND, bool GRAD>
__global__ void __launch_bounds__(32 * kRowWarps, 2)
    row_pass_kernel(const T* src, T* dst, int groups, Tables<T> tb, const T* mk, int rev) {
  using F = RowFFT<T, N>;
  using IO = RowIO<T, N>;
  constexpr bool fwd = KIND == E10 || KIND == O10, sine = KIND == O10 || KIND == O01;
  constexpr bool prefetch = sizeof(T) == 4;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5;
  Cx<T>* xb = reinterpret_cast<Cx<T>*>(smem_raw + F::table_bytes() + warp * F::xch_bytes());
  const typename F::Tab t = F::fill_tables(reinterpret_cast<Cx<T>*>(smem_raw), tb, threadIdx.x, 32 * kRowWarps);
  __syncthreads();
  pdl_begin();
  const RowWarp<T, N> w{int(threadIdx.x & 31)};
  const int l = w.l(), stride = gridDim.x * kRowWarps;
  auto row = [&](int grp) { return (size_t(rev ? groups - 1 - grp : grp) * F::ROWS + 2 * w.pencil()) * N; };
  auto load = [&](int grp, Cx<T>* v) {
    if constexpr (fwd) IO::load_pairs(src + row(grp), l, v);
    else IO::template load_spec<sine, GRAD>(src + row(grp), l, v, mk);
  };
  auto transform = [&](int grp, Cx<T>* v) {
    if constexpr (fwd) {
      F::from_pairs(w, v, sine);
      F::forward(w, v, xb, t);
      IO::template store_spec<sine>(dst + row(grp), l, v);
    } else {
      F::inverse(w, v, xb, t);
      F::to_pairs(w, v, sine);
      IO::store_pairs(dst + row(grp), l, v);
    }
  };
  int grp = blockIdx.x * kRowWarps + warp;
  Cx<T> v[F::E];
  if constexpr (prefetch) {
    Cx<T> next[F::E];
    if (grp < groups) load(grp, next);
    for (; grp < groups; grp += stride) {
#pragma unroll
      for (int i = 0; i < F::E; ++i) v[i] = next[i];
      if (grp + stride < groups) load(grp + stride, next);
      transform(grp, v);
    }
  } else {
    for (; grp < groups; grp += stride) {
      load(grp, v);
      transform(grp, v);
    }
  }
}

template <typename T, int N, int KIND, bool GRAD = false>
cudaError_t launch_row_pass_k(const Geom& g, Tables<T> tb, const T* src, T* dst, const T* mk, int sms, bool rev,
                              cudaStream_t s) {
  using F = RowFFT<T, N>;
  auto kern = row_pass_kernel<T, N, KIND, GRAD>;
  static std::atomic<int> cache[kMaxDevices];
  int per_sm = 1;
  static_assert(row_smem<T, N>() <= kSmemPerCta);
  const cudaError_t e = resident_ctas(kern, 32 * kRowWarps, row_smem<T, N>(), cache, &per_sm);
  if (e != cudaSuccess) return e;
  const int groups = g.nx * g.ny / F::ROWS;   // nx ny is a multiple of 16, ROWS divides 16
  const int grid = std::min(per_sm * sms, (groups + kRowWarps - 1) / kRowWarps);
  return launch_dependent(kern, grid, 32 * kRowWarps, row_smem<T, N>(), s, src, dst, groups, tb, mk, int(rev));
}

template <typename T, int N>
cudaError_t launch_row_pass_n(const Geom& g, int kind, Tables<T> tb, const T* src, T* dst, const T* mk, int sms,
                              bool rev, cudaStream_t s) {
  if (mk) {
    if constexpr (sizeof(T) == 8) {
      if (kind == O01) return launch_row_pass_k<T, N, O01, true>(g, tb, src, dst, mk, sms, rev, s);
    }
    return cudaErrorNotSupported;
  }
  switch (kind) {
    case E10: return launch_row_pass_k<T, N, E10>(g, tb, src, dst, mk, sms, rev, s);
    case E01: return launch_row_pass_k<T, N, E01>(g, tb, src, dst, mk, sms, rev, s);
    case O10: return launch_row_pass_k<T, N, O10>(g, tb, src, dst, mk, sms, rev, s);
    default: return launch_row_pass_k<T, N, O01>(g, tb, src, dst, mk, sms, rev, s);
  }
}

// z pass src -> dst (may be the same field).  mk (double, RODFT01): transforms
// -mk[k] row[k + 1], zero at the top, the z derivative of a cosine spectrum.
// Instantiated in row_pass_f32.cu and row_pass_f64.cu.
template <typename T>
cudaError_t launch_row_pass(const Geom& g, int kind, Tables<T> tb, const T* src, T* dst, const T* mk, int sms, bool rev,
                            cudaStream_t s);

#define QUASI_INSTANTIATE_ROW_PASS(T)                                                                              \
  template <>                                                                                                      \
  cudaError_t launch_row_pass<T>(const Geom& g, int kind, Tables<T> tb, const T* src, T* dst, const T* mk, \
                                 int sms, bool rev, cudaStream_t s) {                                              \
    switch (g.nz) {                                                                                                \
      case 16: return launch_row_pass_n<T, 16>(g, kind, tb, src, dst, mk, sms, rev, s);                        \
      case 32: return launch_row_pass_n<T, 32>(g, kind, tb, src, dst, mk, sms, rev, s);                        \
      case 64: return launch_row_pass_n<T, 64>(g, kind, tb, src, dst, mk, sms, rev, s);                        \
      case 96: return launch_row_pass_n<T, 96>(g, kind, tb, src, dst, mk, sms, rev, s);                        \
      case 128: return launch_row_pass_n<T, 128>(g, kind, tb, src, dst, mk, sms, rev, s);                      \
      case 192: return launch_row_pass_n<T, 192>(g, kind, tb, src, dst, mk, sms, rev, s);                      \
      case 256: return launch_row_pass_n<T, 256>(g, kind, tb, src, dst, mk, sms, rev, s);                      \
      case 512: return launch_row_pass_n<T, 512>(g, kind, tb, src, dst, mk, sms, rev, s);                      \
      default: return cudaErrorNotSupported;                                                                       \
    }                                                                                                              \
  }

}  // namespace quasi
