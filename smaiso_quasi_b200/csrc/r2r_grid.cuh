// A whole 3-D transform of a small field in one cooperative launch.
//
// Up to a few MB a transform is launch-bound: its three passes run in 3 us each
// and their launches take as long on the host (one transform of 16x16x32 doubles:
// 9.9 us of host time in three launches).  Here the passes share a launch, with
// two grid-wide barriers in between; rows and column tiles are the ones of
// row_pass.cuh and col_pass.cuh, loaded and stored directly.  Every length is a
// case of a switch inside the kernel, so one kernel per type covers every grid.
#pragma once
#include <cooperative_groups.h>

#include "col_pass.cuh"

namespace quasi {

constexpr int kGridThreads = 128, kGridWarps = kGridThreads / 32;
// Largest field (bytes).  Above it a pass needs more than one wave of CTAs and the
// GPU's time, not the launches', decides.
constexpr size_t kGridBytes = size_t(4) << 20;

template <typename T>
struct GridPasses {
  T* data;
  Geom g;
  int kind[3];
  Tables<T> tb[3];
};

template <typename T, int N>
__device__ __noinline__ void grid_rows(const GridPasses<T>& a, unsigned char* sm) {
  using F = RowFFT<T, N>;
  using IO = RowIO<T, N>;
  const typename F::Tab t = F::fill_tables(reinterpret_cast<Cx<T>*>(sm), a.tb[2], threadIdx.x, kGridThreads);
  __syncthreads();
  const RowWarp<T, N> w{int(threadIdx.x & 31)};
  const int warp = threadIdx.x >> 5, l = w.l(), groups = a.g.nx * a.g.ny / F::ROWS, kind = a.kind[2];
  Cx<T>* xb = reinterpret_cast<Cx<T>*>(sm + F::table_bytes() + warp * F::xch_bytes());
  for (int grp = blockIdx.x * kGridWarps + warp; grp < groups; grp += gridDim.x * kGridWarps) {
    T* row = a.data + (size_t(grp) * F::ROWS + 2 * w.pencil()) * N;
    Cx<T> v[F::E];
    if (is_forward(kind)) {
      IO::load_pairs(row, l, v);
      F::from_pairs(w, v, is_sine(kind));
      F::forward(w, v, xb, t);
      if (is_sine(kind)) IO::template store_spec<true>(row, l, v);
      else IO::template store_spec<false>(row, l, v);
    } else {
      if (is_sine(kind)) IO::template load_spec<true, 0>(row, l, v);
      else IO::template load_spec<false, 0>(row, l, v);
      F::inverse(w, v, xb, t);
      F::to_pairs(w, v, is_sine(kind));
      IO::store_pairs(row, l, v);
    }
  }
}

template <typename T, int N>
__device__ __noinline__ void grid_cols(const GridPasses<T>& a, int axis, unsigned char* sm) {
  using C = ColTile<N, 8>;
  using F = PencilFFT<T, N>;
  using IO = ColIO<T, N>;
  constexpr int SETS = kGridThreads / C::THREADS;
  const typename F::Tab t = F::fill_tables(reinterpret_cast<Cx<T>*>(sm), a.tb[axis], threadIdx.x, kGridThreads);
  __syncthreads();
  const int set = threadIdx.x / C::THREADS, kind = a.kind[axis];
  const C w(threadIdx.x % C::THREADS, 1 + set);
  const int l = w.l(), kt = a.g.nz / 16, tiles = (axis == 1 ? a.g.nx : a.g.ny) * kt;
  const int stride = axis == 1 ? a.g.nz : a.g.ny * a.g.nz;
  const size_t outer = axis == 1 ? size_t(a.g.ny) * a.g.nz : size_t(a.g.nz);
  Cx<T>* xb = reinterpret_cast<Cx<T>*>(sm + F::table_bytes()) + set * C::XCH;
  for (int tile = blockIdx.x * SETS + set; tile < tiles; tile += gridDim.x * SETS) {
    T* p = a.data + (tile / kt) * outer + (tile % kt) * 16 + 2 * w.g;
    Cx<T> v[F::E];
    if (is_forward(kind)) {
      IO::load_pos(p, stride, l, v, is_sine(kind));
      F::forward(w, v, xb, t);
      if (is_sine(kind)) IO::store_index(p, stride, l, v);
      else IO::store_spec(p, stride, l, v, false);
    } else {
      if (is_sine(kind)) IO::load_index(p, stride, l, v);
      else IO::load_spec(p, stride, l, v, false);
      F::inverse(w, v, xb, t);
      IO::store_pos(p, stride, l, v, is_sine(kind));
    }
  }
}

// Shared memory of one pass along an axis of length n.
template <typename T>
inline size_t grid_pass_smem(int axis, int n) {
  switch (n) {
#define QUASI_GRID_SMEM(N)                                                                                    \
  case N:                                                                                                     \
    if (axis == 2) return N < 16 ? 0 : RowFFT<T, (N < 16 ? 16 : N)>::table_bytes() +                          \
                                           kGridWarps * RowFFT<T, (N < 16 ? 16 : N)>::xch_bytes();            \
    return PencilFFT<T, N>::table_bytes() +                                                                   \
           size_t(kGridThreads / ColTile<N, 8>::THREADS) * ColTile<N, 8>::XCH * sizeof(Cx<T>);
    QUASI_GRID_SMEM(8) QUASI_GRID_SMEM(16) QUASI_GRID_SMEM(32) QUASI_GRID_SMEM(64) QUASI_GRID_SMEM(96)
    QUASI_GRID_SMEM(128) QUASI_GRID_SMEM(192) QUASI_GRID_SMEM(256)
#undef QUASI_GRID_SMEM
    default: return 0;
  }
}

template <typename T>
__global__ void __launch_bounds__(kGridThreads, sizeof(T) == 8 ? 3 : 4) r2r_grid_kernel(const GridPasses<T> a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  auto cols = [&](int axis, int n) {
    switch (n) {
      case 8: return grid_cols<T, 8>(a, axis, smem_raw);
      case 16: return grid_cols<T, 16>(a, axis, smem_raw);
      case 32: return grid_cols<T, 32>(a, axis, smem_raw);
      case 64: return grid_cols<T, 64>(a, axis, smem_raw);
      case 96: return grid_cols<T, 96>(a, axis, smem_raw);
      case 128: return grid_cols<T, 128>(a, axis, smem_raw);
      case 192: return grid_cols<T, 192>(a, axis, smem_raw);
      default: return grid_cols<T, 256>(a, axis, smem_raw);
    }
  };
  switch (a.g.nz) {
    case 16: grid_rows<T, 16>(a, smem_raw); break;
    case 32: grid_rows<T, 32>(a, smem_raw); break;
    case 64: grid_rows<T, 64>(a, smem_raw); break;
    case 96: grid_rows<T, 96>(a, smem_raw); break;
    case 128: grid_rows<T, 128>(a, smem_raw); break;
    case 192: grid_rows<T, 192>(a, smem_raw); break;
    default: grid_rows<T, 256>(a, smem_raw); break;
  }
  cooperative_groups::grid_group grid = cooperative_groups::this_grid();
  grid.sync();
  cols(1, a.g.ny);
  grid.sync();
  cols(0, a.g.nx);
}

// Whether the one-launch form covers a grid (lengths above 256 need tiles of more
// threads than its CTAs have), and whether a transform takes it.
inline bool grid_lengths(const Geom& g) { return g.nx <= 256 && g.ny <= 256 && g.nz <= 256; }
template <typename T>
inline bool grid_form(const Geom& g) {
  return grid_lengths(g) && size_t(g.nx) * g.ny * g.nz * sizeof(T) <= kGridBytes;
}

// The transform in place; every CTA of a cooperative launch is resident.
template <typename T>
cudaError_t launch_r2r_grid(GridPasses<T> a, int sms, cudaStream_t s) {
  const int n[3] = {a.g.nx, a.g.ny, a.g.nz};
  size_t smem = 0;
  for (int axis = 0; axis < 3; ++axis) smem = std::max(smem, grid_pass_smem<T>(axis, n[axis]));
  // one CTA per SM is resident whatever its shared memory (at most 48 KB here)
  auto kern = r2r_grid_kernel<T>;
  static std::atomic<int> cache[kMaxDevices];
  int per_sm = 1;
  cudaError_t e = resident_ctas(kern, kGridThreads, size_t(64) << 10, cache, &per_sm);
  if (e != cudaSuccess) return e;
  const int work = std::max(a.g.nx * a.g.ny / 4, std::max(a.g.nx, a.g.ny) * (a.g.nz / 16));
  const int grid = std::max(1, std::min(per_sm * sms, work));
  void* args[] = {&a};
  return cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kern), dim3(grid), dim3(kGridThreads), args, smem, s);
}

}  // namespace quasi
