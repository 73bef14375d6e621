// Passes of one field along x and y on tiles that the threads load and store
// themselves, one tile each: for fields of up to 16 MB, and for pairs of floats
// whose address (8- but not 16-byte aligned) the tensor copies of col_batch_kernel
// do not take.  The tiles and transforms are the ones of col_pass.cuh.
//
// Bound: latency, and the launch on the host.  Without tensor maps and waits a
// transform of 64x64x128 doubles takes 10.4 us (12.1 through col_batch_kernel) and
// 7.8 us of host time in its three launches (8.5).
#pragma once
#include "col_pass.cuh"

namespace quasi {

template <typename T, int N>
constexpr size_t col_direct_smem() {
  using C = ColTile<N, 8>;
  return PencilFFT<T, N>::table_bytes() + size_t(col_cta<N, 8>() / C::THREADS) * C::XCH * sizeof(Cx<T>);
}

template <typename T, int N>
__global__ void __launch_bounds__(col_cta<N, 8>())
    col_direct_kernel(T* data, Geom g, int axis, int kind, int tiles, Tables<T> tb) {
  using C = ColTile<N, 8>;
  using F = PencilFFT<T, N>;
  using IO = ColIO<T, N>;
  constexpr int NT = col_cta<N, 8>(), SETS = NT / C::THREADS;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const typename F::Tab t = F::fill_tables(reinterpret_cast<Cx<T>*>(smem_raw), tb, threadIdx.x, NT);
  __syncthreads();
  pdl_begin();
  const int set = threadIdx.x / C::THREADS, tile = blockIdx.x * SETS + set;
  const C w(threadIdx.x % C::THREADS, 1 + set);
  if (tile >= tiles) return;
  const int l = w.l(), kt = g.nz / 16, stride = axis == 1 ? g.nz : g.ny * g.nz;
  const size_t outer = axis == 1 ? size_t(g.ny) * g.nz : size_t(g.nz);
  Cx<T>* xb = reinterpret_cast<Cx<T>*>(smem_raw + F::table_bytes()) + set * C::XCH;
  T* p = data + (tile / kt) * outer + (tile % kt) * 16 + 2 * w.g;
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

template <typename T, int N>
cudaError_t launch_col_direct_n(const Geom& g, int axis, int kind, T* data, Tables<T> tb, cudaStream_t s) {
  auto kern = col_direct_kernel<T, N>;
  constexpr size_t smem = col_direct_smem<T, N>();
  constexpr int NT = col_cta<N, 8>(), SETS = NT / ColTile<N, 8>::THREADS;
  static_assert(smem <= kSmemPerCta);
  static std::atomic<int> cache[kMaxDevices];
  int per_sm = 1;
  const cudaError_t e = resident_ctas(kern, NT, smem, cache, &per_sm);
  if (e != cudaSuccess) return e;
  const int tiles = (axis == 1 ? g.nx : g.ny) * (g.nz / 16);
  return launch_dependent(kern, (tiles + SETS - 1) / SETS, NT, smem, s, data, g, axis, kind, tiles, tb);
}

// One pass of a plain field in place along axis 0 or 1.
template <typename T>
cudaError_t launch_col_direct(const Geom& g, int axis, int kind, T* data, Tables<T> tb, cudaStream_t s) {
#define QUASI_COL_DIRECT(N) launch_col_direct_n<T, N>(g, axis, kind, data, tb, s)
  QUASI_COL_LENGTHS(axis == 1 ? g.ny : g.nx, QUASI_COL_DIRECT)
#undef QUASI_COL_DIRECT
}

}  // namespace quasi
