// Real-space stages of the step in float.
#include "row_stage.cuh"

namespace quasi {
using QT = float;

#define QUASI_DENSITY(N) launch_rows<DensitySmem<QT, N>>(density_stage_kernel<QT, N>, g, sms, s, a, tb, tb64)
// 16 or 12 warps per SM
template <int N>
cudaError_t stress(const Geom& g, const StressStage<QT>& a, Tables<QT> tb, int sms, cudaStream_t s) {
  using S = StressSmem<QT, N>;
  if constexpr (kSixteenFit<S>)
    if (sixteen_warps(stage_groups<S>(g), sms))
      return launch_rows<S, 4>(stress_stage_kernel<QT, N, 4>, g, sms, s, a, tb);
  return launch_rows<S, 3>(stress_stage_kernel<QT, N, 3>, g, sms, s, a, tb);
}
template <int N>
cudaError_t stress_stb(const Geom& g, const StressStb& a, Tables<QT> tb, Tables<double> tb64, int sms, cudaStream_t s) {
  using S = StressStbSmem<N>;
  if constexpr (kSixteenFit<S>)
    if (sixteen_warps(stage_groups<S>(g), sms))
      return launch_rows<S, 4>(stress_stb_kernel<N, 4>, g, sms, s, a, tb, tb64);
  return launch_rows<S, 3>(stress_stb_kernel<N, 3>, g, sms, s, a, tb, tb64);
}
template <int N>
cudaError_t nonlinear(const Geom& g, const NonlinearStage<QT>& a, Tables<QT> tb, int sms, cudaStream_t s) {
  using S = NonlinearSmem<QT, N>;
  if constexpr (kSixteenFit<S>)
    if (sixteen_warps(stage_groups<S>(g), sms))
      return launch_rows<S, 4>(nonlinear_stage_kernel<QT, N, 4>, g, sms, s, a, tb);
  return launch_rows<S, 3>(nonlinear_stage_kernel<QT, N, 3>, g, sms, s, a, tb);
}
#define QUASI_STRESS(N) stress<N>(g, a, tb, sms, s)
#define QUASI_STRESS_STB(N) stress_stb<N>(g, a, tb, tb64, sms, s)
#define QUASI_NONLINEAR(N) nonlinear<N>(g, a, tb, sms, s)

template <>
cudaError_t launch_density_stage<QT>(const Geom& g, const DensityStage<QT>& a, Tables<QT> tb, Tables<double> tb64,
                                     int sms, cudaStream_t s) {
  QUASI_ROW_LENGTHS(g.nz, QUASI_DENSITY)
}
template <>
cudaError_t launch_stress_stage<QT>(const Geom& g, const StressStage<QT>& a, Tables<QT> tb, int sms, cudaStream_t s) {
  QUASI_ROW_LENGTHS(g.nz, QUASI_STRESS)
}
template <>
cudaError_t launch_nonlinear_stage<QT>(const Geom& g, const NonlinearStage<QT>& a, Tables<QT> tb, int sms,
                                       cudaStream_t s) {
  QUASI_ROW_LENGTHS(g.nz, QUASI_NONLINEAR)
}
cudaError_t launch_stress_stb(const Geom& g, const StressStb& a, Tables<QT> tb, Tables<double> tb64, int sms,
                              cudaStream_t s) {
  QUASI_ROW_LENGTHS(g.nz, QUASI_STRESS_STB)
}
}  // namespace quasi
