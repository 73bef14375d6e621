// Real-space stages of the step in float.
#include "row_stage.cuh"

namespace quasi {
using QT = float;

#define QUASI_DENSITY(N) launch_rows<DensitySmem<QT, N>>(density_stage_kernel<QT, N>, g, sms, s, a, tb, tb64)
#define QUASI_STRESS(N)                                                                          \
  (sixteen_warps<StressSmem<QT, N>>(stage_groups<StressSmem<QT, N>>(g), sms)                      \
       ? launch_rows<StressSmem<QT, N>, 4>(stress_stage_kernel<QT, N, 4>, g, sms, s, a, tb)       \
       : launch_rows<StressSmem<QT, N>, 3>(stress_stage_kernel<QT, N, 3>, g, sms, s, a, tb))
#define QUASI_STRESS_STB(N)                                                                      \
  (sixteen_warps<StressStbSmem<N>>(stage_groups<StressStbSmem<N>>(g), sms)                        \
       ? launch_rows<StressStbSmem<N>, 4>(stress_stb_kernel<N, 4>, g, sms, s, a, tb, tb64)        \
       : launch_rows<StressStbSmem<N>, 3>(stress_stb_kernel<N, 3>, g, sms, s, a, tb, tb64))
#define QUASI_NONLINEAR(N)                                                                       \
  (sixteen_warps<NonlinearSmem<QT, N>>(stage_groups<NonlinearSmem<QT, N>>(g), sms)                \
       ? launch_rows<NonlinearSmem<QT, N>, 4>(nonlinear_stage_kernel<QT, N, 4>, g, sms, s, a, tb) \
       : launch_rows<NonlinearSmem<QT, N>, 3>(nonlinear_stage_kernel<QT, N, 3>, g, sms, s, a, tb))

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
