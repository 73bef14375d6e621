// Real-space stages of the step in double.
#include "row_stage.cuh"

namespace quasi {
using QT = double;

#define QUASI_DENSITY(N) launch_rows<DensitySmem<QT, N>>(density_stage_kernel<QT, N>, g, sms, s, a, tb, tb64)
#define QUASI_STRESS(N) \
  launch_rows<StressSmem<QT, N>>(stress_stage_kernel<QT, N, stage_ctas<QT, N>()>, g, sms, s, a, tb)
#define QUASI_NONLINEAR(N) \
  launch_rows<NonlinearSmem<QT, N>>(nonlinear_stage_kernel<QT, N, stage_ctas<QT, N>()>, g, sms, s, a, tb)

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

#define QUASI_GRADIENT(N) launch_rows<GradientSmem<N>>(gradient_stage_kernel<N>, g, sms, s, a, tb)
cudaError_t launch_gradient_stage(const Geom& g, const GradientStage& a, Tables<double> tb, int sms, cudaStream_t s) {
  QUASI_ROW_LENGTHS(g.nz, QUASI_GRADIENT)
}
}  // namespace quasi
