// Column passes and x stages in double.
#include "col_pass.cuh"

namespace quasi {
using QT = double;

template <>
cudaError_t launch_col_batch<QT>(const Geom& g, int axis, bool forward, const ColJobs<QT>& jobs, int njobs,
                                 Tables<QT> tb, const double* vq, QT scale, const ColWait& wait, bool narrow, int sms,
                                 cudaStream_t s) {
  QUASI_COL_LENGTHS(axis == 1 ? g.ny : g.nx, QUASI_COL_BATCH)
}
template <>
cudaError_t launch_density_x<QT>(const Geom& g, const DensityX<QT>& a, Tables<double> tb64, Tables<QT> tb, int sms,
                                 cudaStream_t s) {
  QUASI_COL_LENGTHS(g.nx, QUASI_DENSITY_X)
}
template <>
cudaError_t launch_update_x<QT>(const Geom& g, const UpdateX<QT>& a, Tables<double> tb64, Tables<QT> tb, int sms,
                                cudaStream_t s) {
  QUASI_COL_LENGTHS(g.nx, QUASI_UPDATE_X)
}
template <>
cudaError_t launch_project_x<QT>(const Geom& g, const ProjectX<QT>& a, Tables<QT> tb, int sms, cudaStream_t s) {
  QUASI_COL_LENGTHS(g.nx, QUASI_PROJECT_X)
}
}  // namespace quasi
