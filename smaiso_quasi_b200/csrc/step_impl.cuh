// The quasi-incompressible smectic-isotropic time step (quasi.cpp:1014-1965)
// and its stability variant (quasi-stb.cpp:983-1968) as a short sequence of
// kernels, each doing everything that happens to a field between two changes of
// the axis (row_stage.cuh: along z; col_pass.cuh: along x, and the y passes):
//
//   y  rho law            forward
//   x  density_x          forward, filter -> rho^, inverse (rho, grad rho)
//   y  rho, grad rho      inverse
//   z  density_stage      rho, divv; forward (divv)
//   z  stress_stage       df, stress; forward (S)
//   y  S, divv            forward
//   x  project_x          forward, projection, inverse (p, v)
//   y  p, v               inverse
//   z  nonlinear_stage    v, p, N; forward (N)
//   y  N                  forward
//   x  update_x           forward, update -> psi^, inverse (psi, d_x psi; df, lap, grad lap psi)
//   y  psi, grad psi; df, lap, grad lap psi   inverse
//   z  gradient_stage     psi, grad psi, rho law; forward (rho law)
//
// Three passes per transform are three trips through HBM, and every stage in
// between is two more; fused this way a field makes one trip per axis change.
// At 256^3 the FP32 step moves 150 fields' worth of float data in 15 launches
// (245 in 75 before), FP64 in 13.
//
// Two transforms of the reference's step are not made because they return their
// input: divv = iCT(scale CT(divv)) (quasi.cpp:1888-1900) is divv, and the x
// passes of a forward and an inverse transform with pointwise work in between
// meet in one kernel.
//
// Templated on the storage/transform type T (double: the plain FP64 form;
// float: the FP32 form).  Wavenumbers, spectral constants, the semi-implicit
// update and all reductions are evaluated in double in both forms (the projection
// takes its wavenumbers rounded to T), and both keep in double quasi-stb's sh, and
// what the density is built from: the carried spectral state
// psi^, psi and grad psi (and their transforms), the density law, rho^ with
// its Gaussian filter, rho and the divv difference quotient.  The quotient
// (rho - rho_old)/dt (quasi.cpp:1279) amplifies step-to-step rounding noise of
// rho by 1/dt = 1000, and the rounding errors of a float transform of psi^ lie
// next to psi's own spectrum (|q| = q0): the density law's demodulation
// sqrt(q0^2 psi^2 + |grad psi|^2) moves them to the low wavenumbers that the
// Gaussian filter keeps.
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "row_stage.cuh"
#include "tc_pass.cuh"

namespace quasi {

enum Variant : int { kQuasi = 0, kStb = 1 };

template <typename T>
struct StepCtx {
  Geom g;
  // per-axis wavenumbers, quasi.cpp:397-431, and the density filter exp(-1.57^2 8 q^2) per axis
  XTables x;
  const double *vqy, *vqz, *vsz;   // vsz[k] = vqz[k + 1]
  double ep, alpha, beta, gamma, q0, kp, rho0, rho_s, rho_m, nu, dt, scale;
  int variant, divv_switch, n0;   // n0: planes per emulated MPI rank (quasi.cpp:1641-1690)
  int* nloop;                     // device counter of completed steps
  // Buffers of the step from s to s + 1 completed steps.  psiq rotates through
  // three buffers, Nq, psi, rho, the density scratch and grad rho's spectra
  // through two (one captured graph per phase of the rotation).
  double *psiq, *psiq_old, *psiq_new, *rhoq;
  double *psi, *psi_old, *psi_new;   // psi_new is psi_old's buffer
  double *gx, *gy, *gz;
  double *rho, *rho_new;   // after s and s + 1 steps
  // law: the rho law's z pass for this step, then rho's spectrum; law_next: where
  // this step's last stage leaves the next one's (FP64: until then the cosine
  // spectrum of the previous rho, whose z derivative is grad_z rho)
  double *law, *law_next;
  T *Nq, *Nq_old;
  T *rdx, *rdy, *rdz;      // spectra of grad rho of the previous step's rho^ (FP64: rdz unused)
  T *rdx_new, *rdy_new, *rdz_new;
  T *divvq, *Sx, *Sy, *Sz;
  T *vx, *vy, *vz, *divv, *p, *df;
  T *dfs, *lap, *ldx, *ldy, *ldz;   // spectra between the steps
  T *base, *grad;                   // N without velocity and pressure; the pressure's factor
  T *mu, *dtpsi;                    // quasi-stb
  // launch settings
  int sms;
  bool narrow;
  const tc::Tables4* tc;            // tensor-core y passes (BF16X3_TC), or nullptr
  int* err;
};

// The FP32 form holds its float fields apart from the double state.
template <typename T> constexpr bool kStateCopy = !std::is_same<T, double>::value;

template <typename T>
struct AxisTables {
  Tables<T> t[3];
};

#define QUASI_TRY(...)                        \
  do {                                        \
    cudaError_t e_ = (__VA_ARGS__);           \
    if (e_ != cudaSuccess) return e_;         \
  } while (0)

// y passes of up to kMaxJobs fields.  In the tensor-core form plain float cosine
// passes go to the tensor cores where the length allows it.
template <typename T>
struct YBatch {
  ColJobs<T> jobs{};
  int n = 0;
  void add(T* src, T* dst, int op = kColCos, T* dst2 = nullptr) { jobs.job[n++] = ColJob<T>{src, dst, dst2, op}; }
  void add(T* f, int op = kColCos) { add(f, f, op); }
};
template <typename T, typename C>
cudaError_t y_passes(const StepCtx<C>& c, bool forward, const YBatch<T>& b, const Tables<T>& tb, cudaStream_t s) {
  YBatch<T> rest = b;
  if constexpr (std::is_same<T, float>::value) {
    if (c.tc) {
      rest.n = 0;
      for (int j = 0; j < b.n; ++j) {
        const ColJob<T>& jb = b.jobs.job[j];
        cudaError_t e = cudaErrorNotSupported;
        if (jb.op == kColCos)
          e = tc::launch_tc_pass(c.g.nx, c.g.ny, c.g.nz, 1, forward ? E10 : E01, *c.tc, jb.src, jb.dst, c.err, c.sms,
                                 s);
        if (e == cudaErrorNotSupported) rest.jobs.job[rest.n++] = jb;
        else if (e != cudaSuccess) return e;
      }
      if (!rest.n) return cudaSuccess;
    }
  }
  return launch_col_batch<T>(c.g, 1, forward, rest.jobs, rest.n, tb, c.vqy, T(1), ColWait{c.err}, c.narrow, c.sms, s);
}

// One plain pass of a field in place along x (0), y (1) or z (2).
template <typename T, typename C>
cudaError_t plain_pass(const StepCtx<C>& c, int axis, bool forward, T* f, const Tables<T>& tb, cudaStream_t s,
                       T scale = T(1)) {
  if (axis == 2)
    return launch_row_pass<T>(c.g, forward ? E10 : E01, tb, f, f, static_cast<const T*>(nullptr), c.sms, true, s);
  YBatch<T> b;
  b.add(f);
  return launch_col_batch<T>(c.g, axis, forward, b.jobs, 1, tb, nullptr, scale, ColWait{c.err}, c.narrow, c.sms, s);
}
// Forward cosine transform in place, times scale.
template <typename T, typename C>
cudaError_t forward3(const StepCtx<C>& c, T* f, const AxisTables<T>& tb, cudaStream_t s, T scale = T(1)) {
  for (int a = 2; a >= 0; --a) QUASI_TRY(plain_pass<T>(c, a, true, f, tb.t[a], s, a ? T(1) : scale));
  return cudaSuccess;
}

// From psi^: psi and grad psi (into psi, c.gx, c.gy, c.gz), the spectra of the
// next step's df, lap and grad lap psi, and its rho law (into law).  quasi-stb: the
// spectrum of sh in double (into lap, FP32: into law, which has no other use there).
// update: N^ and the new psi^ first (quasi.cpp:1944-1962), and the step counter
// after; else psi^ is taken from psiq (after the pre-loop or a checkpoint).
template <typename T>
cudaError_t enqueue_update(const StepCtx<T>& c, const AxisTables<T>& tb, const AxisTables<double>& tb64, bool update,
                           double* psiq, double* psi, double* law, cudaStream_t s) {
  UpdateX<T> u{};
  u.in = u.Nq = c.Nq;
  u.Nq_old = c.Nq_old;
  u.psiq = c.psiq;
  u.psiq_old = c.psiq_old;
  u.psiq_new = psiq;
  u.out0 = psi;
  u.out1 = c.gx;
  const bool quasi = c.variant == kQuasi;
  T* outs[5] = {c.dfs, c.lap, c.ldx, c.ldy, c.ldz};
  for (int o = 0; o < 5; ++o) u.out[o] = outs[o];
  double* sh = law;
  if constexpr (!kStateCopy<T>) sh = c.lap;
  u.sh = sh;
  u.x = c.x;
  u.ep = c.ep; u.alpha = c.alpha; u.q0 = c.q0; u.rho_m = c.rho_m; u.dt = c.dt; u.scale = c.scale;
  u.nloop = c.nloop;
  u.variant = c.variant;
  u.from_spec = !update;
  QUASI_TRY(launch_update_x<T>(c.g, u, tb64.t[0], tb.t[0], c.sms, s));
  // grad_y and grad_z share the x pass of psi, grad_z also its y pass
  YBatch<double> yd;
  yd.add(psi, psi, kColBoth, c.gy);
  yd.add(c.gx);
  YBatch<T> yt;
  if (quasi) {
    yt.add(c.dfs);
    yt.add(c.lap);
    yt.add(c.ldx);
    yt.add(c.ldy, kColSine);
    yt.add(c.ldz);
  } else {
    yd.add(sh);
  }
  if constexpr (!kStateCopy<T>) {
    for (int j = 0; j < yt.n; ++j) yd.jobs.job[yd.n++] = yt.jobs.job[j];
    QUASI_TRY(y_passes(c, false, yd, tb64.t[1], s));
  } else {
    QUASI_TRY(y_passes(c, false, yd, tb64.t[1], s));
    if (quasi) QUASI_TRY(y_passes(c, false, yt, tb.t[1], s));
  }
  GradientStage gs{psi, c.gy, c.gx, psi, c.gx, c.gy, c.gz, quasi ? law : nullptr, c.vqz, c.kp, c.q0, c.rho0,
                   update ? c.nloop : nullptr};
  return launch_gradient_stage(c.g, gs, tb64.t[2], c.sms, s);
}

// rho^ from `law` (or, from_spec, from memory) -> the spectra of rho (in law) and
// of grad rho for the next step, after their x and y passes.
template <typename T>
cudaError_t enqueue_density(const StepCtx<T>& c, const AxisTables<T>& tb, const AxisTables<double>& tb64,
                            bool from_spec, double* law, T* rdx, T* rdy, T* rdz, cudaStream_t s) {
  DensityX<T> d{};
  d.in = d.out0 = law;
  d.rhoq = c.rhoq;
  if constexpr (!kStateCopy<T>) d.out1 = rdx;
  d.gx = rdx; d.gy = rdy; d.gz = rdz;
  d.x = c.x;
  d.scale = c.scale;
  d.from_spec = from_spec;
  QUASI_TRY(launch_density_x<T>(c.g, d, tb64.t[0], tb.t[0], c.sms, s));
  YBatch<double> yd;
  if constexpr (!kStateCopy<T>) {
    yd.add(law, law, kColBoth, rdy);
    yd.add(rdx);
    return y_passes(c, false, yd, tb64.t[1], s);
  } else {
    yd.add(law);
    QUASI_TRY(y_passes(c, false, yd, tb64.t[1], s));
    YBatch<T> yt;
    yt.add(rdx);
    yt.add(rdy, kColSine);
    yt.add(rdz);
    return y_passes(c, false, yt, tb.t[1], s);
  }
}

// One time step, enqueued on `s` (captured into a CUDA graph by the caller).
// tb64: the FP64 twiddles of the double transforms (the same tables as tb in
// the FP64 form).
template <typename T>
cudaError_t enqueue_step(const StepCtx<T>& c, const AxisTables<T>& tb, const AxisTables<double>& tb64,
                         cudaStream_t s) {
  const Geom g = c.g;
  const bool quasi = c.variant == kQuasi;
  YBatch<T> ys;
  if (quasi) {
    // a5 density + filter quasi.cpp:1237-1268 in double
    YBatch<double> yl;
    yl.add(c.law);
    QUASI_TRY(y_passes(c, true, yl, tb64.t[1], s));
    QUASI_TRY(enqueue_density<T>(c, tb, tb64, false, c.law, c.rdx_new, c.rdy_new, c.rdz_new, s));
    DensityStage<T> d{};
    d.rdx = c.rdx; d.rdy = c.rdy; d.rdz = c.rdz;
    if constexpr (!kStateCopy<T>) d.rdz = c.law_next;
    d.rho_s = c.law; d.rho_old = c.rho; d.rho = c.rho_new;
    d.v[0] = c.vx; d.v[1] = c.vy; d.v[2] = c.vz;
    d.grad = c.grad; d.divv = c.divv; d.divv_s = c.divvq;
    d.vqz = c.vqz;
    d.dt = c.dt;
    d.cp = c.kp / (c.rho_s * c.rho_s);
    d.divv_switch = c.divv_switch;
    d.nloop = c.nloop;
    QUASI_TRY(launch_density_stage<T>(g, d, tb.t[2], tb64.t[2], c.sms, s));
    ys.add(c.divvq);
  }
  // a7 stress quasi.cpp:1298-1330; quasi-stb: rho == 1, divv == 0, grad rho == 0 (quasi-stb.cpp:1232)
  if constexpr (kStateCopy<T>) {
    if (!quasi) {
      const StressStb st{c.law, c.psi, {c.gx, c.gy, c.gz}, c.mu, c.base, {c.Sx, c.Sy, c.Sz}, c.vqz, c.beta, c.gamma};
      QUASI_TRY(launch_stress_stb(g, st, tb.t[2], tb64.t[2], c.sms, s));
    }
  }
  if (quasi || !kStateCopy<T>) {
    StressStage<T> st{};
    st.lap_s = c.lap; st.df_s = quasi ? c.dfs : c.lap;
    st.ld[0] = c.ldx; st.ld[1] = c.ldy; st.ld[2] = c.ldz;
    st.rho = c.rho_new; st.psi = c.psi;
    st.g[0] = c.gx; st.g[1] = c.gy; st.g[2] = c.gz;
    st.df = quasi ? c.df : c.mu; st.base = c.base;
    st.s[0] = c.Sx; st.s[1] = c.Sy; st.s[2] = c.Sz;
    st.ep = c.ep; st.beta = c.beta; st.gamma = c.gamma;
    st.variant = c.variant;
    st.vqz = c.vqz;
    QUASI_TRY(launch_stress_stage<T>(g, st, tb.t[2], c.sms, s));
  }
  ys.add(c.Sx);
  ys.add(c.Sy, kColSine);
  ys.add(c.Sz);
  QUASI_TRY(y_passes(c, true, ys, tb.t[1], s));
  // a8 pressure, a9 velocity quasi.cpp:1336-1884
  ProjectX<T> p{};
  p.in[0] = c.Sx; p.in[1] = c.Sy; p.in[2] = c.Sz; p.in[3] = c.divvq;
  p.out[0] = c.p; p.out[1] = c.vx; p.out[2] = c.vy; p.out[3] = c.vz;
  p.x = c.x;
  p.nu = c.nu; p.scale = c.scale;
  p.variant = c.variant; p.n0 = c.n0;
  QUASI_TRY(launch_project_x<T>(g, p, tb.t[0], c.sms, s));
  YBatch<T> yv;
  if (quasi) yv.add(c.p);
  yv.add(c.vx);
  yv.add(c.vy, kColSine);
  yv.add(c.vz);
  QUASI_TRY(y_passes(c, false, yv, tb.t[1], s));
  // a11 nonlinear term quasi.cpp:1905-1939
  NonlinearStage<T> n{};
  n.v[0] = c.vx; n.v[1] = c.vy; n.v[2] = c.vz; n.p = c.p;
  n.g[0] = c.gx; n.g[1] = c.gy; n.g[2] = c.gz;
  n.base = c.base; n.grad = c.grad; n.mu = c.mu; n.dtpsi = c.dtpsi; n.out = c.Nq;
  n.vqz = c.vqz;
  n.variant = c.variant; n.divv_switch = c.divv_switch; n.nloop = c.nloop;
  QUASI_TRY(launch_nonlinear_stage<T>(g, n, tb.t[2], c.sms, s));
  YBatch<T> yn;
  yn.add(c.Nq);
  QUASI_TRY(y_passes(c, true, yn, tb.t[1], s));
  // a12 update + iCT quasi.cpp:1944-1965, a3 / a4 of the next step quasi.cpp:1036-1232
  return enqueue_update<T>(c, tb, tb64, true, c.psiq_new, c.psi_new, c.law_next, s);
}

// ---------------------------------------------------------------------------
// a14 pre-loop: psiq = scale CT(psi); psi = iCT(psiq); Nq = CT(beta psi^3 - gamma psi^5)
// quasi.cpp:905-951
// ---------------------------------------------------------------------------
template <typename T>
__global__ void init_state_kernel(StepCtx<T> c, size_t n) {
  for (size_t id = blockIdx.x * size_t(blockDim.x) + threadIdx.x; id < n; id += size_t(gridDim.x) * blockDim.x) {
    const double ps = c.psi[id];
    c.psiq_old[id] = c.psiq[id];   // quasi.cpp:939
    c.psi_old[id] = ps;            // quasi.cpp:948
    c.Nq_old[id] = T(c.beta * ps * ps * ps - c.gamma * ps * ps * ps * ps * ps);
    c.divv[id] = c.divvq[id] = T(0);
    c.rhoq[id] = 0.0;
    // grad rho of rho^ = 0
    c.rdx[id] = c.rdy[id] = T(0);
    if constexpr (kStateCopy<T>) c.rdz[id] = T(0);
    else c.law_next[id] = 0.0;
    c.vx[id] = c.vy[id] = c.vz[id] = c.p[id] = T(0);
    c.rho[id] = c.rho_new[id] = c.variant == kQuasi ? 0.0 : 1.0;
  }
}

// The projection psiq = scale CT(psi), psi = iCT(psiq) runs in double in both
// forms (quasi_set_psi leaves the initial psi in c.psi).
template <typename T>
cudaError_t enqueue_init(const StepCtx<T>& c, const AxisTables<T>& tb, const AxisTables<double>& tb64,
                         cudaStream_t s) {
  const size_t n = size_t(c.g.nx) * c.g.ny * c.g.nz;
  QUASI_TRY(cudaMemcpyAsync(c.psiq, c.psi, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  QUASI_TRY(forward3<double>(c, c.psiq, tb64, s, c.scale));
  QUASI_TRY(cudaMemsetAsync(c.nloop, 0, sizeof(int), s));
  QUASI_TRY(enqueue_update<T>(c, tb, tb64, false, c.psiq, c.psi, c.law, s));
  init_state_kernel<T><<<592, 256, 0, s>>>(c, n);
  QUASI_TRY(cudaGetLastError());
  return forward3<T>(c, c.Nq_old, tb, s);
}

// The spectra that a step expects, from a loaded state (psiq, rhoq).
template <typename T>
cudaError_t enqueue_resume(const StepCtx<T>& c, const AxisTables<T>& tb, const AxisTables<double>& tb64,
                           cudaStream_t s) {
  if (c.variant == kQuasi)
    QUASI_TRY(enqueue_density<T>(c, tb, tb64, true, c.law_next, c.rdx, c.rdy, c.rdz, s));
  return enqueue_update<T>(c, tb, tb64, false, c.psiq, c.psi, c.law, s);
}

// double field -> storage type (the float copies a checkpoint holds)
template <typename T>
__global__ void to_storage_kernel(const double* src, T* dst, size_t n) {
  for (size_t id = blockIdx.x * size_t(blockDim.x) + threadIdx.x; id < n; id += size_t(gridDim.x) * blockDim.x)
    dst[id] = T(src[id]);
}

}  // namespace quasi
