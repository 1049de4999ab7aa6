// Dispatch of the local H|psi>: each of the three kernels by its own dimensions to the form compiled for
// them, else to the run-time forms.
#include "hkpsi_kernels.cuh"

namespace cpwb {

// square planes (with their y tile, plane_tile) and line lengths with a compiled form (hkpsi_planes_*.cu,
// hkpsi_lines_*.cu)
#define CPWB_FOR_PLANES(X) X(4, 8, 32) X(5, 8, 40) X(8, 12, 32) X(12, 12, 32)
#define CPWB_FOR_LINES(X)                                                                              \
  X(4, 4) X(3, 6) X(4, 5) X(4, 6) X(4, 8) X(6, 6) X(5, 8) X(6, 8) X(5, 10) X(6, 9) X(8, 8) X(8, 9)     \
  X(8, 10) X(8, 12) X(10, 10) X(9, 12) X(8, 16) X(12, 12) X(10, 16) X(12, 16) X(16, 16)

#define CPWB_DECLARE(R1, R2, TC) CPWB_PLANES(extern, double, R1, R2, TC) CPWB_PLANES(extern, float, R1, R2, TC)
CPWB_FOR_PLANES(CPWB_DECLARE)
#undef CPWB_DECLARE
CPWB_PLANES(extern, double, 0, 0, 0)
CPWB_PLANES(extern, float, 0, 0, 0)
#define CPWB_DECLARE(R1, R2) \
  CPWB_LINES(extern, double, R1, R2) CPWB_LINES(extern, float, R1, R2) CPWB_DENSITY(extern, R1, R2)
CPWB_FOR_LINES(CPWB_DECLARE)
#undef CPWB_DECLARE

static bool is_split(const FftDim& d, int r1, int r2) { return d.r1 == r1 && d.r2 == r2; }
static bool square(const LocalPlan& p, int r1, int r2, int tc) {
  return p.tcol == tc && is_split(p.dx, r1, r2) && is_split(p.dy, r1, r2);
}

template <typename T>
cudaError_t launch_inverse_xy(CPWB_INV_ARGS(T)) {
#define CPWB_TRY(R1, R2, TC)                                                                                   \
  if (square(p, R1, R2, TC))                                                                                    \
    return kern::launch_a_impl<T, R1, R2, R1, R2, TC>(p, nbc, band0, psi, ldpsi, plane_start, pw_idx, pw_pos,  \
                                                      twx, twy, W, st);
  CPWB_FOR_PLANES(CPWB_TRY)
#undef CPWB_TRY
  return kern::launch_a_impl<T, 0, 0, 0, 0, 0>(p, nbc, band0, psi, ldpsi, plane_start, pw_idx, pw_pos, twx, twy, W,
                                               st);
}
template cudaError_t launch_inverse_xy<double>(CPWB_INV_ARGS(double));
template cudaError_t launch_inverse_xy<float>(CPWB_INV_ARGS(float));

template <typename T>
cudaError_t launch_forward_xy(CPWB_C_ARGS(T)) {
#define CPWB_TRY(R1, R2, TC)                                                                                    \
  if (square(p, R1, R2, TC))                                                                                     \
    return kern::launch_c_impl<T, R1, R2, R1, R2, TC>(p, nbc, band0, psi, ldpsi, hpsi, ldh, plane_start, pw_idx, \
                                                      pw_pos, ekpg, twx, twy, W, st);
  CPWB_FOR_PLANES(CPWB_TRY)
#undef CPWB_TRY
  return kern::launch_c_impl<T, 0, 0, 0, 0, 0>(p, nbc, band0, psi, ldpsi, hpsi, ldh, plane_start, pw_idx, pw_pos,
                                               ekpg, twx, twy, W, st);
}
template cudaError_t launch_forward_xy<double>(CPWB_C_ARGS(double));
template cudaError_t launch_forward_xy<float>(CPWB_C_ARGS(float));

// Kernel B: the register form where the kept planes lie in the outer quarters of the lines and the length
// is compiled, else the staged form, else (its shared memory does not fit) the plain one.
template <typename T>
static cudaError_t launch_z(const LocalPlan& p, int nbc, const T* vr, const C2<T>* twz, C2<T>* W, cudaStream_t st) {
  int nsm = 148, dev = 0, smax = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (in_quarters(p.kd3, p.dz.r1, p.dz.r2)) {
#define CPWB_TRY(R1, R2) \
  if (is_split(p.dz, R1, R2)) return kern::launch_z_impl<T, R1, R2>(p, nbc, vr, twz, W, nsm, st);
    CPWB_FOR_LINES(CPWB_TRY)
#undef CPWB_TRY
  }
  cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  const size_t sm_pipe = kern::smem_columns_pipe<T>(p, p.cb);
  const long long tiles = (p.plane + p.cb - 1) / p.cb;
  cudaError_t e;
  if (sm_pipe > (size_t)smax) {
    const size_t sm_co = smem_columns<T>(p);
    auto* kb = kern::k_z_vloc<T>;
    if ((e = smem_limit((const void*)kb, sm_co)) != cudaSuccess) return e;
    kb<<<dim3((unsigned)tiles, nbc), kern::kThreadsCols, sm_co, st>>>(p, vr, twz, W);
  } else {
    auto* kb = kern::k_z_vloc_pipe<T>;
    if ((e = smem_limit((const void*)kb, sm_pipe)) != cudaSuccess) return e;
    const int g = kern::band_groups(p, tiles, nbc, nsm), per = (nbc + g - 1) / g;
    kb<<<dim3((unsigned)tiles, (unsigned)((nbc + per - 1) / per)), kern::kThreadsCols, sm_pipe, st>>>(p, nbc, per, vr,
                                                                                                 twz, W);
  }
  return cudaGetLastError();
}

bool has_line_form(const LocalPlan& p) {
  if (!in_quarters(p.kd3, p.dz.r1, p.dz.r2)) return false;
#define CPWB_TRY(R1, R2) \
  if (is_split(p.dz, R1, R2)) return true;
  CPWB_FOR_LINES(CPWB_TRY)
#undef CPWB_TRY
  return false;
}

cudaError_t launch_density_z(const LocalPlan& p, int nbc, int groups, const double* occ, const C2<double>* twz,
                             const C2<double>* W, double* rho, double* part, cudaStream_t st) {
#define CPWB_TRY(R1, R2) \
  if (is_split(p.dz, R1, R2)) return kern::launch_density_impl<R1, R2>(p, nbc, groups, occ, twz, W, rho, part, st);
  CPWB_FOR_LINES(CPWB_TRY)
#undef CPWB_TRY
  return cudaErrorInvalidValue;
}

template <typename T>
cudaError_t launch_spinor_z(const LocalPlan& p, int nbc, const T* vu, const T* vd, const T* vr, const T* vi,
                            const C2<T>* twz, C2<T>* W, cudaStream_t st) {
  int nsm = 148, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
#define CPWB_TRY(R1, R2) \
  if (is_split(p.dz, R1, R2)) return kern::launch_spinor_impl<T, R1, R2>(p, nbc, vu, vd, vr, vi, twz, W, nsm, st);
  CPWB_FOR_LINES(CPWB_TRY)
#undef CPWB_TRY
  return cudaErrorInvalidValue;
}
#define CPWB_SPINOR(T)                                                                                      \
  template cudaError_t launch_spinor_z<T>(const LocalPlan&, int, const T*, const T*, const T*, const T*,    \
                                          const C2<T>*, C2<T>*, cudaStream_t);
CPWB_SPINOR(double)
CPWB_SPINOR(float)

template <typename T>
cudaError_t launch_local(const LocalPlan& p, int nbc, int band0, const C2<double>* psi, long long ldpsi,
                         C2<double>* hpsi, long long ldh, const int* plane_start, const int* pw_idx,
                         const int* pw_pos, const double* ekpg, const T* vr, const C2<T>* twx, const C2<T>* twy,
                         const C2<T>* twz, C2<T>* W, cudaStream_t st, cudaEvent_t* ev) {
  cudaError_t e;
  if (ev) cudaEventRecord(ev[0], st);
  if ((e = launch_inverse_xy<T>(p, nbc, band0, psi, ldpsi, plane_start, pw_idx, pw_pos, twx, twy, W, st)) != cudaSuccess)
    return e;
  if (ev) cudaEventRecord(ev[1], st);
  if ((e = launch_z<T>(p, nbc, vr, twz, W, st)) != cudaSuccess) return e;
  if (ev) cudaEventRecord(ev[2], st);
  e = launch_forward_xy<T>(p, nbc, band0, psi, ldpsi, hpsi, ldh, plane_start, pw_idx, pw_pos, ekpg, twx, twy, W, st);
  if (ev) cudaEventRecord(ev[3], st);
  return e;
}
#define CPWB_LOCAL(T)                                                                                              \
  template cudaError_t launch_local<T>(const LocalPlan&, int, int, const C2<double>*, long long, C2<double>*,       \
                                       long long, const int*, const int*, const int*, const double*, const T*,     \
                                       const C2<T>*, const C2<T>*, const C2<T>*, C2<T>*, cudaStream_t, cudaEvent_t*);
CPWB_LOCAL(double)
CPWB_LOCAL(float)

}  // namespace cpwb
