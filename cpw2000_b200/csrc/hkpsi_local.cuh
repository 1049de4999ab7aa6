// Local part of H|psi>: G-sphere scatter, pruned inverse 3D FFT, V_loc(r)
// multiply, pruned forward 3D FFT, gather and kinetic diagonal, for a chunk
// of bands. Restates the per-band loop of Src/hk_psi/reference/hk_psi_c16.f90
// (:176-223) with the Goedecker pruning of Src/fft/_cfft/cfft_wf_c16.f
// (:110-410), re-organised for the GPU as three kernels per band chunk:
//
//   A  one CTA per (band, kept z-plane): scatter the plane's coefficients
//      into shared memory, inverse FFT along x on the 2kd2+1 kept rows,
//      inverse FFT along y on every column, write the plane to the slab W.
//   B  one CTA per (run of xy columns, group of bands): inverse FFT along z of the
//      2kd3+1 kept planes, multiply by V(r)/N, forward FFT along z, keep the
//      2kd3+1 planes. The inverse's second pass, the multiply and the
//      forward's first pass share registers.
//   C  one CTA per (band, kept z-plane): forward FFT along y keeping the kept
//      rows, forward FFT along x, gather the sphere, add ekpg*psi.
//
// Slab W layout: [band][zi][y][x storage] (x fastest), zi = compact index of the
// kept z planes; x is stored in the order the inverse's second pass leaves it in
// (slab_column), so that A writes and C reads whole rows. Every 1D transform of
// length n = r1*r2 is two register passes with one shared-memory exchange
// (four-step), twiddles W_n^k from a table in shared memory. Kernels A and C are
// compiled for the square planes in use, B for every line length, each by itself:
// a box whose lengths differ still runs B's compiled form.
#pragma once
#include <stdlib.h>

#include <map>
#include <mutex>
#include <utility>

#include "cplx.cuh"

namespace cpwb {

// Raise, never lower, the dynamic shared memory a kernel may take. Function attributes are
// process-wide: host threads that launch one kernel with different sizes (contexts of different
// k-points in flight) must not lower each other's limit between the setting and the launch.
inline cudaError_t smem_limit(const void* f, size_t bytes) {
  static std::mutex mu;
  static std::map<std::pair<int, const void*>, size_t> cur;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(mu);
  size_t& v = cur[{dev, f}];
  if (bytes <= v) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) v = bytes;
  return e;
}

struct FftDim {
  int n, r1, r2;
};

// One k-point of a batch: its wavefunction blocks, its plane lists (relative to the
// batch's common kept planes and rows) and its kinetic diagonal.
struct KDesc {
  const C2<double>* psi;
  C2<double>* hpsi;
  long long ldpsi, ldh;
  const int* plane_start;
  const int* pw_idx;
  const int* pw_pos;
  const double* ekpg;     // null: no kinetic term
};

struct LocalPlan {
  // batch mode (null for one k-point): global band b of a launch is band bref[b].y of
  // k-point bref[b].x, described by kdesc[bref[b].x]; the per-call pointer arguments
  // of kernels A and C are then ignored
  const KDesc* kdesc;
  const int2* bref;
  int bgroups;            // kernel B band grouping: 0 = heuristic, else target CTAs per SM
  int n1, n2, n3;         // FFT box
  int kd1, kd2, kd3;      // sphere half-widths (largest |k_j| of the basis)
  int nx, ny, nz;         // 2*kd+1
  FftDim dx, dy, dz;
  int rowp;               // shared-memory row stride (complex elements) in A/C
  int tcol;               // columns per batch in the y passes of A/C
  int cb;                 // columns per CTA in B
  long long plane;        // n1*n2
  int accum;              // kernel C adds its result to hpsi instead of storing it (ladd)
};

__host__ __device__ __forceinline__ int kept_to_idx(int i, int kd, int n, int nk) {
  return i <= kd ? i : n - nk + i;
}
__host__ __device__ __forceinline__ int idx_to_kept(int z, int kd, int n, int nk) {
  return z <= kd ? z : (z >= n - kd ? z - (n - nk) : -1);
}

// The column y * n1 + x of the box that column c of the slab holds: storage position r2 k1 + k2 of a
// row is x = k1 + r1 k2.
__host__ __device__ __forceinline__ int slab_column(const LocalPlan& p, long long c) {
  const int y = (int)c / p.n1, pp = (int)c - y * p.n1, k1 = pp / p.dx.r2;
  return y * p.n1 + k1 + p.dx.r1 * (pp - k1 * p.dx.r2);
}

// The storage position of natural index x in a row of the slab.
__host__ __device__ __forceinline__ int slab_slot(int x, int r1, int r2) {
  const int q = x / r1;
  return r2 * (x - q * r1) + q;
}

// Shared-memory footprint in bytes of kernels A/C and B; esz is the size of one complex element.
inline size_t plane_smem_bytes(size_t esz, const LocalPlan& p) {
  return esz * ((size_t)p.ny * p.rowp + (size_t)p.n2 * p.tcol + p.n1 + p.n2);
}
template <typename T> inline size_t smem_planes(const LocalPlan& p) { return plane_smem_bytes(sizeof(C2<T>), p); }
// Columns per y tile of kernels A/C: 32, or fewer and equal tiles of at most 40 where the last one of 32
// would be at most a quarter full (every tile costs four barrier-separated phases: 40 columns in one
// tile, 72 in two of 36; 144 stay with 32, since four of 36 made C 4-8 % slower: a warp's columns
// straddle two rows). 16, 8, 4 while the plane does not fit the shared memory of a CTA; false when it
// does not fit at all.
inline bool plane_tile(size_t esz, LocalPlan& p, size_t smem_block) {
  const int tiles = (p.n1 + 39) / 40, tail = p.n1 % 32;
  p.tcol = tail > 0 && tail <= 8 && p.n1 > 32 ? ((p.n1 + tiles - 1) / tiles + 3) / 4 * 4 : 32;
  while (p.tcol > 4 && plane_smem_bytes(esz, p) > smem_block) p.tcol = p.tcol > 32 ? 32 : p.tcol / 2;
  return plane_smem_bytes(esz, p) <= smem_block;
}
template <typename T> inline size_t smem_columns(const LocalPlan& p) {
  return sizeof(C2<T>) * ((size_t)p.n3 * p.cb + p.n3);
}
// Staged (pipelined) form of kernel B: a column tile, two kept-plane buffers, the z-twiddles
// and the potential columns; esz is the size of one complex element.
inline size_t smem_columns_pipe_bytes(size_t esz, const LocalPlan& p, int cb) {
  return esz * ((size_t)p.n3 * cb + 2 * (size_t)p.nz * cb + p.n3) + esz / 2 * (size_t)p.n3 * cb;
}
// Column tile of kernel B's run-time forms: 32 columns on short columns, 16 on columns of 128 points or
// more and wherever the staged form would leave room for only one CTA per SM. The tile is then
// halved while even the plain form does not fit.
inline int column_tile(size_t esz, const LocalPlan& p, size_t smem_block, size_t smem_sm) {
  int cb = 32;
  if (p.n3 >= 128 || 2 * (smem_columns_pipe_bytes(esz, p, cb) + 1024) > smem_sm) cb = 16;
  while (cb > 4 && esz * ((size_t)p.n3 * cb + p.n3) > smem_block) cb /= 2;
  return cb;
}

// Launch the three kernels for bands [band0, band0+nbc). psi/hpsi are
// complex128 column-major with leading dimensions ldpsi/ldh. W holds nbc
// slabs. ekpg may be null (no kinetic term). If ev is not null, ev[0..3] are
// recorded before A, after A, after B and after C (stage timers). Returns a
// cudaError_t.
template <typename T>
cudaError_t launch_local(const LocalPlan& p, int nbc, int band0, const C2<double>* psi, long long ldpsi,
                         C2<double>* hpsi, long long ldh, const int* plane_start, const int* pw_idx,
                         const int* pw_pos, const double* ekpg, const T* vr, const C2<T>* twx,
                         const C2<T>* twy, const C2<T>* twz, C2<T>* W, cudaStream_t st,
                         cudaEvent_t* ev = nullptr);

// Kernel A alone for bands [band0, band0+nbc): the kept z-planes of every band,
// inverse-transformed in x and y, into W (density / adjoint path).
template <typename T>
cudaError_t launch_inverse_xy(const LocalPlan& p, int nbc, int band0, const C2<double>* psi, long long ldpsi,
                              const int* plane_start, const int* pw_idx, const int* pw_pos, const C2<T>* twx,
                              const C2<T>* twy, C2<T>* W, cudaStream_t st);

// Kernel C alone for bands [band0, band0+nbc) from W.
template <typename T>
cudaError_t launch_forward_xy(const LocalPlan& p, int nbc, int band0, const C2<double>* psi, long long ldpsi,
                              C2<double>* hpsi, long long ldh, const int* plane_start, const int* pw_idx,
                              const int* pw_pos, const double* ekpg, const C2<T>* twx, const C2<T>* twy,
                              const C2<T>* W, cudaStream_t st);

// The register forms of the z stages exist for the plan's z lines (compiled length, kept planes in the
// outer quarters of the line). Only then may the next two be called:
bool has_line_form(const LocalPlan& p);
// the density's (groups band groups; part: a box each when there are several, else null and rho is added to)
cudaError_t launch_density_z(const LocalPlan& p, int nbc, int groups, const double* occ, const C2<double>* twz,
                             const C2<double>* W, double* rho, double* part, cudaStream_t st);
// the non-collinear one (down slabs nbc slabs after the up slabs)
template <typename T>
cudaError_t launch_spinor_z(const LocalPlan& p, int nbc, const T* vu, const T* vd, const T* vr, const T* vi,
                            const C2<T>* twz, C2<T>* W, cudaStream_t st);

}  // namespace cpwb
