// Adjoint of H|psi> for fixed wavefunctions (Hellmann-Feynman):
//
//  * density      rho(r) = sum_n f_n |psi_n(r)|^2 on the FFT box, with psi_n(r) the
//                 unscaled backward transform -- what Src/omp/charge_by_fft.f90
//                 (:185-199) accumulates; rho/N is dE/dV(r) for E = sum_n f_n <psi_n|H|psi_n>.
//  * local term   dE/dtau_aj = sum_r g(r) dV(r)/dtau_aj for V(r) = sum_G V(G) e^{iG.r},
//                 V(G) = sum_a e^{-2 pi i m.tau_a} v_t(G); with FG = sum_r g e^{-iG.r}:
//                 dE/dtau_aj = Re sum_G (-2 pi i m_j) e^{-2 pi i m.tau_a} v_t(G) conj(FG(G))
//                 (the structure-factor derivative of Src/ALFA/for_str_local_force.f90:102-145).
//  * KB term      P = X^H psi, Y = psi diag(f) P^H; dE/dtau_aj = -4 pi
//                 sum_{projectors of a} xnlkb Im sum_G conj(X) G_j Y -- the dhd(1..4) products of
//                 Src/ALFA/for_str_nl_kb.f90:289-362 written with the projectors of
//                 proj_nl_kb_c16 (d/dtau of e^{-2 pi i G.tau} is -2 pi i G), the bands summed first.
// Positions tau are lattice coordinates; derivatives are covariant (per lattice
// coordinate). Band-block recomputation: the density recomputes psi(r) chunk by
// chunk through the slab, nothing real-space is kept between calls.
#include <cufft.h>
#include <math.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "../../include/cpw_b200.h"
#include "context.hpp"

namespace cpwb {
namespace {

using Z = cuDoubleComplex;
constexpr int kDensThreads = 256;
constexpr int kDensCB = 32;

// rho += the band groups' boxes, in order
__global__ void k_add_boxes(long long n, int groups, const double* __restrict__ part, double* __restrict__ rho) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    double s = rho[t];
    for (int g = 0; g < groups; ++g) s += part[(size_t)g * n + t];
    rho[t] = s;
  }
}

// Run-time form of the density's z stage (line lengths without a compiled one, hkpsi_kernels.cuh): inverse z
// of the kept planes of every band of the chunk, |.|^2 accumulated with
// the band weights; one CTA per 32 xy-columns; rho += the chunk's contribution
__global__ void __launch_bounds__(kDensThreads)
k_dens_z(LocalPlan p, int nbc, const double* __restrict__ occ, const C2<double>* __restrict__ twz,
         const C2<double>* __restrict__ W, double* __restrict__ rho) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int cb = kDensCB, n3 = p.n3, r1 = p.dz.r1, r2 = p.dz.r2;
  C2<double>* Cs = reinterpret_cast<C2<double>*>(smem_raw);
  double* acc = reinterpret_cast<double*>(Cs + (size_t)n3 * cb);
  C2<double>* sz = reinterpret_cast<C2<double>*>(acc + (size_t)n3 * cb);
  const long long c0 = (long long)blockIdx.x * cb;
  const int ncol = (int)min((long long)cb, p.plane - c0);
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < n3; i += nt) sz[i] = twz[i];
  for (int i = tid; i < n3 * cb; i += nt) acc[i] = 0.0;
  for (int b = 0; b < nbc; ++b) {
    const C2<double>* Wb = W + (size_t)b * p.nz * (size_t)p.plane + c0;
    const double f = occ[b];
    __syncthreads();
    for (int it = tid; it < cb * p.nz; it += nt) {
      const int cl = it % cb, zi = it / cb;
      if (cl < ncol) Cs[(size_t)kept_to_idx(zi, p.kd3, n3, p.nz) * cb + cl] = Wb[(size_t)zi * p.plane + cl];
    }
    __syncthreads();
    for (int it = tid; it < cb * r2; it += nt) {
      const int cl = it % cb, n2i = it / cb;
      if (cl < ncol) {
        radix_dispatch(r1, [&](auto rc_) {
          constexpr int RR = decltype(rc_)::value;
          C2<double> v[RR];
#pragma unroll
          for (int a = 0; a < RR; ++a) {
            const int z = r2 * a + n2i;
            v[a] = idx_to_kept(z, p.kd3, n3, p.nz) >= 0 ? Cs[(size_t)z * cb + cl] : mk<double>(0.0, 0.0);
          }
          DFT<RR, +1, double>::run(v);
#pragma unroll
          for (int a = 0; a < RR; ++a)
            Cs[(size_t)(r2 * a + n2i) * cb + cl] = a == 0 ? v[0] : cmulc<double>(v[a], sz[n2i * a]);
        });
      }
    }
    __syncthreads();
    for (int it = tid; it < cb * r1; it += nt) {
      const int cl = it % cb, k1 = it / cb;
      if (cl < ncol) {
        radix_dispatch(r2, [&](auto rc_) {
          constexpr int RR = decltype(rc_)::value;
          C2<double> v[RR];
#pragma unroll
          for (int a = 0; a < RR; ++a) v[a] = Cs[(size_t)(r2 * k1 + a) * cb + cl];
          DFT<RR, +1, double>::run(v);
#pragma unroll
          for (int a = 0; a < RR; ++a) acc[(size_t)(k1 + r1 * a) * cb + cl] += f * (v[a].x * v[a].x + v[a].y * v[a].y);
        });
      }
    }
  }
  __syncthreads();
  for (int it = tid; it < cb * n3; it += nt) {
    const int cl = it % cb, z = it / cb;
    if (cl < ncol) rho[(size_t)z * p.plane + slab_column(p, c0 + cl)] += acc[(size_t)z * cb + cl];
  }
}

__device__ __forceinline__ double block_sum3(double v, double* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  }
  return v;   // valid in thread 0
}

__device__ __forceinline__ int freq(int i, int n) { return i <= (n - 1) / 2 ? i : i - n; }

// dE/dtau_aj = Re sum_G (-2 pi i m_j) e^{-2 pi i m.tau_a} v_t(G) conj(FG(G)) = 2 pi sum_G m_j Im(w),
// w = px(m1) py(m2) pz(m3) c(G), c = v_t conj(FG). A CTA takes kSgRows rows (y, z) of the box for a tile of
// kSgAtoms atoms of one species: it stages c of its rows in shared memory, a thread contracts its atom's
// phases px with four rows at a time (S0 = sum px c, S1 = sum m1 px c: 8 FMAs for one broadcast load) and
// multiplies the row sums by py pz. Bound: FP64 FMAs, 8 per point and atom. (One CTA per atom that walked
// the whole box took 2.8 ms for 64 atoms on a 96^3 box, on 64 of the SMs; this takes 65 us.)
constexpr int kSgAtoms = 32, kSgGroups = 8, kSgQuad = 4, kSgRows = kSgGroups * kSgQuad;

// phases e^{-2 pi i m tau} of every atom slot: tab[axis offset + i][slots]; slots beyond the tile's atoms are
// zero
__global__ void k_sg_phases(int n1, int n2, int n3, int slots, const int* __restrict__ atom_of,
                            const double* __restrict__ tau, Z* __restrict__ tab) {
  const int n = n1 + n2 + n3;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n * slots; t += gridDim.x * blockDim.x) {
    const int sl = t % slots, i = t / slots, a = atom_of[sl];
    const int axis = i < n1 ? 0 : i < n1 + n2 ? 1 : 2;
    const int k = axis == 0 ? freq(i, n1) : axis == 1 ? freq(i - n1, n2) : freq(i - n1 - n2, n3);
    double c = 0.0, s = 0.0;
    if (a >= 0) sincospi(-2.0 * k * tau[3 * a + axis], &s, &c);
    tab[t] = make_cuDoubleComplex(c, s);
  }
}

__global__ void __launch_bounds__(kSgAtoms* kSgGroups)
k_structure_grad(int n1, int n2, int n3, int slots, const Z* __restrict__ FG, const double* __restrict__ vgt,
                 const int* __restrict__ tile_type, const Z* __restrict__ tab, double* __restrict__ part) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Z* cs = reinterpret_cast<Z*>(smem_raw);                 // kSgRows x n1
  const int tid = threadIdx.x, at = tid % kSgAtoms, grp = tid / kSgAtoms;
  const long long rows = (long long)n2 * n3, r0 = (long long)blockIdx.x * kSgRows;
  const int nr = (int)min((long long)kSgRows, rows - r0);
  const double* v = vgt + (size_t)tile_type[blockIdx.y] * rows * n1;
  for (int i = tid; i < kSgRows * n1; i += kSgAtoms * kSgGroups) {
    Z c = make_cuDoubleComplex(0.0, 0.0);
    if (i < nr * n1) {
      const double vt = v[r0 * n1 + i];
      if (vt != 0.0) {
        const Z f = FG[r0 * n1 + i];
        c = make_cuDoubleComplex(vt * f.x, -vt * f.y);
      }
    }
    cs[i] = c;
  }
  __syncthreads();
  const int sl = blockIdx.y * kSgAtoms + at;
  Z s0[kSgQuad], s1[kSgQuad];
#pragma unroll
  for (int q = 0; q < kSgQuad; ++q) s0[q] = s1[q] = make_cuDoubleComplex(0.0, 0.0);
  const Z* c = cs + (size_t)grp * kSgQuad * n1;
#pragma unroll 2
  for (int x = 0; x < n1; ++x) {
    const Z p = tab[(size_t)x * slots + sl];
    const double m = freq(x, n1);
    const Z mp = make_cuDoubleComplex(m * p.x, m * p.y);
#pragma unroll
    for (int q = 0; q < kSgQuad; ++q) {
      const Z u = c[q * n1 + x];
      s0[q].x = fma(p.x, u.x, fma(-p.y, u.y, s0[q].x));
      s0[q].y = fma(p.x, u.y, fma(p.y, u.x, s0[q].y));
      s1[q].x = fma(mp.x, u.x, fma(-mp.y, u.y, s1[q].x));
      s1[q].y = fma(mp.x, u.y, fma(mp.y, u.x, s1[q].y));
    }
  }
  double g[3] = {0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < kSgQuad; ++q) {
    const long long r = r0 + grp * kSgQuad + q;
    if (r < rows) {
      const int y = (int)(r % n2), z = (int)(r / n2);
      const Z ph = cuCmul(tab[(size_t)(n1 + y) * slots + sl], tab[(size_t)(n1 + n2 + z) * slots + sl]);
      const double w0 = ph.x * s0[q].y + ph.y * s0[q].x;
      g[0] += ph.x * s1[q].y + ph.y * s1[q].x;
      g[1] += freq(y, n2) * w0;
      g[2] += freq(z, n3) * w0;
    }
  }
  __syncthreads();
  double* red = reinterpret_cast<double*>(smem_raw);      // [group][axis][atom]
  for (int k = 0; k < 3; ++k) red[(grp * 3 + k) * kSgAtoms + at] = g[k];
  __syncthreads();
  if (grp < 3) {
    double t = 0.0;
    for (int w = 0; w < kSgGroups; ++w) t += red[(w * 3 + grp) * kSgAtoms + at];
    part[((size_t)blockIdx.x * 3 + grp) * slots + sl] = t;
  }
}

// out(a, j) = 2 pi sum of the row chunks' parts, one warp per (slot, axis), in a fixed order
__global__ void k_sg_sum(int chunks, int slots, const int* __restrict__ atom_of, const double* __restrict__ part,
                         double* __restrict__ out) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x & 31;
  if (w >= 3 * slots) return;
  const int sl = w / 3, j = w % 3, a = atom_of[sl];
  double t = 0.0;
  for (int c = lane; c < chunks; c += 32) t += part[((size_t)c * 3 + j) * slots + sl];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0 && a >= 0) out[3 * a + j] = 6.283185307179586476925286766559005768 * t;
}

__global__ void k_to_complex(long long n, const double* __restrict__ g, Z* __restrict__ z) {
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    z[t] = make_cuDoubleComplex(g[t], 0.0);
}

// c[slice][a][j] = sum_i Im(conj(X_ia) Y_ia) G_ij over the slice's plane waves, one CTA per projector and slice
__global__ void __launch_bounds__(256) k_nl_contract(int m, const int* __restrict__ kgvb, const Z* __restrict__ X,
                                                     const Z* __restrict__ Y, double* __restrict__ c, int nanl) {
  const int a = blockIdx.x, rows = (m + gridDim.y - 1) / gridDim.y;
  const int i1 = min(m, ((int)blockIdx.y + 1) * rows);
  __shared__ double sh[32];
  double s[3] = {0, 0, 0};
  const Z* x = X + (size_t)a * m;
  const Z* y = Y + (size_t)a * m;
#pragma unroll 2
  for (int i = blockIdx.y * rows + threadIdx.x; i < i1; i += 256) {
    const Z p = x[i], q = y[i];
    const double w = p.x * q.y - p.y * q.x;
    s[0] += w * kgvb[3 * i];
    s[1] += w * kgvb[3 * i + 1];
    s[2] += w * kgvb[3 * i + 2];
  }
  for (int j = 0; j < 3; ++j) {
    const double t = block_sum3(s[j], sh);
    if (threadIdx.x == 0) c[3 * ((size_t)blockIdx.y * nanl + a) + j] = t;
  }
}

// w(i) = sum_n f_n |c_n(i)|^2 (the kinetic stress weight of plane wave i)
__global__ void k_band_weights(int m, int nb, const Z* __restrict__ psi, long long ld, const double* __restrict__ f,
                               double* __restrict__ w) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int n = 0; n < nb; ++n) {
      const Z c = psi[(size_t)n * ld + i];
      s += f[n] * (c.x * c.x + c.y * c.y);
    }
    w[i] = s;
  }
}

// M(n, a) = f_n conj(P(a, n)) xnlkb(a) (xnl null: without the last factor), M (nb x nanl) column-major
__global__ void k_stress_m(int nanl, int nb, const Z* __restrict__ P, const double* __restrict__ f,
                           const double* __restrict__ xnl, Z* __restrict__ M) {
  const long long n = (long long)nanl * nb;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x) {
    const int a = (int)(t / nb), b = (int)(t - (long long)a * nb);
    const Z p = P[(size_t)b * nanl + a];
    const double s = xnl ? f[b] * xnl[a] : f[b];
    M[(size_t)a * nb + b] = make_cuDoubleComplex(s * p.x, -s * p.y);
  }
}

}  // namespace

// The two blocks the strain derivative of E = sum_n f_n <psi_n|H|psi_n> needs besides the
// density: w(i) = sum_n f_n |c_n(i)|^2 (kinetic) and Y = psi diag(f) P^H diag(xnlkb)
// (mtxd x nanl, KB term: dE = 2 Re sum conj(dX) Y for a change dX of the projectors).
int stress_inputs_device(cpw_b200_ctx* c, int nb, const void* psi, long long ldpsi, const double* occ, double* w,
                         void* y, cudaStream_t st) {
  if (!c->have_basis) return fail(kNotReady, "stress inputs: basis must be set");
  const int na = c->nanl, m = c->mtxd;
  if (nb < 0 || ldpsi < m) return fail(kBadArg, "stress inputs: invalid block");
  if (m == 0) return kOk;
  int s;
  DevBuf P, M, docc, dxnl;
  if ((s = docc.ensure(sizeof(double) * std::max(nb, 1)))) return s;
  cudaError_t e;
  if (nb > 0 && (e = cudaMemcpyAsync(docc.p, occ, sizeof(double) * nb, cudaMemcpyHostToDevice, st)) != cudaSuccess)
    return cuda_fail(e, "stress inputs occ");
  if (nb == 0) {
    if ((e = cudaMemsetAsync(w, 0, sizeof(double) * m, st)) != cudaSuccess) return cuda_fail(e, "stress inputs");
  } else {
    k_band_weights<<<std::min(1184, (m + 255) / 256), 256, 0, st>>>(m, nb, (const Z*)psi, ldpsi,
                                                                   (const double*)docc.p, w);
  }
  if (na > 0) {
    if (nb == 0) {
      if ((e = cudaMemsetAsync(y, 0, sizeof(Z) * (size_t)m * na, st)) != cudaSuccess) return cuda_fail(e, "stress");
    } else {
      if ((s = P.ensure(sizeof(Z) * (size_t)na * nb)) || (s = M.ensure(sizeof(Z) * (size_t)na * nb)) ||
          (s = dxnl.ensure(sizeof(double) * na)))
        return s;
      if ((e = cudaMemcpyAsync(dxnl.p, c->xnl_h.data(), sizeof(double) * na, cudaMemcpyHostToDevice, st)) !=
          cudaSuccess)
        return cuda_fail(e, "stress inputs xnlkb");
      cublasSetStream(c->blas, st);
      const Z one = make_cuDoubleComplex(1, 0), zero = make_cuDoubleComplex(0, 0);
      cublasStatus_t bs = cublasZgemm(c->blas, CUBLAS_OP_C, CUBLAS_OP_N, na, nb, m, &one, (const Z*)c->anl.p, m,
                                      (const Z*)psi, (int)ldpsi, &zero, (Z*)P.p, na);
      if (bs != CUBLAS_STATUS_SUCCESS) return fail(kCublas, "stress inputs zgemm P");
      k_stress_m<<<std::max(1, std::min(1184, (na * nb + 255) / 256)), 256, 0, st>>>(
          na, nb, (const Z*)P.p, (const double*)docc.p, (const double*)dxnl.p, (Z*)M.p);
      bs = cublasZgemm(c->blas, CUBLAS_OP_N, CUBLAS_OP_N, m, na, nb, &one, (const Z*)psi, (int)ldpsi, (const Z*)M.p,
                       nb, &zero, (Z*)y, m);
      if (bs != CUBLAS_STATUS_SUCCESS) return fail(kCublas, "stress inputs zgemm Y");
    }
  }
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return cuda_fail(e, "stress inputs");
  return kOk;
}

int density_device(cpw_b200_ctx* c, int nb, const void* psi, long long ldpsi, const double* occ, void* rho,
                   cudaStream_t st) {
  if (!c->have_basis) return fail(kNotReady, "density: basis must be set");
  if (nb < 0 || ldpsi < c->mtxd) return fail(kBadArg, "density: bad neig or leading dimension");
  LocalPlan p = c->plan;
  // the y tile of a context with FP32 transforms was fitted for their element size
  int smax = 0;
  cudaDeviceGetAttribute(&smax, cudaDevAttrMaxSharedMemoryPerBlockOptin, c->device);
  if (!plane_tile(sizeof(C2<double>), p, (size_t)smax))
    return fail(kUnsupported, "density: plane does not fit in shared memory");
  cudaError_t e = cudaMemsetAsync(rho, 0, sizeof(double) * (size_t)p.plane * p.n3, st);
  if (e != cudaSuccess) return cuda_fail(e, "density memset");
  if (nb == 0 || c->mtxd == 0) return kOk;
  const size_t per_band = sizeof(C2<double>) * (size_t)p.nz * (size_t)p.plane;
  const int chunk = (int)std::max<size_t>(1, std::min<size_t>((size_t)nb, c->slab_budget / per_band));
  int s;
  if ((s = c->slab.ensure(per_band * (size_t)chunk))) return s;
  // small boxes have few column tiles: their bands are split over groups of CTAs, each with its own box
  const long long box = p.plane * p.n3, tiles = (p.plane + 15) / 16;
  const int groups = has_line_form(p) ? (int)std::max(1LL, std::min<long long>(std::min(chunk, 8), 592 / tiles)) : 1;
  const size_t occ_bytes = (sizeof(double) * (size_t)nb + 255) & ~(size_t)255;
  if ((s = c->adj.ensure(occ_bytes + (groups > 1 ? sizeof(double) * (size_t)groups * box : 0)))) return s;
  const double* docc = (const double*)c->adj.p;
  double* part = groups > 1 ? (double*)((char*)c->adj.p + occ_bytes) : nullptr;
  if ((e = cudaMemcpyAsync(c->adj.p, occ, sizeof(double) * nb, cudaMemcpyHostToDevice, st)) != cudaSuccess)
    return cuda_fail(e, "density occ");
  const size_t sm = (sizeof(C2<double>) + sizeof(double)) * (size_t)p.n3 * kDensCB + sizeof(C2<double>) * p.n3;
  if ((e = smem_limit((const void*)k_dens_z, (size_t)sm)) != cudaSuccess)
    return cuda_fail(e, "density attribute");
  for (int b0 = 0; b0 < nb; b0 += chunk) {
    const int nbc = std::min(chunk, nb - b0);
    e = launch_inverse_xy<double>(p, nbc, b0, (const C2<double>*)psi, ldpsi, (const int*)c->plane_start.p,
                                  (const int*)c->pw_idx.p, (const int*)c->pw_pos.p, (const C2<double>*)c->tw64[0].p,
                                  (const C2<double>*)c->tw64[1].p, (C2<double>*)c->slab.p, st);
    if (e != cudaSuccess) return cuda_fail(e, "density inverse xy");
    if (has_line_form(p)) {
      e = launch_density_z(p, nbc, groups, docc + b0, (const C2<double>*)c->tw64[2].p, (const C2<double>*)c->slab.p,
                           (double*)rho, part, st);
      if (e == cudaSuccess && groups > 1) {
        k_add_boxes<<<1184, 256, 0, st>>>(box, groups, part, (double*)rho);
        e = cudaGetLastError();
      }
      if (e != cudaSuccess) return cuda_fail(e, "density z");
      continue;
    }
    const unsigned grid = (unsigned)((p.plane + kDensCB - 1) / kDensCB);
    k_dens_z<<<grid, kDensThreads, sm, st>>>(p, nbc, docc + b0, (const C2<double>*)c->tw64[2].p,
                                             (const C2<double>*)c->slab.p, (double*)rho);
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(e, "density z");
  }
  e = cudaStreamSynchronize(st);
  return e == cudaSuccess ? kOk : cuda_fail(e, "density");
}

// The context's complex transform of the current box, kept between calls (a plan costs milliseconds).
static int box_plan(cpw_b200_ctx* c, cufftHandle* out) {
  const LocalPlan& p = c->plan;
  const int n[3] = {p.n3, p.n2, p.n1};
  if (!c->fft_plan || memcmp(c->fft_n, n, sizeof n)) {
    adjoint_release(c);
    cufftHandle h;
    if (cufftPlan3d(&h, n[0], n[1], n[2], CUFFT_Z2Z) != CUFFT_SUCCESS) return fail(kCuda, "cufftPlan3d failed");
    c->fft_plan = new cufftHandle(h);
    memcpy(c->fft_n, n, sizeof n);
  }
  *out = *(cufftHandle*)c->fft_plan;
  return kOk;
}

void adjoint_release(cpw_b200_ctx* c) {
  if (!c->fft_plan) return;
  cufftDestroy(*(cufftHandle*)c->fft_plan);
  delete (cufftHandle*)c->fft_plan;
  c->fft_plan = nullptr;
}

int structure_grad_device(cpw_b200_ctx* c, const void* g, int natom, const int* atom_type, const double* tau,
                          int ntype, const void* vgt, double* dedtau, cudaStream_t st) {
  if (!c->have_basis) return fail(kNotReady, "structure gradient: basis (box) must be set");
  const LocalPlan& p = c->plan;
  const long long ntot = (long long)p.n1 * p.n2 * p.n3;
  for (int a = 0; a < natom; ++a)
    if (atom_type[a] < 0 || atom_type[a] >= ntype) return fail(kBadArg, "structure gradient: atom type out of range");
  // tiles of kSgAtoms atoms of one species, padded with empty slots
  std::vector<int> atom_of, tile_type;
  for (int t = 0; t < ntype; ++t) {
    int used = 0;
    for (int a = 0; a < natom; ++a) {
      if (atom_type[a] != t) continue;
      if (used % kSgAtoms == 0) tile_type.push_back(t);
      atom_of.push_back(a);
      ++used;
    }
    while (atom_of.size() % kSgAtoms) atom_of.push_back(-1);
  }
  const int slots = (int)atom_of.size(), tiles = (int)tile_type.size(), nsum = p.n1 + p.n2 + p.n3;
  const int chunks = (int)(((long long)p.n2 * p.n3 + kSgRows - 1) / kSgRows);
  // FG, phases, parts, result, positions, slot and tile lists in the context's buffer
  const size_t o_tab = sizeof(Z) * (size_t)ntot, o_part = o_tab + sizeof(Z) * (size_t)nsum * slots;
  const size_t o_out = o_part + sizeof(double) * 3 * (size_t)chunks * slots;
  const size_t o_tau = o_out + sizeof(double) * 3 * (size_t)natom, o_atom = o_tau + sizeof(double) * 3 * (size_t)natom;
  const size_t o_type = o_atom + sizeof(int) * (size_t)slots;
  int s;
  if ((s = c->adj.ensure(o_type + sizeof(int) * (size_t)tiles + 16))) return s;
  char* base = (char*)c->adj.p;
  Z* fg = (Z*)base;
  cufftHandle plan;
  if ((s = box_plan(c, &plan))) return s;
  k_to_complex<<<1184, 256, 0, st>>>(ntot, (const double*)g, fg);
  cufftSetStream(plan, st);
  if (cufftExecZ2Z(plan, (cufftDoubleComplex*)fg, (cufftDoubleComplex*)fg, CUFFT_FORWARD) != CUFFT_SUCCESS)
    return fail(kCuda, "cufftExecZ2Z failed");
  cudaError_t e = cudaSuccess;
  if (natom > 0) {
    if ((e = cudaMemcpyAsync(base + o_tau, tau, sizeof(double) * 3 * natom, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (e = cudaMemcpyAsync(base + o_atom, atom_of.data(), sizeof(int) * slots, cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (e = cudaMemcpyAsync(base + o_type, tile_type.data(), sizeof(int) * tiles, cudaMemcpyHostToDevice, st)) != cudaSuccess)
      return cuda_fail(e, "structure gradient upload");
    const size_t sm = std::max(sizeof(Z) * (size_t)kSgRows * p.n1, sizeof(double) * 3 * kSgGroups * kSgAtoms);
    if ((e = smem_limit((const void*)k_structure_grad, sm)) != cudaSuccess)
      return cuda_fail(e, "structure gradient attribute");
    const int* d_atom = (const int*)(base + o_atom);
    k_sg_phases<<<std::min(1184, (nsum * slots + 255) / 256), 256, 0, st>>>(
        p.n1, p.n2, p.n3, slots, d_atom, (const double*)(base + o_tau), (Z*)(base + o_tab));
    k_structure_grad<<<dim3(chunks, tiles), kSgAtoms * kSgGroups, sm, st>>>(
        p.n1, p.n2, p.n3, slots, fg, (const double*)vgt, (const int*)(base + o_type), (const Z*)(base + o_tab),
        (double*)(base + o_part));
    k_sg_sum<<<(3 * slots + 7) / 8, 256, 0, st>>>(chunks, slots, d_atom, (const double*)(base + o_part),
                                                  (double*)(base + o_out));
    if ((e = cudaGetLastError()) == cudaSuccess)
      e = cudaMemcpyAsync(dedtau, base + o_out, sizeof(double) * 3 * natom, cudaMemcpyDeviceToHost, st);
  }
  const cudaError_t e2 = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return cuda_fail(e, "structure gradient");
  return e2 == cudaSuccess ? kOk : cuda_fail(e2, "structure gradient");
}

int nl_grad_device(cpw_b200_ctx* c, int nb, const void* psi, long long ldpsi, const double* occ,
                   const int* proj_atom, int natom, double* dedtau, cudaStream_t st) {
  if (!c->have_basis) return fail(kNotReady, "projector gradient: basis must be set");
  for (int a = 0; a < 3 * natom; ++a) dedtau[a] = 0.0;
  const int na = c->nanl, m = c->mtxd;
  if (na == 0 || nb == 0 || m == 0) return kOk;
  for (int a = 0; a < na; ++a)
    if (proj_atom[a] < 0 || proj_atom[a] >= natom) return fail(kBadArg, "projector gradient: proj_atom out of range");
  // With Y = psi diag(f) P^H the sum over bands goes first: sum_n f_n Im(conj(P_an) Q_jan) =
  // Im sum_i conj(X_ia) G_ij Y_ia, one product of the size of P's in place of the three X^H (G_j psi).
  // The work space is kept, so Y is made in blocks of projectors of at most 512 MB (64 projectors at least, a tile
  // of the product). us for 4 and 128 bands: 26,398 plane waves, 256 projectors, one block of 108 MB, 214 and
  // 535; 89,137, 864, blocks of 64 MB, 256 MB, 512 MB and whole (1.2 GB): 1,738, 1,667, 1,525, 1,474 and 5,411,
  // 5,379, 5,139, 5,100. The contraction's plane waves are split into slices, which fill the SMs for few projectors too.
  const size_t colY = sizeof(Z) * (size_t)m;
  const int most = std::max(64, (int)std::min<size_t>((size_t)na, (size_t)(512 << 20) / colY / 32 * 32));
  const int blocks = (na + most - 1) / most, per = std::min(na, ((na + blocks - 1) / blocks + 31) / 32 * 32);
  const int slices = std::max(1, std::min(16, (592 + per - 1) / per));       // about four CTAs per SM in the contraction
  const size_t zP = sizeof(Z) * (size_t)na * nb, zY = colY * per;
  int s;
  if ((s = c->adj.ensure(zY + 2 * zP + sizeof(double) * (3 * (size_t)na * slices + nb)))) return s;
  char* base = (char*)c->adj.p;
  Z* Y = (Z*)base;
  Z* P = (Z*)(base + zY);
  Z* M = (Z*)(base + zY + zP);
  double* docc = (double*)(base + zY + 2 * zP);
  double* dc = docc + nb;
  cudaError_t e = cudaMemcpyAsync(docc, occ, sizeof(double) * nb, cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess) return cuda_fail(e, "projector gradient occ");
  cublasSetStream(c->blas, st);
  const Z one = make_cuDoubleComplex(1, 0), zero = make_cuDoubleComplex(0, 0);
  cublasStatus_t bs = cublasZgemm(c->blas, CUBLAS_OP_C, CUBLAS_OP_N, na, nb, m, &one, (const Z*)c->anl.p, m,
                                  (const Z*)psi, (int)ldpsi, &zero, P, na);
  if (bs != CUBLAS_STATUS_SUCCESS) return fail(kCublas, "projector gradient zgemm P");
  k_stress_m<<<(int)std::max(1LL, std::min(1184LL, ((long long)na * nb + 255) / 256)), 256, 0, st>>>(
      na, nb, P, docc, nullptr, M);
  for (int a0 = 0; a0 < na; a0 += per) {
    const int n = std::min(per, na - a0);
    bs = cublasZgemm(c->blas, CUBLAS_OP_N, CUBLAS_OP_N, m, n, nb, &one, (const Z*)psi, (int)ldpsi, M + (size_t)a0 * nb,
                     nb, &zero, Y, m);
    if (bs != CUBLAS_STATUS_SUCCESS) return fail(kCublas, "projector gradient zgemm Y");
    k_nl_contract<<<dim3(n, slices), 256, 0, st>>>(m, (const int*)c->kgvb.p, (const Z*)c->anl.p + (size_t)a0 * m, Y,
                                                   dc + 3 * (size_t)a0, na);
  }
  std::vector<double> ch(3 * (size_t)na * slices);
  e = cudaMemcpyAsync(ch.data(), dc, sizeof(double) * ch.size(), cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) return cuda_fail(e, "projector gradient copy");
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return cuda_fail(e, "projector gradient");
  const double fpi = 12.566370614359172953850573533118011537;
  for (int a = 0; a < na; ++a)
    for (int j = 0; j < 3; ++j) {
      double t = 0.0;
      for (int k = 0; k < slices; ++k) t += ch[3 * ((size_t)k * na + a) + j];
      dedtau[3 * proj_atom[a] + j] += -fpi * c->xnl_h[a] * t;
    }
  return kOk;
}

}  // namespace cpwb
