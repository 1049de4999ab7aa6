// Kernel templates A, B, C of the local H|psi> (design in hkpsi_local.cuh).
//
// Template parameters of A and C fix the radix pairs of the plane (RX1*RX2 = n1, RY1*RY2 = n2) and the
// column batch width TC at compile time; 0 means "taken from the LocalPlan at run time". The
// compile-time forms get constant index arithmetic and register allocation sized for their own
// radices; the all-zero form serves any supported box. B has a compiled form per line length and
// two run-time forms.
#pragma once
#include <algorithm>

#include "hkpsi_local.cuh"

namespace cpwb {
namespace kern {

constexpr int kThreadsPlanes = 256;
constexpr int kThreadsCols = 256;
// CTAs per SM asked of the register allocator for kernels A and C (fwd): the passes wait on shared memory
// and on the plane's loads, so small planes want as many CTAs as their shared memory lets in. us per launch
// with this bound, before -> after:
//   Up to 64 points (10 to 40 KB a plane). 40 x 40 (320 threads; 2,560 bands FP32, 160 FP64): C FP32 three -> five 541
//   -> 404 (six the same), A FP32 four -> six 361 -> 326; C FP64 two -> three 60 -> 52 (four 52 with the read-ahead
//   gather that takes three to 46), A FP64 three -> four 36 -> 35. 32 x 32 x 96 (256 threads, 1,000 bands), no
//   bound -> this one: A FP32 139 -> 128, C FP32 157 and both FP64 205 and 236 unchanged.
//   FP32 planes of 65 to 127 points (64 KB at 96, three to an SM). 96 x 96 (160 bands): C with 384 threads in three
//   CTAs 164, 256 in three 179, 256 in four 210; A in three 139, in four 160 (spills).
//   FP64 planes of 128 points or more take over 200 KB of shared memory, one CTA per SM whatever the
//   registers: no cap. The others: two CTAs of 384 threads in 80 registers.
// The run-time form (n1 = 0) would take the registers of its largest radix, one CTA of 256 threads per SM in
// FP64: it is held to two (three: 72 x 80 C 89 -> 105), in FP32 to three, or to five where a plane's shared
// memory lets them in (many: 64 x 50, 91 bands, C 96 -> 83, A 81 -> 72; 48 bands of 48 x 48 42 -> 38 for
// both, 72 x 72 76 -> 73; 80 x 80, which would hold four, 98 -> 111).
template <typename T> constexpr int plane_min_blocks(int nt, int n1, bool fwd, bool many) {
  if (n1 == 0) return sizeof(T) == 8 ? 2 : many ? 5 : 3;
  if (n1 <= 64) return sizeof(T) == 8 ? (fwd ? 3 : 4) : fwd ? 5 : 6;
  if (n1 < 128 && sizeof(T) == 4) return 3;
  return sizeof(T) == 8 && n1 >= 128 ? 1 : nt >= 320 ? 2 : 1;
}
constexpr size_t kManyPlaneBytes = 44 * 1024;   // five CTAs to an SM

template <typename T> __device__ __forceinline__ C2<T> czero() { return mk<T>(T(0), T(0)); }

// ---------------------------------------------------------------------------
// A: scatter + inverse x + inverse y, one CTA per (band, kept z-plane)
// ---------------------------------------------------------------------------
// PR: the kept x and y indices lie in the outer quarters of their lines (in_quarters below), so that
// the first pass of each transform reads and multiplies those points alone.
template <typename T, int RX1, int RX2, int RY1, int RY2, int TC, bool PR, int NT = kThreadsPlanes, bool MANY = false>
__global__ void __launch_bounds__(NT, plane_min_blocks<T>(NT, RX1 * RX2, false, MANY))
k_inv_xy(LocalPlan p, int band0, const C2<double>* __restrict__ psi, long long ldpsi,
         const int* __restrict__ plane_start, const int* __restrict__ pw_idx,
         const int* __restrict__ pw_pos, const C2<T>* __restrict__ twx,
         const C2<T>* __restrict__ twy, C2<T>* __restrict__ W) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tc = TC ? TC : p.tcol;
  const int r1x = RX1 ? RX1 : p.dx.r1, r2x = RX2 ? RX2 : p.dx.r2;
  const int r1y = RY1 ? RY1 : p.dy.r1, r2y = RY2 ? RY2 : p.dy.r2;
  const int n1 = RX1 ? RX1 * RX2 : p.n1, n2 = RY1 ? RY1 * RY2 : p.n2;
  const int ny = p.ny, rowp = p.rowp;
  C2<T>* R = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* Tb = R + (size_t)ny * rowp;
  C2<T>* sx = Tb + (size_t)n2 * tc;
  C2<T>* sy = sx + n1;
  const int zi = blockIdx.x, b = blockIdx.y;
  const int tid = threadIdx.x, nt = NT;     // every launch uses NT threads

  const C2<double>* ps = psi + (size_t)(band0 + b) * ldpsi;
  if (p.kdesc) {      // batch of k-points: this band's own basis and block
    const int2 r = p.bref[band0 + b];
    const KDesc& D = p.kdesc[r.x];
    ps = D.psi + (size_t)r.y * D.ldpsi;
    plane_start = D.plane_start;
    pw_idx = D.pw_idx;
    pw_pos = D.pw_pos;
  }
  const int e0 = plane_start[zi], e1 = plane_start[zi + 1];
  // the first kPre sphere points of this thread are loaded before the plane is cleared, so
  // that their gather latency overlaps the clearing
  constexpr int kPre = 2;
  int pre_pos[kPre];
  C2<double> pre_v[kPre];
#pragma unroll
  for (int j = 0; j < kPre; ++j) {
    const int e = e0 + tid + j * nt;
    pre_pos[j] = -1;
    if (e < e1) {
      pre_pos[j] = pw_pos[e];
      pre_v[j] = ps[pw_idx[e]];
    }
  }
  for (int i = tid; i < n1; i += nt) sx[i] = twx[i];
  for (int i = tid; i < n2; i += nt) sy[i] = twy[i];
  if constexpr (PR) {
    // the points that pass 1 reads: the outer quarters of every row
    const int half = quarter(r1x) * r2x, per = 2 * half;
    for (int i = tid; i < ny * per; i += nt) {
      const int row = i / per, x = i - row * per;
      R[row * rowp + (x < half ? x : n1 - per + x)] = czero<T>();
    }
  } else {
    for (int i = tid; i < ny * rowp; i += nt) R[i] = czero<T>();
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPre; ++j)
    if (pre_pos[j] >= 0)
      R[(pre_pos[j] >> 16) * rowp + (pre_pos[j] & 0xffff)] = mk<T>(T(pre_v[j].x), T(pre_v[j].y));
  for (int e = e0 + tid + kPre * nt; e < e1; e += nt) {
    const int pos = pw_pos[e];
    const C2<double> v = ps[pw_idx[e]];
    R[(pos >> 16) * rowp + (pos & 0xffff)] = mk<T>(T(v.x), T(v.y));
  }
  __syncthreads();

  // inverse x, pass 1: lines (row, n2) with the row index fastest across lanes
  for (int it = tid; it < ny * r2x; it += nt) {
    const int row = it % ny, n2i = it / ny;
    C2<T>* line = R + (size_t)row * rowp + n2i;
    with_radix<RX1>(r1x, [&](auto rc_) {
      constexpr int RR = decltype(rc_)::value;
      constexpr unsigned M = PR ? quarter_bits(RR) : (1u << RR) - 1;
      C2<T> v[RR];
#pragma unroll
      for (int a = 0; a < RR; ++a)
        if ((M >> a) & 1) v[a] = line[r2x * a];
      DFTM<M, RR, +1, T>::run(v);
#pragma unroll
      for (int a = 0; a < RR; ++a) line[r2x * a] = a == 0 ? v[0] : cmulc<T>(v[a], sx[n2i * a]);
    });
  }
  __syncthreads();
  // inverse x, pass 2: lines (row, k1), contiguous block of r2x, permuted in place
  for (int it = tid; it < ny * r1x; it += nt) {
    const int row = it % ny, k1 = it / ny;
    C2<T>* line = R + (size_t)row * rowp + r2x * k1;
    with_radix<RX2>(r2x, [&](auto rc_) {
      constexpr int RR = decltype(rc_)::value;
      C2<T> v[RR];
#pragma unroll
      for (int a = 0; a < RR; ++a) v[a] = line[a];
      DFT<RR, +1, T>::run(v);
#pragma unroll
      for (int a = 0; a < RR; ++a) line[a] = v[a];
    });
  }
  __syncthreads();

  // inverse y on every column, in batches of tc storage positions. The slab keeps the x storage order
  // of pass 2 (slab_x): a warp stores 32 neighbouring columns of a row in 512 contiguous bytes. Stored in
  // x order its 32 pieces of 16 bytes fell r1x columns apart, and the stores took two thirds of the
  // L1 data path that bounds this kernel.
  C2<T>* Wp = W + ((size_t)b * p.nz + zi) * (size_t)p.plane;
  for (int pb = 0; pb < n1; pb += tc) {
    const int ncol = min(tc, n1 - pb);
    for (int it = tid; it < tc * r2y; it += nt) {
      const int pl = it % tc, n2i = it / tc;
      if (pl < ncol) {
        with_radix<RY1>(r1y, [&](auto rc_) {
          constexpr int RR = decltype(rc_)::value;
          C2<T> v[RR];
          if constexpr (PR) {
            constexpr int Q = quarter(RR);
            const C2<T>* lo = R + (size_t)n2i * rowp + pb + pl;       // row of y <= kd2
            const C2<T>* hi = lo - (ptrdiff_t)(n2 - ny) * rowp;       // row of y >= n2 - kd2
#pragma unroll
            for (int a = 0; a < Q; ++a) v[a] = r2y * a + n2i <= p.kd2 ? lo[(size_t)(r2y * a) * rowp] : czero<T>();
#pragma unroll
            for (int a = RR - Q; a < RR; ++a)
              v[a] = r2y * a + n2i >= n2 - p.kd2 ? hi[(size_t)(r2y * a) * rowp] : czero<T>();
            DFTM<quarter_bits(RR), RR, +1, T>::run(v);
          } else {
#pragma unroll
            for (int a = 0; a < RR; ++a) {
              const int yi = idx_to_kept(r2y * a + n2i, p.kd2, n2, ny);
              v[a] = yi >= 0 ? R[(size_t)yi * rowp + pb + pl] : czero<T>();
            }
            DFT<RR, +1, T>::run(v);
          }
#pragma unroll
          for (int a = 0; a < RR; ++a)
            Tb[(size_t)(r2y * a + n2i) * tc + pl] = a == 0 ? v[0] : cmulc<T>(v[a], sy[n2i * a]);
        });
      }
    }
    __syncthreads();
    for (int it = tid; it < tc * r1y; it += nt) {
      const int pl = it % tc, k1 = it / tc;
      if (pl < ncol) {
        with_radix<RY2>(r2y, [&](auto rc_) {
          constexpr int RR = decltype(rc_)::value;
          C2<T> v[RR];
#pragma unroll
          for (int a = 0; a < RR; ++a) v[a] = Tb[(size_t)(r2y * k1 + a) * tc + pl];
          DFT<RR, +1, T>::run(v);
#pragma unroll
          for (int a = 0; a < RR; ++a) Wp[(size_t)(k1 + r1y * a) * n1 + pb + pl] = v[a];
        });
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// B: inverse z, V(r)/N, forward z, one CTA per (band, CB xy-columns)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(kThreadsCols, 1)
k_z_vloc(LocalPlan p, const T* __restrict__ vr, const C2<T>* __restrict__ twz, C2<T>* __restrict__ W) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int cb = p.cb, r1 = p.dz.r1, r2 = p.dz.r2, n3 = p.n3;
  C2<T>* Cs = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* sz = Cs + (size_t)n3 * cb;
  const long long c0 = (long long)blockIdx.x * cb;
  const int b = blockIdx.y;
  const int ncol = (int)min((long long)cb, p.plane - c0);
  const int tid = threadIdx.x, nt = blockDim.x;
  C2<T>* Wb = W + (size_t)b * p.nz * (size_t)p.plane + c0;

  for (int i = tid; i < n3; i += nt) sz[i] = twz[i];
  for (int it = tid; it < cb * p.nz; it += nt) {
    const int cl = it % cb, zi = it / cb;
    if (cl < ncol) Cs[(size_t)kept_to_idx(zi, p.kd3, n3, p.nz) * cb + cl] = Wb[(size_t)zi * p.plane + cl];
  }
  __syncthreads();
  // inverse pass 1 (reads only kept planes; the others are zero)
  for (int it = tid; it < cb * r2; it += nt) {
    const int cl = it % cb, n2i = it / cb;
    if (cl < ncol) {
      with_radix<0>(r1, [&](auto rc_) {
        constexpr int RR = decltype(rc_)::value;
        C2<T> v[RR];
#pragma unroll
        for (int a = 0; a < RR; ++a) {
          const int z = r2 * a + n2i;
          v[a] = idx_to_kept(z, p.kd3, n3, p.nz) >= 0 ? Cs[(size_t)z * cb + cl] : czero<T>();
        }
        DFT<RR, +1, T>::run(v);
#pragma unroll
        for (int a = 0; a < RR; ++a)
          Cs[(size_t)(r2 * a + n2i) * cb + cl] = a == 0 ? v[0] : cmulc<T>(v[a], sz[n2i * a]);
      });
    }
  }
  __syncthreads();
  // inverse pass 2 -> multiply V(r)/N -> forward pass 1, in registers
  for (int it = tid; it < cb * r1; it += nt) {
    const int cl = it % cb, k1 = it / cb;
    if (cl < ncol) {
      with_radix<0>(r2, [&](auto rc_) {
        constexpr int RR = decltype(rc_)::value;
        C2<T> v[RR];
        T vz[RR];
        const int vc = slab_column(p, c0 + cl);
#pragma unroll
        for (int a = 0; a < RR; ++a) vz[a] = vr[(size_t)(k1 + r1 * a) * p.plane + vc];
#pragma unroll
        for (int a = 0; a < RR; ++a) v[a] = Cs[(size_t)(r2 * k1 + a) * cb + cl];
        DFT<RR, +1, T>::run(v);
#pragma unroll
        for (int a = 0; a < RR; ++a) v[a] = scal<T>(v[a], vz[a]);
        DFT<RR, -1, T>::run(v);
#pragma unroll
        for (int a = 0; a < RR; ++a)
          Cs[(size_t)(r2 * k1 + a) * cb + cl] = a == 0 ? v[0] : cmul<T>(v[a], sz[k1 * a]);
      });
    }
  }
  __syncthreads();
  // forward pass 2, keep the kept planes
  for (int it = tid; it < cb * r2; it += nt) {
    const int cl = it % cb, m2 = it / cb;
    if (cl < ncol) {
      with_radix<0>(r1, [&](auto rc_) {
        constexpr int RR = decltype(rc_)::value;
        C2<T> v[RR];
#pragma unroll
        for (int a = 0; a < RR; ++a) v[a] = Cs[(size_t)(r2 * a + m2) * cb + cl];
        DFT<RR, -1, T>::run(v);
#pragma unroll
        for (int a = 0; a < RR; ++a) {
          const int zi = idx_to_kept(m2 + r2 * a, p.kd3, n3, p.nz);
          if (zi >= 0) Wb[(size_t)zi * p.plane + cl] = v[a];
        }
      });
    }
  }
}


// ---------------------------------------------------------------------------
// B (pipelined): one CTA per (CB xy-columns, band group). The V(r)/N tile of
// the columns is loaded into shared memory once; the kept planes of band b+1
// stream in with cp.async while band b is transformed, so global latency
// overlaps the butterflies. Same arithmetic as k_z_vloc.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void cp_async_bytes(void* smem, const void* gmem, int bytes) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem));
  else if (bytes == 8)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem));
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// shared memory of k_z_vloc_pipe: work columns, two staging buffers of kept planes, twiddles, V tile
template <typename T> inline size_t smem_columns_pipe(const LocalPlan& p, int cb) {
  return smem_columns_pipe_bytes(sizeof(C2<T>), p, cb);
}

template <typename T>
__global__ void __launch_bounds__(kThreadsCols, 1)
k_z_vloc_pipe(LocalPlan p, int nbc, int bands_per_group, const T* __restrict__ vr, const C2<T>* __restrict__ twz,
              C2<T>* __restrict__ W) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int cb = p.cb, r1 = p.dz.r1, r2 = p.dz.r2, n3 = p.n3, nz = p.nz;
  C2<T>* Cs = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* Ws = Cs + (size_t)n3 * cb;
  C2<T>* sz = Ws + 2 * (size_t)nz * cb;
  T* Vs = reinterpret_cast<T*>(sz + n3);
  const long long c0 = (long long)blockIdx.x * cb;
  const int ncol = (int)min((long long)cb, p.plane - c0);
  const int b_lo = blockIdx.y * bands_per_group;
  const int b_hi = min(nbc, b_lo + bands_per_group);
  if (b_lo >= b_hi) return;
  const int tid = threadIdx.x, nt = kThreadsCols;

  auto stage = [&](int b, int buf) {
    const C2<T>* Wb = W + (size_t)b * nz * (size_t)p.plane + c0;
    C2<T>* dst = Ws + (size_t)buf * nz * cb;
    for (int it = tid; it < cb * nz; it += nt) {
      const int cl = it % cb, zi = it / cb;
      if (cl < ncol) cp_async_bytes(dst + (size_t)zi * cb + cl, Wb + (size_t)zi * p.plane + cl, (int)sizeof(C2<T>));
    }
  };
  for (int i = tid; i < n3; i += nt) sz[i] = twz[i];
  for (int it = tid; it < cb * n3; it += nt) {
    const int cl = it % cb, z = it / cb;
    if (cl < ncol)
      cp_async_bytes(Vs + (size_t)z * cb + cl, vr + (size_t)z * p.plane + slab_column(p, c0 + cl), (int)sizeof(T));
  }
  stage(b_lo, 0);
  cp_async_commit();
  if (b_lo + 1 < b_hi) stage(b_lo + 1, 1);
  cp_async_commit();

  for (int b = b_lo; b < b_hi; ++b) {
    const int buf = (b - b_lo) & 1;
    cp_async_wait<1>();     // every group but the newest (band b+1) has landed
    __syncthreads();
    const C2<T>* Wsb = Ws + (size_t)buf * nz * cb;
    // inverse pass 1 straight from the staged kept planes
    for (int it = tid; it < cb * r2; it += nt) {
      const int cl = it % cb, n2i = it / cb;
      if (cl < ncol) {
        with_radix<0>(r1, [&](auto rc_) {
          constexpr int RR = decltype(rc_)::value;
          C2<T> v[RR];
#pragma unroll
          for (int a = 0; a < RR; ++a) {
            const int zi = idx_to_kept(r2 * a + n2i, p.kd3, n3, nz);
            v[a] = zi >= 0 ? Wsb[(size_t)zi * cb + cl] : czero<T>();
          }
          DFT<RR, +1, T>::run(v);
#pragma unroll
          for (int a = 0; a < RR; ++a)
            Cs[(size_t)(r2 * a + n2i) * cb + cl] = a == 0 ? v[0] : cmulc<T>(v[a], sz[n2i * a]);
        });
      }
    }
    __syncthreads();
    // the staging buffer of band b is free: prefetch band b+2 into it
    if (b + 2 < b_hi) stage(b + 2, buf);
    cp_async_commit();
    // inverse pass 2 -> V/N -> forward pass 1, in registers
    for (int it = tid; it < cb * r1; it += nt) {
      const int cl = it % cb, k1 = it / cb;
      if (cl < ncol) {
        with_radix<0>(r2, [&](auto rc_) {
          constexpr int RR = decltype(rc_)::value;
          C2<T> v[RR];
#pragma unroll
          for (int a = 0; a < RR; ++a) v[a] = Cs[(size_t)(r2 * k1 + a) * cb + cl];
          DFT<RR, +1, T>::run(v);
#pragma unroll
          for (int a = 0; a < RR; ++a) v[a] = scal<T>(v[a], Vs[(size_t)(k1 + r1 * a) * cb + cl]);
          DFT<RR, -1, T>::run(v);
#pragma unroll
          for (int a = 0; a < RR; ++a)
            Cs[(size_t)(r2 * k1 + a) * cb + cl] = a == 0 ? v[0] : cmul<T>(v[a], sz[k1 * a]);
        });
      }
    }
    __syncthreads();
    // forward pass 2, kept planes back to the slab
    C2<T>* Wb = W + (size_t)b * nz * (size_t)p.plane + c0;
    for (int it = tid; it < cb * r2; it += nt) {
      const int cl = it % cb, m2 = it / cb;
      if (cl < ncol) {
        with_radix<0>(r1, [&](auto rc_) {
          constexpr int RR = decltype(rc_)::value;
          C2<T> v[RR];
#pragma unroll
          for (int a = 0; a < RR; ++a) v[a] = Cs[(size_t)(r2 * a + m2) * cb + cl];
          DFT<RR, -1, T>::run(v);
#pragma unroll
          for (int a = 0; a < RR; ++a) {
            const int zi = idx_to_kept(m2 + r2 * a, p.kd3, n3, nz);
            if (zi >= 0) Wb[(size_t)zi * p.plane + cl] = v[a];
          }
        });
      }
    }
  }
  cp_async_wait<0>();
}

// ---------------------------------------------------------------------------
// B (register form): one CTA per (CB xy-columns, band group) with one thread per line of the outer
// passes, for kept planes in the outer quarters of the z lines (in_quarters). A thread owns the same
// column and line index j in the inverse's first and the forward's last pass, so it reads its kept
// points of the slab straight into registers (those of band b + 1 while band b is transformed: no
// staging buffers), starts from the nonzero half of the line (DFTM), keeps only the kept outputs of the
// last pass, and needs two barriers per band: what pass 1 of band b + 1 overwrites in shared memory the
// same thread has read in the last pass of band b.
// ---------------------------------------------------------------------------
// CTAs per SM asked of the register allocator for a thread budget of `regs` registers. k_z_band: 168 (FP64)
// and 80 (FP32) leave room for the transformed line and the next band's points at once; against 112 and 64
// (more CTAs per SM): 6.2 -> 5.9 ms and 3.64 -> 3.46 ms on 480 bands of a 144^3 box, within 1 % elsewhere.
template <int R2, int CB> constexpr int z_min_blocks(int regs) { return std::max(1, 65536 / (CB * R2 * regs)); }
template <typename T, int R1, int R2, int CB>
__global__ void __launch_bounds__(CB * R2, (z_min_blocks<R2, CB>(sizeof(T) == 8 ? 168 : 80)))
k_z_band(LocalPlan p, int nbc, int per, const T* __restrict__ vr, const C2<T>* __restrict__ twz, C2<T>* __restrict__ W) {
  constexpr int N3 = R1 * R2, NT = CB * R2, Q = quarter(R1);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<T>* Cs = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* sz = Cs + N3 * CB;
  T* Vs = reinterpret_cast<T*>(sz + N3);
  const int tid = threadIdx.x, cl = tid % CB, j = tid / CB;
  const size_t pl = (size_t)p.plane;
  const long long col = (long long)blockIdx.x * CB + cl;
  const bool ok = col < p.plane;
  const int b_lo = blockIdx.y * per, b_hi = min(nbc, b_lo + per);
  if (b_lo >= b_hi) return;
  const int kd = p.kd3, skip = N3 - p.nz;
  C2<T>* Wb = W + (size_t)b_lo * p.nz * pl + col;
  const size_t band = (size_t)p.nz * pl;

  C2<T> nx[2 * Q];       // kept points z = R2 a + j, a < Q and a >= R1 - Q, of the next band
  auto load = [&](const C2<T>* w) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int z = R2 * q + j;
      nx[q] = ok && z <= kd ? w[z * pl] : czero<T>();
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int z = R2 * (R1 - Q + q) + j;
      nx[Q + q] = ok && z >= N3 - kd ? w[(z - skip) * pl] : czero<T>();
    }
  };
  load(Wb);
  for (int i = tid; i < N3; i += NT) sz[i] = twz[i];
  {
    // all of the thread's V values in flight at once
    const T* vc = vr + (ok ? slab_column(p, col) : 0);
    T v[R1];
#pragma unroll
    for (int a = 0; a < R1; ++a) v[a] = ok ? vc[(R2 * a + j) * pl] : T(0);
#pragma unroll
    for (int a = 0; a < R1; ++a) Vs[(R2 * a + j) * CB + cl] = v[a];
  }
  __syncthreads();

  for (int b = b_lo; b < b_hi; ++b, Wb += band) {
    {
      C2<T> v[R1];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        v[q] = nx[q];
        v[R1 - Q + q] = nx[Q + q];
      }
      DFTM<quarter_bits(R1), R1, +1, T>::run(v);
#pragma unroll
      for (int a = 0; a < R1; ++a) Cs[(R2 * a + j) * CB + cl] = a == 0 ? v[0] : cmulc<T>(v[a], sz[j * a]);
    }
    if (b + 1 < b_hi) load(Wb + band);
    __syncthreads();
    if (R1 == R2 || j < R1) {
      C2<T> v[R2];
#pragma unroll
      for (int a = 0; a < R2; ++a) v[a] = Cs[(R2 * j + a) * CB + cl];
      DFT<R2, +1, T>::run(v);
#pragma unroll
      for (int a = 0; a < R2; ++a) v[a] = scal<T>(v[a], Vs[(j + R1 * a) * CB + cl]);
      DFT<R2, -1, T>::run(v);
#pragma unroll
      for (int a = 0; a < R2; ++a) Cs[(R2 * j + a) * CB + cl] = a == 0 ? v[0] : cmul<T>(v[a], sz[j * a]);
    }
    __syncthreads();
    {
      C2<T> v[R1];
#pragma unroll
      for (int a = 0; a < R1; ++a) v[a] = Cs[(R2 * a + j) * CB + cl];
      DFT<R1, -1, T>::run(v);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int z = R2 * q + j, zh = R2 * (R1 - Q + q) + j;
        if (ok && z <= kd) Wb[z * pl] = v[q];
        if (ok && zh >= N3 - kd) Wb[(zh - skip) * pl] = v[R1 - Q + q];
      }
    }
  }
}
template <typename T, int R1, int R2, int CB> constexpr size_t smem_z_band() {
  return (size_t)R1 * R2 * (CB * (sizeof(C2<T>) + sizeof(T)) + sizeof(C2<T>));
}

// The inverse half of B for the density: rho(r) += sum_b occ_b |psi_b(r)|^2. Thread and memory layout of
// k_z_band; the sum over the CTA's bands of a point stays in a register of the thread that owns its
// line in the second pass. part: null = add to rho, else the band groups' own boxes (summed by the caller).
// 128 bands on 96 x 96 x 96: 304 us, the general form with its sums in shared memory 743.
template <int R1, int R2, int CB>
__global__ void __launch_bounds__(CB * R2, (z_min_blocks<R2, CB>(128)))
k_z_density(LocalPlan p, int nbc, int per, const double* __restrict__ occ, const C2<double>* __restrict__ twz,
            const C2<double>* __restrict__ W, double* __restrict__ rho, double* __restrict__ part) {
  using T = double;
  constexpr int N3 = R1 * R2, NT = CB * R2, Q = quarter(R1);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<T>* Cs = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* sz = Cs + N3 * CB;
  const int tid = threadIdx.x, cl = tid % CB, j = tid / CB;
  const size_t pl = (size_t)p.plane;
  const long long col = (long long)blockIdx.x * CB + cl;
  const bool ok = col < p.plane;
  const int b_lo = blockIdx.y * per, b_hi = min(nbc, b_lo + per);
  const int kd = p.kd3, skip = N3 - p.nz;
  const size_t band = (size_t)p.nz * pl;
  const C2<T>* Wb = W + (size_t)b_lo * band + col;
  C2<T> nx[2 * Q];
  auto load = [&](const C2<T>* w) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int z = R2 * q + j, zh = R2 * (R1 - Q + q) + j;
      nx[q] = ok && z <= kd ? w[z * pl] : czero<T>();
      nx[Q + q] = ok && zh >= N3 - kd ? w[(zh - skip) * pl] : czero<T>();
    }
  };
  if (b_lo < b_hi) load(Wb);
  for (int i = tid; i < N3; i += NT) sz[i] = twz[i];
  T acc[R2];
#pragma unroll
  for (int a = 0; a < R2; ++a) acc[a] = T(0);
  __syncthreads();
  for (int b = b_lo; b < b_hi; ++b, Wb += band) {
    {
      C2<T> v[R1];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        v[q] = nx[q];
        v[R1 - Q + q] = nx[Q + q];
      }
      DFTM<quarter_bits(R1), R1, +1, T>::run(v);
#pragma unroll
      for (int a = 0; a < R1; ++a) Cs[(R2 * a + j) * CB + cl] = a == 0 ? v[0] : cmulc<T>(v[a], sz[j * a]);
    }
    if (b + 1 < b_hi) load(Wb + band);
    const T f = occ[b];
    __syncthreads();
    if (R1 == R2 || j < R1) {
      C2<T> v[R2];
#pragma unroll
      for (int a = 0; a < R2; ++a) v[a] = Cs[(R2 * j + a) * CB + cl];
      DFT<R2, +1, T>::run(v);
#pragma unroll
      for (int a = 0; a < R2; ++a) acc[a] += f * (v[a].x * v[a].x + v[a].y * v[a].y);
    }
    __syncthreads();
  }
  if (ok && (R1 == R2 || j < R1)) {
    const int vc = slab_column(p, col);
#pragma unroll
    for (int a = 0; a < R2; ++a) {
      const size_t o = (j + R1 * a) * pl + vc;
      if (part)
        part[(size_t)blockIdx.y * N3 * pl + o] = acc[a];
      else
        rho[o] += acc[a];
    }
  }
}

// The non-collinear z stage of one spinor per step: both components' columns are transformed, multiplied by
// [[V1+V2, V3-iV4], [V3+iV4, V1-V2]] and transformed back. One thread per (component, line, column); the
// four potential columns are staged once per CTA and serve its bands, the kept points of the next spinor
// are loaded while this one is transformed. Up slabs at W, down slabs nbc slabs later. Bound: latency of
// the FP64 passes. 80 spinors on 40 x 40 x 40, FP64: 84 us in 168 registers (three CTAs), 76 in 128 (four);
// the general form that transforms one spinor per CTA through shared memory 495. Lines above 64 points hold
// more and would spill in 128.
template <typename T, int R1, int R2, int CB>
__global__ void __launch_bounds__(2 * CB * R2, (z_min_blocks<R2, 2 * CB>(sizeof(T) == 4 ? 96 : R1 * R2 <= 64 ? 128 : 168)))
k_z_spinor_band(LocalPlan p, int nbc, int per, const T* __restrict__ vu, const T* __restrict__ vd,
                const T* __restrict__ vr, const T* __restrict__ vi, const C2<T>* __restrict__ twz, C2<T>* __restrict__ W) {
  constexpr int N3 = R1 * R2, NT = 2 * CB * R2, Q = quarter(R1);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  C2<T>* Call = reinterpret_cast<C2<T>*>(smem_raw);          // [component][z][column]
  C2<T>* sz = Call + 2 * N3 * CB;
  T* Vs = reinterpret_cast<T*>(sz + N3);                     // [vu, vd, vr, vi][z][column]
  const int tid = threadIdx.x, cl = tid % CB, j = (tid / CB) % R2, s = tid / (CB * R2);
  const size_t pl = (size_t)p.plane;
  const long long col = (long long)blockIdx.x * CB + cl;
  const bool ok = col < p.plane;
  const int b_lo = blockIdx.y * per, b_hi = min(nbc, b_lo + per);
  if (b_lo >= b_hi) return;
  const int kd = p.kd3, skip = N3 - p.nz;
  const size_t band = (size_t)p.nz * pl;
  C2<T>* Cs = Call + s * N3 * CB;
  const C2<T>* Co = Call + (1 - s) * N3 * CB;
  C2<T>* Wb = W + ((size_t)s * nbc + b_lo) * band + col;
  C2<T> nx[2 * Q];
  auto load = [&](const C2<T>* w) {
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int z = R2 * q + j, zh = R2 * (R1 - Q + q) + j;
      nx[q] = ok && z <= kd ? w[z * pl] : czero<T>();
      nx[Q + q] = ok && zh >= N3 - kd ? w[(zh - skip) * pl] : czero<T>();
    }
  };
  load(Wb);
  for (int i = tid; i < N3; i += NT) sz[i] = twz[i];
  {
    const int vc = ok ? slab_column(p, col) : 0;
    const T* src[4] = {vu, vd, vr, vi};
#pragma unroll
    for (int k = 0; k < 2; ++k)
      for (int z = j; z < N3; z += R2) Vs[((2 * s + k) * N3 + z) * CB + cl] = ok ? src[2 * s + k][z * pl + vc] : T(0);
  }
  __syncthreads();
  const T* Va = Vs + s * N3 * CB;                            // this component's diagonal term
  const T* Vr = Vs + 2 * N3 * CB;
  const T* Vi = Vr + N3 * CB;
  const T sgn = s == 0 ? T(1) : T(-1);                       // V3 - i V4 acts on down, V3 + i V4 on up
  for (int b = b_lo; b < b_hi; ++b, Wb += band) {
    {
      C2<T> v[R1];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        v[q] = nx[q];
        v[R1 - Q + q] = nx[Q + q];
      }
      DFTM<quarter_bits(R1), R1, +1, T>::run(v);
#pragma unroll
      for (int a = 0; a < R1; ++a) Cs[(R2 * a + j) * CB + cl] = a == 0 ? v[0] : cmulc<T>(v[a], sz[j * a]);
    }
    if (b + 1 < b_hi) load(Wb + band);
    __syncthreads();
    C2<T> v[R2];
    const bool mid = R1 == R2 || j < R1;
    if (mid) {
#pragma unroll
      for (int a = 0; a < R2; ++a) v[a] = Cs[(R2 * j + a) * CB + cl];
      DFT<R2, +1, T>::run(v);
#pragma unroll
      for (int a = 0; a < R2; ++a) Cs[(R2 * j + a) * CB + cl] = v[a];
    }
    __syncthreads();
    if (mid) {
#pragma unroll
      for (int a = 0; a < R2; ++a) {
        const C2<T> o = Co[(R2 * j + a) * CB + cl];
        const int z = (j + R1 * a) * CB + cl;
        const T d = Va[z], xr = Vr[z], xi = sgn * Vi[z];
        v[a] = mk<T>(d * v[a].x + xr * o.x - xi * o.y, d * v[a].y + xr * o.y + xi * o.x);
      }
      DFT<R2, -1, T>::run(v);
    }
    __syncthreads();
    if (mid) {
#pragma unroll
      for (int a = 0; a < R2; ++a) Cs[(R2 * j + a) * CB + cl] = a == 0 ? v[0] : cmul<T>(v[a], sz[j * a]);
    }
    __syncthreads();
    {
      C2<T> w[R1];
#pragma unroll
      for (int a = 0; a < R1; ++a) w[a] = Cs[(R2 * a + j) * CB + cl];
      DFT<R1, -1, T>::run(w);
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const int z = R2 * q + j, zh = R2 * (R1 - Q + q) + j;
        if (ok && z <= kd) Wb[z * pl] = w[q];
        if (ok && zh >= N3 - kd) Wb[(zh - skip) * pl] = w[R1 - Q + q];
      }
    }
  }
}

// ---------------------------------------------------------------------------
// C: forward y + forward x + gather + kinetic, one CTA per (band, kept z-plane)
// ---------------------------------------------------------------------------
template <typename T, int RX1, int RX2, int RY1, int RY2, int TC, bool PR, int NT = kThreadsPlanes, bool MANY = false>
__global__ void __launch_bounds__(NT, plane_min_blocks<T>(NT, RX1 * RX2, true, MANY))
k_fwd_xy(LocalPlan p, int band0, const C2<double>* __restrict__ psi, long long ldpsi,
         C2<double>* __restrict__ hpsi, long long ldh, const int* __restrict__ plane_start,
         const int* __restrict__ pw_idx, const int* __restrict__ pw_pos,
         const double* __restrict__ ekpg, const C2<T>* __restrict__ twx,
         const C2<T>* __restrict__ twy, const C2<T>* __restrict__ W) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tc = TC ? TC : p.tcol;
  const int r1x = RX1 ? RX1 : p.dx.r1, r2x = RX2 ? RX2 : p.dx.r2;
  const int r1y = RY1 ? RY1 : p.dy.r1, r2y = RY2 ? RY2 : p.dy.r2;
  const int n1 = RX1 ? RX1 * RX2 : p.n1, n2 = RY1 ? RY1 * RY2 : p.n2;
  const int ny = p.ny, rowp = p.rowp;
  C2<T>* R = reinterpret_cast<C2<T>*>(smem_raw);
  C2<T>* Tb = R + (size_t)ny * rowp;
  C2<T>* sx = Tb + (size_t)n2 * tc;
  C2<T>* sy = sx + n1;
  const int zi = blockIdx.x, b = blockIdx.y;
  const int tid = threadIdx.x, nt = NT;     // every launch uses NT threads
  for (int i = tid; i < n1; i += nt) sx[i] = twx[i];
  for (int i = tid; i < n2; i += nt) sy[i] = twy[i];
  const C2<double>* ps = psi + (size_t)(band0 + b) * ldpsi;
  C2<double>* hp = hpsi + (size_t)(band0 + b) * ldh;
  if (p.kdesc) {      // batch of k-points: this band's own basis and block
    const int2 r = p.bref[band0 + b];
    const KDesc& D = p.kdesc[r.x];
    ps = D.psi + (size_t)r.y * D.ldpsi;
    hp = D.hpsi + (size_t)r.y * D.ldh;
    plane_start = D.plane_start;
    pw_idx = D.pw_idx;
    pw_pos = D.pw_pos;
    ekpg = D.ekpg;
  }
  const int e0 = plane_start[zi], e1 = plane_start[zi + 1];

  // FP64 planes of up to 64 points: each thread's first point of the final gather (often the only one) is
  // read ahead, its index here, psi and the kinetic term between the y and x transforms
  constexpr bool kFirst = sizeof(T) == 8 && RX1 > 0 && RX1 * RX2 <= 64;
  const bool first = kFirst && e0 + tid < e1;
  int fi = 0, fp = 0;
  if (first) {
    fi = pw_idx[e0 + tid];
    fp = pw_pos[e0 + tid];
  }
  const C2<T>* Wp = W + ((size_t)b * p.nz + zi) * (size_t)p.plane;
  if (tid == 0 && p.plane * sizeof(C2<T>) % 16 == 0) {
    // bring the plane into L2 while the first tiles are transformed
    const char* w = reinterpret_cast<const char*>(Wp);
    const size_t bytes = (size_t)p.plane * sizeof(C2<T>);
    for (size_t o = 0; o < bytes; o += 16384)
      asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(w + o), "r"((unsigned)min((size_t)16384, bytes - o)) : "memory");
  }
  __syncthreads();      // the twiddles
  // Where a large FP64 plane leaves one CTA per SM and every thread has one line per pass, the next
  // tile's points are loaded while this one is transformed: nothing else hides their latency there
  // (144 x 144: 4.47 -> 4.28 ms per 480 bands).
  constexpr bool kAhead = sizeof(T) == 8 && RX1 * RX2 >= 128 && TC * RY2 == NT;
  C2<T> ahead[kAhead ? RY1 : 1];
  if constexpr (kAhead) {
#pragma unroll
    for (int a = 0; a < RY1; ++a) ahead[a] = Wp[(size_t)(RY2 * a + tid / TC) * n1 + tid % TC];
  }
  for (int xb = 0; xb < n1; xb += tc) {
    const int ncol = min(tc, n1 - xb);
    // pass 1 from the slab (a warp reads neighbouring columns of a row), pass 2 into the kept rows
    for (int it = tid; it < tc * r2y; it += nt) {
      const int xl = it % tc, n2i = it / tc;
      if (xl < ncol) {
        with_radix<RY1>(r1y, [&](auto rc_) {
          constexpr int RR = decltype(rc_)::value;
          C2<T> v[RR];
#pragma unroll
          for (int a = 0; a < RR; ++a) {
            if constexpr (kAhead)
              v[a] = ahead[a];
            else
              v[a] = Wp[(size_t)(r2y * a + n2i) * n1 + xb + xl];
          }
          DFT<RR, -1, T>::run(v);
#pragma unroll
          for (int a = 0; a < RR; ++a)
            Tb[(size_t)(r2y * a + n2i) * tc + xl] = a == 0 ? v[0] : cmul<T>(v[a], sy[n2i * a]);
          if constexpr (kAhead) {
            if (xb + tc + xl < n1) {
#pragma unroll
              for (int a = 0; a < RR; ++a) ahead[a] = Wp[(size_t)(r2y * a + n2i) * n1 + xb + tc + xl];
            }
          }
        });
      }
    }
    if (sizeof(T) == 8 && !kFirst && xb == 0 && ekpg) {
      // bring the psi values and kinetic terms of the final gather into L2, so that its dependent
      // loads do not wait on HBM at the end of the CTA (FP64 only: in FP32 the extra registers cost a
      // CTA per SM on 96-point lines)
      for (int e = e0 + tid; e < e1; e += nt) {
        const int i = pw_idx[e];
        asm volatile("prefetch.global.L2 [%0];" ::"l"(ps + i));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(ekpg + i));
      }
    }
    __syncthreads();
    for (int it = tid; it < tc * r1y; it += nt) {
      const int xl = it % tc, k1 = it / tc;
      if (xl < ncol) {
        with_radix<RY2>(r2y, [&](auto rc_) {
          constexpr int RR = decltype(rc_)::value;
          C2<T> v[RR];
#pragma unroll
          for (int a = 0; a < RR; ++a) v[a] = Tb[(size_t)(r2y * k1 + a) * tc + xl];
          DFT<RR, -1, T>::run(v);
          if constexpr (PR) {
            constexpr int Q = quarter(RR);
            C2<T>* lo = R + (size_t)k1 * rowp + xb + xl;
            C2<T>* hi = lo - (ptrdiff_t)(n2 - ny) * rowp;
#pragma unroll
            for (int a = 0; a < Q; ++a)
              if (k1 + r1y * a <= p.kd2) lo[(size_t)(r1y * a) * rowp] = v[a];
#pragma unroll
            for (int a = RR - Q; a < RR; ++a)
              if (k1 + r1y * a >= n2 - p.kd2) hi[(size_t)(r1y * a) * rowp] = v[a];
          } else {
#pragma unroll
            for (int a = 0; a < RR; ++a) {
              const int yi = idx_to_kept(k1 + r1y * a, p.kd2, n2, ny);
              if (yi >= 0) R[(size_t)yi * rowp + xb + xl] = v[a];
            }
          }
        });
      }
    }
    __syncthreads();
  }

  C2<double> fs = czero<double>();
  double fe = 0.0;
  if (first && ekpg) {
    fs = ps[fi];
    fe = ekpg[fi];
  }
  // forward x on the kept rows (row index fastest across lanes). The points lie in the slab's storage
  // order: slot(x) is where natural index x is (run-time radices: from a table in the tile buffer, which
  // is free by now and at least n1 shorts long: two rows of 32 columns, or more rows).
  unsigned short* sslot = reinterpret_cast<unsigned short*>(Tb);
  if constexpr (RX1 == 0) {
    for (int i = tid; i < n1; i += nt) sslot[i] = (unsigned short)slab_slot(i, r1x, r2x);
    __syncthreads();
  }
  auto slot = [&](int x) { return RX1 ? slab_slot(x, r1x, r2x) : (int)sslot[x]; };
  for (int it = tid; it < ny * r2x; it += nt) {
    const int row = it % ny, n2i = it / ny;
    C2<T>* line = R + (size_t)row * rowp;
    with_radix<RX1>(r1x, [&](auto rc_) {
      constexpr int RR = decltype(rc_)::value;
      C2<T> v[RR];
      int at[RR];
#pragma unroll
      for (int a = 0; a < RR; ++a) {
        at[a] = RX1 && RX1 == RX2 ? RX1 * n2i + a : slot(r2x * a + n2i);
        v[a] = line[at[a]];
      }
      DFT<RR, -1, T>::run(v);
#pragma unroll
      for (int a = 0; a < RR; ++a) line[at[a]] = a == 0 ? v[0] : cmul<T>(v[a], sx[n2i * a]);
    });
  }
  __syncthreads();
  for (int it = tid; it < ny * r1x; it += nt) {
    const int row = it % ny, k1 = it / ny;
    C2<T>* line = R + (size_t)row * rowp;
    with_radix<RX2>(r2x, [&](auto rc_) {
      constexpr int RR = decltype(rc_)::value;
      constexpr unsigned M = PR ? quarter_bits(RR) : (1u << RR) - 1;
      C2<T> v[RR];
      int at[RR];
#pragma unroll
      for (int a = 0; a < RR; ++a) {
        at[a] = RX1 && RX1 == RX2 ? RX1 * a + k1 : slot(r2x * k1 + a);
        v[a] = line[at[a]];
      }
      DFT<RR, -1, T>::run(v);
#pragma unroll
      for (int a = 0; a < RR; ++a)
        if ((M >> a) & 1) line[at[a]] = v[a];       // frequency k1 + r1x a
    });
  }
  __syncthreads();

  // gather the sphere and add the kinetic diagonal
  for (int e = e0 + tid; e < e1; e += nt) {
    const bool f = kFirst && e == e0 + tid;
    const int pos = f ? fp : pw_pos[e];
    const int x = pos & 0xffff, q = x / r1x;
    const C2<T> v = R[(size_t)(pos >> 16) * rowp + slot(r2x * (x - q * r1x) + q)];
    const int i = f ? fi : pw_idx[e];
    C2<double> out = mk<double>(double(v.x), double(v.y));
    if (ekpg) {
      const C2<double> s = f ? fs : ps[i];
      const double ek = f ? fe : ekpg[i];
      out.x += ek * s.x;
      out.y += ek * s.y;
    }
    if (p.accum) {
      const C2<double> h0 = hp[i];
      out.x += h0.x;
      out.y += h0.y;
    }
    hp[i] = out;
  }
}

// Threads of kernels A and C: one per line of the larger y pass.
template <int RY1, int RY2, int TC> constexpr int plane_threads() { return TC && RY1 ? TC * RY2 : kThreadsPlanes; }

// Launch kernel A alone (scatter + inverse x + inverse y into the slab W).
template <typename T, int RX1, int RX2, int RY1, int RY2, int TC>
cudaError_t launch_a_impl(const LocalPlan& p, int nbc, int band0, const C2<double>* psi, long long ldpsi,
                          const int* plane_start, const int* pw_idx, const int* pw_pos, const C2<T>* twx,
                          const C2<T>* twy, C2<T>* W, cudaStream_t st) {
  constexpr int NT = plane_threads<RY1, RY2, TC>();
  const size_t sm = smem_planes<T>(p);
  const bool pr = in_quarters(p.kd1, p.dx.r1, p.dx.r2) && in_quarters(p.kd2, p.dy.r1, p.dy.r2);
  auto* k = pr ? k_inv_xy<T, RX1, RX2, RY1, RY2, TC, true, NT> : k_inv_xy<T, RX1, RX2, RY1, RY2, TC, false, NT>;
  if constexpr (RX1 == 0 && sizeof(T) == 4)
    if (sm <= kManyPlaneBytes)
      k = pr ? k_inv_xy<T, RX1, RX2, RY1, RY2, TC, true, NT, true> : k_inv_xy<T, RX1, RX2, RY1, RY2, TC, false, NT, true>;
  cudaError_t e = smem_limit((const void*)k, sm);
  if (e != cudaSuccess) return e;
  k<<<dim3(p.nz, nbc), NT, sm, st>>>(p, band0, psi, ldpsi, plane_start, pw_idx, pw_pos, twx, twy, W);
  return cudaGetLastError();
}

// Launch kernel C alone (forward y + forward x from the slab W, gather).
template <typename T, int RX1, int RX2, int RY1, int RY2, int TC>
cudaError_t launch_c_impl(const LocalPlan& p, int nbc, int band0, const C2<double>* psi, long long ldpsi,
                          C2<double>* hpsi, long long ldh, const int* plane_start, const int* pw_idx,
                          const int* pw_pos, const double* ekpg, const C2<T>* twx, const C2<T>* twy, const C2<T>* W,
                          cudaStream_t st) {
  constexpr int NT = plane_threads<RY1, RY2, TC>();
  const size_t sm = smem_planes<T>(p);
  const bool pr = in_quarters(p.kd1, p.dx.r2, p.dx.r1) && in_quarters(p.kd2, p.dy.r2, p.dy.r1);
  auto* k = pr ? k_fwd_xy<T, RX1, RX2, RY1, RY2, TC, true, NT> : k_fwd_xy<T, RX1, RX2, RY1, RY2, TC, false, NT>;
  if constexpr (RX1 == 0 && sizeof(T) == 4)
    if (sm <= kManyPlaneBytes)
      k = pr ? k_fwd_xy<T, RX1, RX2, RY1, RY2, TC, true, NT, true> : k_fwd_xy<T, RX1, RX2, RY1, RY2, TC, false, NT, true>;
  cudaError_t e = smem_limit((const void*)k, sm);
  if (e != cudaSuccess) return e;
  k<<<dim3(p.nz, nbc), NT, sm, st>>>(p, band0, psi, ldpsi, hpsi, ldh, plane_start, pw_idx, pw_pos, ekpg, twx, twy, W);
  return cudaGetLastError();
}

// Band groups of kernel B: every CTA stages its V tile once (about 0.7 of a band's time) and then takes
// `per` bands; the split whose busiest SM finishes first. About three CTAs of an SM overlap: fewer take
// as long as one, more share it. p.bgroups > 0: that many CTAs per SM instead.
inline int band_groups(const LocalPlan& p, long long tiles, int nbc, int nsm) {
  if (p.bgroups > 0)
    return (int)std::max(1LL, std::min((long long)nbc, ((long long)p.bgroups * nsm + tiles - 1) / tiles));
  int best = 1;
  double cost = 1e300;
  for (int g = 1; g <= std::min(nbc, 64); ++g) {
    const double ctas = (double)((tiles * g + nsm - 1) / nsm);
    const double c = std::max(1.0, ctas / 3.0) * ((nbc + g - 1) / g + 0.7);
    if (c < cost * 0.99) {
      cost = c;
      best = g;
    }
  }
  return best;
}

// Launch the register form of kernel B for a z split R1 x R2.
template <typename T, int R1, int R2>
cudaError_t launch_z_impl(const LocalPlan& p, int nbc, const T* vr, const C2<T>* twz, C2<T>* W, int nsm,
                          cudaStream_t st) {
  constexpr int CB = 16;
  constexpr size_t sm = smem_z_band<T, R1, R2, CB>();
  auto* k = k_z_band<T, R1, R2, CB>;
  cudaError_t e = smem_limit((const void*)k, sm);
  if (e != cudaSuccess) return e;
  const long long tiles = (p.plane + CB - 1) / CB;
  const int g = band_groups(p, tiles, nbc, nsm), per = (nbc + g - 1) / g;
  k<<<dim3((unsigned)tiles, (unsigned)((nbc + per - 1) / per)), CB * R2, sm, st>>>(p, nbc, per, vr, twz, W);
  return cudaGetLastError();
}

// Launch the density's z stage. groups: band groups (part holds a box for each when there are several).
template <int R1, int R2>
cudaError_t launch_density_impl(const LocalPlan& p, int nbc, int groups, const double* occ, const C2<double>* twz,
                                const C2<double>* W, double* rho, double* part, cudaStream_t st) {
  constexpr int CB = 16;
  constexpr size_t sm = (size_t)R1 * R2 * (CB + 1) * sizeof(C2<double>);
  auto* k = k_z_density<R1, R2, CB>;
  cudaError_t e = smem_limit((const void*)k, sm);
  if (e != cudaSuccess) return e;
  const int per = (nbc + groups - 1) / groups;
  k<<<dim3((unsigned)((p.plane + CB - 1) / CB), groups), CB * R2, sm, st>>>(p, nbc, per, occ, twz, W, rho, part);
  return cudaGetLastError();
}

// Launch the non-collinear z stage for a z split R1 x R2.
template <typename T, int R1, int R2>
cudaError_t launch_spinor_impl(const LocalPlan& p, int nbc, const T* vu, const T* vd, const T* vr, const T* vi,
                               const C2<T>* twz, C2<T>* W, int nsm, cudaStream_t st) {
  constexpr int CB = 8;
  constexpr size_t sm = (size_t)R1 * R2 * (CB * (2 * sizeof(C2<T>) + 4 * sizeof(T)) + sizeof(C2<T>));
  auto* k = k_z_spinor_band<T, R1, R2, CB>;
  cudaError_t e = smem_limit((const void*)k, sm);
  if (e != cudaSuccess) return e;
  const long long tiles = (p.plane + CB - 1) / CB;
  const int g = band_groups(p, tiles, nbc, nsm), per = (nbc + g - 1) / g;
  k<<<dim3((unsigned)tiles, (unsigned)((nbc + per - 1) / per)), 2 * CB * R2, sm, st>>>(p, nbc, per, vu, vd, vr, vi, twz,
                                                                                  W);
  return cudaGetLastError();
}

}  // namespace kern

#define CPWB_INV_ARGS(T)                                                                                     \
  const LocalPlan &p, int nbc, int band0, const C2<double>*psi, long long ldpsi, const int *plane_start,     \
      const int *pw_idx, const int *pw_pos, const C2<T>*twx, const C2<T>*twy, C2<T>*W, cudaStream_t st

#define CPWB_LAUNCH_ARGS(T)                                                                                  \
  const LocalPlan &p, int nbc, int band0, const C2<double>*psi, long long ldpsi, C2<double>*hpsi,            \
      long long ldh, const int *plane_start, const int *pw_idx, const int *pw_pos, const double *ekpg,       \
      const T *vr, const C2<T>*twx, const C2<T>*twy, const C2<T>*twz, C2<T>*W, cudaStream_t st,             \
      cudaEvent_t *ev

#define CPWB_C_ARGS(T)                                                                                       \
  const LocalPlan &p, int nbc, int band0, const C2<double>*psi, long long ldpsi, C2<double>*hpsi,            \
      long long ldh, const int *plane_start, const int *pw_idx, const int *pw_pos, const double *ekpg,       \
      const C2<T>*twx, const C2<T>*twy, const C2<T>*W, cudaStream_t st
#define CPWB_Z_ARGS(T) const LocalPlan &p, int nbc, const T *vr, const C2<T>*twz, C2<T>*W, int nsm, cudaStream_t st

// kernels A and C for planes r1 r2 x r1 r2, kernel B for z lines of r1 r2 points
#define CPWB_PLANES(EXTERN, T, R1, R2, TC)                                                           \
  EXTERN template cudaError_t kern::launch_a_impl<T, R1, R2, R1, R2, TC>(CPWB_INV_ARGS(T));          \
  EXTERN template cudaError_t kern::launch_c_impl<T, R1, R2, R1, R2, TC>(CPWB_C_ARGS(T));
#define CPWB_LINES(EXTERN, T, R1, R2)                                                                       \
  EXTERN template cudaError_t kern::launch_z_impl<T, R1, R2>(CPWB_Z_ARGS(T));                               \
  EXTERN template cudaError_t kern::launch_spinor_impl<T, R1, R2>(                                          \
      const LocalPlan&, int, const T*, const T*, const T*, const T*, const C2<T>*, C2<T>*, int, cudaStream_t);
#define CPWB_DENSITY(EXTERN, R1, R2)                                                                        \
  EXTERN template cudaError_t kern::launch_density_impl<R1, R2>(const LocalPlan&, int, int, const double*,  \
                                                                const C2<double>*, const C2<double>*,       \
                                                                double*, double*, cudaStream_t);

}  // namespace cpwb
