// Kleinman-Bylander projector products P = X^H psi, hpsi += (X D) P (hk_psi_nl_c16.f90:82-97) as exact
// integer GEMMs modulo small coprime numbers on the 5th-generation tensor cores (kind::i8), put
// together with the Chinese remainder theorem. The scheme is "Ozaki scheme II" (Ozaki, Uchino,
// Imamura 2025): where the slice form (oz.cu) needs s (s + 1) / 2 products of s slices, this one
// needs one product per modulus.
//
//   * every real row a of one operand and b of the other is scaled by a power of two so that its
//     2-norm is at most 2^beta, and rounded to integers;
//   * for each modulus p_l the residues (signed bytes) are multiplied with exact int32 accumulation,
//     so that  sum a b  is known modulo P = p_1 ... p_L;
//   * |sum a b| <= 2^(beta_a + beta_b) < P / 4 (Cauchy-Schwarz), so the residues determine it.
// The only error is the rounding of the operands, ~0.4 2^-beta |a| |b| for a row pair: it follows the rows'
// norms, where a ZGEMM's follows sum |a_k b_k|. Projectors fall off with the plane wave's energy by orders of
// magnitude, so the projection is balanced first: plane wave k of X is divided and that of psi multiplied by the
// power of two at the norm of X's row k. Then |a| |b| is near sum |a_k b_k| whatever psi weighs, and X is
// held to 57 (L = 9: 34) bits of numbers of like size. Results do not depend on the tiling, the K splits or the
// other bands. L = 15 (beta 57 for X and X D, 58 for psi and P) takes the place of the FP64 ZGEMMs, L = 9 (beta 34
// and 35) that of split TF32. X D X^H psi, 2-norm of the error over that of the result, 26,398 plane waves and 256
// projectors (ZGEMM, L = 15, split TF32, L = 9):
//   psi                                  norm-wise                        median over the elements
//   1 / (1 + ekpg)^2                     1.4e-15 8.2e-16 2.1e-7 6.7e-9    1.3e-15 1.2e-15 2.1e-7 9.5e-9
//   one plane wave, 1e-6 of the others   1.4e-15 4.6e-16 2.1e-7 2.1e-9    2.0e-15 1.7e-15 2.5e-7 8.2e-9
//   the highest 30 % of energies alone   1.1e-15 9.4e-16 2.1e-7 7.7e-9    1.1e-15 9.4e-16 2.1e-7 7.7e-9
// (without the balance 4.4e-12 and 3.8e-5 in the last row, 1.8e-16 and 1.4e-9 in the first).
//
// Complex products take three real ones per modulus (exact in residues, where the sums below cannot
// cancel digits away):
//   1. P = X^H psi (M na, N nb, K' = m bytes): T0 = Xr psi_r, T1 = Xi psi_i, T2 = (Xr - Xi)(psi_r + psi_i)
//        Re P = T0 + T1, Im P = T2 - T0 + T1
//   2. hpsi += (X D) P (M m, N nb, K' = na bytes): T0 = Xr Pr, T1 = Xi Pi, T2 = (Xr + Xi)(Pr + Pi)
//        Re = T0 - T1, Im = T2 - T0 - T1
// The three byte planes of X and of X D are converted once per projector set, those of psi and P on
// each call.
//
// What bounds it: kind::i8 products run at 4,096 multiply-adds per clock and SM here (counted by the
// tensor pipe's active cycles), so 2.3 P/s over the GPU. 480 bands of a 216-atom cell (88,951 plane
// waves, 864 projectors): FP64 ZGEMMs 17.0 ms; this form 4.6 ms, of which the two residue GEMMs take
// 2.9 ms (2.4 P/s: the tensor pipe's rate), the conversion of psi 0.86 + 0.1 ms and the reconstruction
// 0.75 ms (15 moduli; with 9 in place of split TF32: 5.9 -> 3.1 ms). Four real products per modulus
// (two rows per complex one) take 3.8 ms in the GEMMs.
//
// Operand tiles: 128 rows (X side) or nt rows (psi / P side) x 128 bytes of K', in the
// 128-byte-swizzled K-major order that the tensor cores read; tile (modulus, plane, row block, K
// block). Residues of the products are stored as [K split][modulus, plane][band / 4][row][4 bands].
#include <stdint.h>
#include <stdlib.h>

#include <algorithm>
#include <type_traits>
#include <utility>

#include "context.hpp"
#include "mma_i8.cuh"

namespace cpwb {
namespace crt {

using namespace mma8;

constexpr int kMaxL = 16;
// pairwise coprime, the largest first: residues are signed bytes
__host__ __device__ constexpr int modulus(int l) {
  constexpr int p[kMaxL] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197, 193};
  return p[l];
}
// floor(u / p) = (u * reciprocal) >> 39 for u < 2^31 (128 < p <= 256)
__host__ __device__ constexpr uint32_t reciprocal(int p) { return (uint32_t)((1ull << 39) / (unsigned)p + (p == 256 ? 0 : 1)); }
__host__ __device__ constexpr int pow2_mod(int e, int p) {      // 2^e mod p, symmetric
  int r = 1;
  for (int i = 0; i < e; ++i) r = r * 2 % p;
  return r > p / 2 ? r - p : r;
}

constexpr int BM = 128;
constexpr int KB = 128;                 // bytes of K' per block
constexpr int kATile = BM * KB;
constexpr int kMaxNt = 256;             // columns per output tile
constexpr int kMaxStages = 8;
constexpr int kMaxKb = 512;             // K blocks per int32 accumulation: 127^2 * 65,536 < 2^30.0
constexpr int kDrainWarps = 8;
constexpr int kThreads = 32 * (2 + kDrainWarps);
constexpr int kTmemCols = 512;          // two accumulators of 256 columns
constexpr int kBarBytes = 256;
constexpr int kNanScale = INT32_MIN;    // row or column with a NaN or an infinity

// the low bytes of four words
__device__ __forceinline__ uint32_t pack4(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
}

// ------------------------------------------------------------------ residue GEMM
struct GemmArgs {
  const int8_t* a;          // [lc][tile_m][kb] tiles of 16 KB, lc = 3 modulus + plane
  const int8_t* b;          // [lc][tile_n][kb] tiles of nt * 128 bytes
  uint32_t* r;              // [split][lc][n / 4][ldr] residues in [0, p) of 4 columns
  int N, nt, tiles_m, tiles_n;
  int nkb, kb_per_split, nsplit, L;
  int stages;
  long long ldr;            // tiles_m * 128
  int p[kMaxL];
  uint32_t rcp[kMaxL], off[kMaxL];
  int* err;
  unsigned long long wait_ns;
};

struct Item {
  int lc, mt, nt, split, kb0, nblk;
};

// consecutive items share the modulus, plane and K range, then the X tile
__device__ __forceinline__ Item item_of(const GemmArgs& g, int it) {
  Item w;
  w.nt = it % g.tiles_n;
  it /= g.tiles_n;
  w.mt = it % g.tiles_m;
  it /= g.tiles_m;
  w.split = it % g.nsplit;
  w.lc = it / g.nsplit;
  w.kb0 = w.split * g.kb_per_split;
  w.nblk = min(g.nkb, w.kb0 + g.kb_per_split) - w.kb0;
  return w;
}

// Persistent: one CTA per SM loops over (modulus, K range, output tile). Warp 0 streams the tiles of
// both operands through a ring of stages, warp 1 issues the products (M 128, N nt, K 32) into one of
// two TMEM accumulators, warps 2-9 reduce the other one modulo p and store its residues, so that the
// drain (4 integer instructions per value, one 128-byte store per warp and 4 columns) runs beside the
// next tile's products.
__global__ void __launch_bounds__(kThreads, 1) k_crt_gemm(const __grid_constant__ GemmArgs g) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* ring = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t bytes_b = (uint32_t)g.nt * KB;
  const uint32_t stage_bytes = kATile + bytes_b;
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + (size_t)g.stages * stage_bytes);
  uint64_t* empty = full + kMaxStages;
  uint64_t* accf = empty + kMaxStages;       // [2] accumulator complete (MMA -> drain)
  uint64_t* acce = accf + 2;                 // [2] accumulator read (drain -> MMA)
  uint64_t* done = acce + 2;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
  __shared__ volatile int failed;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nitems = 3 * g.L * g.nsplit * g.tiles_m * g.tiles_n;
  const size_t nkb = (size_t)g.nkb;

  if (threadIdx.x == 0) {
    failed = 0;
    for (int i = 0; i < g.stages; ++i) {
      mbar_init(smem_u32(&full[i]), 1);
      mbar_init(smem_u32(&empty[i]), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&accf[i]), 1);
      mbar_init(smem_u32(&acce[i]), kDrainWarps);
    }
    mbar_init(smem_u32(done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tslot)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n");
  const uint32_t tmem = *tslot;

  if (warp == 0) {
    if (lane == 0) {
      int s = 0;
      uint32_t ph = 1;                       // parity of the "empty" phase waited for (first round passes)
      long long issued = 0;
      for (int it = blockIdx.x; it < nitems && !failed; it += gridDim.x) {
        const Item w = item_of(g, it);
        const int8_t* a = g.a + (((size_t)w.lc * g.tiles_m + w.mt) * nkb + w.kb0) * kATile;
        const int8_t* b = g.b + (((size_t)w.lc * g.tiles_n + w.nt) * nkb + w.kb0) * bytes_b;
        for (int i = 0; i < w.nblk; ++i) {
          if (!mbar_wait(smem_u32(&empty[s]), ph, &failed, g.wait_ns)) {
            failed = 1;
            atomicExch(g.err, 1);
            break;
          }
          const uint32_t st = smem_u32(ring) + (uint32_t)s * stage_bytes, fb = smem_u32(&full[s]);
          mbar_expect_tx(fb, stage_bytes);
          bulk_load(st, a + (size_t)i * kATile, kATile, fb);
          bulk_load(st + kATile, b + (size_t)i * bytes_b, bytes_b, fb);
          ++issued;
          if (++s == g.stages) {
            s = 0;
            ph ^= 1;
          }
        }
      }
      // copies still in flight land before the CTA may exit
      for (long long i = (issued > g.stages ? issued - g.stages : 0); i < issued; ++i)
        if (!mbar_wait(smem_u32(&full[i % g.stages]), (uint32_t)((i / g.stages) & 1), nullptr)) atomicExch(g.err, 1);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = instr_desc_i8(BM, g.nt);
      int s = 0, nit = 0;
      uint32_t ph = 0;
      for (int it = blockIdx.x; it < nitems && !failed; it += gridDim.x, ++nit) {
        const Item w = item_of(g, it);
        const int buf = nit & 1;
        // the item before the previous one has been read out of this accumulator
        if (nit >= 2 && !mbar_wait(smem_u32(&acce[buf]), (uint32_t)((nit / 2 - 1) & 1), &failed, g.wait_ns)) {
          failed = 1;
          atomicExch(g.err, 1);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;\n");
        const uint32_t tacc = tmem + (uint32_t)(buf * 256);
        bool ok = true;
        for (int i = 0; i < w.nblk; ++i) {
          if (!mbar_wait(smem_u32(&full[s]), ph, &failed, g.wait_ns)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;\n");
          const uint32_t st = smem_u32(ring) + (uint32_t)s * stage_bytes;
          const uint64_t da = smem_desc(st), db = smem_desc(st + kATile);
#pragma unroll
          for (int ks = 0; ks < KB / 32; ++ks)
            mma_i8(tacc, da + (uint64_t)(2 * ks), db + (uint64_t)(2 * ks), idesc, (i == 0 && ks == 0) ? 0u : 1u);
          mma_commit(smem_u32(&empty[s]));
          if (++s == g.stages) {
            s = 0;
            ph ^= 1;
          }
        }
        if (!ok) {
          failed = 1;
          atomicExch(g.err, 1);
          break;
        }
        mma_commit(smem_u32(&accf[buf]));
      }
      // every MMA of this thread completes before TMEM is freed
      mma_commit(smem_u32(done));
      if (!mbar_wait(smem_u32(done), 0u, nullptr)) atomicExch(g.err, 1);
    }
  } else {
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const uint32_t lane_base = tmem + ((uint32_t)(32 * quarter) << 16);
    const int ncol = g.nt / 2;                // columns of this warp's half: a multiple of 8
    int nit = 0;
    for (int it = blockIdx.x; it < nitems; it += gridDim.x, ++nit) {
      const Item w = item_of(g, it);
      const int buf = nit & 1;
      if (!mbar_wait_warp(smem_u32(&accf[buf]), (uint32_t)((nit / 2) & 1), &failed, g.wait_ns)) {
        failed = 1;
        atomicExch(g.err, 1);
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;\n");
      const uint32_t p = (uint32_t)g.p[w.lc / 3], rcp = g.rcp[w.lc / 3], off = g.off[w.lc / 3];
      const int n0 = w.nt * g.nt + half * ncol, n4 = (g.N + 3) / 4;
      uint32_t* out = g.r + (((size_t)w.split * 3 * g.L + w.lc) * n4 + n0 / 4) * g.ldr + w.mt * BM + 32 * quarter + lane;
      const uint32_t tcol = lane_base + (uint32_t)(buf * 256 + half * ncol);
      const int nq = min(ncol / 4, n4 - n0 / 4);       // groups of 4 columns to store
      auto store = [&](const uint32_t* v) {
        uint32_t b[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint32_t u = v[t] + off;                 // off: a multiple of p, u < 2^31
          b[t] = u - (__umulhi(u, rcp) >> 7) * p;
        }
        *out = pack4(b[0], b[1], b[2], b[3]);
        out += g.ldr;
      };
      int q = 0;
      for (; q + 4 <= nq; q += 4) {
        uint32_t v[2][8];
        tmem_ld8(tcol + 4 * q, v[0]);
        tmem_ld8(tcol + 4 * q + 8, v[1]);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        store(v[0]);
        store(v[0] + 4);
        store(v[1]);
        store(v[1] + 4);
      }
      for (; q < nq; q += 2) {
        uint32_t v[8];
        tmem_ld8(tcol + 4 * q, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        store(v);
        if (q + 1 < nq) store(v + 4);
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&acce[buf]));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTmemCols));
}

// ------------------------------------------------------------------ operands to residues
// Norm of a row or column: the exponent e with |x|_2 < 2^e. The squares are summed as they are and
// scaled by 2^-600 and 2^600, for rows whose squares would overflow or underflow. A NaN or infinity
// marks the row: everything computed from it becomes NaN.
constexpr double kDown = 2.409919865102884e-181, kUp = 4.149515568880993e+180;      // 2^-600, 2^600
struct Norm {
  double ss, hi, lo, mx;
};
__device__ __forceinline__ void norm_add(Norm& n, double v) {
  n.ss = fma(v, v, n.ss);
  n.hi = fma(v * kDown, v * kDown, n.hi);
  n.lo = fma(v * kUp, v * kUp, n.lo);
  const double a = fabs(v);
  n.mx = (a > n.mx || a != a) ? a : n.mx;     // a NaN replaces the maximum and stays
}
__device__ __forceinline__ Norm norm_join(Norm a, Norm b) {
  Norm r;
  r.ss = a.ss + b.ss;
  r.hi = a.hi + b.hi;
  r.lo = a.lo + b.lo;
  r.mx = (b.mx > a.mx || b.mx != b.mx) ? b.mx : a.mx;
  return r;
}
// the power of two s that scales the row to a norm of at most 2^beta (kNanScale: not finite)
__device__ __forceinline__ int norm_scale(Norm n, int beta) {
  if (!(n.mx < __longlong_as_double(0x7ff0000000000000LL))) return kNanScale;
  if (n.mx == 0.0) return 0;
  int e;
  const double margin = 1.0 + 1e-9;             // of the sum's rounding
  if (n.mx < 1e-130) {
    frexp(sqrt(n.lo) * margin, &e);
    e -= 600;
  } else if (n.mx < 1e130) {
    frexp(sqrt(n.ss) * margin, &e);
  } else {
    frexp(sqrt(n.hi) * margin, &e);
    e += 600;
  }
  return beta - e;
}
__device__ __forceinline__ Norm warp_norm(Norm n) {
  for (int o = 16; o > 0; o >>= 1) {
    Norm b;
    b.ss = __shfl_xor_sync(0xffffffffu, n.ss, o);
    b.hi = __shfl_xor_sync(0xffffffffu, n.hi, o);
    b.lo = __shfl_xor_sync(0xffffffffu, n.lo, o);
    b.mx = __shfl_xor_sync(0xffffffffu, n.mx, o);
    n = norm_join(n, b);
  }
  return n;
}
// over the block, for every thread (sh: 32 entries)
__device__ __forceinline__ Norm block_norm(Norm n, Norm* sh) {
  n = warp_norm(n);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = n;
  __syncthreads();
  Norm r = sh[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) r = norm_join(r, sh[w]);
  return r;
}

// y = round(v 2^s) split as y0 + y1 2^20 + y2 2^40 (|v 2^s| <= 2^62)
struct Limbs {
  int y0, y1, y2;
};
struct Scale {
  double f1, f2;        // 2^s as a product: s alone can leave the range of a double
};
__device__ __forceinline__ double pow2(int e) { return __longlong_as_double((long long)(e + 1023) << 52); }
__device__ __forceinline__ Scale scale_of(int s) {
  Scale f;
  if (s == kNanScale) {
    f.f1 = f.f2 = 0.0;
    return f;
  }
  f.f1 = pow2(s / 2);
  f.f2 = pow2(s - s / 2);
  return f;
}
__device__ __forceinline__ Limbs limbs(double v, Scale f) {
  const double t = f.f1 == 0.0 ? 0.0 : v * f.f1 * f.f2;     // NaN rows convert as zeros
  const long long y = __double2ll_rn(t);
  Limbs r;
  r.y0 = (int)(y & 0xFFFFF);
  r.y1 = (int)((y >> 20) & 0xFFFFF);
  r.y2 = (int)(y >> 40);
  return r;
}
// (y + h) mod p_l in [0, p_l), h = p_l / 2: less h it is the signed byte that is multiplied
template <int l> __device__ __forceinline__ uint32_t residue(Limbs y) {
  constexpr int p = modulus(l), h = p / 2;
  if constexpr (p == 256) {
    return (uint32_t)(y.y0 + h) & 0xff;
  } else {
    constexpr int c1 = pow2_mod(20, p), c2 = pow2_mod(40, p);
    constexpr uint32_t rcp = reciprocal(p);
    // |y0 + y1 c1 + y2 c2| < 2^20 + 127 (2^20 + 2^22) < p 2^22; u < 2^31
    const uint32_t u = (uint32_t)(y.y0 + y.y1 * c1 + y.y2 * c2 + (p << 22) + h);
    return u - (__umulhi(u, rcp) >> 7) * (uint32_t)p;
  }
}

// The bytes of 8 complex numbers in the three planes (re, im, re + im or re - im) modulo p_0 .. p_{L-1}:
// put(3 l + plane, 8 bytes)
template <int L, bool DIFF, int l = 0, class F>
__device__ __forceinline__ void residues8(const Limbs (&re)[8], const Limbs (&im)[8], F&& put) {
  if constexpr (l < L) {
    constexpr uint32_t p = modulus(l), h = p / 2;
    uint32_t a[8], b[8], c[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      a[u] = residue<l>(re[u]);
      b[u] = residue<l>(im[u]);
      uint32_t t = DIFF ? a[u] - b[u] + h : a[u] + b[u] - h;      // in (-p, 2 p), modulo 2^32
      t = min(t, t + p);
      c[u] = min(t, t - p) - h;
      a[u] -= h;
      b[u] -= h;
    }
    put(3 * l, make_uint2(pack4(a[0], a[1], a[2], a[3]), pack4(a[4], a[5], a[6], a[7])));
    put(3 * l + 1, make_uint2(pack4(b[0], b[1], b[2], b[3]), pack4(b[4], b[5], b[6], b[7])));
    put(3 * l + 2, make_uint2(pack4(c[0], c[1], c[2], c[3]), pack4(c[4], c[5], c[6], c[7])));
    residues8<L, DIFF, l + 1>(re, im, put);
  }
}
// offset of the 8-byte piece c (0..15) of row r inside a 128-byte-row swizzled tile
__device__ __forceinline__ int swz8(int r, int c) { return r * KB + (((c >> 1) ^ (r & 7)) << 4) + ((c & 1) << 3); }

constexpr int kNormChunk = 4096;       // complex numbers per block of the column norms

// Norms of 32 rows of a complex block (m rows, K columns): a warp takes every kRowThreads / 32-th column of them, warp
// 0 returns the sum
constexpr int kRowThreads = 256;
__device__ __forceinline__ Norm row_norm(int m, int K, const double2* __restrict__ x, long long ldx) {
  __shared__ Norm sh[kRowThreads];
  const int lane = threadIdx.x & 31, i = blockIdx.x * 32 + lane;
  Norm n{0.0, 0.0, 0.0, 0.0};
  if (i < m) {
#pragma unroll 8
    for (int k = threadIdx.x >> 5; k < K; k += kRowThreads / 32) {
      const double2 v = x[(size_t)k * ldx + i];
      norm_add(n, v.x);
      norm_add(n, v.y);
    }
  }
  sh[threadIdx.x] = n;
  __syncthreads();
  if (threadIdx.x < 32)
    for (int t = 1; t < kRowThreads / 32; ++t) n = norm_join(n, sh[32 * t + lane]);
  return n;
}

// Weights of the plane waves: w = the power of two above the norm of X's row, and its inverse. Zero where the row is
// zero (a NaN or an infinity of psi stays one there, as in the product with the zeros).
__global__ void __launch_bounds__(kRowThreads) k_crt_weights(int m, int K, const double2* __restrict__ x, long long ldx,
                                                             double* __restrict__ w, double* __restrict__ winv) {
  const Norm n = row_norm(m, K, x, ldx);
  const int i = blockIdx.x * 32 + threadIdx.x;
  if (threadIdx.x >= 32 || i >= m) return;
  const int s = norm_scale(n, 0), e = s == kNanScale ? 0 : max(-900, min(900, -s));
  w[i] = n.mx == 0.0 ? 0.0 : pow2(e);
  winv[i] = n.mx == 0.0 ? 0.0 : pow2(-e);
}

// partial norms of the columns of a complex block with weighted rows: part[chunk][ncol]
__global__ void __launch_bounds__(256) k_crt_norm_cols(int m, int ncol, const double2* __restrict__ x, long long ldx,
                                                       const double* __restrict__ w, Norm* __restrict__ part) {
  __shared__ Norm sh[32];
  const int col = blockIdx.x, k0 = blockIdx.y * kNormChunk, k1 = min(m, k0 + kNormChunk);
  const double2* c = x + (size_t)col * ldx;
  Norm n{0.0, 0.0, 0.0, 0.0};
#pragma unroll 4
  for (int k = k0 + threadIdx.x; k < k1; k += 256) {
    const double2 v = c[k];
    const double f = w[k];
    norm_add(n, v.x * f);
    norm_add(n, v.y * f);
  }
  n = block_norm(n, sh);
  if (threadIdx.x == 0) part[(size_t)blockIdx.y * ncol + col] = n;
}

// the rows' scale exponents
__global__ void __launch_bounds__(kRowThreads) k_crt_norm_rows(int m, int K, const double2* __restrict__ x,
                                                               long long ldx, int beta, int* __restrict__ s) {
  const Norm n = row_norm(m, K, x, ldx);
  const int i = blockIdx.x * 32 + threadIdx.x;
  if (threadIdx.x < 32 && i < m) s[i] = norm_scale(n, beta);
}

// Columns of a complex block along K' (contiguous): column n becomes row n of the three planes. One
// block converts 2,048 complex numbers of one column, staged through shared memory so that its loads
// are coalesced (16-byte loads of 8 consecutive numbers per thread would touch 32 lines each). Rows weighted as
// in the norms (w null: not).
constexpr int kConvPer = 256 * 8;
template <int L, bool DIFF>
__global__ void __launch_bounds__(256) k_crt_conv_cols(int m, int ncol, const double2* __restrict__ x, long long ldx,
                                                       const double* __restrict__ w, const Norm* __restrict__ part,
                                                       int nchunk, int beta, int rows, int tiles, int nkb,
                                                       int8_t* __restrict__ out, int* __restrict__ sout) {
  __shared__ double2 buf[256 * 9];
  const int col = blockIdx.y, k0 = blockIdx.x * kConvPer, tid = threadIdx.x;
  Norm n{0.0, 0.0, 0.0, 0.0};
  for (int c = 0; c < nchunk; ++c) n = norm_join(n, part[(size_t)c * ncol + col]);
  const int s = norm_scale(n, beta);
  if (blockIdx.x == 0 && tid == 0) sout[col] = s;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int t = tid + 256 * j, k = k0 + t;
    double2 v = k < m ? x[(size_t)col * ldx + k] : make_double2(0.0, 0.0);
    if (w && k < m) {
      const double f = w[k];
      v.x *= f;
      v.y *= f;
    }
    buf[(t >> 3) * 9 + (t & 7)] = v;
  }
  __syncthreads();
  const int ch = (k0 >> 3) + tid, kb = ch >> 4;        // 8-byte piece of the row, its K block
  if (kb >= nkb) return;
  const Scale f = scale_of(s);
  Limbs re[8], im[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const double2 v = buf[tid * 9 + u];
    re[u] = limbs(v.x, f);
    im[u] = limbs(v.y, f);
  }
  int8_t* o = out + ((size_t)(col / rows) * nkb + kb) * rows * KB + swz8(col % rows, ch & 15);
  const size_t plane = (size_t)tiles * nkb * rows * KB;
  residues8<L, DIFF>(re, im, [&](int lc, uint2 w) { *reinterpret_cast<uint2*>(o + lc * plane) = w; });
}

// Rows of a complex block (m x K, columns strided): row i of the X-side planes of the expansion. One block
// converts the 128 complex numbers of one K block of 16 rows, staged through shared memory: its loads are
// 256 contiguous bytes per column and a warp stores two whole rows of a tile (a thread per row stored
// pieces of 8 bytes that lie 128 apart).
template <int L>
__global__ void __launch_bounds__(256) k_crt_conv_rows(int m, int K, const double2* __restrict__ x, long long ldx,
                                                       const int* __restrict__ s, int tiles, int nkb,
                                                       int8_t* __restrict__ out) {
  constexpr int kRow = 16 * 9 + 1;        // a row's 16 pieces of 8 numbers, spread over the banks
  __shared__ double2 buf[16 * kRow];
  const int i0 = blockIdx.x * 16, kb = blockIdx.y, tid = threadIdx.x;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int t = tid + 256 * j, row = t & 15, k = t >> 4, kk = kb * KB + k;
    buf[row * kRow + (k >> 3) * 9 + (k & 7)] =
        i0 + row < m && kk < K ? x[(size_t)kk * ldx + i0 + row] : make_double2(0.0, 0.0);
  }
  __syncthreads();
  const int row = tid >> 4, c = tid & 15, i = i0 + row;
  if (i >= m) return;
  const Scale f = scale_of(s[i]);
  Limbs re[8], im[8];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    const double2 v = buf[row * kRow + c * 9 + u];
    re[u] = limbs(v.x, f);
    im[u] = limbs(v.y, f);
  }
  int8_t* o = out + ((size_t)(i / BM) * nkb + kb) * kATile + swz8(i % BM, c);
  const size_t plane = (size_t)tiles * nkb * kATile;
  residues8<L, false>(re, im, [&](int lc, uint2 w) { *reinterpret_cast<uint2*>(o + lc * plane) = w; });
}

// ------------------------------------------------------------------ residues to numbers
// x = sum_l r_l w_l - k P with w_l = 1 mod p_l and 0 modulo the others, |x| < P / 4. The weights are
// kept to their leading 80 bits (four limbs of 20): what is dropped is below 2^-66 of P, far below
// the operands' rounding (2^-beta of the norms).
struct Weights {
  uint32_t w[kMaxL][4], P[4];
  float f3, f2;             // 2^(60 + drop) / P and 2^(40 + drop) / P
  int drop;                 // dropped low bits
};

// limb sums s[plane][limb] = sum_l r_l w_l of the three planes, four columns from one word per plane
struct Sums {
  uint32_t s[3][4];
};
__device__ __forceinline__ void add_residue(uint32_t (&s)[4], uint32_t r, const uint32_t (&w)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) s[j] += r * w[j];
}
// the number with the residues a s0 + b s1 + c s2, in units of 2^drop
__device__ __forceinline__ double crt_value(const Sums& S, int a, int b, int c, const Weights& W) {
  long long t[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) t[j] = (long long)a * S.s[0][j] + (long long)b * S.s[1][j] + (long long)c * S.s[2][j];
  const int k = __float2int_rn(fmaf((float)t[3], W.f3, (float)t[2] * W.f2));
#pragma unroll
  for (int j = 0; j < 4; ++j) t[j] -= (long long)k * W.P[j];
  long long lo = (t[1] << 20) + t[0], hi = (t[3] << 20) + t[2];
  hi += lo >> 40;
  lo &= (1LL << 40) - 1;
  return fma((double)hi, 1099511627776.0, (double)lo);       // 2^40
}
__device__ __forceinline__ double scaled(double x, int sa, int sb, int drop) {
  if (sa == kNanScale || sb == kNanScale) return __longlong_as_double(0x7ff8000000000000LL);
  const int e = drop - sa - sb;
  return e > -900 && e < 800 ? x * pow2(e) : ldexp(x, e);
}

// P(a, n) from the residues of the projection (K splits summed), one row and four bands per thread, and
// the partial norms of its columns: part[row block][nb]
template <int L>
__global__ void __launch_bounds__(128) k_crt_p(const __grid_constant__ Weights W, int na, int nb, int nsplit,
                                               const uint32_t* __restrict__ r, long long ldr,
                                               const int* __restrict__ sa, const int* __restrict__ sb,
                                               double2* __restrict__ P, Norm* __restrict__ part) {
  __shared__ Norm sh[32];
  const int a = blockIdx.x * 128 + threadIdx.x, n4 = (nb + 3) / 4, q4 = blockIdx.y;
  Sums S[4] = {};
  if (a < na) {
    // three moduli at a time: the nine words of a split are loaded together, so that their latencies
    // overlap (one modulus at a time: 83 us for the 256 x 160 P of a 64-atom cell over 18 splits)
#pragma unroll
    for (int l0 = 0; l0 < L; l0 += 3) {
      uint32_t even[9], odd[9];             // 16-bit sums over the splits (at most 257 of them)
#pragma unroll
      for (int c = 0; c < 9; ++c) even[c] = odd[c] = 0;
      const uint32_t* rp = r + ((size_t)3 * l0 * n4 + q4) * ldr + a;
#pragma unroll 2
      for (int sp = 0; sp < nsplit; ++sp, rp += (size_t)3 * L * n4 * ldr) {
        uint32_t w[9];
#pragma unroll
        for (int c = 0; c < 9; ++c) w[c] = rp[(size_t)c * n4 * ldr];
#pragma unroll
        for (int c = 0; c < 9; ++c) {
          even[c] += w[c] & 0x00FF00FF;
          odd[c] += (w[c] >> 8) & 0x00FF00FF;
        }
      }
#pragma unroll
      for (int c = 0; c < 9; ++c) {
        const uint32_t p = modulus(l0 + c / 3), rcp = reciprocal(modulus(l0 + c / 3));
        const uint32_t v[4] = {even[c] & 0xFFFF, odd[c] & 0xFFFF, even[c] >> 16, odd[c] >> 16};
#pragma unroll
        for (int t = 0; t < 4; ++t) add_residue(S[t].s[c % 3], v[t] - (__umulhi(v[t], rcp) >> 7) * p, W.w[l0 + c / 3]);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const int n = 4 * q4 + t;
    Norm nm{0.0, 0.0, 0.0, 0.0};
    if (a < na && n < nb) {
      double2 v;
      v.x = scaled(crt_value(S[t], 1, 1, 0, W), sa[a], sb[n], W.drop);       // Re = T0 + T1
      v.y = scaled(crt_value(S[t], -1, 1, 1, W), sa[a], sb[n], W.drop);      // Im = T2 - T0 + T1
      P[(size_t)n * na + a] = v;
      norm_add(nm, v.x);
      norm_add(nm, v.y);
    }
    nm = block_norm(nm, sh);
    if (threadIdx.x == 0 && n < nb) part[(size_t)blockIdx.x * nb + n] = nm;
  }
}

// hpsi(:, n) += X D P (:, n) from the residues of the expansion, one row and four bands per thread
template <int L>
__global__ void __launch_bounds__(128) k_crt_out(const __grid_constant__ Weights W, int m, int nb,
                                                 const uint32_t* __restrict__ r, long long ldr,
                                                 const int* __restrict__ sa, const int* __restrict__ sb,
                                                 double2* __restrict__ hpsi, long long ldh) {
  const int i = blockIdx.x * 128 + threadIdx.x, n4 = (nb + 3) / 4, q4 = blockIdx.y;
  if (i >= m) return;
  Sums S[4] = {};
  const uint32_t* rp = r + (size_t)q4 * ldr + i;
  const size_t plane = (size_t)n4 * ldr;
  // the words of the next three moduli are loaded while those of this group are summed
  uint32_t w[9], wn[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) w[c] = rp[c * plane];
#pragma unroll
  for (int l0 = 0; l0 < L; l0 += 3) {
    if (l0 + 3 < L) {
#pragma unroll
      for (int c = 0; c < 9; ++c) wn[c] = rp[(3 * l0 + 9 + c) * plane];
    }
#pragma unroll
    for (int c = 0; c < 9; ++c)
#pragma unroll
      for (int t = 0; t < 4; ++t) add_residue(S[t].s[c % 3], (w[c] >> (8 * t)) & 0xff, W.w[l0 + c / 3]);
#pragma unroll
    for (int c = 0; c < 9; ++c) w[c] = wn[c];
  }
  const int si = sa[i];
  double2* h = hpsi + (size_t)4 * q4 * ldh + i;
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (4 * q4 + t < nb) {
      const int sn = sb[4 * q4 + t];
      double2 o = h[(size_t)t * ldh];
      o.x += scaled(crt_value(S[t], 1, -1, 0, W), si, sn, W.drop);       // Re = T0 - T1
      o.y += scaled(crt_value(S[t], -1, -1, 1, W), si, sn, W.drop);      // Im = T2 - T0 - T1
      h[(size_t)t * ldh] = o;
    }
}

// ------------------------------------------------------------------ host side
using u128 = unsigned __int128;

struct Plan {
  Weights w;
  int beta_a, beta_b;       // bits of the X-side and psi-side rows
};

int inverse_mod(int a, int p) {
  for (int x = 1; x < p; ++x)
    if ((long long)a * x % p == 1) return x;
  return 0;
}

Plan make_plan(int L) {
  Plan pl{};
  u128 P = 1;
  for (int l = 0; l < L; ++l) P *= (unsigned)modulus(l);
  int bits = 0;
  for (u128 t = P; t; t >>= 1) ++bits;                 // 2^(bits - 1) <= P < 2^bits
  pl.beta_a = (bits - 3) / 2;                          // beta_a + beta_b = bits - 3: products below P / 4
  pl.beta_b = bits - 3 - pl.beta_a;
  const int drop = std::max(0, bits - 80);
  pl.w.drop = drop;
  auto limb = [&](u128 v, int j) { return (uint32_t)((v >> (drop + 20 * j)) & 0xFFFFF); };
  for (int l = 0; l < L; ++l) {
    const u128 q = P / (unsigned)modulus(l);
    const u128 w = q * (unsigned)inverse_mod((int)(q % (unsigned)modulus(l)), modulus(l));
    for (int j = 0; j < 4; ++j) pl.w.w[l][j] = limb(w, j);
  }
  for (int j = 0; j < 4; ++j) pl.w.P[j] = limb(P, j);
  const double Pd = (double)(unsigned long long)(P >> 64) * 18446744073709551616.0 + (double)(unsigned long long)P;
  pl.w.f3 = (float)(ldexp(1.0, 60 + drop) / Pd);
  pl.w.f2 = (float)(ldexp(1.0, 40 + drop) / Pd);
  return pl;
}

template <class F> void with_moduli(int L, F f) {
  if (L == 15)
    f(std::integral_constant<int, 15>{});
  else
    f(std::integral_constant<int, 9>{});
}

// columns per tile: the fewest tiles of at most kMaxNt, as even as multiples of 16 allow
int tile_cols(int n) {
  const int t = (n + kMaxNt - 1) / kMaxNt;
  return ((n + t - 1) / t + 15) / 16 * 16;
}

cudaError_t launch_gemm(GemmArgs g, int nsm, cudaStream_t st) {
  const size_t stage = kATile + (size_t)g.nt * KB;
  g.stages = (int)std::max<size_t>(2, std::min<size_t>(kMaxStages, (size_t)(220 * 1024 - 1024 - kBarBytes) / stage));
  const size_t smem = 1024 + g.stages * stage + kBarBytes;
  for (int l = 0; l < g.L; ++l) {
    const uint32_t p = (uint32_t)modulus(l);
    g.p[l] = (int)p;
    g.rcp[l] = reciprocal((int)p);
    g.off[l] = (uint32_t)(((1u << 30) + p - 1) / p * p);
  }
  cudaError_t e = smem_limit((const void*)k_crt_gemm, smem);
  if (e != cudaSuccess) return e;
  const int items = 3 * g.L * g.nsplit * g.tiles_m * g.tiles_n;
  k_crt_gemm<<<std::min(items, nsm), kThreads, smem, st>>>(g);
  return cudaGetLastError();
}

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

int num_sms() {
  int dev = 0, nsm = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  return nsm;
}

}  // namespace crt

// One buffer: planes of X, planes of X D, row scales of both and weights, partial norms (each cudaMalloc costs a
// few hundred microseconds). Rows past the last one of a tile stay undefined: what they give is not read.
struct CrtPlanes {
  size_t b1, b2, bs, total;
};
static CrtPlanes planes_of(int m, int na, int L) {
  using namespace crt;
  CrtPlanes y{};
  const size_t row = 3 * (size_t)L * kATile;
  y.b1 = row * ((na + BM - 1) / BM) * ((m + KB - 1) / KB);
  y.b2 = row * ((m + BM - 1) / BM) * ((na + KB - 1) / KB);
  y.bs = align256(sizeof(int) * ((size_t)na + m)) + align256(2 * sizeof(double) * (size_t)m);
  y.total = y.b1 + y.b2 + y.bs + sizeof(Norm) * (size_t)((m + kNormChunk - 1) / kNormChunk) * na;
  return y;
}
size_t crt_plane_bytes(int m, int na, int L) { return planes_of(m, na, L).total; }

// Convert X (anl, m x na, ld m) and X D (anld) once per projector set, on st: a call on another stream is ordered
// behind it as behind any earlier call, whose slab and scratch it shares.
int crt_prepare(CrtOperands& o, int m, int na, int L, const void* anl, const void* anld, cudaStream_t st) {
  using namespace crt;
  o.L = 0;
  const Plan pl = make_plan(L);
  o.nkb1 = (m + KB - 1) / KB;
  o.nkb2 = (na + KB - 1) / KB;
  o.tiles1 = (na + BM - 1) / BM;
  o.tiles2 = (m + BM - 1) / BM;
  const int nchunk = (m + kNormChunk - 1) / kNormChunk;
  const CrtPlanes y = planes_of(m, na, L);
  if (int s = o.buf.ensure(y.total)) return s;
  o.a1 = (int8_t*)o.buf.p;
  o.a2 = o.a1 + y.b1;
  o.s1 = (int*)(o.a2 + y.b2);
  o.s2 = o.s1 + na;
  o.w = (double*)(o.a2 + y.b2 + align256(sizeof(int) * ((size_t)na + m)));
  Norm* part = (Norm*)(o.a2 + y.b2 + y.bs);
  k_crt_weights<<<(m + 31) / 32, kRowThreads, 0, st>>>(m, na, (const double2*)anl, m, o.w, o.w + m);
  k_crt_norm_cols<<<dim3(na, nchunk), 256, 0, st>>>(m, na, (const double2*)anl, m, o.w + m, part);
  k_crt_norm_rows<<<(m + 31) / 32, kRowThreads, 0, st>>>(m, na, (const double2*)anld, m, pl.beta_a, o.s2);
  with_moduli(L, [&](auto lc) {
    constexpr int LL = decltype(lc)::value;
    k_crt_conv_cols<LL, true><<<dim3((o.nkb1 * KB + kConvPer - 1) / kConvPer, na), 256, 0, st>>>(
        m, na, (const double2*)anl, m, o.w + m, part, nchunk, pl.beta_a, BM, o.tiles1, o.nkb1, o.a1, o.s1);
    k_crt_conv_rows<LL><<<dim3((m + 15) / 16, o.nkb2), 256, 0, st>>>(m, na, (const double2*)anld, m, o.s2, o.tiles2,
                                                                     o.nkb2, o.a2);
  });
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "projector residues");
  o.m = m;
  o.na = na;
  o.L = L;
  return kOk;
}

namespace crt {
// columns per tile and K splits of one call
struct Sizes {
  int nt, tn, kbps, nsplit;
};
Sizes sizes_of(const CrtOperands& o, int nb, int nsm) {
  Sizes z{};
  z.nt = tile_cols(nb);
  z.tn = (nb + z.nt - 1) / z.nt;
  // K splits of the projection: at most kMaxKb blocks each; among up to 16 more, the count whose
  // waves over the SMs finish first (an item costs its K blocks plus about 6 for its drain)
  const int nmin = (o.nkb1 + kMaxKb - 1) / kMaxKb;
  long long best = -1;
  for (int ns = nmin; ns <= std::min(o.nkb1, nmin + 16); ++ns) {
    const int per = (o.nkb1 + ns - 1) / ns, eff = (o.nkb1 + per - 1) / per;
    const long long items = 3LL * o.L * eff * o.tiles1 * z.tn;
    const long long cost = (items + nsm - 1) / nsm * (per + 6);
    if (best < 0 || cost < best) {
      best = cost;
      z.kbps = per;
      z.nsplit = eff;
    }
  }
  return z;
}

// byte offsets of a call's buffers; the residues of the expansion take the place of psi's planes, which
// the projection has read by then
struct Layout {
  size_t part, b1r2, r1, p, b2, sb, total;
};
Layout layout_of(const CrtOperands& o, const Sizes& z, int nb) {
  const size_t ld1 = (size_t)o.tiles1 * BM, ld2 = (size_t)o.tiles2 * BM;
  const int nchunk = (o.m + kNormChunk - 1) / kNormChunk;
  const size_t n4 = (nb + 3) / 4, cols = (size_t)z.tn * z.nt, planes = 3 * (size_t)o.L;
  Layout y{};
  size_t at = 0;
  auto take = [&](size_t bytes) {
    const size_t here = at;
    at += align256(bytes);
    return here;
  };
  y.part = take(sizeof(Norm) * (size_t)std::max(nchunk, o.tiles1) * nb);
  y.b1r2 = take(std::max(planes * o.nkb1 * cols * KB, planes * n4 * ld2 * 4));
  y.r1 = take(z.nsplit * planes * n4 * ld1 * 4);
  y.p = take(sizeof(double2) * (size_t)o.na * nb);
  y.b2 = take(planes * o.nkb2 * cols * KB);
  y.sb = take(sizeof(int) * 2 * (size_t)nb);
  y.total = at;
  return y;
}
}  // namespace crt

// The buffers of a call on nb bands: allocated (or, under stream capture, only checked). A failure
// leaves the caller its other path.
int crt_reserve(CrtScratch& t, const CrtOperands& o, int nb, bool may_allocate) {
  using namespace crt;
  const size_t need = layout_of(o, sizes_of(o, nb, num_sms()), nb).total;
  if (!may_allocate) return t.buf.p && t.buf.bytes >= need ? kOk : kNotReady;
  return t.buf.ensure(need);
}

// hpsi += X D X^H psi; hpsi already holds the local part. After crt_reserve for nb bands. A wait that gives up
// sets the error flag of tcs (made by tc_error_flag), which tc_check_error reports.
int crt_nl_apply(CrtScratch& t, const CrtOperands& o, int nb, const void* psi, long long ldpsi, void* hpsi,
                 long long ldh, const TcScratch& tcs, cudaStream_t st, cudaEvent_t t0, cudaEvent_t t1,
                 cudaEvent_t t2) {
  using namespace crt;
  const int nsm = num_sms(), m = o.m, na = o.na, L = o.L;
  const Sizes z = sizes_of(o, nb, nsm);
  const Layout y = layout_of(o, z, nb);
  const Plan pl = make_plan(L);
  const int nchunk = (m + kNormChunk - 1) / kNormChunk;
  int8_t* base = (int8_t*)t.buf.p;
  int8_t* b1 = base + y.b1r2;
  int8_t* b2 = base + y.b2;
  double2* P = (double2*)(base + y.p);
  Norm* part = (Norm*)(base + y.part);
  int* sb1 = (int*)(base + y.sb);
  int* sb2 = sb1 + nb;
  GemmArgs g1{};
  g1.a = o.a1;
  g1.b = b1;
  g1.r = (uint32_t*)(base + y.r1);
  g1.N = nb;
  g1.nt = z.nt;
  g1.tiles_m = o.tiles1;
  g1.tiles_n = z.tn;
  g1.nkb = o.nkb1;
  g1.kb_per_split = z.kbps;
  g1.nsplit = z.nsplit;
  g1.L = L;
  g1.ldr = (long long)o.tiles1 * BM;
  g1.err = (int*)tcs.err.p;
  g1.wait_ns = tcs.wait_ns;
  GemmArgs g2 = g1;
  g2.a = o.a2;
  g2.b = b2;
  g2.r = (uint32_t*)(base + y.b1r2);
  g2.tiles_m = o.tiles2;
  g2.nkb = o.nkb2;
  g2.kb_per_split = o.nkb2;
  g2.nsplit = 1;
  g2.ldr = (long long)o.tiles2 * BM;
  const int n4 = (nb + 3) / 4;
  cudaError_t e = cudaSuccess;
  if (t0) cudaEventRecord(t0, st);
  with_moduli(L, [&](auto lc) {
    constexpr int LL = decltype(lc)::value;
    k_crt_norm_cols<<<dim3(nb, nchunk), 256, 0, st>>>(m, nb, (const double2*)psi, ldpsi, o.w, part);
    k_crt_conv_cols<LL, false><<<dim3((o.nkb1 * KB + kConvPer - 1) / kConvPer, nb), 256, 0, st>>>(
        m, nb, (const double2*)psi, ldpsi, o.w, part, nchunk, pl.beta_b, z.nt, z.tn, o.nkb1, b1, sb1);
    if ((e = launch_gemm(g1, nsm, st)) != cudaSuccess) return;
    k_crt_p<LL><<<dim3(o.tiles1, n4), 128, 0, st>>>(pl.w, na, nb, z.nsplit, g1.r, g1.ldr, o.s1, sb1, P, part);
    k_crt_conv_cols<LL, false><<<dim3((o.nkb2 * KB + kConvPer - 1) / kConvPer, nb), 256, 0, st>>>(
        na, nb, P, na, nullptr, part, o.tiles1, pl.beta_b, z.nt, z.tn, o.nkb2, b2, sb2);
    if (t1) cudaEventRecord(t1, st);
    if ((e = launch_gemm(g2, nsm, st)) != cudaSuccess) return;
    k_crt_out<LL><<<dim3(o.tiles2, n4), 128, 0, st>>>(pl.w, m, nb, g2.r, g2.ldr, o.s2, sb2, (double2*)hpsi, ldh);
    if (t2) cudaEventRecord(t2, st);
  });
  if (e == cudaSuccess) e = cudaGetLastError();
  return e == cudaSuccess ? kOk : cuda_fail(e, "projector products (residues)");
}

}  // namespace cpwb
