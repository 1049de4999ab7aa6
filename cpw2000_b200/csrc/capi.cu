// extern "C" entry points declared in include/cpw_b200.h.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <atomic>
#include <mutex>
#include <thread>
#include <string>
#include <vector>

#include "../../include/cpw_b200.h"
#include "context.hpp"

using namespace cpwb;
using C2d = C2<double>;

namespace {

int check_ctx(cpw_b200_ctx* c) { return c ? kOk : fail(kBadArg, "null context"); }

// size_fft of Src/ALFA/size_fft.f90, used for the reference's mxdwrk check.
void size_fft(const int* kmscr, int ns[3]) {
  static const int prim[11] = {2, 4, 6, 8, 10, 12, 16, 18, 20, 24, 32};
  static const int sec[6] = {36, 40, 48, 50, 54, 64};
  for (int n = 0; n < 3; ++n) {
    const int need = 2 * kmscr[n] + 1;
    int v = 0;
    if (need < 32) {
      for (int j = 0; j < 11; ++j) {
        v = prim[j];
        if (need <= v) break;
      }
    } else {
      const int k = (int)(logf((float)need) / logf(2.0f));
      for (int j = 0; j < 6; ++j) {
        v = (1 << (k - 5)) * sec[j];
        if (need <= v) break;
      }
    }
    ns[n] = v;
  }
}

std::mutex g_default_mu;
cpw_b200_ctx* g_default = nullptr;

int default_ctx(cpw_b200_ctx** out) {
  std::lock_guard<std::mutex> lk(g_default_mu);
  if (!g_default) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return cuda_fail(e, "cudaGetDevice");
    int s = cpw_b200_create(&g_default, dev);
    if (s) return s;
    // the drop-in entry points (hk_psi_c16_, hk_psi_nl_c16_, ditsp_c16_, ...) take no context: a
    // host code that links them unchanged selects their form by environment, read once here
    int mode = CPW_B200_FP64;
    if (const char* v = getenv("CPW_B200_DROPIN_PRECISION")) {
      if (!strcmp(v, "mixed")) {
        mode = CPW_B200_MIXED;
      } else if (!strcmp(v, "mixed_tc")) {
        mode = CPW_B200_MIXED_TC;
      } else if (strcmp(v, "fp64") != 0) {
        cpw_b200_destroy(g_default);
        g_default = nullptr;
        return fail(kBadArg, "CPW_B200_DROPIN_PRECISION must be fp64, mixed or mixed_tc");
      }
    }
    if (!s && mode != CPW_B200_FP64) s = cpw_b200_set_precision(g_default, mode);
    if (const char* v = getenv("CPW_B200_DROPIN_PROJECTOR_SLICES"); !s && v) s = cpw_b200_set_projector_slices(g_default, atoi(v));
    if (s) {
      cpw_b200_destroy(g_default);
      g_default = nullptr;
      return s;
    }
  }
  *out = g_default;
  return kOk;
}

template <typename T> bool same(const std::vector<T>& v, const T* p, size_t n) {
  return v.size() == n && (n == 0 || memcmp(v.data(), p, n * sizeof(T)) == 0);
}

// Copy the leading mtxd rows of ncol complex(8) columns with leading dimension ld.
int h2d_cols(void* dst, long long ldd, const double* src, long long lds, long long rows, long long cols,
             cudaStream_t st) {
  if (rows == 0 || cols == 0) return kOk;
  cudaError_t e = cudaMemcpy2DAsync(dst, ldd * 16, src, lds * 16, rows * 16, cols, cudaMemcpyHostToDevice, st);
  return e == cudaSuccess ? kOk : cuda_fail(e, "cudaMemcpy2D H2D");
}
int d2h_cols(double* dst, long long ldd, const void* src, long long lds, long long rows, long long cols,
             cudaStream_t st) {
  if (rows == 0 || cols == 0) return kOk;
  cudaError_t e = cudaMemcpy2DAsync(dst, ldd * 16, src, lds * 16, rows * 16, cols, cudaMemcpyDeviceToHost, st);
  return e == cudaSuccess ? kOk : cuda_fail(e, "cudaMemcpy2D D2H");
}


// H|psi> of host blocks (ld mxddim) through the device buffers h_in / h_out, pipelined over
// band chunks: every chunk's copy to the device is issued first on its own stream (the caller
// checks its other inputs on the host meanwhile), chunk k is computed once its copy landed, and
// its copy back runs on a third stream while chunk k+1 is computed (with page-locked host
// arrays the three overlap; pageable arrays degrade to staged copies). Every band's H|psi>
// depends on that band only; its projector products take the form of its chunk's size (residues
// or ZGEMMs of the same accuracy, both within one call where the end chunks are too small).
struct DropinPipe {
  int m = 0, nb = 0, chunk = 0, nchunk = 0;
  long long ldh = 0;
  std::vector<int> start;     // band boundaries of the chunks (nchunk + 1)
};

int dropin_stage_in(cpw_b200_ctx* c, int m, int nb, int nanl, const double* psi, long long ldh_host, DropinPipe* pp) {
  // Four chunks where even their half-size ends (nb / 6 bands) pay for residue GEMMs, which read the X planes
  // once per chunk: 480 bands of Si216 28.6 ms in six chunks, 26.8 in four. Else six (Si64's 160 bands, ZGEMMs
  // beside the local kernels: 4 and 6 within the spread).
  int kChunks = c->precision != 2 && c->nl_slices == 0 && residues_pay(c->precision, m, nanl, nb / 6) ? 4 : 6;
  constexpr int kMinChunk = 16;
  if (const char* v = getenv("CPW_B200_DROPIN_CHUNKS")) kChunks = std::max(1, atoi(v));
  DropinPipe& p = *pp;
  p.m = m;
  p.nb = nb;
  p.ldh = ldh_host;
  p.chunk = std::max(kMinChunk, (nb + kChunks - 1) / kChunks);
  p.nchunk = (nb + p.chunk - 1) / p.chunk;
  // the first chunk's copy-in and the last chunk's copy-out are the transfers no compute hides:
  // with 3 or more chunks those two are half the size of the others (CPW_B200_DROPIN_EVEN=1:
  // equal chunks)
  p.start.assign(1, 0);
  const char* even = getenv("CPW_B200_DROPIN_EVEN");
  if (p.nchunk >= 3 && !(even && atoi(even))) {
    const double unit = (double)nb / (p.nchunk - 1);
    for (int k = 1; k < p.nchunk; ++k) p.start.push_back((int)lround(unit * (k - 0.5)));
  } else {
    for (int k = 1; k < p.nchunk; ++k) p.start.push_back(k * p.chunk);
  }
  p.start.push_back(nb);
  cudaError_t e;
  if (!c->s_in && (e = cudaStreamCreateWithFlags(&c->s_in, cudaStreamNonBlocking)) != cudaSuccess)
    return cuda_fail(e, "hk_psi_c16 stream");
  if (!c->s_out && (e = cudaStreamCreateWithFlags(&c->s_out, cudaStreamNonBlocking)) != cudaSuccess)
    return cuda_fail(e, "hk_psi_c16 stream");
  while ((int)c->ev_pipe.size() < 2 * p.nchunk + 1) {
    cudaEvent_t ev;
    if ((e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) return cuda_fail(e, "event");
    c->ev_pipe.push_back(ev);
  }
  // the copy-in stream starts after any earlier work on the compute stream (h_in reuse)
  cudaEvent_t start = c->ev_pipe[2 * p.nchunk];
  if ((e = cudaEventRecord(start, c->stream)) != cudaSuccess || (e = cudaStreamWaitEvent(c->s_in, start, 0)) != cudaSuccess)
    return cuda_fail(e, "hk_psi_c16 pipeline");
  C2d* din = (C2d*)c->h_in.p;
  for (int k = 0; k < p.nchunk; ++k) {
    const int b0 = p.start[k], nbc = p.start[k + 1] - b0;
    if (int s = h2d_cols(din + (size_t)b0 * m, m, psi + 2 * (size_t)b0 * ldh_host, ldh_host, m, nbc, c->s_in)) return s;
    if ((e = cudaEventRecord(c->ev_pipe[2 * k], c->s_in)) != cudaSuccess) return cuda_fail(e, "hk_psi_c16 pipeline");
  }
  return kOk;
}

int dropin_wait(cpw_b200_ctx* c) {
  cudaError_t e;
  if ((e = cudaStreamSynchronize(c->s_out)) != cudaSuccess) return cuda_fail(e, "hk_psi_c16");
  if ((e = cudaStreamSynchronize(c->stream)) != cudaSuccess) return cuda_fail(e, "hk_psi_c16");
  return tc_check_error(c);
}

// FP64 projector products of a chunked call: P_k = X^H psi_k of every chunk on the projection
// stream as soon as the chunk's copy landed (it needs psi_k only), so that the compute stream
// runs the local kernels of chunk k and then only the expansion Hpsi_k += (X D) P_k. A 40-band
// ZGEMM is much less efficient than a 160-band one; this takes the projections off the path.
int dropin_nl_setup(cpw_b200_ctx* c, const DropinPipe& p) {
  cudaError_t e;
  if (!c->s_nl && (e = cudaStreamCreateWithFlags(&c->s_nl, cudaStreamNonBlocking)) != cudaSuccess)
    return cuda_fail(e, "hk_psi_c16 stream");
  if (!c->blas_nl) {
    if (cublasCreate(&c->blas_nl) != CUBLAS_STATUS_SUCCESS) {
      c->blas_nl = nullptr;
      return fail(kCublas, "cublasCreate failed");
    }
    cublasSetPointerMode(c->blas_nl, CUBLAS_POINTER_MODE_HOST);
  }
  while ((int)c->ev_nl.size() < p.nchunk) {
    cudaEvent_t ev;
    if ((e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming)) != cudaSuccess) return cuda_fail(e, "event");
    c->ev_nl.push_back(ev);
  }
  return c->proj.ensure((size_t)c->nanl * p.nb * sizeof(C2d));
}

int dropin_compute_out(cpw_b200_ctx* c, const DropinPipe& p, double* hpsi, bool wait = true) {
  cudaError_t e;
  const int m = p.m;
  C2d* din = (C2d*)c->h_in.p;
  C2d* dout = (C2d*)c->h_out.p;
  // Chunks that pay for residue GEMMs take them on the compute stream, where the projections beside the
  // local kernels would be ZGEMMs: 480 bands of Si216 35.1 -> 28.6 ms per call. (Chunks of Si64 with 160 bands do not.)
  int most = 0;
  for (int k = 0; k < p.nchunk; ++k) most = std::max(most, p.start[k + 1] - p.start[k]);
  const bool split_nl = p.nchunk > 1 && c->nanl > 0 && !(c->precision == 2 && (c->tc_ready || c->tc_pending)) &&
                        !ctx_residues(c, most, c->stream);
  if (split_nl) {
    if (int s = dropin_nl_setup(c, p)) return s;
    // the projection stream starts after earlier work on the compute stream (proj reuse)
    cudaEvent_t start = c->ev_pipe[2 * p.nchunk];
    if ((e = cudaEventRecord(start, c->stream)) != cudaSuccess || (e = cudaStreamWaitEvent(c->s_nl, start, 0)) != cudaSuccess)
      return cuda_fail(e, "hk_psi_c16 pipeline");
  }
  const cuDoubleComplex one = make_cuDoubleComplex(1.0, 0.0), zero = make_cuDoubleComplex(0.0, 0.0);
  for (int k = 0; k < p.nchunk; ++k) {
    const int b0 = p.start[k], nbc = p.start[k + 1] - b0;
    cudaEvent_t in_done = c->ev_pipe[2 * k], out_ready = c->ev_pipe[2 * k + 1];
    if ((e = cudaStreamWaitEvent(c->stream, in_done, 0)) != cudaSuccess) return cuda_fail(e, "hk_psi_c16 pipeline");
    if (split_nl) {
      cuDoubleComplex* pk = (cuDoubleComplex*)c->proj.p + (size_t)b0 * c->nanl;
      if ((e = cudaStreamWaitEvent(c->s_nl, in_done, 0)) != cudaSuccess) return cuda_fail(e, "hk_psi_c16 pipeline");
      cublasSetStream(c->blas_nl, c->s_nl);
      ++c->forms[kFormZgemm];
      // P_k = X^H psi_k (hk_psi_nl_c16.f90:82)
      if (cublasZgemm(c->blas_nl, CUBLAS_OP_C, CUBLAS_OP_N, c->nanl, nbc, m, &one, (const cuDoubleComplex*)c->anl.p, m,
                      (const cuDoubleComplex*)(din + (size_t)b0 * m), m, &zero, pk, c->nanl) != CUBLAS_STATUS_SUCCESS)
        return fail(kCublas, "hk_psi_c16: zgemm X^H psi");
      if ((e = cudaEventRecord(c->ev_nl[k], c->s_nl)) != cudaSuccess) return cuda_fail(e, "hk_psi_c16 pipeline");
      if (int s = ctx_hkpsi_device(c, nbc, din + (size_t)b0 * m, m, dout + (size_t)b0 * m, m, c->stream, true, false))
        return s;
      if ((e = cudaStreamWaitEvent(c->stream, c->ev_nl[k], 0)) != cudaSuccess) return cuda_fail(e, "hk_psi_c16 pipeline");
      cublasSetStream(c->blas, c->stream);
      // Hpsi_k += (X D) P_k (hk_psi_nl_c16.f90:87-96)
      if (cublasZgemm(c->blas, CUBLAS_OP_N, CUBLAS_OP_N, m, nbc, c->nanl, &one, (const cuDoubleComplex*)c->anld.p, m,
                      pk, c->nanl, &one, (cuDoubleComplex*)(dout + (size_t)b0 * m), m) != CUBLAS_STATUS_SUCCESS)
        return fail(kCublas, "hk_psi_c16: zgemm X D P");
    } else if (int s = ctx_hkpsi_device(c, nbc, din + (size_t)b0 * m, m, dout + (size_t)b0 * m, m, c->stream, true,
                                        true)) {
      return s;
    }
    if ((e = cudaEventRecord(out_ready, c->stream)) != cudaSuccess || (e = cudaStreamWaitEvent(c->s_out, out_ready, 0)) != cudaSuccess)
      return cuda_fail(e, "hk_psi_c16 pipeline");
    if (int s = d2h_cols(hpsi + 2 * (size_t)b0 * p.ldh, p.ldh, dout + (size_t)b0 * m, m, m, nbc, c->s_out)) return s;
  }
  return wait ? dropin_wait(c) : kOk;
}

// wait for copies already issued (an error path must not leave them reading freed buffers)
void dropin_abandon(cpw_b200_ctx* c) {
  if (c->s_in) cudaStreamSynchronize(c->s_in);
}

// ---- host-side content checks of the drop-in's inputs ----
// The drop-in keeps host shadows of what it uploaded and compares the caller's arrays with them
// on every call. The projectors of a large cell are over a gigabyte (Si216: 88,951 x 864 complex),
// so the compare and the shadow copy are split over host threads; in hk_psi_c16 the compare runs
// while the device already computes with the previous call's arrays.
unsigned host_threads(size_t bytes) {
  unsigned nt = std::thread::hardware_concurrency();
  if (nt == 0) nt = 1;
  const size_t by_size = std::max<size_t>(1, bytes >> 23);     // at least 8 MB per thread
  return (unsigned)std::min<size_t>(std::min<size_t>(nt, 32), by_size);
}

// runs f(c0, c1) over [0, n) split into contiguous ranges, one per thread
template <class F> void par_ranges(size_t n, unsigned nt, F f) {
  nt = (unsigned)std::max<size_t>(1, std::min<size_t>(nt, n));
  if (nt <= 1) {
    f((size_t)0, n);
    return;
  }
  std::vector<std::thread> th;
  th.reserve(nt);
  for (unsigned t = 0; t < nt; ++t) th.emplace_back(f, n * t / nt, n * (t + 1) / nt);
  for (auto& x : th) x.join();
}

// true when ncol columns of `rows` doubles at h (leading dimension ld doubles) equal the packed shadow
bool cols_equal(const std::vector<double>& sh, const double* h, size_t rows, size_t ld, size_t ncol) {
  if (sh.size() != rows * ncol) return false;
  if (rows == 0 || ncol == 0) return true;
  std::atomic<bool> diff(false);
  const unsigned nt = host_threads(rows * ncol * 8);
  if (ld == rows || ncol < nt) {
    // one contiguous run per column (or a single flat run): split the bytes of each column
    for (size_t j = 0; j < ncol && !diff.load(std::memory_order_relaxed); ++j) {
      const double* a = sh.data() + j * rows;
      const double* b = h + j * ld;
      const size_t n = (ld == rows) ? rows * ncol : rows;
      par_ranges(n, host_threads(n * 8), [&](size_t i0, size_t i1) {
        if (memcmp(a + i0, b + i0, (i1 - i0) * 8)) diff = true;
      });
      if (ld == rows) break;
    }
  } else {
    par_ranges(ncol, nt, [&](size_t c0, size_t c1) {
      for (size_t j = c0; j < c1 && !diff.load(std::memory_order_relaxed); ++j)
        if (memcmp(sh.data() + j * rows, h + j * ld, rows * 8)) diff = true;
    });
  }
  return !diff.load();
}

void cols_copy(std::vector<double>& sh, const double* h, size_t rows, size_t ld, size_t ncol) {
  sh.resize(rows * ncol);
  if (rows == 0 || ncol == 0) return;
  par_ranges(ncol, host_threads(rows * ncol * 8), [&](size_t c0, size_t c1) {
    for (size_t j = c0; j < c1; ++j) memcpy(sh.data() + j * rows, h + j * ld, rows * 8);
  });
}

// the caller's projectors equal the ones on the device (compared with the host shadows)
bool dropin_proj_same(cpw_b200_ctx* c, const double* anlga, const double* xnlkb, int nanl, int mxddim) {
  if (c->sh_nanl != nanl) return false;
  if (nanl == 0) return true;
  if (!same(c->sh_xnl, xnlkb, (size_t)nanl)) return false;
  return cols_equal(c->sh_anl, anlga, 2 * (size_t)c->mtxd, 2 * (size_t)mxddim, (size_t)nanl);
}

int dropin_proj_upload(cpw_b200_ctx* c, const double* anlga, const double* xnlkb, int nanl, int mxddim) {
  if (int s = ctx_set_projectors(c, nanl, anlga, mxddim, xnlkb, false)) {
    c->sh_nanl = -1;
    return s;
  }
  c->sh_nanl = nanl;
  c->sh_xnl.assign(xnlkb, xnlkb + nanl);
  cols_copy(c->sh_anl, anlga, 2 * (size_t)c->mtxd, 2 * (size_t)mxddim, (size_t)nanl);
  return kOk;
}

// Bring the default context in line with the k-point arguments of a drop-in call: the
// k-point arrays are compared with the previous call's shadows and re-uploaded only when
// they changed. The projectors are uploaded at once when lnewanl is set (the reference's
// "anlga recalculated" hint, hk_psi_c16.f90:74; the library only reads it), the basis changed
// or nanl changed; otherwise they are compared by content, now (defer false) or, with defer,
// by the caller while the device computes (*pending then tells it to). The potential is the
// caller's next step (sync_dropin_potential).
int sync_dropin_kpoint(cpw_b200_ctx* c, int m, int ng, const int* kgv, const double* ekpg, const int* isort,
                       const int* kmscr, const double* anlga, const double* xnlkb, int nanl, int mxddim,
                       bool lnewanl, bool defer, bool* pending) {
  *pending = false;
  std::vector<int> kg((size_t)3 * m);
  for (int i = 0; i < m; ++i) {
    const int it = isort[i];
    if (it < 1 || it > ng) return fail(kBadArg, "isort out of range of kgv");
    for (int j = 0; j < 3; ++j) kg[3 * (size_t)i + j] = kgv[3 * (size_t)(it - 1) + j];
  }
  const bool kchanged = !c->have_basis || c->sh_mtxd != m || !same(c->sh_kmscr, kmscr, 7) ||
                        !same(c->sh_isort, isort, (size_t)m) || !same(c->sh_kgv, kg.data(), kg.size()) ||
                        !same(c->sh_ekpg, ekpg, (size_t)m);
  int s;
  if (kchanged) {
    // the compact kgv(3, mtxd) of the basis with isort = 1..mtxd is what the device needs
    std::vector<int> iota(m);
    for (int i = 0; i < m; ++i) iota[i] = i + 1;
    c->sh_mtxd = -1;
    c->sh_nanl = -1;
    if ((s = ctx_set_basis(c, m, iota.data(), kg.data(), m, ekpg, kmscr))) return s;
    c->sh_mtxd = m;
    c->sh_kmscr.assign(kmscr, kmscr + 7);
    c->sh_isort.assign(isort, isort + m);
    c->sh_kgv = kg;
    c->sh_ekpg.assign(ekpg, ekpg + m);
    c->sh_vscr.clear();
  }
  if (kchanged || lnewanl || c->sh_nanl != nanl) return dropin_proj_upload(c, anlga, xnlkb, nanl, mxddim);
  if (defer) {
    *pending = true;
    return kOk;
  }
  if (!dropin_proj_same(c, anlga, xnlkb, nanl, mxddim)) return dropin_proj_upload(c, anlga, xnlkb, nanl, mxddim);
  return kOk;
}

// vscr against the shadow of the potential on the device; uploads it when it differs
int sync_dropin_potential(cpw_b200_ctx* c, const double* vscr, const int* kmscr, int mxdscr, bool* uploaded) {
  const size_t nv = (size_t)kmscr[6] * kmscr[4] * kmscr[5];
  *uploaded = false;
  if (c->have_pot && same(c->sh_vscr, vscr, nv)) return kOk;
  if (int s = ctx_set_potential(c, vscr, mxdscr)) return s;
  c->sh_vscr.assign(vscr, vscr + nv);
  *uploaded = true;
  return kOk;
}

[[noreturn]] void stop_like_fortran(const char* routine) {
  printf("\n   STOPPED in %s:  %s\n", routine, cpwb::last_error());
  fflush(stdout);
  exit(1);
}

}  // namespace

extern "C" {

const char* cpw_b200_last_error(void) { return cpwb::last_error(); }
int cpw_b200_version(void) { return 10000; }

int cpw_b200_create(cpw_b200_ctx** out, int device) {
  if (!out) return fail(kBadArg, "create: null output pointer");
  *out = nullptr;
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return cuda_fail(e, "cudaSetDevice");
  cpw_b200_ctx* c = new cpw_b200_ctx();
  c->device = device;
  e = cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete c;
    return cuda_fail(e, "cudaStreamCreate");
  }
  cublasStatus_t bs = cublasCreate(&c->blas);
  if (bs != CUBLAS_STATUS_SUCCESS) {
    cudaStreamDestroy(c->stream);
    delete c;
    return fail(kCublas, "cublasCreate failed");
  }
  cublasSetStream(c->blas, c->stream);
  *out = c;
  return kOk;
}

int cpw_b200_destroy(cpw_b200_ctx* c) {
  if (!c) return kOk;
  cudaSetDevice(c->device);
  cudaStreamSynchronize(c->stream);
  if (c->s_in) cudaStreamSynchronize(c->s_in);
  if (c->s_out) cudaStreamSynchronize(c->s_out);
  if (c->s_nl) cudaStreamSynchronize(c->s_nl);
  for (cudaEvent_t e : c->ev_pipe) cudaEventDestroy(e);
  for (cudaEvent_t e : c->ev_nl) cudaEventDestroy(e);
  for (cudaEvent_t e : c->ov_ev)
    if (e) cudaEventDestroy(e);
  if (c->s_in) cudaStreamDestroy(c->s_in);
  if (c->s_out) cudaStreamDestroy(c->s_out);
  if (c->blas_nl) cublasDestroy(c->blas_nl);
  if (c->s_nl) cudaStreamDestroy(c->s_nl);
  ditsp_release(c);
  adjoint_release(c);
  if (c->blas) cublasDestroy(c->blas);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
  return kOk;
}

void* cpw_b200_stream(cpw_b200_ctx* c) { return c ? (void*)c->stream : nullptr; }

int cpw_b200_synchronize(cpw_b200_ctx* c) {
  if (int s = check_ctx(c)) return s;
  cudaSetDevice(c->device);
  cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) return cuda_fail(e, "synchronize");
  return tc_check_error(c);   // a bounded device wait that gave up reports CPW_B200_TIMEOUT
}

int cpw_b200_set_precision(cpw_b200_ctx* c, int mode) {
  if (int s = check_ctx(c)) return s;
  if (mode != CPW_B200_FP64 && mode != CPW_B200_MIXED && mode != CPW_B200_MIXED_TC)
    return fail(kBadArg, "set_precision: unknown mode");
  if ((mode != 0) != (c->precision != 0) && c->have_basis) {
    // shared-memory tiling depends on the element size: caller must set the k-point again
    c->have_basis = false;
    c->have_pot = false;
  }
  c->precision = mode;
  return kOk;
}

int cpw_b200_set_slab_budget(cpw_b200_ctx* c, long long bytes) {
  if (int s = check_ctx(c)) return s;
  if (bytes <= 0) return fail(kBadArg, "set_slab_budget: bytes must be positive");
  c->slab_budget = (size_t)bytes;
  return kOk;
}

int cpw_b200_set_wait_limits(cpw_b200_ctx* c, long long mbarrier_ns, long long grid_polls) {
  if (int s = check_ctx(c)) return s;
  c->tcs.wait_ns = mbarrier_ns < 0 ? 2000000000ull : (unsigned long long)mbarrier_ns;
  c->grid_polls = grid_polls < 0 ? (1LL << 24) : grid_polls;
  return kOk;
}

int cpw_b200_wait_selftest(cpw_b200_ctx* c, long long limit_ns, void* stream) {
  if (int s = check_ctx(c)) return s;
  if (limit_ns < 0 || limit_ns > 2000000000LL) return fail(kBadArg, "wait_selftest: limit outside 0 .. 2 s");
  cudaSetDevice(c->device);
  return tc_wait_selftest(c, (unsigned long long)limit_ns, stream ? (cudaStream_t)stream : c->stream);
}

int cpw_b200_form_counts(cpw_b200_ctx* c, long long* counts, int n) {
  if (!c) {
    if (int s = default_ctx(&c)) return s;
  }
  for (int i = 0; i < n; ++i) counts[i] = i < kNumForms ? c->forms[i] : 0;
  return kOk;
}

int cpw_b200_set_projector_slices(cpw_b200_ctx* c, int slices) {
  if (int s = check_ctx(c)) return s;
  if (slices < 0 || slices > 8) return fail(kBadArg, "set_projector_slices: slices outside 0..8");
  c->nl_slices = slices;
  c->oz_nl_ready = false;
  return kOk;
}

int cpw_b200_zgemm_i8(cpw_b200_ctx* c, int transa, int m, int n, int k, const void* a, long long lda, const void* b,
                      long long ldb, double alpha, int accumulate, void* cm, long long ldc, int slices, void* stream) {
  return cpw_b200_zgemm_i8_tri(c, transa, m, n, k, a, lda, b, ldb, alpha, accumulate, cm, ldc, slices, 0, stream);
}

int cpw_b200_zgemm_i8_tri(cpw_b200_ctx* c, int transa, int m, int n, int k, const void* a, long long lda,
                          const void* b, long long ldb, double alpha, int accumulate, void* cm, long long ldc,
                          int slices, int tri, void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  if (tri < 0 || tri > 2) return fail(kBadArg, "zgemm_i8: tri must be 0, 1 or 2");
  if (transa != 'N' && transa != 'C') return fail(kBadArg, "zgemm_i8: transa must be 'N' or 'C'");
  if (m < 0 || n < 0 || k < 0) return fail(kBadArg, "zgemm_i8: negative dimension");
  const bool conj = transa == 'C';
  if ((conj ? lda < std::max(k, 1) : lda < std::max(m, 1)) || ldb < std::max(k, 1) || ldc < std::max(m, 1))
    return fail(kBadArg, "zgemm_i8: leading dimension too small");
  cudaSetDevice(c->device);
  return oz_zgemm(c->ozs, conj, m, n, k, a, lda, b, ldb, alpha, accumulate != 0, cm, ldc, slices, c->tcs.wait_ns,
                  stream ? (cudaStream_t)stream : c->stream, tri);
}

int cpw_b200_timing_begin(cpw_b200_ctx* c) {
  if (int s = check_ctx(c)) return s;
  c->timer.on = true;
  c->timer.used = 0;
  c->timer.recs.clear();
  return kOk;
}

int cpw_b200_timing_end(cpw_b200_ctx* c, double* ms, long long* launches, int nstage) {
  if (int s = check_ctx(c)) return s;
  c->timer.on = false;
  for (int k = 0; k < nstage; ++k) {
    ms[k] = 0.0;
    launches[k] = 0;
  }
  for (const auto& r : c->timer.recs) {
    cudaError_t e = cudaEventSynchronize(r.b);
    if (e != cudaSuccess) return cuda_fail(e, "timing_end");
    float t = 0.f;
    e = cudaEventElapsedTime(&t, r.a, r.b);
    if (e != cudaSuccess) return cuda_fail(e, "timing_end");
    if (r.stage >= 0 && r.stage < nstage) {
      ms[r.stage] += t;
      launches[r.stage] += 1;
    }
  }
  c->timer.recs.clear();
  c->timer.used = 0;
  return kOk;
}

int cpw_b200_set_kpoint(cpw_b200_ctx* c, int mtxd, const int* isort, const int* kgv, int ng, const double* ekpg,
                        const int* kmscr) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return ctx_set_basis(c, mtxd, isort, kgv, ng, ekpg, kmscr);
}

int cpw_b200_set_potential(cpw_b200_ctx* c, const double* vscr, long long mxdscr) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return ctx_set_potential(c, vscr, mxdscr);
}

int cpw_b200_set_projectors(cpw_b200_ctx* c, int nanl, const double* anlga, int mxddim, const double* xnlkb) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return ctx_set_projectors(c, nanl, anlga, mxddim, xnlkb, false);
}

int cpw_b200_set_projectors_device(cpw_b200_ctx* c, int nanl, const void* anlga, int ld, const void* xnlkb) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return ctx_set_projectors(c, nanl, (const double*)anlga, ld, (const double*)xnlkb, true);
}

int cpw_b200_proj_nl_kb_device(cpw_b200_ctx* c, const double* rkpt, int ntype, const int* natom, const double* rat,
                               int mxdatm, const double* adot, const int* nqnl, const double* delqnl,
                               const double* vkb, int mxdlqp, const int* nkb, int nanl, double* xnlkb,
                               void* anlga, long long ldanl) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return ctx_proj_nl_kb(c, rkpt, ntype, natom, rat, mxdatm, adot, nqnl, delqnl, vkb, mxdlqp, nkb, nanl, xnlkb, anlga,
                        ldanl);
}

int cpw_b200_proj_nl_kb_der_device(cpw_b200_ctx* c, int nder, const double* rkpt, int ntype, const int* natom,
                                   const double* rat, int mxdatm, const double* adot, const int* nqnl,
                                   const double* delqnl, const double* vkb, int mxdlqp, const int* nkb, int nanl,
                                   double* xnlkb, void* anlga, long long ld, long long mxdanl, void* danlgadrk,
                                   void* d2anlgadrk2) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return ctx_proj_nl_kb_der(c, nder, rkpt, ntype, natom, rat, mxdatm, adot, nqnl, delqnl, vkb, mxdlqp, nkb, nanl,
                            xnlkb, anlga, ld, mxdanl, danlgadrk, d2anlgadrk2);
}

int cpw_b200_hamilt_kb_device(cpw_b200_ctx* c, int mtxd, const double* hdiag, const int* isort, const double* qmod,
                              int ng, const int* kgv, const double* phase, const double* conj, const int* inds,
                              const int* kmax, const int* indv, const double* ek, const double* sfact,
                              const double* veff, const int* nqnl, const double* delqnl, const double* vkb,
                              const int* nkb, int ntype, const double* adot, void* hamk, long long ldh, int mxdtyp,
                              int mxdgve, int mxdnst, int mxdcub, int mxdlqp, int mxddim) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return hamilt_kb_device(c, mtxd, hdiag, isort, qmod, ng, kgv, phase, conj, inds, kmax, indv, ek, sfact, veff, nqnl,
                          delqnl, vkb, nkb, ntype, adot, hamk, ldh, mxdtyp, mxdgve, mxdnst, mxdcub, mxdlqp, mxddim);
}

int cpw_b200_pot_local(cpw_b200_ctx* c, double* vscr, double* vmax, double* vmin, double* cmax, const double* veff,
                       int* kmscr, int idshift, int ng, const int* kgv, const double* phase, const double* conj, int ns,
                       const int* inds, int mxdscr, int mxdgve, int mxdnst, int install) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  // the checks of pot_local.f90:104-120 and the bounds it assumes
  if (ng < 0 || ng > mxdgve) return fail(kBadArg, "pot_local: ng out of range of mxdgve");
  if (ns < 0 || ns > mxdnst) return fail(kBadArg, "pot_local: ns out of range of mxdnst");
  if (idshift < 0) return fail(kBadArg, "pot_local: idshift < 0");
  for (int i = 0; i < ng; ++i)
    if (inds[i] < 1 || inds[i] > ns) return fail(kBadArg, "pot_local: inds out of range 1..ns");
  int n[3];
  size_fft(kmscr, n);
  const long long mxdwrk =
      4LL * std::max((long long)n[0] * n[1], std::max((long long)n[0] * n[2], (long long)n[1] * n[2]));
  if (mxdwrk > mxdscr) {
    char buf[160];
    snprintf(buf, sizeof buf, "pot_local: mxdwrk = %lld is greater than mxdscr = %d", mxdwrk, mxdscr);
    return fail(kBadArg, buf);
  }
  const int id = n[0] + idshift;
  if (vscr && (long long)id * n[1] * n[2] > mxdscr) return fail(kBadArg, "pot_local: vscr (mxdscr) smaller than id*n2*n3");
  kmscr[3] = n[0];
  kmscr[4] = n[1];
  kmscr[5] = n[2];
  kmscr[6] = id;
  cudaSetDevice(c->device);
  return ctx_pot_local(c, n[0], n[1], n[2], id, ng, kgv, veff, phase, conj, inds, vscr, vmax, vmin, cmax, install != 0);
}

int cpw_b200_hk_psi_kin_device(cpw_b200_ctx* c, int neig, const void* psi, long long ldpsi, void* hpsi, long long ldh,
                               int ladd, int nspin, void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  return ctx_hkpsi_kin_device(c, neig, psi, ldpsi, hpsi, ldh, ladd != 0, nspin, st);
}

int cpw_b200_hk_psi_loc_c16_device(cpw_b200_ctx* c, int neig, const void* psi, long long ldpsi, void* hpsi,
                                   long long ldh, int ladd, int nspin, void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  return ctx_hkpsi_loc_general(c, neig, psi, ldpsi, hpsi, ldh, ladd != 0, nspin, st);
}

int cpw_b200_set_potential_spin(cpw_b200_ctx* c, const double* vscr_sp, long long mxdscr, int nsp) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return ctx_set_potential_spin(c, vscr_sp, mxdscr, nsp);
}

int cpw_b200_set_projectors_spin(cpw_b200_ctx* c, int nanlsp, const double* anlsp, long long ld, const double* xnlkbsp) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return ctx_set_projectors_spin(c, nanlsp, anlsp, ld, xnlkbsp);
}

int cpw_b200_hk_psi_spin_device(cpw_b200_ctx* c, int neig, const void* psi_sp, long long ldpsi, void* hpsi_sp,
                                long long ldh, void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  return ctx_hkpsi_spin_device(c, neig, psi_sp, ldpsi, hpsi_sp, ldh, st);
}

int cpw_b200_hk_psi_device(cpw_b200_ctx* c, int neig, const void* psi, long long ldpsi, void* hpsi, long long ldh,
                           void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  return ctx_hkpsi_device(c, neig, psi, ldpsi, hpsi, ldh, st, true, true);
}

int cpw_b200_hk_psi_loc_device(cpw_b200_ctx* c, int neig, const void* psi, long long ldpsi, void* hpsi,
                               long long ldh, void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  return ctx_hkpsi_device(c, neig, psi, ldpsi, hpsi, ldh, st, false, false);
}

int cpw_b200_hk_psi_c16(const int* mtxd, const int* neig, const double* psi, double* hpsi, int* lnewanl,
                        const int* ng, const int* kgv, const double* ekpg, const int* isort, const double* vscr,
                        const int* kmscr, const double* anlga, const double* xnlkb, const int* nanl,
                        const int* mxddim, const int* mxdbnd, const int* mxdanl, const int* mxdgve,
                        const int* mxdscr) {
  // argument checks of hk_psi_c16.f90:110-119 plus the array bounds it assumes
  if (*ng > *mxdgve) return fail(kBadArg, "hk_psi_c16: ng > mxdgve");
  if (*mtxd < 0 || *mtxd > *mxddim) return fail(kBadArg, "hk_psi_c16: mtxd out of range of mxddim");
  if (*neig < 0 || *neig > *mxdbnd) return fail(kBadArg, "hk_psi_c16: neig out of range of mxdbnd");
  if (*nanl < 0 || *nanl > *mxdanl) return fail(kBadArg, "hk_psi_c16: nanl out of range of mxdanl");
  {
    int ns[3];
    size_fft(kmscr, ns);
    const long long mxdwrk =
        4LL * std::max((long long)ns[0] * ns[1], std::max((long long)ns[0] * ns[2], (long long)ns[1] * ns[2]));
    if (mxdwrk > *mxdscr) {
      char buf[160];
      snprintf(buf, sizeof buf, "hk_psi_c16: mxdwrk = %lld is greater than mxdscr = %d", mxdwrk, *mxdscr);
      return fail(kBadArg, buf);
    }
    if ((long long)kmscr[6] * kmscr[4] * kmscr[5] > *mxdscr)
      return fail(kBadArg, "hk_psi_c16: vscr (mxdscr) smaller than id*n2*n3");
  }
  cpw_b200_ctx* c;
  if (int s = default_ctx(&c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  const int m = *mtxd, nb = *neig;
  int s;
  // start the wavefunction copies (device buffers sized by mtxd and neig alone), then bring
  // the context in line with the k-point arguments on the host while they travel
  DropinPipe pipe;
  const bool go = m > 0 && nb > 0;
  if (go) {
    const size_t bytes = (size_t)m * nb * 16;
    if ((s = c->h_in.ensure(bytes)) || (s = c->h_out.ensure(bytes)) ||
        (s = dropin_stage_in(c, m, nb, *nanl, psi, *mxddim, &pipe))) {
      dropin_abandon(c);
      return s;
    }
  }
  // lnewanl is only read: a caller may pass a literal (berry_derivative.f90:229 passes .TRUE.)
  bool proj_pending = false;
  if ((s = sync_dropin_kpoint(c, m, *ng, kgv, ekpg, isort, kmscr, anlga, xnlkb, *nanl, *mxddim, *lnewanl != 0, go,
                              &proj_pending))) {
    dropin_abandon(c);
    return s;
  }
  bool uploaded = false;
  const bool pot_pending = go && c->have_pot;
  if (!pot_pending) {
    if ((s = sync_dropin_potential(c, vscr, kmscr, *mxdscr, &uploaded))) {
      dropin_abandon(c);
      return s;
    }
  }
  if (!go) return kOk;
  if (!pot_pending && !proj_pending) return dropin_compute_out(c, pipe, hpsi);
  // the potential and the projectors on the device are the previous call's: compute with them
  // while vscr and anlga/xnlkb are compared on the host (an SCF changes vscr only between
  // iterations, the projectors only with the k-point); if either changed, upload it and compute
  // again from the wavefunctions already on the device
  if ((s = dropin_compute_out(c, pipe, hpsi, false))) {
    dropin_wait(c);
    return s;
  }
  const size_t nv = (size_t)kmscr[6] * kmscr[4] * kmscr[5];
  const bool vsame = !pot_pending || cols_equal(c->sh_vscr, vscr, nv, nv, 1);
  const bool psame = !proj_pending || dropin_proj_same(c, anlga, xnlkb, *nanl, *mxddim);
  if (vsame && psame) return dropin_wait(c);
  if ((s = dropin_wait(c))) return s;
  if (!vsame && (s = sync_dropin_potential(c, vscr, kmscr, *mxdscr, &uploaded))) return s;
  if (!psame && (s = dropin_proj_upload(c, anlga, xnlkb, *nanl, *mxddim))) return s;
  return dropin_compute_out(c, pipe, hpsi);
}

void hk_psi_c16_(const int* mtxd, const int* neig, const double* psi, double* hpsi, int* lnewanl, const int* ng,
                 const int* kgv, const double* ekpg, const int* isort, const double* vscr, const int* kmscr,
                 const double* anlga, const double* xnlkb, const int* nanl, const int* mxddim, const int* mxdbnd,
                 const int* mxdanl, const int* mxdgve, const int* mxdscr) {
  int s = cpw_b200_hk_psi_c16(mtxd, neig, psi, hpsi, lnewanl, ng, kgv, ekpg, isort, vscr, kmscr, anlga, xnlkb, nanl,
                              mxddim, mxdbnd, mxdanl, mxdgve, mxdscr);
  if (s) stop_like_fortran("hk_psi_c16");
}

namespace {
// the spinor drop-in keeps its own context and host shadows of its k-point, potential and
// projectors (compared by content on every call, like the scalar drop-in's)
struct SpinDropin {
  cpw_b200_ctx* c = nullptr;
  std::vector<int> isort, kgv, kmscr;
  std::vector<double> ekpg, vscr, anl, xnl;
  int nanl = -1;
};
SpinDropin g_spin;
std::mutex g_spin_mu;
}  // namespace

int cpw_b200_hk_psi_spin_c16(const int* mtxd, const int* neig, const double* psi_sp, double* hpsi_sp, int* lnewanl,
                             const int* ng, const int* kgv, const double* ekpg, const int* isort,
                             const double* vscr_sp, const int* kmscr, const int* nsp, const double* anlsp,
                             const double* xnlkbsp, const int* nanlsp, const int* mxddim, const int* mxdbnd,
                             const int* mxdasp, const int* mxdgve, const int* mxdscr, const int* mxdnsp) {
  // argument checks of hk_psi_spin_c16.f90 and the array bounds it assumes
  if (*ng > *mxdgve) return fail(kBadArg, "hk_psi_spin_c16: ng > mxdgve");
  if (*nsp > *mxdnsp) return fail(kBadArg, "hk_psi_spin_c16: nsp is greater than mxdnsp");
  if (*nsp != 1 && *nsp != 2 && *nsp != 4) return fail(kBadArg, "hk_psi_spin_c16: nsp is an incorrect value, should be 1,2,4");
  if (*mtxd < 0 || *mtxd > *mxddim) return fail(kBadArg, "hk_psi_spin_c16: mtxd out of range of mxddim");
  if (*neig < 0 || *neig > *mxdbnd) return fail(kBadArg, "hk_psi_spin_c16: neig out of range of mxdbnd");
  if (*nanlsp < 0 || *nanlsp > *mxdasp) return fail(kBadArg, "hk_psi_spin_c16: nanlsp out of range of mxdasp");
  {
    int ns[3];
    size_fft(kmscr, ns);
    const long long mxdwrk =
        4LL * std::max((long long)ns[0] * ns[1], std::max((long long)ns[0] * ns[2], (long long)ns[1] * ns[2]));
    if (mxdwrk > *mxdscr) {
      char buf[160];
      snprintf(buf, sizeof buf, "hk_psi_spin_c16: mxdwrk = %lld is greater than mxdscr = %d", mxdwrk, *mxdscr);
      return fail(kBadArg, buf);
    }
    if ((long long)kmscr[6] * kmscr[4] * kmscr[5] > *mxdscr)
      return fail(kBadArg, "hk_psi_spin_c16: vscr_sp (mxdscr) smaller than id*n2*n3");
  }
  std::lock_guard<std::mutex> lk(g_spin_mu);
  SpinDropin& d = g_spin;
  int s;
  if (!d.c) {
    int dev = 0;
    cudaGetDevice(&dev);
    if ((s = cpw_b200_create(&d.c, dev))) return s;
  }
  cpw_b200_ctx* c = d.c;
  cudaSetDevice(c->device);
  const int m = *mtxd, nb = *neig;
  bool new_basis = !(d.isort.size() == (size_t)m && same(d.isort, isort, m) && same(d.ekpg, ekpg, m) &&
                     same(d.kmscr, kmscr, 7) && same(d.kgv, kgv, 3 * (size_t)*ng));
  if (new_basis) {
    if ((s = ctx_set_basis(c, m, isort, kgv, *ng, ekpg, kmscr))) return s;
    d.isort.assign(isort, isort + m);
    d.ekpg.assign(ekpg, ekpg + m);
    d.kmscr.assign(kmscr, kmscr + 7);
    d.kgv.assign(kgv, kgv + 3 * (size_t)*ng);
    d.vscr.clear();
  }
  const size_t nv = (size_t)*mxdscr * *nsp;
  if (new_basis || c->nsp != *nsp || !same(d.vscr, vscr_sp, nv)) {
    if ((s = ctx_set_potential_spin(c, vscr_sp, *mxdscr, *nsp))) return s;
    d.vscr.assign(vscr_sp, vscr_sp + nv);
  }
  // lnewanl (only read) forces the upload; otherwise the spinor projectors are compared by content
  const size_t prow = 4 * (size_t)m, pld = 4 * (size_t)*mxddim;    // doubles per column: 2 mtxd complex rows
  if (new_basis || *lnewanl != 0 || d.nanl != *nanlsp || !same(d.xnl, xnlkbsp, (size_t)*nanlsp) ||
      !cols_equal(d.anl, anlsp, prow, pld, (size_t)*nanlsp)) {
    d.nanl = -1;
    if ((s = ctx_set_projectors_spin(c, *nanlsp, anlsp, 2LL * *mxddim, xnlkbsp))) return s;
    d.nanl = *nanlsp;
    d.xnl.assign(xnlkbsp, xnlkbsp + *nanlsp);
    cols_copy(d.anl, anlsp, prow, pld, (size_t)*nanlsp);
  }
  if (m == 0 || nb == 0) return kOk;
  const size_t rows = 2 * (size_t)m;
  const size_t bytes = rows * nb * 16;
  if ((s = c->h_in.ensure(bytes)) || (s = c->h_out.ensure(bytes))) return s;
  cudaError_t e = cudaMemcpy2DAsync(c->h_in.p, rows * 16, psi_sp, 2 * (size_t)*mxddim * 16, rows * 16, nb,
                                    cudaMemcpyHostToDevice, c->stream);
  if (e != cudaSuccess) return cuda_fail(e, "hk_psi_spin_c16 H2D");
  if ((s = ctx_hkpsi_spin_device(c, nb, c->h_in.p, (long long)rows, c->h_out.p, (long long)rows, c->stream))) return s;
  e = cudaMemcpy2DAsync(hpsi_sp, 2 * (size_t)*mxddim * 16, c->h_out.p, rows * 16, rows * 16, nb,
                        cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  return e == cudaSuccess ? kOk : cuda_fail(e, "hk_psi_spin_c16");
}

void hk_psi_spin_c16_(const int* mtxd, const int* neig, const double* psi_sp, double* hpsi_sp, int* lnewanl,
                      const int* ng, const int* kgv, const double* ekpg, const int* isort, const double* vscr_sp,
                      const int* kmscr, const int* nsp, const double* anlsp, const double* xnlkbsp,
                      const int* nanlsp, const int* mxddim, const int* mxdbnd, const int* mxdasp, const int* mxdgve,
                      const int* mxdscr, const int* mxdnsp) {
  int s = cpw_b200_hk_psi_spin_c16(mtxd, neig, psi_sp, hpsi_sp, lnewanl, ng, kgv, ekpg, isort, vscr_sp, kmscr, nsp,
                                   anlsp, xnlkbsp, nanlsp, mxddim, mxdbnd, mxdasp, mxdgve, mxdscr, mxdnsp);
  if (s) stop_like_fortran("hk_psi_spin_c16");
}

int cpw_b200_ditsp_device(cpw_b200_ctx* c, int ipr, int* ifail, int icmax, int iguess, double epspsi, int* neig,
                          int mtxds, void* psi, long long ldpsi, void* hpsi, double* ei, const double* hamsm,
                          int mxdsml, const double* hdiag, int mxdbnd, long long* ihkpsum, void* stream,
                          double* itlog, int itlog_rows) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  long long ih = 0;
  int s = ditsp_device(c, ipr, ifail, icmax, iguess, epspsi, neig, mtxds, psi, ldpsi, hpsi, hamsm, mxdsml, hdiag,
                       mxdbnd, ei, &ih, st, itlog, itlog_rows);
  if (ihkpsum) *ihkpsum = ih;
  return s;
}

int cpw_b200_ditsp_c16(const int* ipr, int* ifail, const int* icmax, const int* iguess, const double* epspsi,
                       int* lnewanl, int* neig, const int* mtxd, const int* mtxds, double* psi, double* hpsi,
                       double* ei, const double* ekpg, const int* isort, const double* vscr, const int* kmscr,
                       const int* ng, const int* kgv, const double* anlga, const double* xnlkb, const int* nanl,
                       const double* hamsm, const double* hdiag, const int* mxddim, const int* mxdsml,
                       const int* mxdbnd, const int* mxdgve, const int* mxdscr, const int* mxdanl) {
  // argument checks of ditsp_c16.f90:143-210
  *ifail = 0;
  if (*neig < 1) return kOk;
  if (*neig > *mtxds) return fail(kBadArg, "ditsp_c16: neig is greater than mtxds");
  if (*neig > *mxdbnd) return fail(kBadArg, "ditsp_c16: neig is greater than mxdbnd");
  if (3 * *neig > *mxdsml) return fail(kBadArg, "ditsp_c16: 3*neig is greater than mxdsml");
  if (*mtxds > *mxdsml) return fail(kBadArg, "ditsp_c16: mtxds is greater than mxdsml");
  if (*mtxd > *mxddim) return fail(kBadArg, "ditsp_c16: mtxd is greater than mxddim");
  if (*nanl > *mxdanl) return fail(kBadArg, "ditsp_c16: nanl is greater than mxdanl");
  if (*ng > *mxdgve) return fail(kBadArg, "ditsp_c16: ng is greater than mxdgve");
  cpw_b200_ctx* c;
  if (int s = default_ctx(&c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  const int m = *mtxd, nb = *mxdbnd;
  int s;
  bool uploaded = false;
  bool proj_pending = false;
  if ((s = sync_dropin_kpoint(c, m, *ng, kgv, ekpg, isort, kmscr, anlga, xnlkb, *nanl, *mxddim, *lnewanl != 0, false,
                              &proj_pending)) ||
      (s = sync_dropin_potential(c, vscr, kmscr, *mxdscr, &uploaded)))
    return s;
  const size_t bytes = (size_t)m * nb * 16;
  if ((s = c->h_in.ensure(bytes))) return s;
  if ((s = c->h_out.ensure(bytes))) return s;
  if ((s = h2d_cols(c->h_in.p, m, psi, *mxddim, m, nb, c->stream))) return s;
  if ((s = h2d_cols(c->h_out.p, m, hpsi, *mxddim, m, nb, c->stream))) return s;
  long long ih = 0;
  const int sd = ditsp_device(c, *ipr, ifail, *icmax, *iguess, *epspsi, neig, *mtxds, c->h_in.p, m, c->h_out.p, hamsm,
                              *mxdsml, hdiag, nb, ei, &ih, c->stream);
  if (sd != kOk && sd != kNotConverged) return sd;
  if ((s = d2h_cols(psi, *mxddim, c->h_in.p, m, m, nb, c->stream))) return s;
  if ((s = d2h_cols(hpsi, *mxddim, c->h_out.p, m, m, nb, c->stream))) return s;
  cudaError_t e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_fail(e, "ditsp_c16");
  return sd;
}

void ditsp_c16_(const int* ipr, int* ifail, const int* icmax, const int* iguess, const double* epspsi, int* lnewanl,
                int* neig, const int* mtxd, const int* mtxds, double* psi, double* hpsi, double* ei,
                const double* ekpg, const int* isort, const double* vscr, const int* kmscr, const int* ng,
                const int* kgv, const double* anlga, const double* xnlkb, const int* nanl, const double* hamsm,
                const double* hdiag, const int* mxddim, const int* mxdsml, const int* mxdbnd, const int* mxdgve,
                const int* mxdscr, const int* mxdanl) {
  int s = cpw_b200_ditsp_c16(ipr, ifail, icmax, iguess, epspsi, lnewanl, neig, mtxd, mtxds, psi, hpsi, ei, ekpg, isort,
                             vscr, kmscr, ng, kgv, anlga, xnlkb, nanl, hamsm, hdiag, mxddim, mxdsml, mxdbnd, mxdgve,
                             mxdscr, mxdanl);
  // not converged is reported through ifail, as the reference does (ditsp_c16.f90:412)
  if (s != 0 && s != CPW_B200_NOT_CONVERGED) stop_like_fortran("ditsp_c16");
}

int cpw_b200_density_device(cpw_b200_ctx* c, int neig, const void* psi, long long ldpsi, const double* occ,
                            void* rho, void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return density_device(c, neig, psi, ldpsi, occ, rho, stream ? (cudaStream_t)stream : c->stream);
}

int cpw_b200_structure_grad_device(cpw_b200_ctx* c, const void* g, int natom, const int* atom_type, const double* tau,
                                   int ntype, const void* vgt, double* dedtau, void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return structure_grad_device(c, g, natom, atom_type, tau, ntype, vgt, dedtau,
                               stream ? (cudaStream_t)stream : c->stream);
}

int cpw_b200_nl_grad_device(cpw_b200_ctx* c, int neig, const void* psi, long long ldpsi, const double* occ,
                            const int* proj_atom, int natom, double* dedtau, void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return nl_grad_device(c, neig, psi, ldpsi, occ, proj_atom, natom, dedtau, stream ? (cudaStream_t)stream : c->stream);
}

int cpw_b200_stress_inputs_device(cpw_b200_ctx* c, int neig, const void* psi, long long ldpsi, const double* occ,
                                  double* w, void* y, void* stream) {
  if (int s = check_ctx(c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  return stress_inputs_device(c, neig, psi, ldpsi, occ, w, y, stream ? (cudaStream_t)stream : c->stream);
}

int cpw_b200_hk_psi_nl_c16(const int* mtxd, const int* neig, const double* psi, double* hpsi, const double* anlga,
                           const double* xnlkb, const int* nanl, const int* ladd, const int* mxddim,
                           const int* mxdbnd, const int* mxdanl) {
  if (*mtxd < 0 || *mtxd > *mxddim) return fail(kBadArg, "hk_psi_nl_c16: mtxd out of range of mxddim");
  if (*neig < 0 || *neig > *mxdbnd) return fail(kBadArg, "hk_psi_nl_c16: neig out of range of mxdbnd");
  if (*nanl < 0 || *nanl > *mxdanl) return fail(kBadArg, "hk_psi_nl_c16: nanl out of range of mxdanl");
  const int m = *mtxd, nb = *neig, na = *nanl;
  if (m == 0 || nb == 0) return kOk;
  cpw_b200_ctx* c;
  if (int s = default_ctx(&c)) return s;
  const SpareMemory spare(c);
  cudaSetDevice(c->device);
  DevBuf x, xd, p, h, v;
  int s;
  // no projectors: the reference skips both products (the `if(nanl > 0)` of
  // hk_psi_nl_c16.f90:78-98), so hpsi is left as it is even when ladd is false
  if (na == 0) return kOk;
  if ((s = h.ensure((size_t)m * nb * 16)) || (s = x.ensure((size_t)m * na * 16)) || (s = p.ensure((size_t)na * nb * 16)) ||
      (s = v.ensure((size_t)m * nb * 16)) || (s = xd.ensure((size_t)na * 8)))
    return s;
  if ((s = h2d_cols(x.p, m, anlga, *mxddim, m, na, c->stream))) return s;
  if ((s = h2d_cols(v.p, m, psi, *mxddim, m, nb, c->stream))) return s;
  if (*ladd) {
    if ((s = h2d_cols(h.p, m, hpsi, *mxddim, m, nb, c->stream))) return s;
  }
  cudaMemcpyAsync(xd.p, xnlkb, (size_t)na * 8, cudaMemcpyHostToDevice, c->stream);
  cublasSetStream(c->blas, c->stream);
  const cuDoubleComplex one = make_cuDoubleComplex(1.0, 0.0), zero = make_cuDoubleComplex(0.0, 0.0);
  cublasStatus_t bs = cublasZgemm(c->blas, CUBLAS_OP_C, CUBLAS_OP_N, na, nb, m, &one, (const cuDoubleComplex*)x.p,
                                  m, (const cuDoubleComplex*)v.p, m, &zero, (cuDoubleComplex*)p.p, na);
  if (bs != CUBLAS_STATUS_SUCCESS) return fail(kCublas, "hk_psi_nl_c16: zgemm 'c','n'");
  // dhd := Diag(xnlkb) dhd (hk_psi_nl_c16.f90:87-91) as a row scaling of P
  {
    std::vector<double> dz(2 * (size_t)na, 0.0);
    for (int i = 0; i < na; ++i) dz[2 * (size_t)i] = xnlkb[i];
    DevBuf dd;
    if ((s = dd.ensure(dz.size() * 8))) return s;
    cudaMemcpyAsync(dd.p, dz.data(), dz.size() * 8, cudaMemcpyHostToDevice, c->stream);
    bs = cublasZdgmm(c->blas, CUBLAS_SIDE_LEFT, na, nb, (const cuDoubleComplex*)p.p, na,
                     (const cuDoubleComplex*)dd.p, 1, (cuDoubleComplex*)p.p, na);
    if (bs != CUBLAS_STATUS_SUCCESS) return fail(kCublas, "hk_psi_nl_c16: zdgmm");
    const cuDoubleComplex beta = *ladd ? one : zero;
    bs = cublasZgemm(c->blas, CUBLAS_OP_N, CUBLAS_OP_N, m, nb, na, &one, (const cuDoubleComplex*)x.p, m,
                     (const cuDoubleComplex*)p.p, na, &beta, (cuDoubleComplex*)h.p, m);
    if (bs != CUBLAS_STATUS_SUCCESS) return fail(kCublas, "hk_psi_nl_c16: zgemm 'n','n'");
    if ((s = d2h_cols(hpsi, *mxddim, h.p, m, m, nb, c->stream))) return s;
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) return cuda_fail(e, "hk_psi_nl_c16");
  }
  return kOk;
}

void hk_psi_nl_c16_(const int* mtxd, const int* neig, const double* psi, double* hpsi, const double* anlga,
                    const double* xnlkb, const int* nanl, const int* ladd, const int* mxddim, const int* mxdbnd,
                    const int* mxdanl) {
  int s = cpw_b200_hk_psi_nl_c16(mtxd, neig, psi, hpsi, anlga, xnlkb, nanl, ladd, mxddim, mxdbnd, mxdanl);
  if (s) stop_like_fortran("hk_psi_nl_c16");
}

}  // extern "C"
