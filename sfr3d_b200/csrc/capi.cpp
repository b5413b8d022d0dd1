// extern "C" entry points of libsfr3d_b200.so (declared in
// include/sfr3d_b200.h) and the solverC drop-in.
#include <cuda_runtime.h>

#include <algorithm>
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <thread>
#include <tuple>
#include <vector>

#include "internal.h"

using sfr::HostSell;

namespace {

thread_local std::string g_last_error;

int cuda_fail(cudaError_t e) {
  g_last_error = cudaGetErrorString(e);
  return SFR_CUDA_ERROR;
}

#define SFR_CU(expr)                           \
  do {                                         \
    cudaError_t e_ = (expr);                   \
    if (e_ != cudaSuccess) return cuda_fail(e_); \
  } while (0)

struct IoBuffers {
  double *b = nullptr, *x = nullptr, *diag = nullptr;
  size_t cap = 0;  // doubles per buffer
};
std::map<const sfr_system *, IoBuffers> g_io;
std::mutex g_io_mu;

int io_for(sfr_system *s, size_t doubles, IoBuffers **out) {
  std::lock_guard<std::mutex> lk(g_io_mu);
  IoBuffers &io = g_io[s];
  if (io.cap < doubles) {
    cudaFree(io.b);
    cudaFree(io.x);
    cudaFree(io.diag);
    io = IoBuffers{};
    SFR_CU(cudaMalloc(&io.b, sizeof(double) * doubles));
    SFR_CU(cudaMalloc(&io.x, sizeof(double) * doubles));
    SFR_CU(cudaMalloc(&io.diag, sizeof(double) * doubles));
    io.cap = doubles;
  }
  *out = &io;
  return SFR_OK;
}

void io_release(const sfr_system *s) {
  std::lock_guard<std::mutex> lk(g_io_mu);
  auto it = g_io.find(s);
  if (it == g_io.end()) return;
  cudaFree(it->second.b);
  cudaFree(it->second.x);
  cudaFree(it->second.diag);
  g_io.erase(it);
}

int ensure_transpose(sfr_system *s) {
  if (s->at_ready) return SFR_OK;
  if (!s->have_at_host) return SFR_UNSUPPORTED;
  int rc = sfr::upload_sell(s->host_at, &s->At, &s->bytes);
  if (rc != SFR_OK) return rc;
  s->host_at = HostSell{};
  s->have_at_host = false;
  s->at_ready = true;
  if (s->values_set) return sfr::gather_values(s, &s->At, s->stream);
  return SFR_OK;
}

}  // namespace

namespace sfr {
void set_last_error(const char *msg) { g_last_error = msg ? msg : ""; }
}  // namespace sfr

extern "C" {

const char *sfr_status_string(int status) {
  switch (status) {
    case SFR_OK: return "converged";
    case SFR_MAXIT: return "maximum iterations reached";
    case SFR_BREAKDOWN: return "Krylov breakdown (zero or non-finite scalar)";
    case SFR_BAD_INPUT: return "bad input";
    case SFR_CUDA_ERROR: return "CUDA error";
    case SFR_TIMEOUT: return "grid barrier timed out";
    case SFR_UNSUPPORTED: return "unsupported solver/storage/precision";
    default: return "unknown status";
  }
}

const char *sfr_last_error(void) { return g_last_error.c_str(); }

int sfr_gpu_check_device(int32_t device, int32_t *major, int32_t *minor) {
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
    g_last_error = "no CUDA device";
    return SFR_CUDA_ERROR;
  }
  if (device < 0 || device >= n) return SFR_BAD_INPUT;
  int ma = 0, mi = 0;
  SFR_CU(cudaDeviceGetAttribute(&ma, cudaDevAttrComputeCapabilityMajor, device));
  SFR_CU(cudaDeviceGetAttribute(&mi, cudaDevAttrComputeCapabilityMinor, device));
  if (major) *major = ma;
  if (minor) *minor = mi;
  return (ma == 10 && mi == 0) ? SFR_OK : SFR_UNSUPPORTED;
}

int sfr_gpu_wait_selftest(int32_t kind, int32_t absent, uint32_t spin_limit, void *stream) {
  if (spin_limit == 0) return SFR_BAD_INPUT;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (kind == 0 || kind == 1) return sfr::wait_selftest_fused(kind, absent, spin_limit, st);
  if (kind == 2) return sfr::wait_selftest_resident(absent, spin_limit, st);
  return SFR_BAD_INPUT;
}

int sfr_gpu_create(int32_t neq, int32_t nad, const int32_t *ia, const int32_t *ja,
                   int32_t storage, int32_t unsym, int32_t device, sfr_system **out) {
  if (!out) return SFR_BAD_INPUT;
  *out = nullptr;
  auto s = std::make_unique<sfr_system>();
  HostSell a;
  std::string why;
  int32_t nsrc = 0;
  int rc = sfr::build_sell(neq, nad, ia, ja, storage, unsym, &a, &s->host_at, &nsrc, &why);
  if (rc != SFR_OK) {
    g_last_error = why;
    return rc;
  }
  s->have_at_host = true;
  s->device = device;
  s->n = neq;
  s->storage = storage;
  s->unsym = unsym;
  s->nad = nad;
  s->nsrc = nsrc;
  s->bandwidth = a.bandwidth;
  SFR_CU(cudaSetDevice(device));
  SFR_CU(cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking));
  rc = sfr::upload_sell(a, &s->A, &s->bytes);
  if (rc != SFR_OK) return rc;
  SFR_CU(cudaMalloc(&s->d_stage, sizeof(double) * std::max(nsrc, 1)));
  SFR_CU(cudaMalloc(&s->d_diag, sizeof(double) * neq));
  SFR_CU(cudaMalloc(&s->d_diag32, sizeof(float) * neq));
  s->bytes += static_cast<int64_t>(sizeof(double) * std::max(nsrc, 1) + 12 * static_cast<size_t>(neq));
  *out = s.release();
  return SFR_OK;
}

extern "C++" {
namespace sfr {

// After new raw values (d_stage) and diagonal (d_diag) are in place on `st`:
// the SELL copies, the FP32 compensation and diagonal, and the epoch the
// derived operators are keyed on.  a_done: the SELL copy of A, its
// compensation and the FP32 diagonal were written with the values.
int values_refreshed(sfr_system *s, cudaStream_t st, bool a_done) {
  int rc = SFR_OK;
  if (!a_done) {
    rc = gather_values(s, &s->A, st);
    if (rc != SFR_OK) return rc;
    rc = row_compensation(s, s->A, st);
    if (rc != SFR_OK) return rc;
    SFR_CU(convert_diag32(s->d_diag, s->d_diag32, s->n, st));
  }
  if (s->at_ready) {
    rc = gather_values(s, &s->At, st);
    if (rc != SFR_OK) return rc;
  }
  s->values_set = true;
  ++s->values_epoch;
  if (s->tview) s->tview->comp_stale = true;
  return SFR_OK;
}

}  // namespace sfr
}  // extern "C++"

int sfr_gpu_set_values(sfr_system *s, const double *al, const double *ad, const double *au) {
  if (!s || !ad || (!al && s->nsrc > 0)) return SFR_BAD_INPUT;
  SFR_CU(cudaSetDevice(s->device));
  const bool split = s->storage == SFR_CSRC && s->unsym;
  if (split && au) {
    const size_t half = static_cast<size_t>(s->nsrc) / 2;
    SFR_CU(cudaMemcpyAsync(s->d_stage, al, sizeof(double) * half, cudaMemcpyHostToDevice, s->stream));
    SFR_CU(cudaMemcpyAsync(s->d_stage + half, au, sizeof(double) * half, cudaMemcpyHostToDevice,
                           s->stream));
  } else if (s->nsrc > 0) {
    SFR_CU(cudaMemcpyAsync(s->d_stage, al, sizeof(double) * s->nsrc, cudaMemcpyHostToDevice,
                           s->stream));
  }
  SFR_CU(cudaMemcpyAsync(s->d_diag, ad, sizeof(double) * s->n, cudaMemcpyHostToDevice, s->stream));
  const int rc = sfr::values_refreshed(s, s->stream);
  if (rc != SFR_OK) return rc;
  SFR_CU(cudaStreamSynchronize(s->stream));
  return SFR_OK;
}

namespace {

// The device entries take inputs that the caller's stream may still be
// writing: `st` goes on after what is in that stream now.
int follow(sfr_system *s, cudaStream_t caller, cudaStream_t st) {
  if (!s->ev0) SFR_CU(cudaEventCreate(&s->ev0));
  SFR_CU(cudaEventRecord(s->ev0, caller));
  SFR_CU(cudaStreamWaitEvent(st, s->ev0, 0));
  return SFR_OK;
}

}  // namespace

int sfr_gpu_set_values_device(sfr_system *s, int32_t nsrc, const double *d_src,
                              const double *d_ad, void *stream) {
  if (!s || nsrc != s->nsrc || !d_ad || (!d_src && nsrc > 0)) return SFR_BAD_INPUT;
  SFR_CU(cudaSetDevice(s->device));
  int rc = follow(s, static_cast<cudaStream_t>(stream), s->stream);
  if (rc != SFR_OK) return rc;
  if (s->nsrc > 0)
    SFR_CU(cudaMemcpyAsync(s->d_stage, d_src, sizeof(double) * s->nsrc, cudaMemcpyDeviceToDevice,
                           s->stream));
  SFR_CU(cudaMemcpyAsync(s->d_diag, d_ad, sizeof(double) * s->n, cudaMemcpyDeviceToDevice,
                         s->stream));
  rc = sfr::values_refreshed(s, s->stream);
  if (rc != SFR_OK) return rc;
  SFR_CU(cudaStreamSynchronize(s->stream));
  return SFR_OK;
}

// Matrix Market dumps as the reference writes them (WriteMtx.c:26-179 with
// its vendored writer): the diagonal then the stored entries of each row,
// 1-based, "%d %d %30.14e"; values al below the diagonal and, for unsym, au
// above it (csrToCoo).  Only CSRD, as writeCoo.
int sfr_write_coo(const char *path, int32_t neq, const int32_t *ia, const int32_t *ja,
                  const double *au, const double *ad, const double *al, int32_t nad,
                  int32_t storage, int32_t unsym, int32_t bin) {
  if (!path || neq < 0 || nad < 0 || !ia || (nad > 0 && !ja)) {
    g_last_error = "NULL argument or negative size";
    return SFR_BAD_INPUT;
  }
  if (storage != SFR_CSRD) {
    g_last_error = "writeCoo writes CSRD only";
    return SFR_BAD_INPUT;
  }
  if (!bin && (!ad || (nad > 0 && (!al || (unsym && !au))))) {
    g_last_error = "values are NULL";
    return SFR_BAD_INPUT;
  }
  if (ia[neq] - ia[0] != nad) {
    g_last_error = "ia[neq] - ia[0] != nad";
    return SFR_BAD_INPUT;
  }
  std::unique_ptr<FILE, int (*)(FILE *)> f(std::fopen(path, "w"), &std::fclose);
  if (!f) {
    g_last_error = std::string("cannot open ") + path;
    return SFR_BAD_INPUT;
  }
  std::fprintf(f.get(), "%%%%MatrixMarket matrix coordinate real %s\n",
               unsym ? "general" : "symmetric");
  std::fprintf(f.get(), "%d %d %d\n", neq, neq, neq + nad);
  for (int32_t i = 0; i < neq; ++i) {
    const int32_t row = i + 1;
    std::fprintf(f.get(), "%d %d %30.14e\n", row, row, bin ? 1.0 : ad[i]);
    for (int32_t k = ia[i]; k < ia[i + 1]; ++k) {
      const int32_t col = ja[k] + 1;
      double v = 0.0;
      if (bin)
        v = 1.0;
      else if (col < row)
        v = al[k];
      else if (col > row && unsym)
        v = au[k];
      std::fprintf(f.get(), "%d %d %30.14e\n", row, col, v);
    }
  }
  return std::ferror(f.get()) ? SFR_BAD_INPUT : SFR_OK;
}

int sfr_write_coo_b(const char *path, const double *b, int32_t neq) {
  if (!path || !b || neq < 0) {
    g_last_error = "NULL argument or negative size";
    return SFR_BAD_INPUT;
  }
  std::unique_ptr<FILE, int (*)(FILE *)> f(std::fopen(path, "w"), &std::fclose);
  if (!f) {
    g_last_error = std::string("cannot open ") + path;
    return SFR_BAD_INPUT;
  }
  // writeCooB's own banner (WriteMtx.c:171-176: one '%')
  std::fprintf(f.get(), "%%MatrixMarket matrix array real general\n");
  std::fprintf(f.get(), "%d %d\n", neq, 1);
  for (int32_t i = 0; i < neq; ++i) std::fprintf(f.get(), "%.14e\n", b[i]);
  return std::ferror(f.get()) ? SFR_BAD_INPUT : SFR_OK;
}

int sfr_gpu_write_coo(sfr_system *s, const char *path, const int32_t *ia, const int32_t *ja,
                      int32_t bin) {
  if (!s || !ia) {
    g_last_error = "NULL argument";
    return SFR_BAD_INPUT;
  }
  if (s->storage != SFR_CSRD) {
    g_last_error = "writeCoo writes CSRD only";
    return SFR_BAD_INPUT;
  }
  std::vector<double> al(static_cast<size_t>(std::max(s->nsrc, 1))), ad(s->n);
  const int rc = sfr_gpu_get_values(s, al.data(), ad.data(), nullptr);
  if (rc != SFR_OK) return rc;
  // CSRD keeps every stored value in al: above the diagonal too
  return sfr_write_coo(path, s->n, ia, ja, al.data(), ad.data(), al.data(), s->nsrc,
                       s->storage, s->unsym, bin);
}

int sfr_gpu_get_values(sfr_system *s, double *al, double *ad, double *au) {
  if (!s) return SFR_BAD_INPUT;
  if (!s->values_set) {
    g_last_error = "no values were set or assembled";
    return SFR_BAD_INPUT;
  }
  SFR_CU(cudaSetDevice(s->device));
  const bool split = s->storage == SFR_CSRC && s->unsym;
  const size_t first = split ? static_cast<size_t>(s->nsrc) / 2 : static_cast<size_t>(s->nsrc);
  if (al && first > 0)
    SFR_CU(cudaMemcpyAsync(al, s->d_stage, sizeof(double) * first, cudaMemcpyDeviceToHost,
                           s->stream));
  if (au && split)
    SFR_CU(cudaMemcpyAsync(au, s->d_stage + first, sizeof(double) * first,
                           cudaMemcpyDeviceToHost, s->stream));
  if (ad)
    SFR_CU(cudaMemcpyAsync(ad, s->d_diag, sizeof(double) * s->n, cudaMemcpyDeviceToHost,
                           s->stream));
  SFR_CU(cudaStreamSynchronize(s->stream));
  return SFR_OK;
}

int sfr_gpu_set_diagonal(sfr_system *s, const double *ad) {
  if (!s || !ad) return SFR_BAD_INPUT;
  SFR_CU(cudaSetDevice(s->device));
  SFR_CU(cudaMemcpyAsync(s->d_diag, ad, sizeof(double) * s->n, cudaMemcpyHostToDevice, s->stream));
  SFR_CU(sfr::convert_diag32(s->d_diag, s->d_diag32, s->n, s->stream));
  SFR_CU(cudaStreamSynchronize(s->stream));
  ++s->values_epoch;
  return SFR_OK;
}

int sfr_gpu_solve_device(sfr_system *s, int32_t solver, const double *d_b, double *d_x,
                         double tol, uint32_t maxit, int32_t newx, int32_t precision,
                         void *stream, sfr_solve_info *info) {
  if (!s || !d_b || !d_x) return SFR_BAD_INPUT;
  if (!s->values_set) {
    g_last_error = "sfr_gpu_set_values was not called";
    return SFR_BAD_INPUT;
  }
  SFR_CU(cudaSetDevice(s->device));
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : s->stream;
  return sfr::solve_device(s, solver, 1, nullptr, d_b, d_x, tol, maxit, newx, precision, st, info);
}

int sfr_gpu_solve_multi_device(sfr_system *s, int32_t solver, int32_t k, const double *d_ad_k,
                               const double *d_b, double *d_x, double tol, uint32_t maxit,
                               int32_t newx, int32_t precision, void *stream,
                               sfr_solve_info *info) {
  if (!s || !d_b || !d_x || k < 1) return SFR_BAD_INPUT;
  if (!s->values_set) {
    g_last_error = "sfr_gpu_set_values was not called";
    return SFR_BAD_INPUT;
  }
  SFR_CU(cudaSetDevice(s->device));
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : s->stream;
  return sfr::solve_device(s, solver, k, d_ad_k, d_b, d_x, tol, maxit, newx, precision, st, info);
}

int sfr_gpu_solve_multi(sfr_system *s, int32_t solver, int32_t k, const double *ad_k,
                        const double *b, double *x, double tol, uint32_t maxit, int32_t newx,
                        int32_t precision, sfr_solve_info *info) {
  if (!s || !b || !x || k < 1) return SFR_BAD_INPUT;
  if (!s->values_set) {
    g_last_error = "sfr_gpu_set_values was not called";
    return SFR_BAD_INPUT;
  }
  SFR_CU(cudaSetDevice(s->device));
  IoBuffers *io = nullptr;
  const size_t total = static_cast<size_t>(s->n) * k;
  int rc = io_for(s, total, &io);
  if (rc != SFR_OK) return rc;
  SFR_CU(cudaMemcpyAsync(io->b, b, sizeof(double) * total, cudaMemcpyHostToDevice, s->stream));
  if (!newx)
    SFR_CU(cudaMemcpyAsync(io->x, x, sizeof(double) * total, cudaMemcpyHostToDevice, s->stream));
  if (ad_k)
    SFR_CU(cudaMemcpyAsync(io->diag, ad_k, sizeof(double) * total, cudaMemcpyHostToDevice,
                           s->stream));
  rc = sfr::solve_device(s, solver, k, ad_k ? io->diag : nullptr, io->b, io->x, tol, maxit, newx,
                         precision, s->stream, info);
  if (rc == SFR_CUDA_ERROR || rc == SFR_BAD_INPUT || rc == SFR_UNSUPPORTED || rc == SFR_TIMEOUT)
    return rc;
  SFR_CU(cudaMemcpyAsync(x, io->x, sizeof(double) * total, cudaMemcpyDeviceToHost, s->stream));
  SFR_CU(cudaStreamSynchronize(s->stream));
  return rc;
}

int sfr_gpu_solve(sfr_system *s, int32_t solver, const double *b, double *x, double tol,
                  uint32_t maxit, int32_t newx, int32_t precision, sfr_solve_info *info) {
  return sfr_gpu_solve_multi(s, solver, 1, nullptr, b, x, tol, maxit, newx, precision, info);
}

int sfr_gpu_set_engine(sfr_system *s, int32_t engine, int32_t threads, int32_t slices_per_warp) {
  if (!s || engine < 0 || engine > 4) return SFR_BAD_INPUT;
  if (threads != 0 && threads != 128 && threads != 256) return SFR_BAD_INPUT;
  if (slices_per_warp < -1 || slices_per_warp > 64) return SFR_BAD_INPUT;
  s->engine = engine;
  if (threads) s->graph_threads = threads;
  if (slices_per_warp > 0) s->graph_spw = slices_per_warp;
  if (slices_per_warp == -1) s->graph_spw = 0;  // one wave of resident blocks
  return SFR_OK;
}

int sfr_gpu_set_prefetch(sfr_system *s, int32_t rounds) {
  if (!s || rounds < 0 || rounds > 8) return SFR_BAD_INPUT;
  s->graph_pf = rounds;
  return SFR_OK;
}

int sfr_gpu_set_staging(sfr_system *s, int32_t flag) {
  if (!s || flag < 0 || flag > 1) return SFR_BAD_INPUT;
  s->graph_stage = flag;
  return SFR_OK;
}

int sfr_gpu_set_fused(sfr_system *s, int32_t flag) {
  if (!s) return SFR_BAD_INPUT;
  if (flag < 0 || flag > 4) return SFR_BAD_INPUT;
  s->graph_fused = flag;
  return SFR_OK;
}

int sfr_gpu_destroy(sfr_system *s) {
  if (!s) return SFR_OK;
  cudaSetDevice(s->device);
  if (s->tview) sfr_gpu_destroy(s->tview);
  sfr::release_stream_engine(s);
  sfr::release_minres_graph(s);
  sfr::release_bicgstabl2_graph(s);
  sfr::release_gmres_graph(s);
  io_release(s);
  if (!s->borrowed) {
    sfr::free_sell(&s->A);
    sfr::free_sell(&s->At);
    cudaFree(s->d_stage);
    cudaFree(s->d_diag);
    cudaFree(s->d_diag32);
  }
  cudaFree(s->d_comp);
  cudaFree(s->d_rval);
  cudaFree(s->d_rdelta);
  cudaFree(s->d_rbad);
  cudaFree(s->ws.base);
  if (s->ev0) cudaEventDestroy(s->ev0);
  if (s->ev1) cudaEventDestroy(s->ev1);
  if (s->stream) cudaStreamDestroy(s->stream);
  delete s;
  return SFR_OK;
}

namespace {

// The transposed system: shares A^T (uploaded on first use), the diagonal
// and the value staging of `s`; owns its workspace and compensation.
int transpose_view(sfr_system *s, sfr_system **out) {
  int rc = ensure_transpose(s);
  if (rc != SFR_OK) return rc;
  if (!s->tview) {
    auto *t = new sfr_system;
    t->borrowed = true;
    t->device = s->device;
    t->n = s->n;
    t->storage = s->storage;
    t->unsym = s->unsym;
    t->nad = s->nad;
    t->nsrc = s->nsrc;
    t->bandwidth = s->bandwidth;
    t->A = s->At;
    t->d_stage = s->d_stage;
    t->d_diag = s->d_diag;
    t->d_diag32 = s->d_diag32;
    if (cudaStreamCreateWithFlags(&t->stream, cudaStreamNonBlocking) != cudaSuccess) {
      delete t;
      return SFR_CUDA_ERROR;
    }
    s->tview = t;
  }
  sfr_system *t = s->tview;
  t->values_set = s->values_set;
  t->values_epoch = s->values_epoch;
  t->engine = s->engine;
  t->graph_threads = s->graph_threads;
  t->graph_spw = s->graph_spw;
  t->graph_pf = s->graph_pf;
  t->graph_fused = s->graph_fused;
  t->graph_stage = s->graph_stage;
  if (t->comp_stale && s->values_set) {
    rc = sfr::row_compensation(t, t->A, t->stream);
    if (rc != SFR_OK) return rc;
    if (cudaStreamSynchronize(t->stream) != cudaSuccess) return SFR_CUDA_ERROR;
    t->comp_stale = false;
  }
  *out = t;
  return SFR_OK;
}

}  // namespace

int sfr_gpu_solve_transpose(sfr_system *s, int32_t solver, const double *b, double *x, double tol,
                            uint32_t maxit, int32_t newx, int32_t precision,
                            sfr_solve_info *info) {
  if (!s || !b || !x) return SFR_BAD_INPUT;
  if (!s->values_set) return SFR_BAD_INPUT;
  SFR_CU(cudaSetDevice(s->device));
  sfr_system *t = nullptr;
  int rc = transpose_view(s, &t);
  if (rc != SFR_OK) return rc;
  return sfr_gpu_solve_multi(t, solver, 1, nullptr, b, x, tol, maxit, newx, precision, info);
}

int sfr_gpu_adjoint(sfr_system *s, int32_t solver, const double *x, const double *g,
                    double *lam, double *g_al, double *g_ad, double *g_au, double tol,
                    uint32_t maxit, int32_t precision, sfr_solve_info *info) {
  if (!s || !x || !g || !lam) return SFR_BAD_INPUT;
  const bool split = s->storage == SFR_CSRC && s->unsym;
  if (std::all_of(g, g + s->n, [](double v) { return v == 0.0; })) {
    // J does not depend on x: lam = 0 and every gradient is 0 (a Krylov
    // solve of a zero right-hand side would report a breakdown)
    std::fill(lam, lam + s->n, 0.0);
    const size_t nl = split ? static_cast<size_t>(s->nsrc) / 2 : static_cast<size_t>(s->nsrc);
    if (g_al) std::fill(g_al, g_al + nl, 0.0);
    if (g_au && split) std::fill(g_au, g_au + nl, 0.0);
    if (g_ad) std::fill(g_ad, g_ad + s->n, 0.0);
    if (info) *info = sfr_solve_info{};
    return SFR_OK;
  }
  int rc = sfr_gpu_solve_transpose(s, solver, g, lam, tol, maxit, 1, precision, info);
  if (rc != SFR_OK) return rc;
  if (!g_al && !g_ad && !g_au) return SFR_OK;
  IoBuffers *io = nullptr;
  rc = io_for(s, std::max<size_t>(static_cast<size_t>(s->n), static_cast<size_t>(s->nsrc)), &io);
  if (rc != SFR_OK) return rc;
  // io->b = lam, io->x = x, io->diag = gradient of the value source
  double *d_gad = nullptr;
  SFR_CU(cudaMalloc(&d_gad, sizeof(double) * s->n));
  cudaError_t e = cudaMemcpyAsync(io->b, lam, sizeof(double) * s->n, cudaMemcpyHostToDevice,
                                  s->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(io->x, x, sizeof(double) * s->n, cudaMemcpyHostToDevice, s->stream);
  if (e != cudaSuccess) {
    cudaFree(d_gad);
    return cuda_fail(e);
  }
  rc = sfr::adjoint_gradients(s, io->b, io->x, io->diag, d_gad, s->stream);
  if (rc == SFR_OK) {
    const size_t nl = split ? static_cast<size_t>(s->nsrc) / 2 : static_cast<size_t>(s->nsrc);
    if (g_al) e = cudaMemcpyAsync(g_al, io->diag, sizeof(double) * nl, cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess && split && g_au)
      e = cudaMemcpyAsync(g_au, io->diag + nl, sizeof(double) * nl, cudaMemcpyDeviceToHost,
                          s->stream);
    if (e == cudaSuccess && g_ad)
      e = cudaMemcpyAsync(g_ad, d_gad, sizeof(double) * s->n, cudaMemcpyDeviceToHost, s->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
    if (e != cudaSuccess) rc = cuda_fail(e);
  }
  cudaFree(d_gad);
  return rc;
}

int sfr_gpu_adjoint_device(sfr_system *s, int32_t solver, int32_t nsrc, const double *d_x,
                           const double *d_g, double *d_lam, double *d_gsrc, double *d_gad,
                           double tol, uint32_t maxit, int32_t precision, void *stream,
                           sfr_solve_info *info) {
  if (!s || nsrc != s->nsrc || !d_x || !d_g || !d_lam || !d_gad || (!d_gsrc && nsrc > 0))
    return SFR_BAD_INPUT;
  if (!s->values_set) return SFR_BAD_INPUT;
  SFR_CU(cudaSetDevice(s->device));
  sfr_system *t = nullptr;
  int rc = transpose_view(s, &t);
  if (rc != SFR_OK) return rc;
  rc = follow(s, static_cast<cudaStream_t>(stream), t->stream);
  if (rc != SFR_OK) return rc;
  // s->ev0 is behind the caller's stream, so after the wait for this flag
  // everything the gradients read is ready on any stream
  IoBuffers *io = nullptr;
  rc = io_for(s, 1, &io);
  if (rc != SFR_OK) return rc;
  int nonzero = 0;
  rc = sfr::any_nonzero(d_g, s->n, reinterpret_cast<int *>(io->diag), &nonzero, t->stream);
  if (rc != SFR_OK) return rc;
  if (!nonzero) {  // as in sfr_gpu_adjoint
    SFR_CU(cudaMemsetAsync(d_lam, 0, sizeof(double) * s->n, t->stream));
    if (s->nsrc > 0) SFR_CU(cudaMemsetAsync(d_gsrc, 0, sizeof(double) * s->nsrc, t->stream));
    SFR_CU(cudaMemsetAsync(d_gad, 0, sizeof(double) * s->n, t->stream));
    SFR_CU(cudaStreamSynchronize(t->stream));
    if (info) *info = sfr_solve_info{};
    return SFR_OK;
  }
  rc = sfr::solve_device(t, solver, 1, nullptr, d_g, d_lam, tol, maxit, 1, precision, t->stream,
                         info);
  if (rc != SFR_OK) return rc;
  rc = sfr::adjoint_gradients(s, d_lam, d_x, d_gsrc, d_gad, t->stream);
  if (rc != SFR_OK) return rc;
  SFR_CU(cudaStreamSynchronize(t->stream));
  return SFR_OK;
}

int sfr_gpu_spmv(sfr_system *s, const double *d_x, double *d_y, void *stream) {
  if (!s || !d_x || !d_y) return SFR_BAD_INPUT;
  SFR_CU(cudaSetDevice(s->device));
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : s->stream;
  return sfr::spmv_device(s, s->A, s->d_diag, d_x, d_y, nullptr, st);
}

int sfr_gpu_spmv_transpose(sfr_system *s, const double *d_x, double *d_y, void *stream) {
  if (!s || !d_x || !d_y) return SFR_BAD_INPUT;
  SFR_CU(cudaSetDevice(s->device));
  int rc = ensure_transpose(s);
  if (rc != SFR_OK) return rc;
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : s->stream;
  return sfr::spmv_device(s, s->At, s->d_diag, d_x, d_y, nullptr, st);
}

int sfr_gpu_spmv_dot(sfr_system *s, const double *d_x, double *d_y, double *dot_out,
                     void *stream) {
  if (!s || !d_x || !d_y) return SFR_BAD_INPUT;
  SFR_CU(cudaSetDevice(s->device));
  cudaStream_t st = stream ? static_cast<cudaStream_t>(stream) : s->stream;
  IoBuffers *io = nullptr;
  int rc = io_for(s, 1, &io);
  if (rc != SFR_OK) return rc;
  rc = sfr::spmv_device(s, s->A, s->d_diag, d_x, d_y, io->diag, st);
  if (rc != SFR_OK) return rc;
  if (dot_out) {
    SFR_CU(cudaMemcpyAsync(dot_out, io->diag, sizeof(double), cudaMemcpyDeviceToHost, st));
    SFR_CU(cudaStreamSynchronize(st));
  }
  return SFR_OK;
}

int sfr_gpu_dot(const double *d_a, const double *d_b, int32_t n, double *dot_out,
                void *stream) {
  if (!d_a || !d_b || n < 0 || !dot_out) return SFR_BAD_INPUT;
  return sfr::dot_host(d_a, d_b, n, dot_out, static_cast<cudaStream_t>(stream));
}

int sfr_gpu_stats(const sfr_system *s, int64_t *bytes, int64_t *slots, int32_t *bandwidth) {
  if (!s) return SFR_BAD_INPUT;
  if (bytes) *bytes = s->bytes;
  if (slots) *slots = s->A.nslots;
  if (bandwidth) *bandwidth = s->bandwidth;
  return SFR_OK;
}

// ------------------------------------------------------------ solverC ----

namespace {

std::mutex g_shim_mu;
bool g_exit_on_failure = true;
int g_precision = SFR_FP64;
bool g_autotune = false;  // sfr_solverC tunes a pattern's first PCG / BiCGSTAB solve

struct PatternKey {
  const int32_t *ia, *ja;
  int32_t neq, storage, unsym;
  bool operator<(const PatternKey &o) const {
    return std::tie(ia, ja, neq, storage, unsym) < std::tie(o.ia, o.ja, o.neq, o.storage, o.unsym);
  }
};
struct Cached {
  sfr_system *sys = nullptr;
  uint64_t hash = 0;
};
std::map<PatternKey, Cached> g_cache;

// Hash of n 32-bit words: eight xor-multiply lanes over 64-bit words (one
// lane's chain of dependent multiplies would bound the hash to a word per
// multiply latency).
uint64_t words_hash(const int32_t *p, int64_t n, uint64_t seed) {
  constexpr int kLanes = 8;
  constexpr uint64_t kMul = 0x9e3779b97f4a7c15ULL;
  uint64_t h[kLanes];
  for (int l = 0; l < kLanes; ++l) h[l] = (seed + 0x2545f4914f6cdd1dULL) * (l + 1);
  const char *c = reinterpret_cast<const char *>(p);
  const int64_t words = n / 2;  // whole 64-bit words
  int64_t i = 0;
  for (; i + kLanes <= words; i += kLanes) {
    uint64_t w[kLanes];
    std::memcpy(w, c + 8 * i, sizeof(w));
    for (int l = 0; l < kLanes; ++l) h[l] = (h[l] ^ w[l]) * kMul;
  }
  for (; i < words; ++i) {
    uint64_t w;
    std::memcpy(&w, c + 8 * i, sizeof(w));
    h[0] = (h[0] ^ w) * kMul;
  }
  if (n & 1) h[1] = (h[1] ^ static_cast<uint32_t>(p[n - 1])) * kMul;
  h[2] = (h[2] ^ static_cast<uint64_t>(n)) * kMul;
  uint64_t out = seed;
  for (int l = 0; l < kLanes; ++l) {  // combine the lanes, with a final avalanche
    out = (out ^ h[l]) * kMul;
    out ^= out >> 29;
  }
  return out;
}

// Fingerprint of the pattern, checked on every sfr_solverC call so that a
// caller reusing the same ia/ja buffers for another pattern gets a fresh
// upload.  It covers all of ia (the row structure; a large ia is hashed in
// four parts on four threads) and a fixed sample of ja: its first and last
// 512 entries and 65,536 entries evenly spaced between.  A pattern rewritten
// in place with the same row lengths and different columns only at unsampled
// positions goes unseen; sfr_solverC_release() drops every cached pattern.
// (The reference builds its pattern once per run and never rewrites it.)
uint64_t pattern_hash(const int32_t *ia, const int32_t *ja, int32_t n_ia, int64_t n_ja) {
  constexpr int kParts = 4;
  uint64_t out = 1;
  if (n_ia < (1 << 20)) {
    out = words_hash(ia, n_ia, 1);
  } else {
    uint64_t part[kParts];
    const int64_t chunk = (static_cast<int64_t>(n_ia) / kParts) & ~int64_t{1};
    std::vector<std::thread> th;
    for (int t = 0; t < kParts; ++t) {
      const int64_t b = t * chunk, e = t + 1 == kParts ? n_ia : (t + 1) * chunk;
      th.emplace_back([&part, ia, t, b, e] { part[t] = words_hash(ia + b, e - b, t + 2); });
    }
    for (auto &x : th) x.join();
    for (int t = 0; t < kParts; ++t)
      out = words_hash(reinterpret_cast<const int32_t *>(&part[t]), 2, out);
  }
  if (!ja || n_ja <= 0) return out;
  constexpr int64_t kEdge = 512, kSamples = 65536;
  if (n_ja <= 2 * kEdge + kSamples) return words_hash(ja, n_ja, out);
  out = words_hash(ja, kEdge, out);
  out = words_hash(ja + n_ja - kEdge, kEdge, out);
  std::vector<int32_t> sample(kSamples);
  const int64_t span = n_ja - 2 * kEdge;
  for (int64_t i = 0; i < kSamples; ++i) sample[i] = ja[kEdge + span * i / kSamples];
  return words_hash(sample.data(), kSamples, out);
}

}  // namespace

void sfr_set_exit_on_failure(int32_t flag) { g_exit_on_failure = flag != 0; }
void sfr_set_precision(int32_t precision) { g_precision = precision; }
void sfr_set_autotune(int32_t flag) { g_autotune = flag != 0; }

namespace {
void release_dist_cache();
}

void sfr_solverC_release(void) {
  std::lock_guard<std::mutex> lk(g_shim_mu);
  for (auto &kv : g_cache) sfr_gpu_destroy(kv.second.sys);
  g_cache.clear();
  release_dist_cache();
}

// The MPI branch: one rank's share of a row-partitioned system per call.
namespace {
sfr_dist_group *g_group = nullptr;
struct DistCached {
  sfr_dist *d = nullptr;
  uint64_t hash = 0;
};
std::map<PatternKey, DistCached> g_dist_cache;

void release_dist_cache() {
  for (auto &kv : g_dist_cache)
    if (kv.second.d) sfr_gpu_dist_destroy(kv.second.d);
  g_dist_cache.clear();
}

int solverC_mpi(int32_t nEq, int32_t nEqNov, int32_t nAd, int32_t nAdR, int32_t *ia,
                int32_t *ja, double *al, double *ad, double *b, double *x, void *iNeq,
                double tol, uint32_t maxIt, int16_t storage, int16_t solver, FILE *fSolvLog,
                bool fLog, bool newX, bool unSym, const char *name) {
  int32_t kind = 0, nranks = 0, rank = 0;
  sfr_dist_group_info(g_group, &kind, &nranks, &rank);
  const bool known_storage = storage == SFR_CSRD || storage == SFR_CSRC ||
                             storage == SFR_ELLPACK || storage == SFR_CSRDCOO ||
                             storage == SFR_CSRCCOO;
  if (!known_storage || (storage == SFR_CSRDCOO && unSym) ||
      (solver != SFR_PCG && solver != SFR_PBICGSTAB) || !iNeq || kind != 1) {
    fprintf(stderr, "Opcao %d e invalida!!\n", !known_storage ? storage : solver);
    fprintf(stderr, "Arquivo:%s\nFonte:  %s\n", __FILE__, "sfr_solverC (MPI)");
    if (g_exit_on_failure) exit(EXIT_FAILURE);
    return SFR_UNSUPPORTED;
  }
  // the pattern arrays of the storage (Datastruct.c:115-420)
  int64_t n_ia = 0, n_ja = static_cast<int64_t>(nAd) + nAdR;
  if (storage == SFR_ELLPACK) {
    n_ia = 2;
    n_ja = static_cast<int64_t>(nEqNov) * ia[0];
  } else if (storage == SFR_CSRD && unSym) {
    n_ia = nEqNov + 1;
  } else {
    n_ia = 2 * (static_cast<int64_t>(nEqNov) + 1) +
           (storage == SFR_CSRDCOO || storage == SFR_CSRCCOO ? nAdR : 0);
  }
  const uint64_t h = pattern_hash(ia, ja, static_cast<int32_t>(n_ia), n_ja) ^
                     (static_cast<uint64_t>(nEq) << 32) ^ (static_cast<uint64_t>(storage) << 56);
  PatternKey key{ia, ja, nEqNov, storage, unSym ? 1 : 0};
  DistCached &c = g_dist_cache[key];
  int rc = SFR_OK;
  if (!c.d || c.hash != h) {
    if (c.d) sfr_gpu_dist_destroy(c.d);
    c.d = nullptr;
    rc = sfr_gpu_dist_create_storage(g_group, rank, storage, nEq, nEqNov, nAd, nAdR, ia, ja,
                                     unSym ? 1 : 0, static_cast<const sfr_interface *>(iNeq),
                                     &c.d);
    if (rc != SFR_OK) g_dist_cache.erase(key);
    else c.hash = h;
  }
  sfr_solve_info info;
  std::memset(&info, 0, sizeof(info));
  if (rc == SFR_OK) rc = sfr_gpu_dist_set_values(c.d, al, ad);
  if (rc == SFR_OK) {
    sfr_dist *parts[1] = {c.d};
    const double *bs[1] = {b};
    double *xs[1] = {x};
    rc = sfr_gpu_dist_solve(g_group, 1, parts, solver, bs, xs, tol, maxIt, newX ? 1 : 0, &info);
  }
  const bool pcg = solver == SFR_PCG;
  if (rc == SFR_MAXIT) {
    if (rank == 0) {
      printf("name : %s\n", name ? name : "");
      printf(pcg ? " MPIPCG *** WARNING: no convergende reached !\n"
                 : " MPIPBICGSTAB *** WARNING: no convergende reached !\n");
      printf("MAXIT = %d \n", maxIt);
    }
    if (g_exit_on_failure) exit(-2);
    return rc;
  }
  if (rc != SFR_OK) {
    fprintf(stderr, "sfr_solverC: %s (%s)\n", sfr_status_string(rc), g_last_error.c_str());
    if (g_exit_on_failure) exit(-2);
    return rc;
  }
  if (rank == 0 && fLog && fSolvLog) {
    if (pcg)
      fprintf(fSolvLog,
              "MPIPCG: tol %20.2e iteration %d xKx %20.12e norma(x*x) %20.12e time %20.5lf\n",
              tol, info.iters, info.xKx, info.norm_x, info.seconds);
    else
      fprintf(fSolvLog,
              "MPIPBICGSTAB: tol %20.2e iteration %d xKx %20.12e ||x*x|| %20.12e "
              "time %20.5lf\n",
              tol, info.iters, info.xKx, info.norm_x, info.seconds);
  }
  return rc;
}
}  // namespace

int sfr_solverC_set_group(sfr_dist_group *g) {
  std::lock_guard<std::mutex> lk(g_shim_mu);
  if (g) {
    int32_t kind = 0;
    if (sfr_dist_group_info(g, &kind, nullptr, nullptr) != SFR_OK || kind != 1) {
      g_last_error = "solverC takes an NCCL group (one rank per process)";
      return SFR_BAD_INPUT;
    }
  }
  release_dist_cache();
  g_group = g;
  return SFR_OK;
}

int sfr_solverC(void *m, int32_t nEq, int32_t nEqNov, int32_t nAd, int32_t nAdR, int32_t *ia,
                int32_t *ja, double *al, double *ad, double *au, double *b, double *x,
                void *iNeq, void *bOmp, double tol, uint32_t maxIt, int16_t storage,
                int16_t solver, FILE *fSolvLog, bool fLog, bool newX, bool unSym,
                const char *name) {
  (void)m;
  (void)bOmp;
  std::lock_guard<std::mutex> lk(g_shim_mu);
  if (g_group)
    return solverC_mpi(nEq, nEqNov, nAd, nAdR, ia, ja, al, ad, b, x, iNeq, tol, maxIt, storage,
                       solver, fSolvLog, fLog, newX, unSym, name);
  int rc = SFR_OK;
  const bool known = solver == SFR_PCG || solver == SFR_PBICGSTAB || solver == SFR_PBICGSTABL2 ||
                     solver == SFR_GMRES || solver == SFR_MINRES;
  if (!known || nEqNov != nEq) {
    // the reference's ERRO_OP (Erro.h:17-20) for an option this path lacks
    fprintf(stderr, "Opcao %d e invalida!!\n", solver);
    fprintf(stderr, "Arquivo:%s\nFonte:  %s\n", __FILE__, "sfr_solverC");
    if (g_exit_on_failure) exit(EXIT_FAILURE);
    return SFR_UNSUPPORTED;
  }
  const int32_t n_ia = storage == SFR_ELLPACK ? 2 : nEq + 1;
  int64_t n_ja = 0;
  if (storage == SFR_ELLPACK)
    n_ja = static_cast<int64_t>(nEq) * ia[0];
  else
    n_ja = static_cast<int64_t>(ia[nEq]) - ia[0];
  PatternKey key{ia, ja, nEq, storage, unSym ? 1 : 0};
  Cached &c = g_cache[key];
  // A cached pattern takes the new values while the fingerprint of ia/ja is
  // taken on another thread; a changed pattern is rebuilt and takes them
  // again.
  uint64_t h = 0;
  bool uploaded = false;
  // values this call's al (| au) holds
  const int64_t nsrc_now = storage == SFR_ELLPACK ? static_cast<int64_t>(ia[1])
                           : (storage == SFR_CSRC && unSym) ? 2 * n_ja
                                                            : n_ja;
  if (c.sys && c.sys->nsrc == nsrc_now) {  // same sizes: the upload reads within al / au
    std::thread hasher([&] { h = pattern_hash(ia, ja, n_ia, n_ja); });
    rc = sfr_gpu_set_values(c.sys, al, ad, au);
    hasher.join();
    uploaded = rc == SFR_OK && c.hash == h;
  } else {
    h = pattern_hash(ia, ja, n_ia, n_ja);
  }
  if (!c.sys || c.hash != h) {
    if (c.sys) sfr_gpu_destroy(c.sys);
    c.sys = nullptr;
    int dev = 0;
    cudaGetDevice(&dev);
    rc = sfr_gpu_create(nEq, nAd, ia, ja, storage, unSym ? 1 : 0, dev, &c.sys);
    if (rc != SFR_OK) {
      g_cache.erase(key);
      fprintf(stderr, "sfr_solverC: %s (%s)\n", sfr_status_string(rc), g_last_error.c_str());
      if (g_exit_on_failure) exit(EXIT_FAILURE);
      return rc;
    }
    c.hash = h;
  }
  sfr_system *s = c.sys;
  if (!uploaded) rc = sfr_gpu_set_values(s, al, ad, au);
  sfr_solve_info info;
  std::memset(&info, 0, sizeof(info));
  if (rc == SFR_OK && g_autotune && (solver == SFR_PCG || solver == SFR_PBICGSTAB) &&
      !sfr::find_tuned(s, solver, 1, g_precision, true)) {
    // the first solve of this kind on this pattern: time the engines and
    // launch shapes on it (the choice serves every later call); a failed
    // tune leaves the automatic choice
    sfr_tune_result tr;
    sfr_gpu_autotune(s, solver, 1, nullptr, b, tol, maxIt, g_precision, &tr);
  }
  if (rc == SFR_OK)
    rc = sfr_gpu_solve(s, solver, b, x, tol, maxIt, newX ? 1 : 0, g_precision, &info);
  if (rc == SFR_MAXIT) {
    // Cg.c:195-200, Bicgstab.c:225-231, Bicgstab.c:1428-1432,
    // Iters.c:773-777; MINRES only warns (Iters.c:525-529)
    if (solver == SFR_PCG || solver == SFR_PBICGSTAB) printf("name : %s\n", name ? name : "");
    switch (solver) {
      case SFR_PCG: printf("PCG: *** WARNING: no convergende reached !\n"); break;
      case SFR_PBICGSTAB: printf(" PBICGSTAB *** WARNING: no convergende reached !\n"); break;
      case SFR_PBICGSTABL2:
        printf(" PBICGSTAB(2) *** WARNING: no convergende reached !\n");
        break;
      case SFR_GMRES: printf(" GMRES *** WARNING: no convergende reached !\n"); break;
      default: printf("PMINRES: *** WARNING: no convergende reached !\n"); break;
    }
    printf("MAXIT = %d \n", maxIt);
    if (solver != SFR_MINRES) {
      if (g_exit_on_failure) exit(solver == SFR_PBICGSTAB ? -2 : EXIT_FAILURE);
      return rc;
    }
  }
  if (rc != SFR_OK && rc != SFR_MAXIT) {
    fprintf(stderr, "sfr_solverC: %s (%s)\n", sfr_status_string(rc), g_last_error.c_str());
    if (g_exit_on_failure) exit(solver == SFR_PBICGSTAB ? -2 : EXIT_FAILURE);
    return rc;
  }
  if (fLog && fSolvLog) {
    // Cg.c:201-208, Bicgstab.c:235-242, Bicgstab.c:1436-1443,
    // Iters.c:779-788, Iters.c:531-538
    switch (solver) {
      case SFR_PCG:
        fprintf(fSolvLog,
                "PCG: tol %20.2e iteration %d xKx %20.12e norma(x*x) %20.12e time %20.5lf\n",
                tol, info.iters, info.xKx, info.norm_x, info.seconds);
        break;
      case SFR_PBICGSTAB:
        fprintf(fSolvLog,
                "PBICGSTAB: tol %20.2e iteration %d xKx %20.12e ||x*x|| %20.12e time %20.5lf\n",
                tol, info.iters, info.xKx, info.norm_x, info.seconds);
        break;
      case SFR_PBICGSTABL2:
        fprintf(fSolvLog,
                "PBICGSTAB(2): tol %20.2e iteration %d xKx %20.12e norma(x*x) %20.12e "
                "time %20.5lf\n",
                tol, info.iters, info.xKx, info.norm_x, info.seconds);
        break;
      case SFR_GMRES:
        fprintf(fSolvLog,
                "GMRES: tol %20.2e  Cycles %d iteration %d  nKrylov %d  xKx %20.12e  "
                "norma(x*x) %20.12e  time %20.5lf\n",
                tol, (info.iters - 1) / 15, info.iters, 15, info.xKx, info.norm_x,
                info.seconds);
        break;
      default:
        fprintf(fSolvLog,
                "PMINRES: tol %20.2e iteration %d xKx %20.12e norma(x*x) %20.12e time %20.5lf\n",
                tol, info.iters, info.xKx, info.norm_x, info.seconds);
        break;
    }
  }
  return rc;
}

}  // extern "C"
