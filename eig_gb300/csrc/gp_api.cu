/*
 * C ABI of the smartpca hot path: handle management and the pass orchestration
 * (gp_xtx, gp_eigvecs, gp_snp_weights, gp_lsqproj) plus the host-side outlier rule.
 * The numerical work runs in the kernels of the other .cu files on the handle's stream.
 */
#include <cuda_runtime.h>
#include <cusolverDn.h>
#include <math.h>
#include <stdarg.h>
#include <stdlib.h>
#include <sys/mman.h>
#include <unistd.h>
#include <algorithm>
#include <atomic>
#include <memory>
#include <thread>
#include <vector>

#include "gp_geno_gemm.h"
#include "gp_geno_tc.h"
#include "gp_internal.h"

#define GP_VERSION 10000

static char g_open_err[GP_ERRLEN];

extern "C" int gp_version(void) { return GP_VERSION; }

extern "C" const char *gp_last_error(const gp_ctx *ctx) { return ctx ? ctx->err : g_open_err; }

int gp_fail(gp_ctx *ctx, int code, const char *fmt, ...)
{
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(ctx ? ctx->err : g_open_err, GP_ERRLEN, fmt, ap);
  va_end(ap);
  return code;
}

extern "C" int gp_fail_msg(gp_ctx *ctx, int code, const char *fmt, ...)
{
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(ctx ? ctx->err : g_open_err, GP_ERRLEN, fmt, ap);
  va_end(ap);
  return code;
}

cudaError_t gp_memcpy(gp_ctx *ctx, void *dst, const void *src, size_t bytes, cudaMemcpyKind kind,
                      cudaStream_t stream)
{
  if (kind == cudaMemcpyHostToDevice) ctx->h2d_bytes += (int64_t)bytes;
  if (kind == cudaMemcpyDeviceToHost) ctx->d2h_bytes += (int64_t)bytes;
  return cudaMemcpyAsync(dst, src, bytes, kind, stream);
}

/*
 * Fresh pages, Gram and its copy out: 13.5 MB 1.08 ms with threads and 0.91 without, 32 MB 1.27 and
 * 1.58, so from 16 MB on.  Four threads: 72 MB 1.80 ms and 200 MB 3.25, with one 3.0 and 6.8, two 2.1
 * and 4.2, eight 3.8 and 8.7 (they queue for the address space's lock).  Pieces of 1 MB 1.93 and
 * 3.40, of 16 MB 2.08 and 3.49.  Pages that are there already, as an array's that is used again, need
 * none of it: 8.4 MB 0.53 ms with threads and 0.45 without, 32 MB 1.11 and 1.00.
 */
#define OP_PIECE ((size_t)4 << 20)
#define OP_LEAST ((size_t)16 << 20)
#define OP_THREADS 4

struct gp_out_pages::impl {
  std::vector<std::thread> threads;
  std::atomic<size_t> next{0};
  std::unique_ptr<std::atomic<uint8_t>[]> done;
  size_t npieces = 0;

  void run(uint8_t *base, size_t bytes)
  {
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
    for (size_t i; (i = next.fetch_add(1)) < npieces;) {
      /* whole pages that begin in the piece (the first piece's partial page stays as it is) */
      const uintptr_t end = (uintptr_t)base + bytes;
      uintptr_t a = (uintptr_t)base + i * OP_PIECE, b = a + OP_PIECE < end ? a + OP_PIECE : end;
      a = (a + page - 1) / page * page;
      b = (b + page - 1) / page * page;
      if (b > end) b -= page;
#ifdef MADV_POPULATE_WRITE
      if (a < b) (void)madvise((void *)a, b - a, MADV_POPULATE_WRITE); /* a hint: may fail */
#endif
      done[i].store(1, std::memory_order_release);
    }
  }
};

/* whether the pages of [base, base + bytes) are there already, by a few spread evenly */
#define OP_PROBES 4
static bool op_present(const uint8_t *base, size_t bytes)
{
  const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE);
  const uintptr_t first = ((uintptr_t)base + page - 1) / page;
  const uintptr_t last = ((uintptr_t)base + bytes) / page - 1;
  for (uintptr_t i = 0; i < OP_PROBES; ++i) {
    unsigned char in = 0;
    if (mincore((void *)((first + (last - first) * i / (OP_PROBES - 1)) * page), page, &in) != 0 || !(in & 1))
      return false;
  }
  return true;
}

gp_out_pages::gp_out_pages(void *dst, size_t n) : base((uint8_t *)dst), bytes(n), im(NULL)
{
  if (!dst || n < OP_LEAST) return;
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, dst) != cudaSuccess) {
    (void)cudaGetLastError();
    return;
  }
  if (at.type != cudaMemoryTypeUnregistered || op_present(base, n)) return;
  try {
    std::unique_ptr<impl> p(new impl);
    p->npieces = (n + OP_PIECE - 1) / OP_PIECE;
    p->done.reset(new std::atomic<uint8_t>[p->npieces]);
    for (size_t i = 0; i < p->npieces; ++i) p->done[i].store(0, std::memory_order_relaxed);
    impl *q = p.get();
    p->threads.reserve(OP_THREADS);
    im = p.release();
    for (int t = 0; t < OP_THREADS; ++t)
      im->threads.emplace_back([q, this] { q->run(this->base, this->bytes); });
  } catch (...) {
    /* no memory or no thread: the pieces that no thread takes are nobody's to wait for */
    if (im && im->threads.empty()) {
      delete im;
      im = NULL;
    }
  }
}

gp_out_pages::~gp_out_pages()
{
  if (!im) return;
  im->next.store(im->npieces); /* pieces not begun are not needed any more */
  for (std::thread &t : im->threads) t.join();
  delete im;
}

void gp_out_pages::wait(size_t begin, size_t end)
{
  if (!im || end <= begin) return;
  for (size_t i = begin / OP_PIECE; i <= (end - 1) / OP_PIECE; ++i)
    while (!im->done[i].load(std::memory_order_acquire)) std::this_thread::yield();
}

cudaError_t gp_copy_out(gp_ctx *ctx, gp_out_pages &pages, size_t offset, const void *src,
                        size_t bytes)
{
  if (!pages.im)
    return gp_memcpy(ctx, pages.base + offset, src, bytes, cudaMemcpyDeviceToHost, ctx->stream);
  for (size_t a = 0; a < bytes;) {
    const size_t n = bytes - a < 4 * OP_PIECE ? bytes - a : 4 * OP_PIECE;
    pages.wait(offset + a, offset + a + n);
    cudaError_t e = gp_memcpy(ctx, pages.base + offset + a, (const uint8_t *)src + a, n,
                              cudaMemcpyDeviceToHost, ctx->stream);
    if (e != cudaSuccess) return e;
    a += n;
  }
  return cudaSuccess;
}

int gp_cuda_fail(gp_ctx *ctx, cudaError_t e, const char *what)
{
  return gp_fail(ctx, e == cudaErrorMemoryAllocation ? GP_ERR_NOMEM : GP_ERR_CUDA,
                 "%s: %s", what, cudaGetErrorString(e));
}

static int grow(gp_ctx *ctx, void **buf, size_t *cap, size_t bytes)
{
  if (bytes <= *cap && *buf) return GP_OK;
  if (*buf) {
    cudaFree(*buf);
    *buf = NULL;
    *cap = 0;
  }
  size_t want = bytes < 256 ? 256 : bytes;
  cudaError_t e = cudaMalloc(buf, want);
  if (e != cudaSuccess) {
    *buf = NULL;
    return gp_fail(ctx, GP_ERR_NOMEM, "device allocation of %zu bytes failed: %s", want,
                   cudaGetErrorString(e));
  }
  *cap = want;
  return GP_OK;
}

int gp_scratch(gp_ctx *ctx, size_t bytes, void **out)
{
  int rc = grow(ctx, &ctx->d_scratch, &ctx->scratch_cap, bytes);
  *out = ctx->d_scratch;
  return rc;
}

int gp_scratch_aux(gp_ctx *ctx, size_t bytes, void **out)
{
  int rc = grow(ctx, &ctx->d_scratch3, &ctx->scratch3_cap, bytes);
  *out = ctx->d_scratch3;
  return rc;
}

int gp_scratch4(gp_ctx *ctx, size_t bytes, void **out)
{
  ctx->codes4_rows = 0; /* the caller overwrites the codes */
  int rc = grow(ctx, &ctx->d_scratch4, &ctx->scratch4_cap, bytes);
  *out = ctx->d_scratch4;
  return rc;
}

int gp_scratch5(gp_ctx *ctx, size_t bytes, void **out)
{
  int rc = grow(ctx, &ctx->d_scratch5, &ctx->scratch5_cap, bytes);
  *out = ctx->d_scratch5;
  return rc;
}

int gp_scratch2(gp_ctx *ctx, size_t bytes, void **out)
{
  int rc = grow(ctx, &ctx->d_scratch2, &ctx->scratch2_cap, bytes);
  *out = ctx->d_scratch2;
  return rc;
}

/* a handle buffer of at least `bytes` (contents not kept): the allocation stays while it is
 * large enough, so that the per-pass buffers of a run (sample and SNP lists, tables, vectors)
 * cost no cudaFree / cudaMalloc, nor their device synchronisation, after the first pass */
int gp_realloc(gp_ctx *ctx, void **ptr, size_t bytes)
{
  if (bytes < 256) bytes = 256;
  int slot = -1;
  for (int i = 0; i < ctx->ncaps; ++i)
    if (ctx->caps[i].p == ptr) slot = i;
  if (slot >= 0 && *ptr && ctx->caps[slot].bytes >= bytes) return GP_OK;
  if (*ptr) cudaFree(*ptr);
  *ptr = NULL;
  cudaError_t e = cudaMalloc(ptr, bytes);
  if (e != cudaSuccess) {
    *ptr = NULL;
    return gp_fail(ctx, GP_ERR_NOMEM, "device allocation of %zu bytes failed: %s", bytes,
                   cudaGetErrorString(e));
  }
  if (slot < 0 && ctx->ncaps < (int)(sizeof(ctx->caps) / sizeof(ctx->caps[0]))) {
    slot = ctx->ncaps++;
    ctx->caps[slot].p = ptr;
  }
  if (slot >= 0) ctx->caps[slot].bytes = bytes;
  return GP_OK;
}

cudaError_t gp_allow_smem(gp_ctx *ctx, const void *func)
{
  int optin = 0;
  cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin,
                                         ctx->device);
  if (e != cudaSuccess) return e;
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, func);
  if (e != cudaSuccess) return e;
  return cudaFuncSetAttribute(func, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              optin - (int)fa.sharedSizeBytes);
}

extern "C" int gp_open(int device, gp_ctx **out)
{
  if (!out) return gp_fail(NULL, GP_ERR_ARG, "gp_open: out is NULL");
  *out = NULL;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess || ndev == 0)
    return gp_fail(NULL, GP_ERR_CUDA, "gp_open: no CUDA device (%s)", cudaGetErrorString(e));
  if (device < 0 || device >= ndev)
    return gp_fail(NULL, GP_ERR_ARG, "gp_open: device %d out of range", device);
  gp_ctx *ctx = (gp_ctx *)calloc(1, sizeof(gp_ctx));
  if (!ctx) return gp_fail(NULL, GP_ERR_NOMEM, "gp_open: host allocation failed");
  ctx->device = device;
  e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ctx->num_sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    gp_fail(NULL, GP_ERR_CUDA, "gp_open: %s", cudaGetErrorString(e));
    free(ctx);
    return GP_ERR_CUDA;
  }
  if (e == cudaSuccess) e = cudaMalloc((void **)&ctx->d_err, 256);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev_t0);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev_t1);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev_g0);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev_tr0);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev_tr1);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev_c0);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev_c1);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev_g1);
  if (e != cudaSuccess) {
    gp_fail(NULL, GP_ERR_CUDA, "gp_open: %s", cudaGetErrorString(e));
    free(ctx);
    return GP_ERR_CUDA;
  }
  if (cusolverDnCreate(&ctx->solver) != CUSOLVER_STATUS_SUCCESS ||
      cusolverDnSetStream(ctx->solver, ctx->stream) != CUSOLVER_STATUS_SUCCESS) {
    cudaStreamDestroy(ctx->stream);
    free(ctx);
    return gp_fail(NULL, GP_ERR_SOLVER, "gp_open: cusolverDnCreate failed");
  }
  *out = ctx;
  return GP_OK;
}

extern "C" void gp_close(gp_ctx *ctx)
{
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  void *bufs[] = {ctx->d_geno,   ctx->d_rows,    ctx->d_rowmask, ctx->d_cols,    ctx->d_cnt,
                  ctx->d_killed, ctx->d_vtab,    ctx->d_xmean,   ctx->d_xfancy,  ctx->d_kept,
                  ctx->d_xtx,    ctx->d_evals,   ctx->d_evecs,   ctx->d_ffvecs,  ctx->d_fxscal,
                  ctx->d_scratch, ctx->d_scratch2, ctx->d_scratch3, ctx->d_scratch4, ctx->d_scratch5,
                  ctx->d_err,   ctx->d_xtx_keep, ctx->d_rowpop, ctx->d_gtab, ctx->d_gfill,
                  ctx->d_tri,   ctx->d_tt};
  for (size_t i = 0; i < sizeof(bufs) / sizeof(bufs[0]); ++i)
    if (bufs[i]) cudaFree(bufs[i]);
  if (ctx->solver) cusolverDnDestroy(ctx->solver);
  if (ctx->blas) cublasDestroy(ctx->blas);
  if (ctx->ev_t0) cudaEventDestroy(ctx->ev_t0);
  if (ctx->ev_t1) cudaEventDestroy(ctx->ev_t1);
  if (ctx->ev_g0) cudaEventDestroy(ctx->ev_g0);
  if (ctx->ev_tr0) cudaEventDestroy(ctx->ev_tr0);
  if (ctx->ev_tr1) cudaEventDestroy(ctx->ev_tr1);
  if (ctx->ev_c0) cudaEventDestroy(ctx->ev_c0);
  if (ctx->ev_c1) cudaEventDestroy(ctx->ev_c1);
  if (ctx->ev_g1) cudaEventDestroy(ctx->ev_g1);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  free(ctx->h_rows);
  free(ctx);
}

extern "C" int gp_release(gp_ctx *ctx)
{
  if (!ctx) return GP_ERR_ARG;
  GP_CUDA(ctx, cudaSetDevice(ctx->device));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  void **bufs[] = {(void **)&ctx->d_geno,    (void **)&ctx->d_rows,     (void **)&ctx->d_rowmask,
                   (void **)&ctx->d_cols,    (void **)&ctx->d_cnt,      (void **)&ctx->d_killed,
                   (void **)&ctx->d_vtab,    (void **)&ctx->d_xmean,    (void **)&ctx->d_xfancy,
                   (void **)&ctx->d_kept,    (void **)&ctx->d_xtx,      (void **)&ctx->d_evals,
                   (void **)&ctx->d_evecs,   (void **)&ctx->d_ffvecs,   (void **)&ctx->d_fxscal,
                   (void **)&ctx->d_scratch, (void **)&ctx->d_scratch2, (void **)&ctx->d_scratch3,
                   (void **)&ctx->d_scratch4, (void **)&ctx->d_scratch5, (void **)&ctx->d_xtx_keep,
                   (void **)&ctx->d_rowpop,  (void **)&ctx->d_gtab,     (void **)&ctx->d_gfill,
                   (void **)&ctx->d_tri,     (void **)&ctx->d_tt};
  for (size_t i = 0; i < sizeof(bufs) / sizeof(bufs[0]); ++i) {
    if (*bufs[i]) cudaFree(*bufs[i]);
    *bufs[i] = NULL;
  }
  ctx->scratch_cap = ctx->scratch2_cap = ctx->scratch3_cap = ctx->scratch4_cap =
      ctx->scratch5_cap = 0;
  ctx->xtx_cap = 0;
  ctx->tt_n = 0;
  ctx->geno_cap = 0;
  ctx->codes4_rows = 0;
  ctx->keep_cap = 0;
  ctx->keep_valid = 0;
  ctx->nsnp_all = 0;
  ctx->nind_all = 0;
  ctx->rlen_dev = 0;
  ctx->nrows = ctx->ncols = ctx->nkept = ctx->nvec = ctx->nweights = 0;
  ctx->npop = 0;
  ctx->xtx_valid = ctx->eig_valid = ctx->weights_valid = 0;
  return GP_OK;
}

extern "C" int gp_device_bytes(const gp_ctx *ctx, int64_t *bytes)
{
  if (!ctx || !bytes) return GP_ERR_ARG;
  int64_t b = (int64_t)ctx->rlen_dev * ctx->nsnp_all + (int64_t)ctx->scratch_cap +
              (int64_t)ctx->scratch2_cap + (int64_t)ctx->scratch3_cap +
              (int64_t)ctx->scratch4_cap + (int64_t)ctx->scratch5_cap +
              (int64_t)sizeof(double) * ctx->xtx_cap;
  *bytes = b;
  return GP_OK;
}

/* ------------------------------------------------------------------------------------ */

__global__ void k_scale(double *x, int64_t n, double s)
{
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    x[i] = x[i] * s;
}

extern "C" int gp_xtx(gp_ctx *ctx, const gp_xtx_opts *opts, int32_t *n0, int32_t *n1,
                      int32_t *nmiss, uint8_t *killed, double *xmean, double *xfancy,
                      double *XTX, double *trace, int32_t *nused)
{
  if (!ctx || !opts) return GP_ERR_ARG;
  if (!ctx->d_geno || ctx->nrows < 1 || ctx->ncols < 1)
    return gp_fail(ctx, GP_ERR_STATE, "gp_xtx: genotypes, samples and SNPs must be set first");
  if (opts->precision < GP_PREC_FP64 || opts->precision > GP_PREC_SPLIT_FP16)
    return gp_fail(ctx, GP_ERR_ARG, "gp_xtx: unknown precision %d", opts->precision);
  GP_CUDA(ctx, cudaSetDevice(ctx->device));
  const int32_t n = ctx->nrows, nc = ctx->ncols;
  int64_t need = (int64_t)n * n;
  if (need > ctx->xtx_cap) {
    int rc = gp_realloc(ctx, (void **)&ctx->d_xtx, sizeof(double) * (size_t)need);
    if (rc) {
      ctx->xtx_cap = 0;
      return rc;
    }
    ctx->xtx_cap = need;
  }
  ctx->xtx_valid = ctx->eig_valid = ctx->weights_valid = 0;
  ctx->precision = opts->precision;
  gp_out_pages out_pages(XTX, XTX ? sizeof(double) * (size_t)need : 0);
  int rc;
  if (ctx->npop > 0) {
    /* usepopsformissing: the observed counts first (the missing-count rule waits for the
     * fill), then the filled tables, counts and kill flags */
    if (opts->precision != GP_PREC_FP64)
      return gp_fail(ctx, GP_ERR_ARG, "gp_xtx: usepopsformissing runs in FP64 precision only");
    gp_xtx_opts o1 = *opts;
    o1.maxmissing = 0x7FFFFFFF;
    rc = gp_launch_snp_stats(ctx, &o1);
    if (!rc) rc = gp_popfill_pass(ctx, opts);
  } else {
    rc = gp_launch_snp_stats(ctx, opts);
  }
  if (rc) return rc;

  /* FP64 without population fill: exact integer sums on the tensor cores, whose scale comes back
   * with the kill flags, in one copy */
  const bool exact = opts->precision == GP_PREC_FP64 && ctx->npop == 0;
  const size_t part_at = gp_killed_bytes(nc) - sizeof(double) * GP_EXACT_PARTS;
  if (exact) {
    rc = gp_gram_exact_max(ctx, (double *)(ctx->d_killed + part_at));
    if (rc) return rc;
  }
  /* kept-column list (ascending) built from the kill flags */
  std::vector<uint8_t> hk(exact ? gp_killed_bytes(nc) : (size_t)nc);
  GP_CUDA(ctx, gp_memcpy(ctx, hk.data(), ctx->d_killed, hk.size(), cudaMemcpyDeviceToHost,
                         ctx->stream));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  std::vector<int32_t> kept;
  kept.reserve((size_t)nc);
  for (int32_t c = 0; c < nc; ++c)
    if (!hk[(size_t)c]) kept.push_back(c);
  ctx->nkept = (int32_t)kept.size();
  ctx->codes4_rows = 0;
  if (ctx->nkept)
    GP_CUDA(ctx, gp_memcpy(ctx, ctx->d_kept, kept.data(), sizeof(int32_t) * kept.size(),
                                 cudaMemcpyHostToDevice, ctx->stream));

  GP_CUDA(ctx, cudaEventRecord(ctx->ev_g0, ctx->stream));
  ctx->gram_launches = 0;
  /* usepopsformissing's filled values are no linear function of the genotype and keep the
   * FP64-pipe kernel, which also takes over when the device has no room for the digits of one
   * block of SNPs */
  bool symmetric = false;
  if (opts->precision != GP_PREC_FP64) {
    rc = gp_gram_split(ctx, opts->precision);
  } else {
    rc = GP_ERR_NOMEM;
    if (exact && ctx->nkept > 0) {
      double part[GP_EXACT_PARTS];
      memcpy(part, hk.data() + part_at, sizeof part);
      rc = gp_gram_exact(ctx, part);
      symmetric = rc == GP_OK;
    }
    if (rc == GP_ERR_NOMEM) {
      cudaGetLastError();
      rc = gp_gram_fp64(ctx);
    }
  }
  if (rc) return rc;
  GP_CUDA(ctx, cudaEventRecord(ctx->ev_g1, ctx->stream));

  double *d_tr;
  rc = gp_scratch(ctx, sizeof(double), (void **)&d_tr);
  if (rc) return rc;
  rc = gp_launch_symmetrize_trace(ctx, d_tr, symmetric);
  if (rc) return rc;
  double tr = 0.0;
  GP_CUDA(ctx, gp_memcpy(ctx, &tr, d_tr, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
  if (symmetric) {
    rc = gp_tc_check(ctx);
    if (rc) return rc;
  }
  if (n0 || n1 || nmiss) {
    std::vector<int32_t> cnt((size_t)nc * 3);
    GP_CUDA(ctx, gp_memcpy(ctx, cnt.data(), ctx->d_cnt, sizeof(int32_t) * cnt.size(),
                                 cudaMemcpyDeviceToHost, ctx->stream));
    GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    for (int32_t c = 0; c < nc; ++c) {
      if (n0) n0[c] = cnt[3 * (size_t)c];
      if (n1) n1[c] = cnt[3 * (size_t)c + 1];
      if (nmiss) nmiss[c] = cnt[3 * (size_t)c + 2];
    }
  }
  if (killed) memcpy(killed, hk.data(), (size_t)nc);
  if (xmean)
    GP_CUDA(ctx, gp_memcpy(ctx, xmean, ctx->d_xmean, sizeof(double) * nc,
                                 cudaMemcpyDeviceToHost, ctx->stream));
  if (xfancy)
    GP_CUDA(ctx, gp_memcpy(ctx, xfancy, ctx->d_xfancy, sizeof(double) * nc,
                                 cudaMemcpyDeviceToHost, ctx->stream));
  if (XTX)
    GP_CUDA(ctx, gp_copy_out(ctx, out_pages, 0, ctx->d_xtx, sizeof(double) * (size_t)need));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  float gms = 0.f;
  GP_CUDA(ctx, cudaEventElapsedTime(&gms, ctx->ev_g0, ctx->ev_g1));
  ctx->gram_ms = gms;
  ctx->gram_flops = (double)n * (double)(n + 1) * (double)ctx->nkept;
  ctx->trace = tr;
  if (trace) *trace = tr;
  if (nused) *nused = ctx->nkept;
  ctx->xtx_valid = 1;
  return GP_OK;
}

/* ------------------------------------------------------------------------------------ */

/* evecs[j*n + i] = A[(n-1-j)*n + i]: the top nvec eigenvectors (columns) in descending order */
__global__ void k_take_top(double *evecs, const double *A, int32_t n, int32_t nvec)
{
  int64_t total = (int64_t)n * nvec;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int64_t j = idx / n, i = idx - j * n;
    evecs[idx] = A[(int64_t)(n - 1 - j) * n + i];
  }
}

extern "C" int gp_eigvecs(gp_ctx *ctx, int32_t nvec, double *evals, double *evecs)
{
  if (!ctx) return GP_ERR_ARG;
  if (!ctx->xtx_valid) return gp_fail(ctx, GP_ERR_STATE, "gp_eigvecs: no Gram (call gp_xtx)");
  const int32_t n = ctx->nrows;
  if (nvec < 0 || nvec > n) return gp_fail(ctx, GP_ERR_ARG, "gp_eigvecs: nvec %d", nvec);
  GP_CUDA(ctx, cudaSetDevice(ctx->device));
  /* y = trace/(n-1); XTX *= 1/y  (smartpca.c:1230-1236) */
  double y = ctx->trace / (double)(n - 1);
  if (isnan(y)) return gp_fail(ctx, GP_ERR_NODATA, "bad XTX matrix");
  if (y <= 0.0) return gp_fail(ctx, GP_ERR_NODATA, "XTX has zero trace (perhaps no data)");
  int64_t nn = (int64_t)n * n;
  int blocks = (int)((nn + 255) / 256);
  if (blocks > ctx->num_sms * 16) blocks = ctx->num_sms * 16;
  k_scale<<<blocks, 256, 0, ctx->stream>>>(ctx->d_xtx, nn, 1.0 / y);
  GP_LAUNCH_CHECK(ctx, "k_scale");
  ctx->keep_valid = 0;
  if (ctx->keep_gram) {
    /* the scaled Gram for the relatedness scan (the eigensolve overwrites d_xtx) */
    if (ctx->keep_cap < nn) {
      if (ctx->d_xtx_keep) cudaFree(ctx->d_xtx_keep);
      ctx->d_xtx_keep = NULL;
      ctx->keep_cap = 0;
      GP_CUDA(ctx, cudaMalloc((void **)&ctx->d_xtx_keep, sizeof(double) * (size_t)nn));
      ctx->keep_cap = nn;
    }
    GP_CUDA(ctx, cudaMemcpyAsync(ctx->d_xtx_keep, ctx->d_xtx, sizeof(double) * (size_t)nn,
                                 cudaMemcpyDeviceToDevice, ctx->stream));
    ctx->keep_valid = 1;
  }

  int rc = gp_realloc(ctx, (void **)&ctx->d_evals, sizeof(double) * (size_t)n);
  if (rc) return rc;
  int32_t keep = nvec > 0 ? nvec : 1;
  rc = gp_realloc(ctx, (void **)&ctx->d_evecs, sizeof(double) * (size_t)n * keep);
  if (rc) return rc;
  const char *alt = getenv("GP_EIG_SYEVD");
  if (!(alt && alt[0] == '1')) {
    /* tridiagonalisation + bisection + inverse iteration for the top vectors (gp_eig.cu) */
    rc = gp_eig_tridiag(ctx, n, nvec, ctx->d_evals, ctx->d_evecs);
    if (rc) return rc;
    if (evals)
      GP_CUDA(ctx, gp_memcpy(ctx, evals, ctx->d_evals, sizeof(double) * (size_t)n,
                             cudaMemcpyDeviceToHost, ctx->stream));
    if (evecs && nvec > 0)
      GP_CUDA(ctx, gp_memcpy(ctx, evecs, ctx->d_evecs, sizeof(double) * (size_t)n * nvec,
                             cudaMemcpyDeviceToHost, ctx->stream));
    GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    ctx->xtx_valid = 0; /* sytrd overwrote the Gram */
  } else {
    int lwork = 0;
    if (cusolverDnDsyevd_bufferSize(ctx->solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER,
                                    n, ctx->d_xtx, n, ctx->d_evals, &lwork) !=
        CUSOLVER_STATUS_SUCCESS)
      return gp_fail(ctx, GP_ERR_SOLVER, "cusolverDnDsyevd_bufferSize failed");
    uint8_t *ws;
    rc = gp_scratch(ctx, sizeof(double) * (size_t)lwork + 256, (void **)&ws);
    if (rc) return rc;
    int *d_info = (int *)(ws + sizeof(double) * (size_t)lwork);
    if (cusolverDnDsyevd(ctx->solver, CUSOLVER_EIG_MODE_VECTOR, CUBLAS_FILL_MODE_LOWER, n,
                         ctx->d_xtx, n, ctx->d_evals, (double *)ws, lwork,
                         d_info) != CUSOLVER_STATUS_SUCCESS)
      return gp_fail(ctx, GP_ERR_SOLVER, "cusolverDnDsyevd failed to launch");
    int info = 0;
    GP_CUDA(ctx, gp_memcpy(ctx, &info, d_info, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    if (nvec > 0) {
      int64_t tot = (int64_t)n * nvec;
      int b2 = (int)((tot + 255) / 256);
      if (b2 > ctx->num_sms * 16) b2 = ctx->num_sms * 16;
      k_take_top<<<b2, 256, 0, ctx->stream>>>(ctx->d_evecs, ctx->d_xtx, n, nvec);
      GP_LAUNCH_CHECK(ctx, "k_take_top");
    }
    std::vector<double> w((size_t)n);
    GP_CUDA(ctx, gp_memcpy(ctx, w.data(), ctx->d_evals, sizeof(double) * (size_t)n,
                                 cudaMemcpyDeviceToHost, ctx->stream));
    if (evecs && nvec > 0)
      GP_CUDA(ctx, gp_memcpy(ctx, evecs, ctx->d_evecs, sizeof(double) * (size_t)n * nvec,
                                   cudaMemcpyDeviceToHost, ctx->stream));
    GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    ctx->xtx_valid = 0; /* the solver overwrote the Gram with eigenvectors */
    if (info != 0) return gp_fail(ctx, GP_ERR_SOLVER, "eigensolver info = %d", info);
    if (evals)
      for (int32_t i = 0; i < n; ++i) evals[i] = w[(size_t)(n - 1 - i)];
    /* the resident eigenvalues descending, as the tridiagonal path leaves them */
    for (int32_t i = 0; i < n / 2; ++i) std::swap(w[(size_t)i], w[(size_t)(n - 1 - i)]);
    GP_CUDA(ctx, gp_memcpy(ctx, ctx->d_evals, w.data(), sizeof(double) * (size_t)n,
                           cudaMemcpyHostToDevice, ctx->stream));
  }
  ctx->nvec = nvec;
  ctx->eig_valid = 1;
  ctx->weights_valid = 0;
  return GP_OK;
}

/* ------------------------------------------------------------------------------------ */
/*
 * Relatedness of smartrel (src/eigensrc/smartrel.c:578-615): from the scaled Gram of the last
 * pass, R = XTX - sum_{i < K} w_i w_i^T with w_i = sqrt(lambda_i) v_i (subouter, in order),
 * then for rows a < b: y = R_ab / sqrt(R_aa R_bb) + 1/(n-1); pairs with y >= relthresh.
 * Same operation order as the reference, every product and sum rounded on its own.
 */
__global__ void k_rel_weights(const double *evals, const double *evecs, int32_t n, int32_t K,
                              double *w)
{
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < (int64_t)K * n;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = (int32_t)(idx / n);
    w[idx] = __dmul_rn(evecs[idx], __dsqrt_rn(evals[i]));
  }
}

__device__ __forceinline__ double rel_entry(const double *X, const double *w, int32_t n, int32_t K,
                                            int32_t a, int32_t b)
{
  double r = X[(int64_t)a * n + b];
  for (int32_t i = 0; i < K; ++i)
    r = __dsub_rn(r, __dmul_rn(w[(int64_t)i * n + a], w[(int64_t)i * n + b]));
  return r;
}

/* R_aa for every row, once (the scan reads it for both ends of each pair) */
__global__ void k_rel_diag(const double *X, const double *w, int32_t n, int32_t K, double *d)
{
  for (int32_t a = blockIdx.x * blockDim.x + threadIdx.x; a < n; a += gridDim.x * blockDim.x)
    d[a] = rel_entry(X, w, n, K, a, a);
}

__global__ void k_rel_scan(const double *X, const double *w, const double *d, int32_t n,
                           int32_t K, double relthresh, int64_t max_pairs, int32_t *pa,
                           int32_t *pb, double *ps, unsigned long long *count)
{
  const int64_t total = (int64_t)n * (n - 1) / 2;
  const double add = 1.0 / (double)(n - 1);
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total;
       t += (int64_t)gridDim.x * blockDim.x) {
    /* t -> (a, b), a < b, row by row of the strict upper triangle */
    int32_t a = (int32_t)floor(((2.0 * n - 1.0) - sqrt((2.0 * n - 1.0) * (2.0 * n - 1.0) - 8.0 * (double)t)) * 0.5);
    while (a > 0 && (int64_t)a * (2 * (int64_t)n - a - 1) / 2 > t) --a;
    while ((int64_t)(a + 1) * (2 * (int64_t)n - a - 2) / 2 <= t) ++a;
    const int32_t b = (int32_t)(t - (int64_t)a * (2 * (int64_t)n - a - 1) / 2) + a + 1;
    const double y1 = d[a], y2 = d[b];
    const double y = __dadd_rn(__ddiv_rn(rel_entry(X, w, n, K, a, b), __dsqrt_rn(__dmul_rn(y1, y2))), add);
    if (y < relthresh) continue;
    const unsigned long long slot = atomicAdd(count, 1ull);
    if ((int64_t)slot < max_pairs) {
      pa[slot] = a;
      pb[slot] = b;
      ps[slot] = y;
    }
  }
}

extern "C" int gp_keep_gram(gp_ctx *ctx, int32_t keep)
{
  if (!ctx) return GP_ERR_ARG;
  ctx->keep_gram = keep ? 1 : 0;
  return GP_OK;
}

extern "C" int gp_relate(gp_ctx *ctx, int32_t numeigs, double relthresh, int64_t max_pairs,
                         int32_t *pair_a, int32_t *pair_b, double *score, int64_t *npairs)
{
  if (!ctx || !npairs || max_pairs < 0 || (max_pairs > 0 && (!pair_a || !pair_b || !score)))
    return GP_ERR_ARG;
  if (!ctx->keep_valid || !ctx->eig_valid)
    return gp_fail(ctx, GP_ERR_STATE, "gp_relate: no kept Gram (gp_keep_gram before gp_eigvecs)");
  const int32_t n = ctx->nrows, K = numeigs;
  if (K < 0 || K > ctx->nvec) return gp_fail(ctx, GP_ERR_ARG, "gp_relate: numeigs %d > %d", K, ctx->nvec);
  GP_CUDA(ctx, cudaSetDevice(ctx->device));
  const size_t nw = (size_t)K * n;
  size_t bytes = sizeof(double) * (nw + (size_t)n + (size_t)max_pairs) +
                 sizeof(int32_t) * 2 * (size_t)max_pairs + 1024;
  uint8_t *base;
  int rc = gp_scratch(ctx, bytes, (void **)&base);
  if (rc) return rc;
  double *d_w = (double *)base, *d_d = d_w + nw, *d_s = d_d + n;
  int32_t *d_a = (int32_t *)(d_s + max_pairs), *d_b = d_a + max_pairs;
  unsigned long long *d_cnt = (unsigned long long *)(((uintptr_t)(d_b + max_pairs) + 15) & ~(uintptr_t)15);
  GP_CUDA(ctx, cudaMemsetAsync(d_cnt, 0, sizeof(unsigned long long), ctx->stream));
  if (nw) {
    int blocks = (int)((nw + 255) / 256);
    if (blocks > ctx->num_sms * 8) blocks = ctx->num_sms * 8;
    k_rel_weights<<<blocks, 256, 0, ctx->stream>>>(ctx->d_evals, ctx->d_evecs, n, K, d_w);
    GP_LAUNCH_CHECK(ctx, "k_rel_weights");
  }
  if (n > 1) {
    k_rel_diag<<<(n + 255) / 256, 256, 0, ctx->stream>>>(ctx->d_xtx_keep, d_w, n, K, d_d);
    GP_LAUNCH_CHECK(ctx, "k_rel_diag");
    k_rel_scan<<<ctx->num_sms * 8, 256, 0, ctx->stream>>>(ctx->d_xtx_keep, d_w, d_d, n, K,
                                                          relthresh, max_pairs, d_a, d_b, d_s,
                                                          d_cnt);
    GP_LAUNCH_CHECK(ctx, "k_rel_scan");
  }
  unsigned long long cnt = 0;
  GP_CUDA(ctx, gp_memcpy(ctx, &cnt, d_cnt, sizeof cnt, cudaMemcpyDeviceToHost, ctx->stream));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  *npairs = (int64_t)cnt;
  const int64_t got = (int64_t)cnt < max_pairs ? (int64_t)cnt : max_pairs;
  if (got > 0) {
    GP_CUDA(ctx, gp_memcpy(ctx, pair_a, d_a, sizeof(int32_t) * (size_t)got, cudaMemcpyDeviceToHost, ctx->stream));
    GP_CUDA(ctx, gp_memcpy(ctx, pair_b, d_b, sizeof(int32_t) * (size_t)got, cudaMemcpyDeviceToHost, ctx->stream));
    GP_CUDA(ctx, gp_memcpy(ctx, score, d_s, sizeof(double) * (size_t)got, cudaMemcpyDeviceToHost, ctx->stream));
    GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  return GP_OK;
}

/* ------------------------------------------------------------------------------------ */

extern "C" int gp_ridoutlier(const double *evecs, int32_t n, int32_t neigs, double thresh,
                             int32_t mode, int32_t *badlist, int32_t *vecno, double *score)
{
  /* restates ridoutlier (src/eigensrc/smartsubs.c:18-91) with the same operation order */
  if (!evecs || !badlist || n < 0 || neigs < 0) return GP_ERR_ARG;
  if (mode > 1) return 0;
  if (n < 3) return 0;
  std::vector<double> ww((size_t)n), w2((size_t)n);
  std::vector<int> vbad((size_t)n, 0), vno((size_t)n, -1);
  std::vector<double> sc((size_t)n, 0.0);
  for (int32_t i = 0; i < neigs; ++i) {
    memcpy(ww.data(), evecs + (size_t)i * n, sizeof(double) * (size_t)n);
    if (mode == 0) {
      double y1 = 0.0;
      for (int32_t j = 0; j < n; ++j) y1 += ww[(size_t)j];
      y1 = y1 / (double)n;
      for (int32_t j = 0; j < n; ++j) ww[(size_t)j] = ww[(size_t)j] + (-y1);
      double y2 = 0.0;
      for (int32_t j = 0; j < n; ++j) y2 += ww[(size_t)j] * ww[(size_t)j];
      y2 = y2 / (double)n;
      y2 = sqrt(y2);
      double inv = 1.0 / y2;
      for (int32_t j = 0; j < n; ++j) ww[(size_t)j] = ww[(size_t)j] * inv;
      for (int32_t j = 0; j < n; ++j) {
        if (fabs(ww[(size_t)j]) > thresh) {
          vbad[(size_t)j] = 1;
          if (vno[(size_t)j] < 0) {
            vno[(size_t)j] = i;
            sc[(size_t)j] = ww[(size_t)j];
          }
        }
      }
    } else {
      for (int32_t j = 0; j < n; ++j) {
        double yy = ww[(size_t)j];
        ww[(size_t)j] = 0;
        double y1 = 0.0;
        for (int32_t t = 0; t < n; ++t) y1 += ww[(size_t)t];
        y1 = y1 / (double)(n - 1);
        for (int32_t t = 0; t < n; ++t) w2[(size_t)t] = ww[(size_t)t] + (-y1);
        w2[(size_t)j] = 0;
        double y2 = 0.0;
        for (int32_t t = 0; t < n; ++t) y2 += w2[(size_t)t] * w2[(size_t)t];
        y2 = y2 / (double)n;
        y2 = sqrt(y2);
        double zz = yy - y1;
        zz /= y2;
        if (fabs(zz) > thresh) {
          vbad[(size_t)j] = 1;
          if (vno[(size_t)j] < 0) {
            vno[(size_t)j] = i;
            sc[(size_t)j] = zz;
          }
        }
        ww[(size_t)j] = yy;
      }
    }
  }
  int32_t nbad = 0;
  for (int32_t j = 0; j < n; ++j) {
    if (vecno) vecno[j] = vno[(size_t)j];
    if (score) score[j] = sc[(size_t)j];
    if (vbad[(size_t)j] == 1) badlist[nbad++] = j;
  }
  return nbad;
}

/* ------------------------------------------------------------------------------------ */

/* B[r*K + j] = 10 * evecs[j*n + r]   (setfvecs src/qpsubs.c:489-507) */
__global__ void k_fvecs_T(double *B, const double *evecs, int32_t n, int32_t K)
{
  int64_t total = (int64_t)n * K;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int64_t r = idx / K, j = idx - r * K;
    B[idx] = evecs[j * n + r] * 10.0;
  }
}

/* per kept column: record index, value table (vtab) and the fixxrow table
 * r(g) = g*fancy - xmean (src/qpsubs.c:338-348), missing -> 0 */
__global__ void k_kept_tables(const int32_t *kept, int32_t nkept, const int32_t *cols,
                              const double *vtab, const double *xmean, const double *xfancy,
                              int32_t *snprec, double *vt, double *rt, double *ot)
{
  for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nkept; k += gridDim.x * blockDim.x) {
    int32_t c = kept[k];
    snprec[k] = cols[c];
    for (int t = 0; t < 4; ++t) vt[4 * k + t] = vtab[4 * c + t];
    double f = xfancy[c], m = xmean[c];
    for (int g = 0; g < 3; ++g) {
      double x = __dmul_rn((double)g, f);
      rt[4 * k + g] = (x < -0.001) ? 0.0 : __dsub_rn(x, m);
    }
    rt[4 * k + 3] = 0.0;
    ot[4 * k] = ot[4 * k + 1] = ot[4 * k + 2] = 1.0;
    ot[4 * k + 3] = 0.0;
  }
}

/* ffvT[k][j] = fancy_c Yg[k][j] - xmean_c Yo[k][j], c = kept[k]  (X = G fancy - O xmean) */
__global__ void k_combine_gx(double *ffvT, const double *yg, const double *yo, const int32_t *kept,
                             const double *xfancy, const double *xmean, int32_t nk, int32_t K)
{
  int64_t total = (int64_t)nk * K;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int32_t c = kept[idx / K];
    ffvT[idx] = xfancy[c] * yg[idx] - xmean[c] * yo[idx];
  }
}

/* a[k][j] = fancy_c w[k][j], b[k][j] = xmean_c w[k][j], c = kept[k] */
__global__ void k_scale_rows2(double *a, double *b, const double *w, const int32_t *kept,
                              const double *xfancy, const double *xmean, int32_t nk, int32_t K)
{
  int64_t total = (int64_t)nk * K;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int32_t c = kept[idx / K];
    a[idx] = xfancy[c] * w[idx];
    b[idx] = xmean[c] * w[idx];
  }
}

/* ffvecs[j*ncols + kept[k]] = ffvT[k*K + j] (killed columns stay 0) */
__global__ void k_scatter_ffvecs(double *ffvecs, const double *ffvT, const int32_t *kept,
                                 int32_t nkept, int32_t ncols, int32_t K)
{
  int64_t total = (int64_t)nkept * K;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int64_t k = idx / K, j = idx - k * K;
    ffvecs[j * ncols + kept[k]] = ffvT[idx];
  }
}

struct kept_tables {
  int32_t *snprec;
  double *vt, *rt, *ot;
};

static int build_kept_tables(gp_ctx *ctx, uint8_t *base, kept_tables *t)
{
  int32_t nk = ctx->nkept;
  t->vt = (double *)base;
  t->rt = t->vt + 4 * (size_t)nk;
  t->ot = t->rt + 4 * (size_t)nk;
  t->snprec = (int32_t *)(t->ot + 4 * (size_t)nk);
  if (nk == 0) return GP_OK;
  int blocks = (nk + 255) / 256;
  if (blocks > ctx->num_sms * 8) blocks = ctx->num_sms * 8;
  k_kept_tables<<<blocks, 256, 0, ctx->stream>>>(ctx->d_kept, nk, ctx->d_cols, ctx->d_vtab,
                                                 ctx->d_xmean, ctx->d_xfancy, t->snprec, t->vt,
                                                 t->rt, t->ot);
  GP_LAUNCH_CHECK(ctx, "k_kept_tables");
  return GP_OK;
}

/* bytes of the kept-column tables, rounded up so that what follows stays 256-byte aligned */
static size_t kept_tables_bytes(int32_t nk)
{
  size_t b = (size_t)nk * (12 * sizeof(double) + sizeof(int32_t)) + 256;
  return (b + 255) / 256 * 256;
}

/* Whether the products of weights and lsqproject run on the tensor cores: always at the split
 * precisions; at FP64 with 12-bit slices, except after a pass with population fill (its SNP
 * weights take the observed genotypes' table, which is not g fancy - xmean) and for records
 * longer than the SNP-major code builder stages in shared memory. */
static int tc_products(const gp_ctx *ctx, int32_t nk)
{
  if (nk < 1) return 0;
  if (ctx->precision != GP_PREC_FP64) return 1;
  return ctx->npop == 0 && ctx->rlen_dev <= 200 * 1024;
}
static int tc_digits(const gp_ctx *ctx) { return ctx->precision == GP_PREC_FP64 ? 5 : 4; }

static int grid16(const gp_ctx *ctx, int64_t work)
{
  const int64_t b = (work + 255) / 256;
  return (int)(b < ctx->num_sms * 16 ? b : ctx->num_sms * 16);
}

/* out[rows[r]][j] = w[r][j] */
__global__ void k_spread_rows(double *out, const double *w, const int32_t *rows, int32_t n, int32_t K)
{
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < (int64_t)n * K;
       idx += (int64_t)gridDim.x * blockDim.x)
    out[(int64_t)rows[idx / K] * K + idx % K] = w[idx];
}

/* ffvT [nk][K] = fancy (G^T W) - xmean (O^T W) */
static int weights_tc(gp_ctx *ctx, const kept_tables *kt, const double *d_W, int32_t K, double *d_ffvT)
{
  const int32_t n = ctx->nrows, nk = ctx->nkept, ni = ctx->nind_all;
  /* rows that are part of the samples: the resident records serve as the operand all the same,
   * W zero for the other samples, which cost a product term each; gathering the rows' codes of
   * every SNP costs about eight (4,000 of 5,000 samples x 200,000 SNPs: 2.7 ms, the products of
   * all 5,000 0.27 ms each) */
  const bool spread = n < ni && ni <= 8 * (int64_t)n;
  double *d_yg;
  int rc = gp_scratch_aux(ctx, sizeof(double) * (2 * (size_t)nk + (spread ? ni : 0)) * K,
                          (void **)&d_yg);
  if (rc) return rc;
  double *d_yo = d_yg + (size_t)nk * K;
  gp_tc_codes A;
  if (spread) {
    double *d_Wa = d_yo + (size_t)nk * K;
    GP_CUDA(ctx, cudaMemsetAsync(d_Wa, 0, sizeof(double) * (size_t)ni * K, ctx->stream));
    k_spread_rows<<<grid16(ctx, (int64_t)n * K), 256, 0, ctx->stream>>>(d_Wa, d_W, ctx->d_rows, n,
                                                                        K);
    GP_LAUNCH_CHECK(ctx, "k_spread_rows");
    d_W = d_Wa;
    A = {ctx->d_geno, ctx->rlen_dev, kt->snprec, nk, ni};
  } else {
    rc = gp_tc_codes_for(ctx, 0, ctx->d_rows, n, kt->snprec, nk, 1, &A);
    if (rc) return rc;
  }
  gp_tc_panel pw = {d_W, K, 1.0, 1};
  rc = gp_geno_panel_tc_codes(ctx, &A, 1, &pw, K, tc_digits(ctx), d_yg, K);
  if (rc) return rc;
  pw.count = 0;
  rc = gp_geno_panel_tc_codes(ctx, &A, 1, &pw, K, tc_digits(ctx), d_yo, K);
  if (rc) return rc;
  k_combine_gx<<<grid16(ctx, (int64_t)nk * K), 256, 0, ctx->stream>>>(
      d_ffvT, d_yg, d_yo, ctx->d_kept, ctx->d_xfancy, ctx->d_xmean, nk, K);
  GP_LAUNCH_CHECK(ctx, "k_combine_gx");
  return GP_OK;
}

/* Y [rows][K] = G (fancy w) - O (xmean w) for a panel w [nk][K]: the fixxrow products */
static int scores_tc(gp_ctx *ctx, const gp_tc_codes *A, const double *d_w, int32_t K, double *d_Y)
{
  const int32_t nk = ctx->nkept;
  double *tmp;
  int rc = gp_scratch_aux(ctx, sizeof(double) * 2 * (size_t)nk * K, (void **)&tmp);
  if (rc) return rc;
  k_scale_rows2<<<grid16(ctx, (int64_t)nk * K), 256, 0, ctx->stream>>>(
      tmp, tmp + (size_t)nk * K, d_w, ctx->d_kept, ctx->d_xfancy, ctx->d_xmean, nk, K);
  GP_LAUNCH_CHECK(ctx, "k_scale_rows2");
  gp_tc_panel pr[2] = {{tmp, K, 1.0, 1}, {tmp + (size_t)nk * K, K, -1.0, 0}};
  return gp_geno_panel_tc_codes(ctx, A, 2, pr, K, tc_digits(ctx), d_Y, K);
}

extern "C" int gp_snp_weights(gp_ctx *ctx, int32_t numeigs, double *ffvecs, double *fxvecs,
                              double *fxscal)
{
  if (!ctx || !fxscal) return GP_ERR_ARG;
  if (!ctx->eig_valid) return gp_fail(ctx, GP_ERR_STATE, "gp_snp_weights: call gp_eigvecs first");
  if (numeigs < 1 || numeigs > ctx->nvec)
    return gp_fail(ctx, GP_ERR_ARG, "gp_snp_weights: numeigs %d > resident vectors %d", numeigs,
                   ctx->nvec);
  GP_CUDA(ctx, cudaSetDevice(ctx->device));
  const int32_t n = ctx->nrows, nc = ctx->ncols, nk = ctx->nkept, K = numeigs;
  int rc = gp_realloc(ctx, (void **)&ctx->d_ffvecs, sizeof(double) * (size_t)K * nc);
  if (!rc) rc = gp_realloc(ctx, (void **)&ctx->d_fxscal, sizeof(double) * (size_t)K);
  if (rc) return rc;
  gp_out_pages out_pages(ffvecs, ffvecs ? sizeof(double) * (size_t)K * nc : 0);
  size_t off_tab = kept_tables_bytes(nk);
  size_t bytes = off_tab + sizeof(double) * ((size_t)n * K + (size_t)nk * K + (size_t)n * K) + 256;
  uint8_t *base;
  rc = gp_scratch(ctx, bytes, (void **)&base);
  if (rc) return rc;
  kept_tables kt;
  rc = build_kept_tables(ctx, base, &kt);
  if (rc) return rc;
  double *d_B = (double *)(base + off_tab);
  double *d_ffvT = d_B + (size_t)n * K;
  double *d_fxT = d_ffvT + (size_t)nk * K;
  int blocks = (int)(((int64_t)n * K + 255) / 256);
  if (blocks > ctx->num_sms * 16) blocks = ctx->num_sms * 16;
  k_fvecs_T<<<blocks, 256, 0, ctx->stream>>>(d_B, ctx->d_evecs, n, K);
  GP_LAUNCH_CHECK(ctx, "k_fvecs_T");
  int tc = tc_products(ctx, nk);
  const int tc_ran = tc;
  if (tc) {
    rc = gp_tc_begin(ctx);
    if (rc) return rc;
    /* tensor-core exact products: X = G fancy - O xmean, so
     * ffvecs^T = fancy (G^T W) - xmean (O^T W) with W = 10 evecs^T over the rows */
    rc = weights_tc(ctx, &kt, d_B, K, d_ffvT);
    if (rc == GP_ERR_NOMEM && ctx->precision == GP_PREC_FP64) {
      cudaGetLastError();
      tc = 0;
    } else if (rc) {
      return rc;
    }
  }
  if (!tc) {
    /* ffvecs^T[k][j] = sum_r v(r,k) * 10 evec_j[r] */
    rc = gp_geno_gemm_f64(ctx, 0, ctx->d_rows, n, kt.snprec, kt.vt, nk, d_B, K, K, d_ffvT, K);
    if (rc) return rc;
  }
  GP_CUDA(ctx, cudaMemsetAsync(ctx->d_ffvecs, 0, sizeof(double) * (size_t)K * nc, ctx->stream));
  if (nk) {
    int b2 = (int)(((int64_t)nk * K + 255) / 256);
    if (b2 > ctx->num_sms * 16) b2 = ctx->num_sms * 16;
    k_scatter_ffvecs<<<b2, 256, 0, ctx->stream>>>(ctx->d_ffvecs, d_ffvT, ctx->d_kept, nk, nc, K);
    GP_LAUNCH_CHECK(ctx, "k_scatter_ffvecs");
  }
  /* fxvecs^T[i][j] = xrow_i . ffvecs_j  (fixxrow values g fancy - xmean) */
  if (tc) {
    gp_tc_codes A;
    rc = gp_tc_codes_for(ctx, 1, ctx->d_rows, n, kt.snprec, nk, 1, &A);
    if (!rc) rc = scores_tc(ctx, &A, d_ffvT, K, d_fxT);
    if (rc == GP_ERR_NOMEM && ctx->precision == GP_PREC_FP64) {
      cudaGetLastError();
      tc = 0;
    } else if (rc) {
      return rc;
    }
  }
  if (!tc) {
    rc = gp_geno_gemm_f64(ctx, 1, ctx->d_rows, n, kt.snprec, kt.rt, nk, d_ffvT, K, K, d_fxT, K);
    if (rc) return rc;
  }
  if (tc_ran) {
    rc = gp_tc_check(ctx);
    if (rc) return rc;
  }
  std::vector<double> fx((size_t)n * K);
  GP_CUDA(ctx, gp_memcpy(ctx, fx.data(), d_fxT, sizeof(double) * fx.size(),
                               cudaMemcpyDeviceToHost, ctx->stream));
  if (ffvecs)
    GP_CUDA(ctx, gp_copy_out(ctx, out_pages, 0, ctx->d_ffvecs, sizeof(double) * (size_t)K * nc));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  /* fxscal_j = 1/sqrt(sum_i fxvecs^2) in row order (smartpca.c:1504-1525) */
  for (int32_t j = 0; j < K; ++j) {
    double s = 0.0;
    for (int32_t i = 0; i < n; ++i) {
      double y = fx[(size_t)i * K + j];
      if (fxvecs) fxvecs[(size_t)j * n + i] = y;
      s += y * y;
    }
    fxscal[j] = 1.0 / sqrt(s);
  }
  GP_CUDA(ctx, gp_memcpy(ctx, ctx->d_fxscal, fxscal, sizeof(double) * K, cudaMemcpyHostToDevice,
                               ctx->stream));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  ctx->nweights = K;
  ctx->weights_valid = 1;
  return GP_OK;
}

/* ------------------------------------------------------------------------------------ */

/* E[k*K + j] = fxscal_j * ffvecs_j[kept k];  P[k*ldp + pair(a,b)] = E_a E_b (a<=b), then 1 */
/* E[k][j] = fxscal_j ffvecs_j(kept k) and P[k] = (E_a E_b for a <= b in row order, 1):
 * a warp per kept SNP, E of the SNP in shared memory, the pair products written as
 * consecutive doubles (coalesced) from a pair-index table; K <= 64 */
#define EP_THREADS 256
__global__ void __launch_bounds__(EP_THREADS)
k_build_EP(const double *ffvecs, const double *fxscal, const int32_t *kept, int32_t nkept,
           int32_t ncols, int32_t K, double *E, double *P, int32_t ldp)
{
  __shared__ uint8_t pa[64 * 65 / 2], pb[64 * 65 / 2];
  __shared__ double se[EP_THREADS / 32][64];
  const int npair = K * (K + 1) / 2;
  for (int t = threadIdx.x; t < npair; t += blockDim.x) {
    int a = 0, rem = t;
    while (rem >= K - a) {
      rem -= K - a;
      ++a;
    }
    pa[t] = (uint8_t)a;
    pb[t] = (uint8_t)(a + rem);
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t k = (int64_t)blockIdx.x * (blockDim.x >> 5) + warp; k < nkept; k += nw) {
    const int32_t c = kept[k];
    for (int j = lane; j < K; j += 32) {
      const double v = fxscal[j] * ffvecs[(int64_t)j * ncols + c];
      se[warp][j] = v;
      E[k * K + j] = v;
    }
    __syncwarp();
    double *p = P + k * ldp;
    for (int t = lane; t < npair; t += 32) p[t] = se[warp][pa[t]] * se[warp][pb[t]];
    if (lane == 0) p[npair] = 1.0;
    __syncwarp();
  }
}

/*
 * Per sample: check the normal equations for NaN, Cholesky (choldc
 * src/nicksrc/linsubs.c:361-380) and the two triangular solves (cholsl :331-358), with the
 * reference's loop order and no contraction.  Eight lanes per sample, four samples per
 * one-warp CTA.  What bounds it is the FP64 pipe of a warp's own quarter of the SM (an
 * instruction occupies it for about 64 clocks) along the chains of subtractions that the
 * order prescribes: the lanes form the products of a chain side by side and take the columns
 * of a row in turn, and the factor (packed lower triangle over the pair sums it replaces),
 * the pivots, the solution and the products sit in shared memory.  K = 20, 5,000 samples:
 * 493 us with a thread per sample and the factors in global memory, 235 with a thread per
 * sample and shared memory, 185 here; 300 samples: 477, now 106.
 */
#define LSQ_LANES 8
#define LSQ_SAMPLES (32 / LSQ_LANES)
__global__ void __launch_bounds__(32)
k_lsq_solve(const double *co, int32_t ldco, const double *rr, int32_t K, int32_t nproj,
            double *acoef, double *bcoef, int32_t *nobs, int32_t *status, int32_t per,
            const int32_t *d_nproj)
{
  extern __shared__ double lsq_sm[];
  if (d_nproj) nproj = *d_nproj; /* a device-resident loop's batch size */
  const int sub = threadIdx.x & (LSQ_LANES - 1), sm = threadIdx.x / LSQ_LANES;
  const unsigned group = ((1u << LSQ_LANES) - 1u) << (sm * LSQ_LANES);
  double *Lm = lsq_sm + (size_t)sm * per;                    /* row j: L(j, k), k < j */
  double *p = Lm + K * (K - 1) / 2, *x = p + K, *pr = x + K; /* pivots, solution, products */
  for (int32_t q0 = blockIdx.x * LSQ_SAMPLES; q0 < nproj; q0 += gridDim.x * LSQ_SAMPLES) {
    const int32_t q = q0 + sm;
    bool act = q < nproj;
    int bad = 0;
    if (act) {
      const double *c = co + (int64_t)q * ldco, *rq = rr + (int64_t)q * K;
      const int32_t nob = (int32_t)llrint(c[K * (K + 1) / 2]);
      for (int i = 0; i < K; ++i) {
        for (int j = i + sub; j < K; j += LSQ_LANES) {
          const double v = c[j - i];
          bad |= isnan(v);
          *(j == i ? p + i : Lm + j * (j - 1) / 2 + i) = v;
        }
        c += K - i;
      }
      for (int j = sub; j < K; j += LSQ_LANES) {
        const double v = rq[j];
        bad |= isnan(v);
        x[j] = v;
        bcoef[(int64_t)j * nproj + q] = v;
      }
      if (sub == 0) nobs[q] = nob;
      if (nob <= K) {
        act = false;
        if (sub == 0) status[q] = 1;
      }
    }
    bad = (__ballot_sync(0xffffffffu, bad) & group) != 0;
    if (act && bad) {
      act = false;
      if (sub == 0) status[q] = 2;
    }
    for (int i = 0; i < K; ++i) {
      const double *Li = Lm + i * (i - 1) / 2;
      if (act)
        for (int k = sub; k < i; k += LSQ_LANES) pr[k] = __dmul_rn(Li[k], Li[k]);
      __syncwarp();
      if (act) {
        double sum = p[i];
        for (int k = i - 1; k >= 0; --k) sum = __dsub_rn(sum, pr[k]);
        if (sum <= 0.0) {
          act = false; /* every lane of the sample computes the same sum */
          if (sub == 0) status[q] = 2;
        } else {
          const double pi = __dsqrt_rn(sum);
          for (int j = i + 1 + sub; j < K; j += LSQ_LANES) {
            double *Lj = Lm + j * (j - 1) / 2;
            double s = Lj[i];
            for (int k = i - 1; k >= 0; --k) s = __dsub_rn(s, __dmul_rn(Li[k], Lj[k]));
            Lj[i] = __ddiv_rn(s, pi);
          }
          __syncwarp(group); /* every lane has read p[i] */
          if (sub == 0) p[i] = pi;
        }
      }
      __syncwarp();
    }
    for (int i = 0; i < K; ++i) {
      const double *Li = Lm + i * (i - 1) / 2;
      if (act)
        for (int k = sub; k < i; k += LSQ_LANES) pr[k] = __dmul_rn(Li[k], x[k]);
      __syncwarp();
      double sum = 0.0;
      if (act) {
        sum = x[i];
        for (int k = i - 1; k >= 0; --k) sum = __dsub_rn(sum, pr[k]);
        sum = __ddiv_rn(sum, p[i]);
      }
      __syncwarp();
      if (act && sub == 0) x[i] = sum;
      __syncwarp();
    }
    for (int i = K - 1; i >= 0; --i) {
      if (act)
        for (int k = i + 1 + sub; k < K; k += LSQ_LANES)
          pr[k] = __dmul_rn(Lm[k * (k - 1) / 2 + i], x[k]);
      __syncwarp();
      double sum = 0.0;
      if (act) {
        sum = x[i];
        for (int k = i + 1; k < K; ++k) sum = __dsub_rn(sum, pr[k]);
        sum = __ddiv_rn(sum, p[i]);
      }
      __syncwarp();
      if (act && sub == 0) {
        x[i] = sum;
        acoef[(int64_t)i * nproj + q] = sum;
      }
      __syncwarp();
    }
    if (act && sub == 0) status[q] = 0;
  }
}

int gp_launch_lsq_solve(gp_ctx *ctx, const double *co, int32_t ldco, const double *rr, int32_t K,
                        int32_t nproj, double *acoef, double *bcoef, int32_t *nobs,
                        int32_t *status, const int32_t *d_nproj)
{
  /* doubles of one sample; odd, so that the samples' equal elements lie in different banks */
  const int32_t per = (K * (K - 1) / 2 + 3 * K) | 1;
  const size_t smem = sizeof(double) * (size_t)per * LSQ_SAMPLES;
  GP_CUDA(ctx, gp_allow_smem(ctx, (const void *)k_lsq_solve));
  int blocks = (nproj + LSQ_SAMPLES - 1) / LSQ_SAMPLES;
  if (blocks > ctx->num_sms * 32) blocks = ctx->num_sms * 32;
  k_lsq_solve<<<blocks, 32, smem, ctx->stream>>>(co, ldco, rr, K, nproj, acoef, bcoef, nobs, status,
                                                 per, d_nproj);
  GP_LAUNCH_CHECK(ctx, "k_lsq_solve");
  return GP_OK;
}

static int lsqproj_impl(gp_ctx *ctx, int32_t numeigs, const int32_t *samples,
                        const int32_t *sample_pop, int32_t npop, int32_t nproj, double *acoeffs,
                        double *bcoeffs, int32_t *nobs, int32_t *status)
{
  if (!ctx || !acoeffs || (nproj > 0 && !samples)) return GP_ERR_ARG;
  if (!ctx->weights_valid)
    return gp_fail(ctx, GP_ERR_STATE, "gp_lsqproj: call gp_snp_weights first");
  if (numeigs < 1 || numeigs > ctx->nweights || numeigs > 64)
    return gp_fail(ctx, GP_ERR_ARG, "gp_lsqproj: numeigs %d out of range", numeigs);
  if (nproj == 0) return GP_OK;
  for (int32_t q = 0; q < nproj; ++q)
    if (samples[q] < 0 || samples[q] >= ctx->nind_all)
      return gp_fail(ctx, GP_ERR_ARG, "gp_lsqproj: sample %d out of range", samples[q]);
  GP_CUDA(ctx, cudaSetDevice(ctx->device));
  const int32_t K = numeigs, nk = ctx->nkept, nc = ctx->ncols;
  const int32_t npair = K * (K + 1) / 2, ldp = npair + 1;
  size_t off_tab = kept_tables_bytes(nk);
  size_t nE = (size_t)nk * K, nP = (size_t)nk * ldp;
  size_t nco = (size_t)nproj * ldp, nrr = (size_t)nproj * K;
  const bool pf = sample_pop != NULL && npop > 0;
  if (pf && ctx->precision != GP_PREC_FP64)
    return gp_fail(ctx, GP_ERR_ARG, "gp_lsqproj_pops: usepopsformissing runs in FP64 precision only");
  if (pf)
    for (int32_t q = 0; q < nproj; ++q)
      if (sample_pop[q] >= npop)
        return gp_fail(ctx, GP_ERR_ARG, "gp_lsqproj_pops: population %d >= npop %d",
                       sample_pop[q], npop);
  const size_t off_fill = pf ? gp_lsq_fill_work_bytes(nproj, nk, npop) : 0;
  size_t bytes = off_tab + sizeof(double) * (nE + nP + nco + 3 * nrr) +
                 sizeof(int32_t) * (4 * (size_t)nproj) + off_fill + 1024;
  uint8_t *base;
  int rc = gp_scratch(ctx, bytes, (void **)&base);
  if (rc) return rc;
  kept_tables kt;
  rc = build_kept_tables(ctx, base, &kt);
  if (rc) return rc;
  double *d_E = (double *)(base + off_tab);
  double *d_P = d_E + nE, *d_co = d_P + nP, *d_rr = d_co + nco;
  double *d_a = d_rr + nrr, *d_b = d_a + nrr;
  int32_t *d_samp = (int32_t *)(d_b + nrr), *d_nobs = d_samp + nproj, *d_st = d_nobs + nproj;
  int32_t *d_spop = d_st + nproj;
  void *fill_work = (void *)((((uintptr_t)(d_spop + nproj)) + 255) & ~(uintptr_t)255);
  GP_CUDA(ctx, gp_memcpy(ctx, d_samp, samples, sizeof(int32_t) * (size_t)nproj,
                               cudaMemcpyHostToDevice, ctx->stream));
  double *d_raw = NULL, *d_of = NULL, *d_rf = NULL;
  if (pf && nk > 0) {
    GP_CUDA(ctx, gp_memcpy(ctx, d_spop, sample_pop, sizeof(int32_t) * (size_t)nproj,
                           cudaMemcpyHostToDevice, ctx->stream));
    rc = gp_lsq_fill_tables(ctx, d_samp, d_spop, nproj, npop, K, kt.snprec, kt.ot, nk,
                            fill_work, &d_raw, &d_of, &d_rf);
    if (rc) return rc;
  }
  if (nk) {
    int blocks = (nk + EP_THREADS / 32 - 1) / (EP_THREADS / 32);
    if (blocks > ctx->num_sms * 16) blocks = ctx->num_sms * 16;
    k_build_EP<<<blocks, EP_THREADS, 0, ctx->stream>>>(ctx->d_ffvecs, ctx->d_fxscal, ctx->d_kept,
                                                       nk, nc, K, d_E, d_P, ldp);
    GP_LAUNCH_CHECK(ctx, "k_build_EP");
  }
  /* masked normal equations: co = O P (pair sums + observed count), rr = R E */
  int tc = d_raw ? 0 : tc_products(ctx, nk);
  const int tc_ran = tc;
  if (tc) {
    rc = gp_tc_begin(ctx);
    if (rc) return rc;
    gp_tc_codes A;
    /* projecting exactly the analysis rows: the product can reuse their codes */
    const int32_t *d_list = d_samp;
    if (nproj == ctx->nrows && ctx->h_rows &&
        memcmp(samples, ctx->h_rows, sizeof(int32_t) * (size_t)nproj) == 0)
      d_list = ctx->d_rows;
    int ascending = 1;
    for (int32_t q = 1; q < nproj; ++q) ascending &= samples[q] > samples[q - 1];
    rc = gp_tc_codes_for(ctx, 1, d_list, nproj, kt.snprec, nk, ascending, &A);
    gp_tc_panel pc = {d_P, ldp, 1.0, 0};
    if (!rc) rc = gp_geno_panel_tc_codes(ctx, &A, 1, &pc, ldp, tc_digits(ctx), d_co, ldp);
    if (!rc) rc = scores_tc(ctx, &A, d_E, K, d_rr);
    if (rc == GP_ERR_NOMEM && ctx->precision == GP_PREC_FP64) {
      cudaGetLastError();
      tc = 0;
    } else if (rc) {
      return rc;
    }
  }
  if (d_raw) {
    /* usepopsformissing: a filled genotype counts as observed with its fixxrow value */
    rc = gp_geno_gemm_f64_fill(ctx, d_samp, d_spop, nproj, kt.snprec, kt.ot, d_of, npop, nk,
                               d_P, ldp, ldp, d_co, ldp);
    if (rc) return rc;
    rc = gp_geno_gemm_f64_fill(ctx, d_samp, d_spop, nproj, kt.snprec, kt.rt, d_rf, npop, nk,
                               d_E, K, K, d_rr, K);
    if (rc) return rc;
  } else if (!tc) {
    rc = gp_geno_gemm_f64(ctx, 1, d_samp, nproj, kt.snprec, kt.ot, nk, d_P, ldp, ldp, d_co, ldp);
    if (rc) return rc;
    rc = gp_geno_gemm_f64(ctx, 1, d_samp, nproj, kt.snprec, kt.rt, nk, d_E, K, K, d_rr, K);
    if (rc) return rc;
  }
  GP_CUDA(ctx, cudaMemsetAsync(d_a, 0, sizeof(double) * nrr, ctx->stream));
  rc = gp_launch_lsq_solve(ctx, d_co, ldp, d_rr, K, nproj, d_a, d_b, d_nobs, d_st, NULL);
  if (rc) return rc;
  if (tc_ran) {
    rc = gp_tc_check(ctx);
    if (rc) return rc;
  }
  std::vector<int32_t> st((size_t)nproj);
  std::vector<double> ha(nrr);
  GP_CUDA(ctx, gp_memcpy(ctx, ha.data(), d_a, sizeof(double) * nrr, cudaMemcpyDeviceToHost,
                               ctx->stream));
  GP_CUDA(ctx, gp_memcpy(ctx, st.data(), d_st, sizeof(int32_t) * (size_t)nproj,
                               cudaMemcpyDeviceToHost, ctx->stream));
  if (bcoeffs)
    GP_CUDA(ctx, gp_memcpy(ctx, bcoeffs, d_b, sizeof(double) * nrr, cudaMemcpyDeviceToHost,
                                 ctx->stream));
  std::vector<int32_t> hn((size_t)nproj);
  GP_CUDA(ctx, gp_memcpy(ctx, hn.data(), d_nobs, sizeof(int32_t) * (size_t)nproj,
                         cudaMemcpyDeviceToHost, ctx->stream));
  std::vector<double> raw;
  if (d_raw) {
    raw.resize((size_t)nproj);
    GP_CUDA(ctx, gp_memcpy(ctx, raw.data(), d_raw, sizeof(double) * (size_t)nproj,
                           cudaMemcpyDeviceToHost, ctx->stream));
  }
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  for (int32_t q = 0; q < nproj; ++q) {
    if (d_raw && raw[(size_t)q] <= (double)K) {
      /* the coverage check runs on the observed genotypes, before any fill */
      st[(size_t)q] = 1;
      hn[(size_t)q] = (int32_t)raw[(size_t)q];
      if (bcoeffs)
        for (int32_t j = 0; j < K; ++j) bcoeffs[(size_t)j * nproj + q] = 0.0;
    }
    if (nobs) nobs[q] = hn[(size_t)q];
    if (status) status[q] = st[(size_t)q];
    if (st[(size_t)q] == 2) continue; /* left untouched, as the reference keeps regans */
    for (int32_t j = 0; j < K; ++j)
      acoeffs[(size_t)j * nproj + q] = st[(size_t)q] == 1 ? 0.0 : ha[(size_t)j * nproj + q];
  }
  return GP_OK;
}

extern "C" int gp_lsqproj(gp_ctx *ctx, int32_t numeigs, const int32_t *samples, int32_t nproj,
                          double *acoeffs, double *bcoeffs, int32_t *nobs, int32_t *status)
{
  return lsqproj_impl(ctx, numeigs, samples, NULL, 0, nproj, acoeffs, bcoeffs, nobs, status);
}

extern "C" int gp_lsqproj_pops(gp_ctx *ctx, int32_t numeigs, const int32_t *samples,
                               const int32_t *sample_pop, int32_t npop, int32_t nproj,
                               double *acoeffs, double *bcoeffs, int32_t *nobs, int32_t *status)
{
  if (!sample_pop || npop <= 0)
    return gp_fail(ctx, GP_ERR_ARG, "gp_lsqproj_pops: sample populations are required");
  return lsqproj_impl(ctx, numeigs, samples, sample_pop, npop, nproj, acoeffs, bcoeffs, nobs,
                      status);
}

/* ------------------------------------------------------------------------------------ */

extern "C" int gp_timer_start(gp_ctx *ctx)
{
  if (!ctx) return GP_ERR_ARG;
  GP_CUDA(ctx, cudaEventRecord(ctx->ev_t0, ctx->stream));
  return GP_OK;
}

extern "C" int gp_timer_stop(gp_ctx *ctx, double *ms)
{
  if (!ctx || !ms) return GP_ERR_ARG;
  GP_CUDA(ctx, cudaEventRecord(ctx->ev_t1, ctx->stream));
  GP_CUDA(ctx, cudaEventSynchronize(ctx->ev_t1));
  float f = 0.f;
  GP_CUDA(ctx, cudaEventElapsedTime(&f, ctx->ev_t0, ctx->ev_t1));
  *ms = f;
  return GP_OK;
}

extern "C" int gp_last_tridiag_time(const gp_ctx *ctx, double *ms, int32_t *n)
{
  if (!ctx) return GP_ERR_ARG;
  if (ms) *ms = ctx->tridiag_ms;
  if (n) *n = ctx->tridiag_n;
  return GP_OK;
}

extern "C" int gp_last_counts_time(const gp_ctx *ctx, double *ms, int64_t *bytes)
{
  if (!ctx) return GP_ERR_ARG;
  float f = 0.f;
  if (ctx->counts_bytes > 0) {
    if (cudaEventSynchronize(ctx->ev_c1) != cudaSuccess ||
        cudaEventElapsedTime(&f, ctx->ev_c0, ctx->ev_c1) != cudaSuccess)
      return GP_ERR_CUDA;
  }
  if (ms) *ms = f;
  if (bytes) *bytes = ctx->counts_bytes;
  return GP_OK;
}

extern "C" int gp_last_gram_time(const gp_ctx *ctx, double *ms, int32_t *launches, double *flops)
{
  if (!ctx) return GP_ERR_ARG;
  if (ms) *ms = ctx->gram_ms;
  if (launches) *launches = ctx->gram_launches;
  if (flops) *flops = ctx->gram_flops;
  return GP_OK;
}

extern "C" int gp_host_register(void *ptr, size_t bytes)
{
  if (!ptr || !bytes) return GP_ERR_ARG;
  cudaError_t e = cudaHostRegister(ptr, bytes, cudaHostRegisterDefault);
  if (e != cudaSuccess) return gp_fail(NULL, GP_ERR_CUDA, "cudaHostRegister: %s", cudaGetErrorString(e));
  return GP_OK;
}

extern "C" int gp_host_unregister(void *ptr)
{
  if (!ptr) return GP_ERR_ARG;
  cudaError_t e = cudaHostUnregister(ptr);
  if (e != cudaSuccess) return gp_fail(NULL, GP_ERR_CUDA, "cudaHostUnregister: %s", cudaGetErrorString(e));
  return GP_OK;
}

extern "C" int gp_transfer_bytes(gp_ctx *ctx, int64_t *h2d, int64_t *d2h, int32_t reset)
{
  if (!ctx) return GP_ERR_ARG;
  if (h2d) *h2d = ctx->h2d_bytes;
  if (d2h) *d2h = ctx->d2h_bytes;
  if (reset) ctx->h2d_bytes = ctx->d2h_bytes = 0;
  return GP_OK;
}

extern "C" int gp_launch_count(gp_ctx *ctx, int64_t *n, int32_t reset)
{
  if (!ctx) return GP_ERR_ARG;
  if (n) *n = ctx->launches;
  if (reset) ctx->launches = 0;
  return GP_OK;
}
