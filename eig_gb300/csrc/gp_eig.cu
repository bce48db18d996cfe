/*
 * Dense symmetric FP64 eigensolve for the smartpca Gram, on the device: all N eigenvalues
 * and the top nvec eigenvectors (the reference computes every eigenpair with LAPACK dspev,
 * src/eigensrc/eigx.c:97-117, but prints all eigenvalues and uses only the top vectors).
 *
 *   1. Householder tridiagonalisation A = Q T Q^T (k_tridiag_tiled, or k_tridiag above orders of
 *      about 7,600, while the trailing matrix is large, then k_tridiag_smem: LAPACK dsytd2's reflectors and storage;
 *      cuSOLVER sytrd beyond 8,533 rows);
 *   2. all eigenvalues of T by multisection on Sturm counts (the published bisection method:
 *      the count of negative pivots of the LDL^T factorisation of T - x I equals the number
 *      of eigenvalues below x), several lanes per eigenvalue index: FP32 brackets first,
 *      then float-float, checked and finished in FP64 to 3e-14 ||T|| (1e-13 above 6,080);
 *   3. the top nvec eigenvectors of T by inverse iteration, one block per vector: LU with
 *      partial pivoting of the tridiagonal T - lambda I (Gaussian elimination with row
 *      interchanges) and three solves from a fixed pseudo-random start, then modified
 *      Gram-Schmidt over the vectors in order (eigenvalues that are distinct to far more than
 *      eps*||T|| make each iterate converge to its own eigenvector);
 *   4. back-transformation of those nvec vectors only, V = Q Z (k_apply_q: compact WY blocks
 *      of 32 reflectors in float-float; cuSOLVER ormtr when its row slab does not fit).
 */
#include <cuda_runtime.h>
#include <cusolverDn.h>
#include <float.h>
#include <algorithm>
#include <math.h>
#include <stdio.h>
#include <stdlib.h>

#include "gp_internal.h"
#include "gp_tc.cuh"


/*
 * Float-float arithmetic: a value is an unevaluated sum h + l of two FP32 numbers (about 46
 * significant bits), built from the error-free transformations TwoSum (Knuth) and TwoProd
 * with FMA (Dekker / Ogita-Rump-Oishi 2005).  GB300's FP64 pipe issues about 2 FMAs per clock
 * per SM and its FP32 pipe 128, so the tridiagonalisation keeps its trailing matrix and
 * vectors in this form; every operation below is explicitly rounded (no contraction).
 */
struct ff2 {
  float h, l;
};

__device__ __forceinline__ ff2 ff_make(float h, float l)
{
  ff2 r;
  r.h = h;
  r.l = l;
  return r;
}
__device__ __forceinline__ ff2 ff_from_double(double x)
{
  const float h = __double2float_rn(x);
  return ff_make(h, __double2float_rn(x - (double)h));
}
__device__ __forceinline__ double ff_to_double(ff2 a) { return (double)a.h + (double)a.l; }
__device__ __forceinline__ ff2 ff_neg(ff2 a) { return ff_make(-a.h, -a.l); }
/* a + b */
__device__ __forceinline__ ff2 ff_add(ff2 a, ff2 b)
{
  const float s = __fadd_rn(a.h, b.h);
  const float bb = __fsub_rn(s, a.h);
  float err = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, bb)), __fsub_rn(b.h, bb));
  err = __fadd_rn(err, __fadd_rn(a.l, b.l));
  const float h = __fadd_rn(s, err);
  return ff_make(h, __fsub_rn(err, __fsub_rn(h, s)));
}
/* a * b */
__device__ __forceinline__ ff2 ff_mul(ff2 a, ff2 b)
{
  const float p = __fmul_rn(a.h, b.h);
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, e);
  e = __fmaf_rn(a.l, b.h, e);
  const float h = __fadd_rn(p, e);
  return ff_make(h, __fsub_rn(e, __fsub_rn(h, p)));
}
/* a * b + c */
__device__ __forceinline__ ff2 ff_fma(ff2 a, ff2 b, ff2 c)
{
  const float p = __fmul_rn(a.h, b.h);
  float pe = __fmaf_rn(a.h, b.h, -p);
  pe = __fmaf_rn(a.h, b.l, pe);
  pe = __fmaf_rn(a.l, b.h, pe);
  const float s = __fadd_rn(c.h, p);
  const float bb = __fsub_rn(s, c.h);
  float err = __fadd_rn(__fsub_rn(c.h, __fsub_rn(s, bb)), __fsub_rn(p, bb));
  err = __fadd_rn(err, __fadd_rn(c.l, pe));
  const float h = __fadd_rn(s, err);
  return ff_make(h, __fsub_rn(err, __fsub_rn(h, s)));
}
__device__ __forceinline__ ff2 ff_shfl_xor(ff2 a, int o)
{
  return ff_make(__shfl_xor_sync(0xFFFFFFFFu, a.h, o), __shfl_xor_sync(0xFFFFFFFFu, a.l, o));
}
__device__ __forceinline__ ff2 ff_load(const double *p)
{
  const float2 v = *reinterpret_cast<const float2 *>(p);
  return ff_make(v.x, v.y);
}
__device__ __forceinline__ void ff_store(double *p, ff2 a)
{
  *reinterpret_cast<float2 *>(p) = make_float2(a.h, a.l);
}

/* sqrt(a) for a > 0: FP32 root plus one correction, (a - s^2) / 2s */
__device__ __forceinline__ ff2 ff_sqrt(ff2 a)
{
  const float s = sqrtf(a.h);
  const ff2 r = ff_fma(ff_make(-s, 0.f), ff_make(s, 0.f), a);
  return ff_add(ff_make(s, 0.f), ff_make(__fdiv_rn(r.h, 2.f * s), 0.f));
}
/* a / b: FP32 quotient plus one correction from the float-float remainder */
__device__ __forceinline__ ff2 ff_div(ff2 a, ff2 b)
{
  const float q1 = __fdiv_rn(a.h, b.h);
  const ff2 r = ff_fma(ff_neg(b), ff_make(q1, 0.f), a);
  return ff_add(ff_make(q1, 0.f), ff_make(__fdiv_rn(r.h, b.h), 0.f));
}
__device__ __forceinline__ ff2 ff_scale(ff2 a, float s) { return ff_make(a.h * s, a.l * s); }

/* the same count in FP32 (coarse brackets only; verified in FP64 afterwards) */
__device__ __forceinline__ int sturm_count_f(const float *d, const float *e2, int n, float x,
                                             float pivmin)
{
  int cnt = 0;
  float q = d[0] - x;
  if (fabsf(q) < pivmin) q = -pivmin;
  if (q < 0.f) ++cnt;
  for (int i = 1; i < n; ++i) {
    q = (d[i] - x) - __fdividef(e2[i - 1], q);
    if (fabsf(q) < pivmin) q = -pivmin;
    if (q < 0.f) ++cnt;
  }
  return cnt;
}

/*
 * 1/q to ~2^-44 relative with four integer-built pieces and two FP64 FMAs: the mantissa of q
 * (truncated to 23 bits) is inverted by the FP32 approximate reciprocal, the exponent is
 * negated in integer arithmetic, and one Newton step r = r0 + r0 (1 - q r0) refines it.
 * Valid for normal q with |exponent| < 1000 (the Sturm pivots are clamped away from 0).
 * GB300's FP64 pipe is narrow, so this keeps conversions and divisions off it.
 */
__device__ __forceinline__ double rcp_newton(double q)
{
  const unsigned long long qb = (unsigned long long)__double_as_longlong(q);
  const unsigned hi = (unsigned)(qb >> 32);
  const int e = (int)((hi >> 20) & 0x7FFu) - 1023;
  const float f = __uint_as_float(0x3F800000u | (unsigned)((qb >> 29) & 0x7FFFFFull));
  float rf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(f));
  const unsigned rb = __float_as_uint(rf);
  const unsigned er = (unsigned)((int)(rb >> 23) - 127 - e + 1023);
  const unsigned long long r0b =
      ((unsigned long long)((hi & 0x80000000u) | (er << 20) | ((rb & 0x7FFFFFu) >> 3)) << 32) |
      ((unsigned long long)(rb & 7u) << 29);
  const double r0 = __longlong_as_double((long long)r0b);
  return fma(r0, fma(-q, r0, 1.0), r0);
}

/*
 * Sturm count with 4 FP64-pipe operations per step (d - x and three FMAs); the pivot clamp
 * and the sign test work on the bit patterns.
 */
__device__ __forceinline__ int sturm_count_bits(const double *d, const double *e2, int n, double x,
                                                double pivmin)
{
  const unsigned long long piv_bits = (unsigned long long)__double_as_longlong(pivmin);
  const double negpiv = -pivmin;
  int cnt = 0;
  double q = d[0] - x;
  unsigned long long qb = (unsigned long long)__double_as_longlong(q);
  if ((qb & 0x7FFFFFFFFFFFFFFFull) < piv_bits) {
    q = negpiv;
    qb = (unsigned long long)__double_as_longlong(negpiv);
  }
  cnt += (int)(qb >> 63);
  for (int i = 1; i < n; ++i) {
    const double r = rcp_newton(q);
    q = fma(-e2[i - 1], r, d[i] - x);
    qb = (unsigned long long)__double_as_longlong(q);
    if ((qb & 0x7FFFFFFFFFFFFFFFull) < piv_bits) {
      q = negpiv;
      qb = (unsigned long long)__double_as_longlong(negpiv);
    }
    cnt += (int)(qb >> 63);
  }
  return cnt;
}

/* a / b in float-float from the FP32 approximate reciprocal and one remainder correction
 * (relative error ~2^-44; the Sturm brackets below allow for it) */
__device__ __forceinline__ ff2 ff_div_approx(ff2 a, ff2 b)
{
  float rb;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rb) : "f"(b.h));
  const float q1 = __fmul_rn(a.h, rb);
  const ff2 r = ff_fma(ff_neg(b), ff_make(q1, 0.f), a);
  const float q2 = __fmul_rn(r.h, rb);
  const float h = __fadd_rn(q1, q2);
  return ff_make(h, __fsub_rn(q2, __fsub_rn(h, q1)));
}

/* the Sturm count in float-float (d and e2 as hi/lo FP32 pairs; verified in FP64 afterwards) */
__device__ __forceinline__ int sturm_count_ff(const float *dh, const float *dl, const float *eh,
                                              const float *el, int n, ff2 x, float pivmin)
{
  const ff2 nx = ff_neg(x), clamp = ff_make(-pivmin, 0.f);
  ff2 q = ff_add(ff_make(dh[0], dl[0]), nx);
  if (fabsf(q.h) < pivmin) q = clamp;
  int cnt = q.h < 0.f;
  for (int i = 1; i < n; ++i) {
    const ff2 t = ff_add(ff_make(dh[i], dl[i]), nx);
    q = ff_add(t, ff_neg(ff_div_approx(ff_make(eh[i - 1], el[i - 1]), q)));
    if (fabsf(q.h) < pivmin) q = clamp;
    cnt += q.h < 0.f;
  }
  return cnt;
}

/*
 * All eigenvalues by multisection: a warp owns epw consecutive eigenvalue indices and each
 * index gets P = 32/epw lanes (P >= 1), so every warp slot of the GPU has work whatever N is.
 * A step evaluates P interior points of the bracket at once (one Sturm count per lane) and
 * keeps the sub-interval where the count crosses k: log2(P+1) bits per step.  FP32 counts
 * narrow the bracket to ~4e-7 ||T|| (widened by 64 eps_32 ||T||), float-float counts on the
 * FP32 pipe narrow it to ~1e-12 ||T|| (widened by 16 2^-44 ||T||).  The first FP64 count takes
 * the bracket's ends among its points, which checks it (back to the Gershgorin bracket if that
 * fails), and FP64 counts narrow it to tol: n = 5,000 9.2 ms, of 10.1, and 1,000 0.95, of
 * 1.13, with a check of its own and a bracket four times as wide.  (Three points per lane in
 * the FP32 and float-float phases took longer, 12.0 and 1.5 ms: they are bound by issue.)
 * Grid: one CTA of 4 warps per SM; d, e2 and their FP32 hi/lo copies in shared memory
 * (32 N bytes) when they fit (use_smem 2), d, e2 and FP32 copies without the float-float
 * phase (24 N bytes, use_smem 1), else FP64 counts from global memory only.
 */
__global__ void __launch_bounds__(128)
k_multisect(const double *gd, const double *ge2, int n, double gl, double gu, double tnorm,
            double pivmin, double tol, int use_smem, int epw, int P, double *w)
{
  extern __shared__ double sm[];
  const double *d = gd, *e2 = ge2;
  const float *df = NULL, *e2f = NULL, *dl = NULL, *e2l = NULL;
  if (use_smem) {
    double *sd = sm, *se2 = sm + n;
    float *sdf = (float *)(sm + 2 * n), *se2f = sdf + n;
    float *sdl = se2f + n, *se2l = sdl + n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      sd[i] = gd[i];
      sdf[i] = (float)gd[i];
      if (use_smem > 1) sdl[i] = (float)(gd[i] - (double)sdf[i]);
      if (i < n - 1) {
        se2[i] = ge2[i];
        se2f[i] = (float)ge2[i];
        if (use_smem > 1) se2l[i] = (float)(ge2[i] - (double)se2f[i]);
      }
    }
    __syncthreads();
    d = sd;
    e2 = se2;
    df = sdf;
    e2f = se2f;
    if (use_smem > 1) {
      dl = sdl;
      e2l = se2l;
    }
  }
  const int lane = threadIdx.x & 31;
  const int gwarp = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int slot = lane / P, sub = lane - slot * P;
  if (slot >= epw) return;
  const int k = gwarp * epw + slot;
  if (k >= n) return;
  const unsigned gmask = ((P == 32) ? 0xFFFFFFFFu : ((1u << P) - 1u)) << (slot * P);
  const int gshift = slot * P;
  const unsigned gbits = (P == 32) ? 0xFFFFFFFFu : ((1u << P) - 1u);
  double lo = gl, hi = gu;
  if (df) {
    float flo = (float)gl, fhi = (float)gu;
    const float fpiv = fmaxf((float)pivmin, 1e-30f) * 1e6f;
    const float ftol = 4e-7f * (float)tnorm;
    for (int it = 0; it < 64 && fhi - flo > ftol; ++it) {
      const float wdt = fhi - flo;
      const float x = flo + wdt * (float)(sub + 1) / (float)(P + 1);
      const int flag = (x > flo && x < fhi) ? (sturm_count_f(df, e2f, n, x, fpiv) > k) : (x >= fhi);
      const unsigned b = (__ballot_sync(gmask, flag) >> gshift) & gbits;
      const int first = b ? __ffs(b) - 1 : P;
      const float nlo = first == 0 ? flo : flo + wdt * (float)first / (float)(P + 1);
      const float nhi = first == P ? fhi : flo + wdt * (float)(first + 1) / (float)(P + 1);
      if (!(nhi - nlo < wdt)) break;
      flo = nlo;
      fhi = nhi;
    }
    const double margin = 64.0 * (double)FLT_EPSILON * tnorm;
    lo = fmax(gl, (double)flo - margin);
    hi = fmin(gu, (double)fhi + margin);
    if (dl) {
      /* float-float phase: the same multisection with x_j = lo + (hi - lo) j / (P+1) formed
       * identically for a point and for the bracket end it becomes */
      ff2 glo = ff_from_double(lo), ghi = ff_from_double(hi);
      const float fpiv = fmaxf((float)pivmin, 1e-30f);
      const float ftol2 = (float)(1e-12 * tnorm);
      for (int it = 0; it < 64; ++it) {
        const ff2 wdt = ff_add(ghi, ff_neg(glo));
        if (!(wdt.h > ftol2)) break;
        const ff2 x = ff_fma(wdt, ff_make((float)(sub + 1) / (float)(P + 1), 0.f), glo);
        const bool inside = ff_add(x, ff_neg(glo)).h > 0.f && ff_add(ghi, ff_neg(x)).h > 0.f;
        const int flag = inside ? (sturm_count_ff(df, dl, e2f, e2l, n, x, fpiv) > k)
                                : (ff_add(x, ff_neg(ghi)).h >= 0.f);
        const unsigned b = (__ballot_sync(gmask, flag) >> gshift) & gbits;
        const int first = b ? __ffs(b) - 1 : P;
        const ff2 nlo =
            first == 0 ? glo : ff_fma(wdt, ff_make((float)first / (float)(P + 1), 0.f), glo);
        const ff2 nhi =
            first == P ? ghi : ff_fma(wdt, ff_make((float)(first + 1) / (float)(P + 1), 0.f), glo);
        if (!(ff_add(nhi, ff_neg(nlo)).h < wdt.h)) break;
        glo = nlo;
        ghi = nhi;
      }
      const double margin2 = 16.0 * 0x1p-44 * tnorm;
      lo = fmax(gl, ff_to_double(glo) - margin2);
      hi = fmin(gu, ff_to_double(ghi) + margin2);
    }
    if (P == 1) {
      /* one lane: both ends in turn */
      if (sturm_count_bits(d, e2, n, lo, pivmin) > k || sturm_count_bits(d, e2, n, hi, pivmin) <= k) {
        lo = gl;
        hi = gu;
      }
    } else {
      /* P points from end to end: the ends check the bracket, the others narrow it */
      const double wdt = hi - lo, den = (double)(P - 1);
      const double x = sub == P - 1 ? hi : lo + wdt * (double)sub / den;
      const int flag = sturm_count_bits(d, e2, n, x, pivmin) > k;
      const unsigned b = (__ballot_sync(gmask, flag) >> gshift) & gbits;
      if ((b & 1u) || !((b >> (P - 1)) & 1u)) {
        lo = gl;
        hi = gu;
      } else {
        const int first = __ffs(b) - 1;
        const double nhi = first == P - 1 ? hi : lo + wdt * (double)first / den;
        lo = first == 1 ? lo : lo + wdt * (double)(first - 1) / den;
        hi = nhi;
      }
    }
  }
  for (int it = 0; it < 200 && hi - lo > tol; ++it) {
    const double wdt = hi - lo;
    const double x = lo + wdt * (double)(sub + 1) / (double)(P + 1);
    const int flag = (x > lo && x < hi) ? (sturm_count_bits(d, e2, n, x, pivmin) > k) : (x >= hi);
    const unsigned b = (__ballot_sync(gmask, flag) >> gshift) & gbits;
    const int first = b ? __ffs(b) - 1 : P;
    const double nlo = first == 0 ? lo : lo + wdt * (double)first / (double)(P + 1);
    const double nhi = first == P ? hi : lo + wdt * (double)(first + 1) / (double)(P + 1);
    if (!(nhi - nlo < wdt)) break;
    lo = nlo;
    hi = nhi;
  }
  if (sub == 0) w[k] = 0.5 * (lo + hi);
}

/* ---------------------------------------------------------------------------------- */
/*
 * Householder tridiagonalisation A = Q T Q^T of the symmetric n x n matrix (held in full,
 * column-major: element (r, q) at A[q*n + r]), the unblocked algorithm of LAPACK dsytd2
 * (lower) restated for one cooperative launch:
 *   for c = 0 .. n-2:  x = A(c+1:n, c);  (beta, tau, v) = reflector of x (dlarfg: v(c+1) = 1,
 *   beta = -sign(alpha) ||x||, tau = (beta - alpha)/beta, v = x/(alpha - beta) below);
 *   y = A(c+1:n, c+1:n) v;  w = tau y - (tau^2/2)(y.v) v;  A(c+1:n, c+1:n) -= v w^T + w v^T.
 * The rank-2 update of step c is not a pass of its own: it is applied while step c+1 reads the
 * trailing matrix for its product (look-ahead).  Both triangles of the trailing matrix are
 * kept up to date, so the product is a dot of each whole column with v: every block owns an
 * even share of the columns (equal lengths), reads and writes them once, and no block needs
 * another block's columns within the step.  Per step:
 *   A   every block rebuilds, from y and x of step c-1 and column c, the vectors v and w of
 *       step c-1, the pending update of column c, its norm and the reflector (O(n) work done
 *       redundantly instead of a grid-wide reduction); each block writes its share of the
 *       reflector storage of step c-1 (LAPACK's, e(c-1) on the subdiagonal) and of x_c
 *   B   each block, per owned column r: pending update of A(c+1:n, r), written back, and
 *       y(r) = A(c+1:n, r) . v, warp per column (segments when the block has fewer columns
 *       than warps); then its share of y . v
 *   --- grid barrier
 * x and y are double-buffered across steps, so phase A of one step never reads a vector
 * that a faster block is already writing in the next.
 * Every sum has a fixed order (no atomics), so the result is deterministic.  The grid
 * barrier is a monotonic counter with a %globaltimer bound: on expiry the kernel records an
 * error code and returns (the host reports GP_ERR_TIMEOUT).
 * Outputs: d[n], e[n-1], tau[n-1] and the reflectors in the lower triangle of A, as
 * dormtr (lower) reads them.  Shared memory: v(step c-1), w(step c-1), v(step c) over the
 * rows (24 n bytes).
 */
#define TR_THREADS 1024
#define TR_WARPS (TR_THREADS / 32)
#define TR_U 8 /* loads in flight per lane in the product loops */
#define TR_B1_SLOTS 256 /* segment dots of one block in the column pass */
#define TR_ERR_BARRIER 11

/* arrival with release semantics at GPU scope (the block's writes, ordered before it by the
 * block barrier, become visible to a block that acquires the count) */
__device__ __forceinline__ void red_release_gpu(unsigned *p, unsigned v)
{
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned ld_acquire_gpu(const unsigned *p)
{
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

/* grid barrier on a monotonic arrival counter: the k-th barrier of the launch waits until
 * k * gridDim.x blocks have arrived (one release-add per block, acquire loads while
 * waiting, no reset) */
__device__ __forceinline__ bool tr_grid_sync(unsigned *count, unsigned target, int *err)
{
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    volatile int *verr = err;
    red_release_gpu(count, 1u);
    const uint64_t t0 = globaltimer_ns();
    for (unsigned it = 1; ld_acquire_gpu(count) < target; ++it) {
      if ((it & 63u) == 0) {
        if (*verr) {
          ok = 0;
          break;
        }
        if (globaltimer_ns() - t0 > GP_WAIT_NS) {
          atomicExch(err, TR_ERR_BARRIER);
          ok = 0;
          break;
        }
      }
    }
    if (*verr) ok = 0;
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

/* block sum of one float-float per thread (fixed order: warp shuffles, then warp 0's
 * shuffle tree over the warps' sums), as float-float in thread 0 */
__device__ __forceinline__ ff2 ff_block_sum2(ff2 v, ff2 *red)
{
  static_assert(TR_WARPS == 32, "one warp sums the warps' partials");
  for (int o = 16; o; o >>= 1) v = ff_add(v, ff_shfl_xor(v, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  ff2 t = ff_make(0.f, 0.f);
  if (threadIdx.x < 32) {
    t = red[threadIdx.x];
    for (int o = 16; o; o >>= 1) t = ff_add(t, ff_shfl_xor(t, o));
  }
  __syncthreads();
  return t;
}

/* a - (p q + r s) in float-float (the rank-2 update of one element): the two high products
 * exactly (TwoProd with FMA), their cross terms and the errors of two TwoSums gathered in one
 * FP32 term, one renormalisation: 27 FP32 operations against 30 for two ff_fma, of the same
 * error order.  With p = r = 0 or q = s = 0 it returns a normalised a unchanged. */
__device__ __forceinline__ ff2 ff_sub2prod(ff2 a, ff2 p, ff2 q, ff2 r, ff2 s)
{
  const float p1 = __fmul_rn(p.h, q.h);
  float e = __fmaf_rn(p.h, q.h, -p1);
  e = __fmaf_rn(p.h, q.l, e);
  e = __fmaf_rn(p.l, q.h, e);
  const float p2 = __fmul_rn(r.h, s.h);
  e = __fadd_rn(__fmaf_rn(r.h, s.h, -p2), e);
  e = __fmaf_rn(r.h, s.l, e);
  e = __fmaf_rn(r.l, s.h, e);
  const float t1 = __fsub_rn(a.h, p1);
  const float b1 = __fsub_rn(t1, a.h);
  const float r1 = __fadd_rn(__fsub_rn(a.h, __fsub_rn(t1, b1)), __fsub_rn(-p1, b1));
  const float t2 = __fsub_rn(t1, p2);
  const float b2 = __fsub_rn(t2, t1);
  const float r2 = __fadd_rn(__fsub_rn(t1, __fsub_rn(t2, b2)), __fsub_rn(-p2, b2));
  const float low = __fadd_rn(__fsub_rn(a.l, e), __fadd_rn(r1, r2));
  const float h = __fadd_rn(t2, low);
  return ff_make(h, __fsub_rn(low, __fsub_rn(h, t2)));
}

/* a x + b y in float-float: two exact high products, one TwoSum, the cross terms and errors
 * in one FP32 term (19 FP32 operations against 22 for ff_mul + ff_fma) */
__device__ __forceinline__ ff2 ff_dot2(ff2 a, ff2 x, ff2 b, ff2 y)
{
  const float p1 = __fmul_rn(a.h, x.h);
  float e = __fmaf_rn(a.h, x.h, -p1);
  e = __fmaf_rn(a.h, x.l, e);
  e = __fmaf_rn(a.l, x.h, e);
  const float p2 = __fmul_rn(b.h, y.h);
  e = __fadd_rn(__fmaf_rn(b.h, y.h, -p2), e);
  e = __fmaf_rn(b.h, y.l, e);
  e = __fmaf_rn(b.l, y.h, e);
  const float s = __fadd_rn(p1, p2);
  const float bb = __fsub_rn(s, p1);
  const float er = __fadd_rn(__fsub_rn(p1, __fsub_rn(s, bb)), __fsub_rn(p2, bb));
  const float low = __fadd_rn(e, er);
  const float h = __fadd_rn(s, low);
  return ff_make(h, __fsub_rn(low, __fsub_rn(h, s)));
}

/* acc += a x with the accumulator left unnormalised (acc.h the running TwoSum of the high
 * products, acc.l every lower-order term): 12 FP32 operations against 15 for ff_fma.  The dots here
 * take some 40 terms (a lane's share of a tile row at order 5,000; at most 27 of a column in shared
 * memory); normalising the tiled ones every 4, 8 or 16 terms changed neither the eigenvalues' error
 * nor the vectors' residuals in the third digit (orders 2,500 to 5,000) and took 0.5 ms of 93.
 * ff_renorm makes the pair normalised again. */
__device__ __forceinline__ ff2 ff_acc_lazy(ff2 acc, ff2 a, ff2 x)
{
  const float p = __fmul_rn(a.h, x.h);
  float e = __fmaf_rn(a.h, x.h, -p);
  e = __fmaf_rn(a.h, x.l, e);
  e = __fmaf_rn(a.l, x.h, e);
  const float s = __fadd_rn(acc.h, p);
  const float bb = __fsub_rn(s, acc.h);
  const float er = __fadd_rn(__fsub_rn(acc.h, __fsub_rn(s, bb)), __fsub_rn(p, bb));
  return ff_make(s, __fadd_rn(acc.l, __fadd_rn(e, er)));
}
__device__ __forceinline__ ff2 ff_renorm(ff2 a)
{
  const float h = __fadd_rn(a.h, a.l);
  return ff_make(h, __fsub_rn(a.l, __fsub_rn(h, a.h)));
}

/* sum over the warp, the same in every lane: the high parts by TwoSum, the lower-order terms
 * kept aside and added once at the end, so that a level costs a shuffle and one addition of
 * latency */
__device__ __forceinline__ ff2 ff_warp_sum(ff2 v)
{
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const float oh = __shfl_xor_sync(0xFFFFFFFFu, v.h, o), ol = __shfl_xor_sync(0xFFFFFFFFu, v.l, o);
    const float s = __fadd_rn(v.h, oh);
    const float bb = __fsub_rn(s, v.h);
    const float er = __fadd_rn(__fsub_rn(v.h, __fsub_rn(s, bb)), __fsub_rn(oh, bb));
    v = ff_make(s, __fadd_rn(__fadd_rn(v.l, ol), er));
  }
  return ff_renorm(v);
}

/* the (symmetric, full) double matrix to float-float pairs, in place */
__global__ void k_tri_to_ff(double *A, int n)
{
  const int64_t total = (int64_t)n * n;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x)
    ff_store(A + idx, ff_from_double(A[idx]));
}

/* per-step scalars, computed once per block by thread 0 (GB300's FP64 pipe is narrow, so
 * scalar square roots and divisions are not repeated by every thread) */
struct tr_step {
  ff2 beta, tau_c, scale_c;
  int b1_u0, b1_u1;
};

/*
 * A holds the whole matrix as float-float pairs on entry (k_tri_to_ff); vbuf/wbuf hold the
 * updated column x of alternate steps, ybuf [2n] the product y of alternate steps and
 * part_dot2 [2G] the blocks' partial y.v of alternate steps, as float-float pairs in doubles'
 * storage.  On exit the reflectors are FP64 again in A(c+2:n, c) and e on the subdiagonal, as
 * dormtr (lower) reads them; the upper triangle is left in float-float form.
 */
/*
 * Steps 0 .. c_end - 1 (at most n-2) by whole columns.  svp/swp/svc: the block's vectors in shared
 * memory (n pairs each).  tau_pf, scale_pf, e_pf, have_p and target carry the previous step's
 * state.  sph (block 0, thread 0 only; else NULL): phase times as in k_tridiag, sph[5] the last
 * time stamp.  False when the grid barrier failed.
 */
__device__ __forceinline__ bool tr_full_steps(double *A, int n, int c_end, double *d, double *e,
                                              double *tau, double *vbuf, double *wbuf,
                                              double *ybuf, double *part_dot2, unsigned *count,
                                              unsigned &target, int *err, double *svp,
                                              double *swp, double *svc, ff2 &tau_pf,
                                              ff2 &scale_pf, ff2 &e_pf, bool &have_p,
                                              unsigned long long *sph)
{
  __shared__ ff2 red[TR_WARPS];
  __shared__ ff2 sdotp[TR_B1_SLOTS];
  __shared__ tr_step st;
  __shared__ ff2 s_slotf, s_yc;
  const int G = gridDim.x, b = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const ff2 ONE = ff_make(1.f, 0.f), ZERO = ff_make(0.f, 0.f);
  const bool stamp = sph != NULL;
#define TR_STAMP(i)                                    \
  if (stamp) {                                         \
    const unsigned long long t_now = globaltimer_ns(); \
    sph[i] += t_now - sph[5];                          \
    sph[5] = t_now;                                    \
  }
  const int early = (int)((3LL * n) / 10);
  for (int c = 0; c < c_end; ++c) {
    /* ---- A (every block, no grid barrier): v and w of step c-1, the pending update of
     * column c and its norm, rebuilt from y, the stored x of step c-1 and column c; each
     * block also writes its share of the reflector storage and of x_c (double buffer) ---- */
    const int m = n - c - 1;
    double *xcur = (c & 1) ? wbuf : vbuf, *xprev = (c & 1) ? vbuf : wbuf;
    /* y of step c and of step c-1 (double buffer: phase A reads one while B writes the other) */
    double *ycur = ybuf + (int64_t)(c & 1) * n, *yprev = ybuf + (int64_t)((c + 1) & 1) * n;
    if (threadIdx.x == 32) st.b1_u0 = (int)(((int64_t)m * b) / G);
    if (threadIdx.x == 33) st.b1_u1 = (int)(((int64_t)m * (b + 1)) / G);
    /* the block partials of y.v of step c-1 (double buffer: blocks already in step c+1 write
     * the other half), loaded by the last warp ahead of the vector loads so that the two
     * latencies overlap; summed per lane in order, then by a fixed shuffle tree */
    ff2 pacc = ZERO;
    if (have_p && warp == TR_WARPS - 1) {
      const double *pprev = part_dot2 + (size_t)((c + 1) & 1) * G;
#pragma unroll 4
      for (int g = lane; g < G; g += 32) pacc = ff_add(pacc, ff_load(pprev + g));
    }
    /* loads (v_p needs only step c-1's scale; y is kept raw in swp for now) */
#pragma unroll 4
    for (int q = c + threadIdx.x; q < n; q += blockDim.x) {
      ff2 vp = ZERO, yq = ZERO;
      if (have_p) {
        vp = (q == c) ? ONE : ff_mul(ff_load(xprev + q), scale_pf);
        yq = ff_load(yprev + q);
        if (q == c) s_yc = yq; /* swp(c) changes while other warps still need y(c) */
      }
      ff_store(svp + q, vp);
      ff_store(swp + q, yq);
      ff_store(svc + q, ff_load(A + (int64_t)c * n + q));
    }
    if (have_p && warp == TR_WARPS - 1) {
      for (int o = 16; o; o >>= 1) pacc = ff_add(pacc, ff_shfl_xor(pacc, o));
      if (lane == 0) s_slotf = pacc;
    }
    __syncthreads(); /* publishes the partial sum and svp, swp, svc */
    ff2 wpc = ZERO, alpha_pf = ZERO;
    if (have_p) {
      /* every thread forms alpha and w_p(c) of step c-1 from the same values */
      const ff2 dsum = s_slotf;
      alpha_pf = ff_scale(ff_mul(ff_mul(tau_pf, tau_pf), dsum), -0.5f);
      wpc = ff_fma(tau_pf, s_yc, alpha_pf); /* w_p(c); v_p(c) = 1 */
    }
    {
      const int cnt = n - c, per = (cnt + G - 1) / G;
      const int r0 = c + b * per, r1 = min(n, r0 + per);
      ff2 nrm = ZERO;
      for (int q = c + threadIdx.x; q < n; q += blockDim.x) {
        ff2 x = ff_load(svc + q);
        const bool mine = q >= r0 && q < r1;
        if (have_p) {
          const ff2 vp = ff_load(svp + q);
          const ff2 wp = ff_fma(tau_pf, ff_load(swp + q), ff_mul(alpha_pf, vp));
          ff_store(swp + q, wp);
          x = ff_fma(ff_neg(vp), wpc, x);
          x = ff_add(x, ff_neg(wp));
          if (mine) A[(int64_t)(c - 1) * n + q] = ff_to_double(q == c ? e_pf : vp); /* FP64 */
        }
        ff_store(svc + q, x);
        if (mine) ff_store(xcur + q, x);
        if (q >= c + 2) nrm = ff_fma(x, x, nrm);
      }
      const ff2 xn2 = ff_block_sum2(nrm, red); /* thread 0; the sum's barriers publish svc */
      if (threadIdx.x == 0) {
        /* the reflector (dlarfg) in float-float: beta = -sign(alpha) sqrt(alpha^2 + |x|^2),
         * tau = (beta - alpha) / beta, scale = 1 / (alpha - beta) */
        const ff2 alpha = ff_load(svc + c + 1);
        if (xn2.h == 0.f) {
          st.beta = alpha;
          st.tau_c = ZERO;
          st.scale_c = ZERO;
        } else {
          const ff2 nrm2 = ff_sqrt(ff_fma(alpha, alpha, xn2));
          const ff2 beta = alpha.h >= 0.f ? ff_neg(nrm2) : nrm2;
          const ff2 am = ff_add(alpha, ff_neg(beta));
          st.beta = beta;
          st.tau_c = ff_div(ff_neg(am), beta);
          st.scale_c = ff_div(ONE, am);
        }
      }
      __syncthreads();
      if (b == 0 && threadIdx.x == 32) {
        d[c] = ff_to_double(ff_load(svc + c));
        e[c] = ff_to_double(st.beta);
        tau[c] = ff_to_double(st.tau_c);
      }
    }
    const ff2 beta = st.beta, tau_c = st.tau_c;
    const ff2 scale_cf = st.scale_c;
    TR_STAMP(0)
    /* ---- B: pending update + product over whole columns (both triangles are stored),
     * warp per column; the block's columns are an even share of the trailing matrix ---- */
    for (int q = c + 1 + threadIdx.x; q < n; q += blockDim.x)
      ff_store(svc + q, (q == c + 1) ? ONE : ff_mul(ff_load(svc + q), scale_cf));
    __syncthreads();
    {
      const int u0 = st.b1_u0, u1 = st.b1_u1, ncol = u1 - u0;
      /* one piece [qs, qe) of column r: pending update, store and dot with v; the last
       * partial batch is one predicated round of loads, so no piece ends in a chain of
       * dependent single loads */
      auto piece = [&](int r, int qs, int qe) -> ff2 {
        const ff2 vpr = ff_neg(ff_load(svp + r)), wpr = ff_neg(ff_load(swp + r));
        double *col = A + (int64_t)r * n;
        ff2 dot = ZERO;
        for (int qb = qs; qb < qe; qb += 32 * TR_U) {
          ff2 a[TR_U];
#pragma unroll
          for (int u = 0; u < TR_U; ++u) {
            const int qq = qb + lane + 32 * u;
            a[u] = qq < qe ? ff_load(col + qq) : ZERO;
          }
#pragma unroll
          for (int u = 0; u < TR_U; ++u) {
            const int qq = qb + lane + 32 * u;
            if (qq < qe) {
              if (have_p) {
                a[u] = ff_fma(ff_load(svp + qq), wpr, a[u]);
                a[u] = ff_fma(ff_load(swp + qq), vpr, a[u]);
                ff_store(col + qq, a[u]);
              }
              dot = ff_fma(a[u], ff_load(svc + qq), dot);
            }
          }
        }
        for (int o = 16; o; o >>= 1) dot = ff_add(dot, ff_shfl_xor(dot, o));
        return dot;
      };
      /* work items (column, segment): a block with fewer columns than warps splits each into
       * S segments so that every warp works; segment dots are summed in order.  (Equal
       * flattened element ranges per warp measured slower than this split.) */
      const int S = (ncol > 0 && ncol < TR_WARPS) ? (TR_WARPS + ncol - 1) / ncol : 1;
      const int nitem = ncol * S;
      const int seg = ((m + S - 1) / S + 31) & ~31;
      for (int it = warp; it < nitem; it += TR_WARPS) {
        const int j = it / S, sg = it - j * S;
        const int qs = c + 1 + sg * seg, qe = min(n, qs + seg);
        const ff2 dot = piece(c + 1 + u0 + j, qs, qe);
        if (lane == 0) {
          if (S == 1)
            ff_store(ycur + c + 1 + u0 + j, dot);
          else
            sdotp[it] = dot;
        }
      }
      if (S > 1) {
        __syncthreads();
        for (int j = threadIdx.x; j < ncol; j += blockDim.x) {
          ff2 t = sdotp[j * S];
          for (int sg = 1; sg < S; ++sg) t = ff_add(t, sdotp[j * S + sg]);
          ff_store(ycur + c + 1 + u0 + j, t);
        }
      }
      __syncthreads();
      /* the block's share of y . x for the next step's alpha, in column order */
      ff2 dpart = ZERO;
      for (int j = threadIdx.x; j < ncol; j += blockDim.x) {
        const int r = c + 1 + u0 + j;
        dpart = ff_fma(ff_load(ycur + r), ff_load(svc + r), dpart);
      }
      const ff2 ds = ff_block_sum2(dpart, red);
      if (threadIdx.x == 0) ff_store(part_dot2 + (size_t)(c & 1) * G + b, ds);
    }
    TR_STAMP(c < early ? 2 : 1)
    target += G;
    if (!tr_grid_sync(count, target, err)) return false;
    TR_STAMP(4)
    tau_pf = tau_c;
    scale_pf = scale_cf;
    e_pf = beta;
    have_p = true;
  }
#undef TR_STAMP
  return true;
}

/*
 * sqrt(a), a > 0, and a / b from the approximate FP32 reciprocal (square root): two
 * corrections from the float-float remainder (Karp & Markstein 1997) reach the pair's
 * precision; they replace ff_sqrt and ff_div on one thread's critical path, whose rounded FP32
 * divisions are several times longer chains.
 */
__device__ __forceinline__ ff2 ff_sqrt_fast(ff2 a)
{
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a.h));
  const float s = a.h * r, hr = 0.5f * r;
  ff2 x = ff_make(s, 0.f);
  ff2 t = ff_fma(ff_neg(x), x, a);
  x = ff_add(x, ff_make(t.h * hr, 0.f));
  t = ff_fma(ff_neg(x), x, a);
  return ff_add(x, ff_make(t.h * hr, 0.f));
}
__device__ __forceinline__ ff2 ff_div_fast(ff2 a, ff2 b)
{
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b.h));
  ff2 q = ff_make(a.h * r, 0.f);
  ff2 t = ff_fma(ff_neg(b), q, a);
  q = ff_add(q, ff_make(t.h * r, 0.f));
  t = ff_fma(ff_neg(b), q, a);
  return ff_add(q, ff_make(t.h * r, 0.f));
}

/*
 * Pairs of float-float numbers in the packed FP32 instructions (two operations in one issue
 * slot; each is rounded as its scalar form, so every formula below is the scalar one above it,
 * twice).
 */
typedef unsigned long long f2;
struct pf2 {
  f2 h, l;
};
__device__ __forceinline__ f2 f2_make(float a, float b)
{
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_get(f2 a)
{
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b)
{
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b)
{
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c)
{
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
#define F2_MINUS_ONE 0xBF800000BF800000ull
__device__ __forceinline__ f2 f2_sub(f2 a, f2 b) { return f2_fma(b, F2_MINUS_ONE, a); }
__device__ __forceinline__ f2 f2_neg(f2 a) { return a ^ 0x8000000080000000ull; }
__device__ __forceinline__ pf2 pf_make(f2 h, f2 l)
{
  pf2 r;
  r.h = h;
  r.l = l;
  return r;
}
__device__ __forceinline__ pf2 pf_dup(ff2 a)
{
  return pf_make(f2_make(a.h, a.h), f2_make(a.l, a.l));
}
__device__ __forceinline__ ff2 pf_even(pf2 a) { return ff_make(f2_get(a.h).x, f2_get(a.l).x); }
__device__ __forceinline__ ff2 pf_odd(pf2 a) { return ff_make(f2_get(a.h).y, f2_get(a.l).y); }
__device__ __forceinline__ pf2 pf_join(ff2 e, ff2 o)
{
  return pf_make(f2_make(e.h, o.h), f2_make(e.l, o.l));
}
/* ff_add */
__device__ __forceinline__ pf2 pf_add(pf2 a, pf2 b)
{
  const f2 s = f2_add(a.h, b.h);
  const f2 bb = f2_sub(s, a.h);
  f2 err = f2_add(f2_sub(a.h, f2_sub(s, bb)), f2_sub(b.h, bb));
  err = f2_add(err, f2_add(a.l, b.l));
  const f2 h = f2_add(s, err);
  return pf_make(h, f2_sub(err, f2_sub(h, s)));
}
/* ff_mul */
__device__ __forceinline__ pf2 pf_mul(pf2 a, pf2 b)
{
  const f2 p = f2_mul(a.h, b.h);
  f2 e = f2_fma(a.h, b.h, f2_neg(p));
  e = f2_fma(a.h, b.l, e);
  e = f2_fma(a.l, b.h, e);
  const f2 h = f2_add(p, e);
  return pf_make(h, f2_sub(e, f2_sub(h, p)));
}
/* ff_fma */
__device__ __forceinline__ pf2 pf_fma(pf2 a, pf2 b, pf2 c)
{
  const f2 p = f2_mul(a.h, b.h);
  f2 pe = f2_fma(a.h, b.h, f2_neg(p));
  pe = f2_fma(a.h, b.l, pe);
  pe = f2_fma(a.l, b.h, pe);
  const f2 s = f2_add(c.h, p);
  const f2 bb = f2_sub(s, c.h);
  f2 err = f2_add(f2_sub(c.h, f2_sub(s, bb)), f2_sub(p, bb));
  err = f2_add(err, f2_add(c.l, pe));
  const f2 h = f2_add(s, err);
  return pf_make(h, f2_sub(err, f2_sub(h, s)));
}
/* ff_sub2prod, with qn = -q.h and sn = -s.h */
__device__ __forceinline__ pf2 pf_sub2prod(pf2 a, pf2 p, pf2 q, f2 qn, pf2 r, pf2 s, f2 sn)
{
  const f2 m1 = f2_mul(p.h, qn);
  f2 e = f2_fma(p.h, q.h, m1);
  e = f2_fma(p.h, q.l, e);
  e = f2_fma(p.l, q.h, e);
  const f2 m2 = f2_mul(r.h, sn);
  e = f2_add(f2_fma(r.h, s.h, m2), e);
  e = f2_fma(r.h, s.l, e);
  e = f2_fma(r.l, s.h, e);
  const f2 t1 = f2_add(a.h, m1);
  const f2 b1 = f2_sub(t1, a.h);
  const f2 r1 = f2_add(f2_sub(a.h, f2_sub(t1, b1)), f2_sub(m1, b1));
  const f2 t2 = f2_add(t1, m2);
  const f2 b2 = f2_sub(t2, t1);
  const f2 r2 = f2_add(f2_sub(t1, f2_sub(t2, b2)), f2_sub(m2, b2));
  const f2 low = f2_add(f2_sub(a.l, e), f2_add(r1, r2));
  const f2 h = f2_add(t2, low);
  return pf_make(h, f2_sub(low, f2_sub(h, t2)));
}
/* ff_dot2 */
__device__ __forceinline__ pf2 pf_dot2(pf2 a, pf2 x, pf2 b, pf2 y)
{
  const f2 p1 = f2_mul(a.h, x.h);
  f2 e = f2_fma(a.h, x.h, f2_neg(p1));
  e = f2_fma(a.h, x.l, e);
  e = f2_fma(a.l, x.h, e);
  const f2 p2 = f2_mul(b.h, y.h);
  e = f2_add(f2_fma(b.h, y.h, f2_neg(p2)), e);
  e = f2_fma(b.h, y.l, e);
  e = f2_fma(b.l, y.h, e);
  const f2 s = f2_add(p1, p2);
  const f2 bb = f2_sub(s, p1);
  const f2 er = f2_add(f2_sub(p1, f2_sub(s, bb)), f2_sub(p2, bb));
  const f2 low = f2_add(e, er);
  const f2 h = f2_add(s, low);
  return pf_make(h, f2_sub(low, f2_sub(h, s)));
}
/* ff_acc_lazy, with xn = -x.h */
__device__ __forceinline__ pf2 pf_acc_lazy(pf2 acc, pf2 a, pf2 x, f2 xn)
{
  const f2 m = f2_mul(a.h, xn);
  f2 e = f2_fma(a.h, x.h, m);
  e = f2_fma(a.h, x.l, e);
  e = f2_fma(a.l, x.h, e);
  const f2 s = f2_sub(acc.h, m);
  const f2 bb = f2_sub(s, acc.h);
  const f2 er = f2_sub(f2_sub(acc.h, f2_sub(s, bb)), f2_add(m, bb));
  return pf_make(s, f2_add(acc.l, f2_add(e, er)));
}
__device__ __forceinline__ pf2 pf_shfl_xor(pf2 a, int o)
{
  return pf_make(__shfl_xor_sync(0xFFFFFFFFu, a.h, o), __shfl_xor_sync(0xFFFFFFFFu, a.l, o));
}
/* vectors of pairs: indices 2p and 2p + 1 as 16 bytes h, h', l, l' at double 2p */
__device__ __forceinline__ pf2 pv_load(const double *v, int p)
{
  const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(v + 2 * (size_t)p);
  return pf_make(x.x, x.y);
}
__device__ __forceinline__ void pv_store(double *v, int p, pf2 a)
{
  *reinterpret_cast<ulonglong2 *>(v + 2 * (size_t)p) = make_ulonglong2(a.h, a.l);
}
__device__ __forceinline__ ff2 pv_get(const double *v, int q)
{
  const float *f = reinterpret_cast<const float *>(v + (q & ~1)) + (q & 1);
  return ff_make(f[0], f[2]);
}
__device__ __forceinline__ void pv_put(double *v, int q, ff2 a)
{
  float *f = reinterpret_cast<float *>(v + (q & ~1)) + (q & 1);
  f[0] = a.h;
  f[2] = a.l;
}

/* a + b left unnormalised (ff_warp_sum's step) */
__device__ __forceinline__ pf2 pf_add_lazy(pf2 a, pf2 b)
{
  const f2 s = f2_add(a.h, b.h);
  const f2 bb = f2_sub(s, a.h);
  const f2 er = f2_add(f2_sub(a.h, f2_sub(s, bb)), f2_sub(b.h, bb));
  return pf_make(s, f2_add(f2_add(a.l, b.l), er));
}
__device__ __forceinline__ ff2 ff_add_lazy(ff2 a, ff2 b)
{
  const float s = __fadd_rn(a.h, b.h);
  const float bb = __fsub_rn(s, a.h);
  const float er = __fadd_rn(__fsub_rn(a.h, __fsub_rn(s, bb)), __fsub_rn(b.h, bb));
  return ff_make(s, __fadd_rn(__fadd_rn(a.l, b.l), er));
}
/*
 * A float-float value that carries its step: each half next to the step's tag in a 64-bit word, so
 * that a reader polls for the value itself and needs no barrier, fence or second trip to L2 for it.
 * The two words are the elements of one vector access: each is read and written whole, in no
 * order between them, so the reader looks at both tags.  Tags are c + 1 for values of step c,
 * never 0.
 */
__device__ __forceinline__ void tag_store(uint4 *p, ff2 v, unsigned tag)
{
  asm volatile(
      "{\n\t.reg .b64 h, l;\n\tmov.b64 h, {%1, %3};\n\tmov.b64 l, {%2, %3};\n\t"
      "st.relaxed.gpu.global.v2.b64 [%0], {h, l};\n\t}\n" ::"l"(p),
      "r"(__float_as_uint(v.h)), "r"(__float_as_uint(v.l)), "r"(tag)
      : "memory");
}
__device__ __forceinline__ uint4 tag_load(const uint4 *p)
{
  uint4 r;
  asm volatile(
      "{\n\t.reg .b64 h, l;\n\tld.relaxed.gpu.global.v2.b64 {h, l}, [%4];\n\t"
      "mov.b64 {%0, %1}, h;\n\tmov.b64 {%2, %3}, l;\n\t}\n"
      : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
      : "l"(p)
      : "memory");
  return r;
}

/*
 * y and x of the rows q0 + (u / 2) step + u % 2 (u < RPT, at least c and below n): all the loads
 * of a round are in flight together, and a round asks for what is missing only.  False when the wait ran out or another
 * block gave up.
 */
template <int RPT>
__device__ __forceinline__ bool tag_wait(const uint4 *yt, const uint4 *xt, int q0, int step, int c, int n,
                                         unsigned tag, ff2 *y, ff2 *x, int *err)
{
  unsigned need = 0;
#pragma unroll
  for (int u = 0; u < RPT; ++u)
    if (q0 + (u >> 1) * step + (u & 1) >= c && q0 + (u >> 1) * step + (u & 1) < n)
      need |= 3u << (2 * u);
  uint64_t t0 = 0;
  for (unsigned it = 0; need; ++it) {
    uint4 ry[RPT], rx[RPT];
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      if (need & (1u << (2 * u))) ry[u] = tag_load(yt + q0 + (u >> 1) * step + (u & 1));
      if (need & (2u << (2 * u))) rx[u] = tag_load(xt + q0 + (u >> 1) * step + (u & 1));
    }
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      if ((need & (1u << (2 * u))) && ry[u].y == tag && ry[u].w == tag) {
        y[u] = ff_make(__uint_as_float(ry[u].x), __uint_as_float(ry[u].z));
        need &= ~(1u << (2 * u));
      }
      if ((need & (2u << (2 * u))) && rx[u].y == tag && rx[u].w == tag) {
        x[u] = ff_make(__uint_as_float(rx[u].x), __uint_as_float(rx[u].z));
        need &= ~(2u << (2 * u));
      }
    }
    if (it == 0) t0 = globaltimer_ns();
    if ((it & 63u) == 63u) {
      if (*(volatile int *)err) return false;
      if (globaltimer_ns() - t0 > GP_WAIT_NS) {
        atomicExch(err, TR_ERR_BARRIER);
        return false;
      }
    }
  }
  return true;
}

/* one level of ff_warp_sum */
__device__ __forceinline__ ff2 ff_lazy_xor(ff2 v, int o)
{
  const float oh = __shfl_xor_sync(0xFFFFFFFFu, v.h, o), ol = __shfl_xor_sync(0xFFFFFFFFu, v.l, o);
  const float s = __fadd_rn(v.h, oh);
  const float bb = __fsub_rn(s, v.h);
  const float er = __fadd_rn(__fsub_rn(v.h, __fsub_rn(s, bb)), __fsub_rn(oh, bb));
  return ff_make(s, __fadd_rn(__fadd_rn(v.l, ol), er));
}

/*
 * Steps c0 .. n-2 with the trailing matrix (order m = n - c0 <= NT RPT) in shared memory, and
 * the last diagonal entry: block b holds whole columns r = c0 + b, c0 + b + G, .. (both
 * triangles, as float-float pairs; at most 32 columns).  Per step:
 *   A   every block redundantly: y of step c-1 and column c are polled for in global memory
 *       (tagged values, double-buffered); x of step c-1 is still in svc, unscaled, with alpha - beta in the
 *       pivot's place: v = scale x; then y.v, w, the pending update of column c, its norm and
 *       the reflector
 *   B   each warp takes a segment of rows of two owned columns: pending update, written back,
 *       and the dots with x; the owner of column c + 1 publishes it; then the first warp adds
 *       the segments and publishes y = scale (A x)
 * No barrier over the blocks: a block cannot start step c before every block's y of step c-1
 * is there, and a block publishes y of step c only after it has read all of step c-1, so the
 * two buffers suffice; a block without a column after c leaves before step c, since nobody
 * would wait for its reading.  A step is a chain of latencies: four block barriers, one trip
 * through L2, three sums over the block.  Every warp takes part in those sums, so a block has
 * few: with 32 warps their instructions alone took half the step.  A thread's rows come in pairs for
 * the packed FP32 instructions.  Reflectors, d, e and tau are stored as pairs and converted at the end (an
 * FP64 instruction occupies its quarter of the SM for 64 clocks).  n = 1,000: 5.2 ms of
 * 8.2 with the matrix in L2 and a grid barrier per step (5.9 before the packed pairs); n = 180 on 12
 * blocks: 0.50 of 1.34; the last 1,706 columns of 5,000: 12.4 (13.1).
 * Needs every block resident (a cooperative launch), ytag and ctag [2][n] zero.
 */
template <int NT, int RPT>
__device__ __forceinline__ bool tr_smem_steps(double *A, int n, int c0, double *d, double *e,
                                              double *tau, const double *xprev,
                                              const double *yprev0, uint4 *ytag, uint4 *ctag,
                                              unsigned *count, unsigned &target, int *err,
                                              double *smm, ff2 tau_p, ff2 scale_p, ff2 e_p,
                                              bool have_p)
{
  constexpr int NW = NT / 32;
  __shared__ ff2 red[NW], red1[NW];
  __shared__ ff2 sdot[2 * NW];
  __shared__ tr_step st;
  __shared__ ff2 s_yc;
  const int G = gridDim.x, b = blockIdx.x;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const ff2 ONE = ff_make(1.f, 0.f), ZERO = ff_make(0.f, 0.f);
  constexpr int RP = RPT / 2; /* pairs of rows per thread */
  const int m = n - c0, mp = (m + 1) & ~1, np = mp / 2;
  /* vectors of pairs over the rows from c0; column j at j mp */
  double *svp = smm, *swp = smm + mp, *svc = smm + 2 * mp, *cols = smm + 3 * (size_t)mp;
  const int cfirst = have_p ? c0 - 1 : c0; /* first reflector stored as pairs */
  const int nown = c0 + b < n ? (n - 1 - c0 - b) / G + 1 : 0;
  for (int j = 0; j < nown; ++j)
    for (int q = tid; q < mp; q += NT)
      pv_put(cols + (size_t)j * mp, q,
             q < m ? ff_load(A + (int64_t)(c0 + b + j * G) * n + c0 + q) : ZERO);
  for (int q = tid; q < mp; q += NT)
    pv_put(svc, q, have_p && q < m ? ff_load(xprev + c0 + q) : ZERO);
  int j0 = 0; /* first owned column at or after c + 1 */
  /* position from the owner of the last column: at step c < n-1 the blocks at positions below
   * n-1-c own a column after c */
  const int pos = ((n - 1 - c0) % G - b + G) % G;
  __syncthreads();
  bool fail = false;
  for (int c = c0; pos < max(1, n - 1 - c); ++c) {
    /* ---- A ---- */
    const int nact = min(G, max(1, n - 1 - c)); /* blocks in this step */
    const int k = c - c0, P0 = k >> 1, odd = k & 1; /* the pair of c, whose first row may be done */
    ff2 x[RPT], y[RPT];
    const uint4 *yt = ytag + (size_t)((c - 1) & 1) * n, *ct = ctag + (size_t)(c & 1) * n;
#pragma unroll
    for (int u = 0; u < RPT; ++u) {
      const int q = c0 + 2 * (P0 + tid + (u >> 1) * NT) + (u & 1);
      x[u] = y[u] = ZERO;
      if (q < c || q >= n) continue;
      if (c == c0) {
        x[u] = ff_load(A + (int64_t)c * n + q);
        if (have_p) y[u] = ff_load(yprev0 + q);
      }
    }
    if (c > c0)
      fail = !tag_wait<RPT>(yt, ct, c0 + 2 * (P0 + tid), 2 * NT, c, n, (unsigned)c, y, x, err);
    pf2 x2[RP], y2[RP], v2[RP], dacc2 = pf_make(0, 0);
    const pf2 scale2 = pf_dup(scale_p);
#pragma unroll
    for (int u = 0; u < RP; ++u) {
      const int p = P0 + tid + u * NT;
      x2[u] = pf_join(x[2 * u], x[2 * u + 1]);
      y2[u] = pf_join(y[2 * u], y[2 * u + 1]);
      v2[u] = pf_make(0, 0);
      if (p < np && have_p) {
        v2[u] = pf_mul(pv_load(svc, p), scale2);
        if (p == P0) v2[u] = odd ? pf_join(ZERO, ONE) : pf_join(ONE, pf_odd(v2[u]));
        dacc2 = pf_acc_lazy(dacc2, y2[u], v2[u], f2_neg(v2[u].h));
      }
    }
    const ff2 dacc = ff_warp_sum(ff_add_lazy(pf_even(dacc2), pf_odd(dacc2)));
    if (lane == 0) red1[warp] = dacc;
    if (tid == 0) s_yc = odd ? y[1] : y[0];
    if (__syncthreads_or(fail)) {
      fail = true;
      break;
    }
    ff2 dsum = red1[lane & (NW - 1)];
#pragma unroll
    for (int o = NW / 2; o; o >>= 1) dsum = ff_lazy_xor(dsum, o);
    dsum = ff_renorm(dsum);
    const ff2 alpha_p = ff_scale(ff_mul(ff_mul(tau_p, tau_p), dsum), -0.5f);
    const ff2 wpc = ff_fma(tau_p, s_yc, alpha_p); /* w(c) of step c-1, where v(c) = 1 */
    const pf2 tau2 = pf_dup(tau_p), alpha2 = pf_dup(alpha_p), nwpc2 = pf_dup(ff_neg(wpc));
    pf2 nrm2 = pf_make(0, 0);
#pragma unroll
    for (int u = 0; u < RP; ++u) {
      const int p = P0 + tid + u * NT;
      if (p >= np) continue;
      pf2 w = pf_make(0, 0), z = x2[u];
      if (have_p) {
        w = pf_fma(tau2, y2[u], pf_mul(alpha2, v2[u]));
        z = pf_fma(v2[u], nwpc2, z);
        z = pf_add(z, pf_make(f2_neg(w.h), f2_neg(w.l)));
      }
      pv_store(svp, p, v2[u]);
      pv_store(swp, p, w);
      pv_store(svc, p, z);
      if (2 * p < k + 2) z = pf_join(ZERO, 2 * p + 1 < k + 2 ? ZERO : pf_odd(z));
      nrm2 = pf_acc_lazy(nrm2, z, z, f2_neg(z.h));
    }
    const ff2 nrm = ff_warp_sum(ff_add_lazy(pf_even(nrm2), pf_odd(nrm2)));
    if (lane == 0) red[warp] = nrm;
    __syncthreads();
    if (have_p && warp > 0) {
      /* the reflector of step c-1, the blocks in turn by rows, while the first warp forms the
       * next one */
      for (int q = c + pos + (tid - 32) * nact; q < n; q += (NT - 32) * nact)
        ff_store(A + (int64_t)(c - 1) * n + q, q == c ? e_p : pv_get(svp, q - c0));
    }
    if (c == n - 1) {
      if (tid == 0) ff_store(d + c, pv_get(svc, k));
      break;
    }
    if (warp == 0) {
      ff2 xn2 = red[lane & (NW - 1)];
#pragma unroll
      for (int o = NW / 2; o; o >>= 1) xn2 = ff_lazy_xor(xn2, o);
      xn2 = ff_renorm(xn2);
      if (lane == 0) {
        /* the reflector (dlarfg): beta = -sign(alpha) sqrt(alpha^2 + |x|^2), tau = (beta -
         * alpha) / beta, scale = 1 / (alpha - beta) */
        const ff2 alpha = pv_get(svc, k + 1);
        ff2 beta = alpha, tau_c = ZERO, scale_c = ZERO;
        if (xn2.h != 0.f) {
          const ff2 sq = ff_fma(alpha, alpha, xn2);
          /* the approximate instructions flush subnormals: far from them only */
          const bool fast = sq.h > 1e-28f && sq.h < 1e28f;
          const ff2 nrm2 = fast ? ff_sqrt_fast(sq) : ff_sqrt(sq);
          beta = alpha.h >= 0.f ? ff_neg(nrm2) : nrm2;
          const ff2 am = ff_add(alpha, ff_neg(beta));
          tau_c = fast ? ff_div_fast(ff_neg(am), beta) : ff_div(ff_neg(am), beta);
          scale_c = fast ? ff_div_fast(ONE, am) : ff_div(ONE, am);
          pv_put(svc, k + 1, am);
        }
        st.beta = beta;
        st.tau_c = tau_c;
        st.scale_c = scale_c;
        if (pos == 0) {
          ff_store(d + c, pv_get(svc, k));
          ff_store(e + c, beta);
          ff_store(tau + c, tau_c);
        }
      }
    } else if (tid == 32) {
      /* the owned columns from c + 1 on and the segments of a pair of them: a power of two, as
       * many as there are warps for, of at least 64 rows */
      int j = j0;
      if (c0 + b + j * G < c + 1) ++j;
      const int npair = (nown - j + 1) >> 1, rows = n - 1 - c;
      int sh = 0;
      while ((npair << (sh + 1)) <= NW && (rows >> (sh + 1)) >= 64) ++sh;
      st.b1_u0 = j;
      st.b1_u1 = sh;
    }
    __syncthreads();
    const ff2 scale_c = st.scale_c;
    j0 = st.b1_u0;
    const int sh = st.b1_u1, S = 1 << sh;
    tau_p = st.tau_c;
    scale_p = scale_c;
    e_p = st.beta;
    have_p = true;
    /* ---- B: the owned columns r >= c + 1, two at a time ---- */
    const int nc = nown - j0, nitem = ((nc + 1) >> 1) << sh;
    const int pb = (k + 1) >> 1; /* the pair of c + 1, whose first row may be c */
    const int seg = (((np - pb + S - 1) >> sh) + 31) & ~31;
    uint4 *cn = ctag + (size_t)((c + 1) & 1) * n;
    /* an item per warp; with more pairs than warps (sh = 0) the dots of the later pairs wait
     * in registers for the slots of the earlier ones: at most two rounds, 32 columns */
    ff2 dab[2];
#pragma unroll
    for (int rd = 0; rd < 2; ++rd) {
      const int it = warp + rd * NW;
      ff2 da = ZERO, db = ZERO;
      if (it < nitem) {
        const int pi = it >> sh, sg = it & (S - 1);
        const int ja = j0 + 2 * pi, ra = c0 + b + ja * G, rb = ra + G;
        const bool two = rb < n;
        double *ca = cols + (size_t)ja * mp, *cb = two ? ca + mp : ca;
        const pf2 vra = pf_dup(pv_get(svp, ra - c0)), wra = pf_dup(pv_get(swp, ra - c0));
        const pf2 vrb = pf_dup(two ? pv_get(svp, rb - c0) : ZERO);
        const pf2 wrb = pf_dup(two ? pv_get(swp, rb - c0) : ZERO);
        const f2 vran = f2_neg(vra.h), wran = f2_neg(wra.h);
        const f2 vrbn = f2_neg(vrb.h), wrbn = f2_neg(wrb.h);
        const int ps = pb + sg * seg, pe = min(np, ps + seg);
        const bool next = ra == c + 1; /* the first of its block: never the second of a pair */
        pf2 da2 = pf_make(0, 0), db2 = da2;
#pragma unroll 2
        for (int p = ps + lane; p < pe; p += 32) {
          const pf2 vq = pv_load(svp, p), wq = pv_load(swp, p);
          pf2 xq = pv_load(svc, p);
          if (p == pb && !odd) xq = pf_join(ZERO, pf_odd(xq)); /* k + 1 odd: the first row is c */
          const f2 xn = f2_neg(xq.h);
          const pf2 a = pf_sub2prod(pv_load(ca, p), vq, wra, wran, wq, vra, vran);
          pv_store(ca, p, a);
          if (next) {
            const int q = c0 + 2 * p;
            if (q > c) tag_store(cn + q, pf_even(a), (unsigned)(c + 1));
            if (q + 1 < n) tag_store(cn + q + 1, pf_odd(a), (unsigned)(c + 1));
          }
          da2 = pf_acc_lazy(da2, a, xq, xn);
          if (two) {
            const pf2 a2 = pf_sub2prod(pv_load(cb, p), vq, wrb, wrbn, wq, vrb, vrbn);
            pv_store(cb, p, a2);
            db2 = pf_acc_lazy(db2, a2, xq, xn);
          }
        }
        da = ff_add_lazy(pf_even(da2), pf_odd(da2));
        db = ff_add_lazy(pf_even(db2), pf_odd(db2));
#pragma unroll
        for (int o = 16; o; o >>= 1) {
          da = ff_lazy_xor(da, o);
          db = ff_lazy_xor(db, o);
        }
      }
      dab[rd] = lane ? db : da; /* lanes 0 and 1 carry a pair's two sums */
      if (rd == 0) {
        if (lane < 2) sdot[2 * warp + lane] = dab[0];
        if (nitem <= NW) break;
      }
    }
    if (nitem > NW) {
      /* one segment per pair: a warp's own sums are complete */
      if (lane < 2)
#pragma unroll
        for (int rd = 0; rd < 2; ++rd) {
          const int col = 2 * (warp + rd * NW) + lane;
          if (col < nc)
            tag_store(ytag + (size_t)(c & 1) * n + c0 + b + (j0 + col) * G,
                      ff_mul(ff_renorm(dab[rd]), scale_c), (unsigned)(c + 1));
        }
      __syncthreads(); /* the vectors are rewritten by the next step */
      continue;
    }
    __syncthreads();
    if (warp == 0) {
      /* the segments of a column, slots 2 (pair S + segment) + column of the pair, by a tree */
#pragma unroll
      for (int h = 0; h < (2 * NW + 31) / 32; ++h) {
        const int slot = lane + 32 * h;
        ff2 t = slot < 2 * nitem ? sdot[slot] : ZERO;
        for (int o = 1; o < S; o <<= 1) t = ff_lazy_xor(t, 2 * o);
        const int col = 2 * (slot >> (sh + 1)) + (slot & 1);
        if (((slot >> 1) & (S - 1)) == 0 && slot < 2 * nitem && col < nc)
          tag_store(ytag + (size_t)(c & 1) * n + c0 + b + (j0 + col) * G,
                    ff_mul(ff_renorm(t), scale_c), (unsigned)(c + 1));
      }
    }
  }
  if (fail) return false;
  /* when every block's pairs are stored: to FP64 */
  target += G;
  if (!tr_grid_sync(count, target, err)) return false;
  for (int c = cfirst + b; c < n - 1; c += G)
    for (int q = c + 1 + tid; q < n; q += blockDim.x) {
      double *p = A + (int64_t)c * n + q;
      *p = ff_to_double(ff_load(p));
    }
  if (b == 0)
    for (int c = c0 + tid; c < n; c += blockDim.x) {
      d[c] = ff_to_double(ff_load(d + c));
      if (c < n - 1) {
        e[c] = ff_to_double(ff_load(e + c));
        tau[c] = ff_to_double(ff_load(tau + c));
      }
    }
  return true;
}

/* what a launch's last step leaves for the next launch's first (float-float pairs) */
struct tr_state {
  ff2 tau, scale, e;
};

/* steps c0 .. n-2: from the start (c0 = 0), or after the steps of another kernel */
template <int NT, int RPT>
__global__ void __launch_bounds__(NT, 1)
k_tridiag_smem(double *A, int n, int c0, double *d, double *e, double *tau, const double *xprev,
               const double *yprev, uint4 *ytag, uint4 *ctag, const tr_state *state, unsigned *bar,
               int *err)
{
  extern __shared__ double sh[];
  const ff2 ZERO = ff_make(0.f, 0.f);
  unsigned target = 0;
  const bool have_p = c0 > 0;
  tr_smem_steps<NT, RPT>(A, n, c0, d, e, tau, xprev, yprev, ytag, ctag, bar, target, err, sh,
                         have_p ? state->tau : ZERO, have_p ? state->scale : ZERO,
                         have_p ? state->e : ZERO, have_p);
}

/* 256 threads at every order, of 2, 4 or 8 rows each (the loops over a thread's rows are
 * unrolled): 512 threads of 4 rows took 13.7 ms where these take 12.4 at 1,706 rows, 6.8 against 5.2
 * at 1,000; 128 threads 0.54 against 0.50 at 180.  Two rows a thread up to TR_SMALL_ORDER: 0.50 ms
 * against 0.52 at 180, 1.53 against 1.44 at 400 */
#define TR_SMEM_NT 256
#define TR_SMEM_RPT 8
#define TR_SMALL_ORDER 320

/* steps 0 .. c_end - 1 by whole columns in L2: orders whose tiles' shared memory does not fit */
__global__ void __launch_bounds__(TR_THREADS, 1)
k_tridiag(double *A, int n, int c_end, double *d, double *e, double *tau, double *vbuf,
          double *wbuf, double *ybuf, double *part_dot2, tr_state *state, unsigned *bar, int *err,
          unsigned long long *phase_ns)
{
  extern __shared__ double sh[];
  const ff2 ZERO = ff_make(0.f, 0.f);
  unsigned target = 0;
  ff2 tau_pf = ZERO, scale_pf = ZERO, e_pf = ZERO;
  bool have_p = false;
  /* phase_ns (optional, block 0): time in A, B (entry 1; entry 2 for the first 30% of the
   * steps) and the barrier (entry 4) */
  __shared__ unsigned long long s_ph[6];
  const bool stamp = phase_ns != NULL && blockIdx.x == 0 && threadIdx.x == 0;
  if (stamp) {
    for (int i = 0; i < 5; ++i) s_ph[i] = 0ull;
    s_ph[5] = globaltimer_ns();
  }
  if (!tr_full_steps(A, n, c_end, d, e, tau, vbuf, wbuf, ybuf, part_dot2, bar, target, err, sh,
                     sh + n, sh + 2 * n, tau_pf, scale_pf, e_pf, have_p, stamp ? s_ph : NULL))
    return;
  if (stamp)
    for (int i = 0; i < 5; ++i) phase_ns[i] = s_ph[i];
  if (blockIdx.x == 0 && threadIdx.x == 0) *state = {tau_pf, scale_pf, e_pf};
}

/* ---------------------------------------------------------------------------------- */
/*
 * The same reduction (dsytd2, lower) with the trailing matrix held as its lower triangle only,
 * in TT x TT tiles: half the bytes per column step and two thirds of the float-float work of
 * the whole-column step, whose product needs both triangles.  Tile (I, J), I >= J, of the
 * lower triangle is at Tm + tt_tile(I, J)*TT*TT (doubles' storage): 16 bytes per row and pair of
 * columns, the pairs of columns one after the other (TT rows each), elements (i, 2k), (i, 2k+1)
 * as h, h', l, l', the operands of the packed FP32 instructions.  Diagonal tiles are held in
 * full; rows and columns beyond n are zero padding.
 *
 * Work is split into parts: tile row I (TT rows) x column unit u (TT_U columns, u = 0 ..
 * nt*TT/TT_U - 1, in tile column u/(TT/TT_U)).  The blocks form a pr x pc grid: block (a, b)
 * owns the parts of the tile rows in row group a and the column units in column group b
 * (tables computed by the host for each first active tile index J0, balanced so that every
 * block has about the same number of parts).  So the product's index block K (TT indices)
 * has pc row-part contributors (blocks (rg(K), *)) and, for each of its units, pr column-part
 * contributors (blocks (*, cg(u))).  Per step:
 *   A   every block: y of step c-1, the index blocks' partial dots y.v and column c are polled for
 *       as tagged values (tag_store); the pending w of step c-1, the pending update of column c,
 *       its norm, the reflector.  v of step c-1 is still in shared memory
 *   B   each warp takes parts of the block: the pending rank-2 update of step c-1 (written
 *       back), the row dots (two rows per lane) and, off the diagonal, the column dots (a
 *       reduce-scatter over the warp per 8 columns), and column c + 1 published as it is then; the
 *       block sums its parts per tile row and
 *       per column unit in a fixed order and publishes them, one arrival (release) on the
 *       index block's counter per published sum; block K mod G waits (acquire, bounded) for
 *       index block K's pc + (TT/TT_U)*pr arrivals and sums them in a fixed order into y and
 *       the index block's partial y.v, published
 * No barrier over the blocks in a step: every index block's sums have a contribution of every
 * block of its row group and of its units' column groups, so a block starts step c only when
 * every block has published its sums of step c-1 and with that has read all of step c-2: two
 * buffers suffice, and the arrival counters never mix steps.  A grid barrier stands where the tiles
 * change hands (every TT steps) and where a block could have no tile row (see there).
 * Rows and columns up to c keep their values (the pending-update vectors and v are zero there),
 * so that phase A of a block still reading column c never sees it change.  Every sum has a
 * fixed order.
 *
 * What bounds it: in B the FP32 pipe, 53 operations per element and step, and the issue slots.
 * Packed over two columns the operations take half the slots, and with 16 warps instead of 32 the
 * registers hold the next columns while these are worked on (parts of an early step of order
 * 5,000: 69,000 -> 52,000 clocks; 20 and 24 warps spill and are slower).  The chain around them,
 * some 25,000 clocks a step, is A (14,000: y and the column of every block from L2, then the
 * vectors, packed too), the sums, the arrivals and their wait (10,000) and the terms of y, all read
 * before any is added (3,000).  With a grid barrier in every step and the column read from the tiles
 * order 5,000 took 98.8 ms, now 92.5 (3,600: 50.2 -> 46.9, 2,500: 25.5 -> 24.2), 114 before the packed
 * pairs.  Down to the order that fits shared memory these steps beat whole columns (2,500: 28.4 ms),
 * which remain for orders whose vectors leave no room for the slots.
 */
#define TT 64
#define TT_U 16                /* columns per column unit */
#define TT_UPT (TT / TT_U)     /* column units per tile column */
#define TT_MAXG 32             /* row or column groups at most */
#define TT_THREADS 512
#define TT_WARPS (TT_THREADS / 32)
#define TR_ERR_LISTS 12
#define TR_ERR_WAIT 13

__host__ __device__ __forceinline__ int64_t tt_tile(int I, int J)
{
  return (int64_t)I * (I + 1) / 2 + J;
}

/* the lower triangle of the symmetric FP64 matrix A (column-major, both triangles valid) into
 * float-float tiles, padding zero */
__global__ void k_tri_to_tiles(const double *A, int n, int nt, double *Tm)
{
  const int64_t ntiles = (int64_t)nt * (nt + 1) / 2;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    int I = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
    while ((int64_t)(I + 1) * (I + 2) / 2 <= t) ++I;
    while ((int64_t)I * (I + 1) / 2 > t) --I;
    const int J = (int)(t - (int64_t)I * (I + 1) / 2);
    double *tile = Tm + t * (TT * TT);
    for (int idx = threadIdx.x; idx < TT * TT / 2; idx += blockDim.x) {
      const int j = idx / TT * 2, i = idx % TT;
      const int r = I * TT + i, q = J * TT + j;
      const double v0 = (r < n && q < n) ? A[(int64_t)q * n + r] : 0.0;
      const double v1 = (r < n && q + 1 < n) ? A[(int64_t)(q + 1) * n + r] : 0.0;
      pv_store(tile, idx, pf_join(ff_from_double(v0), ff_from_double(v1)));
    }
  }
}

/* sum over the lanes of 8 columns' dots (4 pairs), scattered: lanes 4k .. 4k+3 end with column k */
__device__ __forceinline__ ff2 tt_scatter8(pf2 *cp, int lane)
{
  const bool b4 = (lane & 16) != 0, b3 = (lane & 8) != 0, b2 = (lane & 4) != 0;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const pf2 send = b4 ? cp[k] : cp[k + 2], keep = b4 ? cp[k + 2] : cp[k];
    cp[k] = pf_add_lazy(keep, pf_shfl_xor(send, 16));
  }
  {
    const pf2 send = b3 ? cp[0] : cp[1], keep = b3 ? cp[1] : cp[0];
    cp[0] = pf_add_lazy(keep, pf_shfl_xor(send, 8));
  }
  const ff2 e = pf_even(cp[0]), o = pf_odd(cp[0]);
  const ff2 send = b2 ? e : o, keep = b2 ? o : e;
  ff2 r = ff_add_lazy(keep, ff_shfl_xor(send, 4));
  r = ff_add_lazy(r, ff_shfl_xor(r, 2));
  return ff_renorm(ff_add_lazy(r, ff_shfl_xor(r, 1)));
}

/*
 * y and the column at the indices q + u TT_THREADS (u < TT_POLL, below npad) into sy and sx: tagged
 * values, all the loads of a round in flight together, a round asking for what is missing only.
 * False when the wait ran out or another block gave up.
 */
#define TT_POLL 2 /* indices a thread polls for at a time: 1 took 96 ms, 3 106 (spills), 2 92.5 */
__device__ __forceinline__ bool tt_wait(const uint4 *yt, const uint4 *ct, int q, int npad,
                                        unsigned ytag, unsigned ctag, double *sy, double *sx,
                                        int *err)
{
  unsigned need = 0;
#pragma unroll
  for (int u = 0; u < TT_POLL; ++u)
    if (q + u * TT_THREADS < npad) need |= 3u << (2 * u);
  uint64_t t0 = 0;
  for (unsigned it = 0; need; ++it) {
    uint4 r[2 * TT_POLL];
#pragma unroll
    for (int k = 0; k < 2 * TT_POLL; ++k)
      if (need & (1u << k)) r[k] = tag_load((k & 1 ? ct : yt) + q + (k >> 1) * TT_THREADS);
#pragma unroll
    for (int k = 0; k < 2 * TT_POLL; ++k) {
      const unsigned tag = k & 1 ? ctag : ytag;
      if ((need & (1u << k)) && r[k].y == tag && r[k].w == tag) {
        pv_put(k & 1 ? sx : sy, q + (k >> 1) * TT_THREADS,
               ff_make(__uint_as_float(r[k].x), __uint_as_float(r[k].z)));
        need &= ~(1u << k);
      }
    }
    if (it == 0) t0 = globaltimer_ns();
    if ((it & 63u) == 63u) {
      if (*(volatile int *)err) return false;
      if (globaltimer_ns() - t0 > GP_WAIT_NS) {
        atomicExch(err, TR_ERR_WAIT);
        return false;
      }
    }
  }
  return true;
}

/* two pairs of columns of the lane's rows (lane, lane + 32), from the first pair's address */
__device__ __forceinline__ void tt_load(pf2 a[2][2], const double *p0)
{
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    a[k][0] = pv_load(p0 + (size_t)k * (2 * TT), 0);
    a[k][1] = pv_load(p0 + (size_t)k * (2 * TT), 32);
  }
}

/* a warp's halves of parts (TT_H columns each), h0 .. h1 - 1 in the order of the block's parts:
 * the pending update of step c-1, written back; the row dots with v (rows lane and lane + 32),
 * into one slot rseg[TT] for each tile row that the warp meets, from slot seg on; off the
 * diagonal the column dots with v over the tile's rows into cslot[h][TT_H].  The next columns are
 * read while these are worked on. */
#define TT_H 8
__device__ __forceinline__ void tt_halves(double *Tm, const int4 *items, int h0, int h1, int seg,
                                          int dead, uint4 *cnext, const double *svp, const double *swp,
                                          const double *svc, double *rseg, double *cslot, int lane)
{
  if (h0 >= h1) return;
  const pf2 Z = pf_make(0, 0);
  Tm += 2 * lane;
  auto half = [&](int h) { return Tm + (int64_t)items[h >> 1].z * (TT * TT_H) + (h & 1) * (TT * TT_H); };
  pf2 vr0 = Z, vr1 = Z, pr0 = Z, pr1 = Z, qr0 = Z, qr1 = Z, ra0 = Z, ra1 = Z;
  int I = -1;
  double *p0 = half(h0);
  pf2 a[2][2];
  tt_load(a, p0);
  for (int h = h0; h < h1; ++h) {
    const int4 it = items[h >> 1];
    if (it.x != I) {
      if (I >= 0) {
        ff_store(rseg + seg * TT + lane, ff_add(ff_renorm(pf_even(ra0)), ff_renorm(pf_odd(ra0))));
        ff_store(rseg + seg * TT + lane + 32,
                 ff_add(ff_renorm(pf_even(ra1)), ff_renorm(pf_odd(ra1))));
        ++seg;
      }
      I = it.x;
      const int r = I * TT + lane;
      vr0 = pf_dup(pv_get(svc, r)), vr1 = pf_dup(pv_get(svc, r + 32));
      pr0 = pf_dup(pv_get(svp, r)), pr1 = pf_dup(pv_get(svp, r + 32));
      qr0 = pf_dup(pv_get(swp, r)), qr1 = pf_dup(pv_get(swp, r + 32));
      ra0 = ra1 = Z;
    }
    const int col0 = it.y * TT_U + (h & 1) * TT_H;
    double *pn = h + 1 < h1 ? half(h + 1) : p0;
    if (col0 + TT_H <= dead) { /* every column is at or before c */
      if (lane < TT_H) ff_store(cslot + (size_t)h * TT_H + lane, ff_make(0.f, 0.f));
      tt_load(a, pn);
    } else {
      pf2 cp[4];
#pragma unroll
      for (int cb = 0; cb < 4; cb += 2) {
        pf2 nx[2][2];
        tt_load(nx, cb ? pn : p0 + 2 * (2 * TT));
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int p = col0 / 2 + cb + k;
          const pf2 vpc = pv_load(svp, p), wpc = pv_load(swp, p), vc = pv_load(svc, p);
          const f2 vpn = f2_neg(vpc.h), wpn = f2_neg(wpc.h), vn = f2_neg(vc.h);
          const pf2 a0 = pf_sub2prod(a[k][0], pr0, wpc, wpn, qr0, vpc, vpn);
          const pf2 a1 = pf_sub2prod(a[k][1], pr1, wpc, wpn, qr1, vpc, vpn);
          pv_store(p0 + (size_t)(cb + k) * (2 * TT), 0, a0);
          pv_store(p0 + (size_t)(cb + k) * (2 * TT), 32, a1);
          if (p == dead >> 1) { /* the next step's column */
            const int r = I * TT + lane;
            tag_store(cnext + r, dead & 1 ? pf_odd(a0) : pf_even(a0), (unsigned)dead + 1u);
            tag_store(cnext + r + 32, dead & 1 ? pf_odd(a1) : pf_even(a1), (unsigned)dead + 1u);
          }
          ra0 = pf_acc_lazy(ra0, a0, vc, vn);
          ra1 = pf_acc_lazy(ra1, a1, vc, vn);
          cp[cb + k] = pf_dot2(a0, vr0, a1, vr1);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          a[k][0] = nx[k][0];
          a[k][1] = nx[k][1];
        }
      }
      if (it.w >= 0) {
        const ff2 t = tt_scatter8(cp, lane);
        if ((lane & 3) == 0) ff_store(cslot + (size_t)h * TT_H + (lane >> 2), t);
      }
    }
    p0 = pn;
  }
  ff_store(rseg + seg * TT + lane, ff_add(ff_renorm(pf_even(ra0)), ff_renorm(pf_odd(ra0))));
  ff_store(rseg + seg * TT + lane + 32, ff_add(ff_renorm(pf_even(ra1)), ff_renorm(pf_odd(ra1))));
}

/* shared-memory bytes of k_tridiag_tiled for the bounds of a block's tile rows, column units and
 * parts */
__host__ __device__ inline size_t tt_smem_bytes(int nt, int maxr, int maxc, int maxi)
{
  const size_t npad = (size_t)nt * TT;
  const size_t dbl = 3 * npad + (size_t)(maxr + TT_WARPS) * TT + (size_t)maxi * TT_U;
  const size_t bytes = dbl * sizeof(double) + (size_t)maxi * sizeof(int4) +
                       sizeof(int) * (size_t)(5 * maxr + maxc) + (size_t)nt * (1 + TT_UPT);
  return (bytes + 15) & ~(size_t)15;
}

/*
 * Tm: the tiles (k_tri_to_tiles); A receives the reflectors in FP64 in A(c+2:n, c) and e on the
 * subdiagonal, as dormtr (lower) reads them.  rgt [nt][nt], cgt [nt][nt*TT_UPT]: the row group
 * of each tile row and the column group of each column unit for first active tile index J0
 * (row J0 of each table).  prow [nt][pc][TT], pcol [nt*TT_UPT][pr][TT_U]: the published row
 * and column parts; dotp [2][nt]: the index blocks' partial y.v of alternate steps; kcnt [nt]:
 * arrival counters (zero at launch); yb [2][nt*TT]: y of alternate steps, as a vector of pairs
 * (zero at launch, as dotp).  maxr/maxc/maxi bound a block's tile rows, column units and parts
 * over all J0.  After step cs - 1 the trailing matrix (indices >= cs) goes to
 * A as float-float pairs in whole columns, both triangles, v and y of that step to xlast and
 * ylast and its scalars to *state (v is scaled already, so its scale is 1): k_tridiag_smem does
 * the rest.
 */
__global__ void __launch_bounds__(TT_THREADS, 1)
k_tridiag_tiled(double *A, double *Tm, int n, int nt, int pr, int pc, int maxr, int maxc,
                int maxi, int cs, const unsigned char *rgt, const unsigned char *cgt,
                double *d, double *e, double *tau, uint4 *yt, uint4 *ct, uint4 *dott,
                double *xlast, double *ylast, double *prow, double *pcol, unsigned *kcnt, unsigned *bar, int *err,
                unsigned long long *phase_ns, tr_state *state)
{
  extern __shared__ double sh[];
  const int npad = nt * TT, nu = nt * TT_UPT;
  double *svp = sh, *swp = sh + npad, *svc = sh + 2 * npad; /* vectors of pairs */
  double *rseg = sh + 3 * (size_t)npad;                     /* [maxr + TT_WARPS][TT] */
  double *cslot = rseg + (size_t)(maxr + TT_WARPS) * TT;    /* [maxi][TT_U] */
  int4 *items = reinterpret_cast<int4 *>(cslot + (size_t)maxi * TT_U);
  int *rowl = reinterpret_cast<int *>(items + maxi); /* tile rows */
  int *rowb = rowl + maxr;                           /* first part of each tile row */
  int *rown = rowb + maxr;                           /* parts of each tile row */
  int *segb = rown + maxr;                           /* first row slot of each tile row */
  int *segn = segb + maxr;                           /* row slots of each tile row */
  int *coll = segn + maxr;                           /* column units */
  unsigned char *rg = reinterpret_cast<unsigned char *>(coll + maxc);
  unsigned char *cg = rg + nt;
  __shared__ ff2 red[TT_WARPS];
  __shared__ ff2 s_dot[TT_WARPS];
  __shared__ tr_step st;
  __shared__ ff2 s_slotf, s_dc, s_yc;
  __shared__ int s_nr, s_nc, s_ni, s_ok;
  __shared__ int s_seg[TT_WARPS]; /* each warp's first row slot */
  const int G = gridDim.x, b = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool active = b < pr * pc, all = G == pr * pc;
  const int ga = active ? b / pc : 0, gb = active ? b - (b / pc) * pc : 0;
  const ff2 ONE = ff_make(1.f, 0.f), ZERO = ff_make(0.f, 0.f);
  unsigned *count = bar;
  unsigned target = 0;
  /* the previous step's reflector scalars (block-uniform, kept in shared memory) */
  __shared__ ff2 s_tau_p, s_e_p;
  /* phase_ns (optional, block 0): time in A, B (entry 1; entry 2 for the first 30% of the
   * steps) and the barrier (entry 4), accumulated in shared memory */
  __shared__ unsigned long long s_ph[6];
  const bool stamp = phase_ns != NULL && b == 0 && threadIdx.x == 0;
  if (stamp) {
    for (int i = 0; i < 5; ++i) s_ph[i] = 0ull;
    s_ph[5] = globaltimer_ns();
  }
  if (threadIdx.x == 0) s_tau_p = s_e_p = ZERO;
#define TT_STAMP(i)                                    \
  if (stamp) {                                         \
    const unsigned long long t_now = globaltimer_ns(); \
    s_ph[i] += t_now - s_ph[5];                        \
    s_ph[5] = t_now;                                   \
  }
  const int early = (int)((3LL * n) / 10);
  const unsigned arrivals = (unsigned)(pc + TT_UPT * pr); /* per index block and step */
  for (int q = threadIdx.x; q < 3 * npad; q += TT_THREADS) sh[q] = 0.0; /* padding stays 0 */
  int j0_lists = -1;
  for (int c = 0; c < cs; ++c) {
    const int J0 = (c + 1) / TT;
    if (J0 != j0_lists) {
      /* the block's tile rows, column units and parts from J0 on (row J0 of the tables) */
      for (int I = threadIdx.x; I < nt; I += blockDim.x) rg[I] = rgt[(size_t)J0 * nt + I];
      for (int u = threadIdx.x; u < nu; u += blockDim.x) cg[u] = cgt[(size_t)J0 * nu + u];
      __syncthreads();
      if (threadIdx.x == 0) {
        int nr = 0, nc = 0, ni = 0, bad = 0;
        if (active) {
          for (int I = J0; I < nt; ++I)
            if (rg[I] == ga) {
              if (nr < maxr) rowl[nr++] = I; else bad = 1;
            }
          for (int u = J0 * TT_UPT; u < nu; ++u)
            if (cg[u] == gb) {
              if (nc < maxc) coll[nc++] = u; else bad = 1;
            }
          for (int kr = 0; kr < nr; ++kr) {
            rowb[kr] = ni;
            int k = 0;
            for (; k < nc && coll[k] / TT_UPT <= rowl[kr]; ++k) {
              if (ni < maxi)
                items[ni++] = make_int4(rowl[kr], coll[k],
                                        (int)tt_tile(rowl[kr], coll[k] / TT_UPT) * (TT / TT_H) +
                                            coll[k] % TT_UPT * (TT_U / TT_H),
                                        coll[k] / TT_UPT == rowl[kr] ? -1 : k);
              else
                bad = 1;
            }
            rown[kr] = k;
          }
          /* the warps' shares of the parts' halves in order, and a row slot for every piece of
           * a tile row in a share */
          int seg = 0, w = 0;
          for (int kr = 0; kr < nr; ++kr) {
            const int ha = 2 * rowb[kr], hb = ha + 2 * rown[kr];
            segb[kr] = seg;
            for (int h = ha; h < hb;) {
              while (2 * ni * (w + 1) / TT_WARPS <= h) ++w;
              if (2 * ni * w / TT_WARPS >= ha) s_seg[w] = seg; /* the share begins in this row */
              h = 2 * ni * (w + 1) / TT_WARPS;
              ++seg;
            }
            segn[kr] = seg - segb[kr];
          }
        }
        if (bad) atomicExch(err, TR_ERR_LISTS);
        s_nr = nr;
        s_nc = nc;
        s_ni = ni;
      }
      __syncthreads();
      j0_lists = J0;
    }
    /* ---- A ---- (before step 0 every vector and scalar of the "previous step" is zero) */
    {
      double *t = svp; /* v of step c-1 */
      svp = svc;
      svc = t;
    }
    const ff2 tau_pf = s_tau_p, e_pf = s_e_p;
    uint4 *ycur = yt + (size_t)(c & 1) * npad;
    const uint4 *yprev = yt + (size_t)((c + 1) & 1) * npad, *ccur = ct + (size_t)(c & 1) * npad;
    const int p0 = c / 2, odd = c & 1, np = npad / 2;
    bool fail = false;
    if (c == 0) {
      for (int p = threadIdx.x; p < np; p += TT_THREADS) {
        const int q = 2 * p, I = q / TT;
        const double *a = Tm + tt_tile(I, 0) * (TT * TT) + 2 * (q - I * TT);
        pv_store(svc, p, pf_join(pf_even(pv_load(a, 0)), pf_even(pv_load(a, 1))));
        pv_store(swp, p, pf_make(0, 0));
      }
      if (threadIdx.x == 0) s_yc = s_slotf = ZERO;
    } else {
      for (int q = 2 * p0 + threadIdx.x; q < npad && !fail; q += TT_POLL * TT_THREADS)
        fail = !tt_wait(yprev, ccur, q, npad, (unsigned)c, (unsigned)c + 1u, swp, svc, err);
      if (threadIdx.x == (unsigned)odd) s_yc = pv_get(swp, c); /* its own store */
      if (warp == TT_WARPS - 1) {
        /* y.v of step c-1: its index blocks' partial dots (from (c-1+1)/TT on), in order */
        const uint4 *dprev = dott + (size_t)((c + 1) & 1) * nt;
        ff2 pacc = ZERO;
        for (int k = c / TT + lane; k < nt && !fail; k += 32) {
          uint4 r = tag_load(dprev + k);
          const uint64_t t0 = globaltimer_ns();
          for (unsigned it = 1; r.y != (unsigned)c || r.w != (unsigned)c; ++it) {
            if ((it & 63u) == 0 &&
                (*(volatile int *)err || globaltimer_ns() - t0 > GP_WAIT_NS)) {
              atomicCAS(err, 0, TR_ERR_WAIT);
              fail = true;
              break;
            }
            r = tag_load(dprev + k);
          }
          pacc = ff_add(pacc, ff_make(__uint_as_float(r.x), __uint_as_float(r.z)));
        }
        for (int o = 16; o; o >>= 1) pacc = ff_add(pacc, ff_shfl_xor(pacc, o));
        if (lane == 0) s_slotf = pacc;
      }
    }
    if (__syncthreads_or(fail)) return;
    {
      const ff2 alpha_pf = ff_scale(ff_mul(ff_mul(tau_pf, tau_pf), s_slotf), -0.5f);
      const ff2 wpc = ff_fma(tau_pf, s_yc, alpha_pf);
      const pf2 tau2 = pf_dup(tau_pf), alpha2 = pf_dup(alpha_pf), nwpc2 = pf_dup(ff_neg(wpc));
      const int cnt = n - c, per = (cnt + G - 1) / G;
      const int r0 = c + b * per, r1 = min(n, r0 + per);
      pf2 nrm = pf_make(0, 0);
#pragma unroll 2
      for (int p = p0 + threadIdx.x; p < np; p += TT_THREADS) {
        const pf2 vp = pv_load(svp, p);
        pf2 wp = pf_fma(tau2, pv_load(swp, p), pf_mul(alpha2, vp));
        pf2 x = pf_fma(vp, nwpc2, pv_load(svc, p));
        x = pf_add(x, pf_make(f2_neg(wp.h), f2_neg(wp.l)));
        if (2 * p < c) { /* index c - 1 takes no part any more */
          wp = pf_join(ZERO, pf_odd(wp));
          x = pf_join(ZERO, pf_odd(x));
        }
        pv_store(swp, p, wp);
        pv_store(svc, p, x);
        if (2 * p + 1 >= r0 && 2 * p < r1 && c > 0) {
          for (int q = max(2 * p, r0); q < min(2 * p + 2, r1); ++q)
            A[(int64_t)(c - 1) * n + q] =
                ff_to_double(q == c ? e_pf : (q & 1) ? pf_odd(vp) : pf_even(vp));
        }
        if (2 * p < c + 2) x = pf_join(ZERO, 2 * p + 1 < c + 2 ? ZERO : pf_odd(x));
        nrm = pf_fma(x, x, nrm);
      }
      ff2 t = ff_add(pf_even(nrm), pf_odd(nrm));
      for (int o = 16; o; o >>= 1) t = ff_add(t, ff_shfl_xor(t, o));
      if (lane == 0) red[warp] = t;
      __syncthreads();
      if (warp == 0) {
        t = lane < TT_WARPS ? red[lane] : ZERO;
        for (int o = 16; o; o >>= 1) t = ff_add(t, ff_shfl_xor(t, o));
      }
      if (threadIdx.x == 0) {
        const ff2 xn2 = t, alpha = pv_get(svc, c + 1);
        s_dc = pv_get(svc, c);
        if (xn2.h == 0.f) {
          st.beta = alpha;
          st.tau_c = ZERO;
          st.scale_c = ZERO;
        } else {
          const ff2 nrm2 = ff_sqrt(ff_fma(alpha, alpha, xn2));
          const ff2 beta = alpha.h >= 0.f ? ff_neg(nrm2) : nrm2;
          const ff2 am = ff_add(alpha, ff_neg(beta));
          st.beta = beta;
          st.tau_c = ff_div(ff_neg(am), beta);
          st.scale_c = ff_div(ONE, am);
        }
      }
      __syncthreads();
      if (b == 0 && threadIdx.x == 32) {
        d[c] = ff_to_double(s_dc);
        e[c] = ff_to_double(st.beta);
        tau[c] = ff_to_double(st.tau_c);
      }
    }
    const ff2 beta = st.beta, tau_c = st.tau_c;
    TT_STAMP(0)
    /* ---- B ---- v of step c; the vectors zero at indices J0*TT .. c (rows and columns up to
     * c keep their values, and take no part in the dots) */
    {
      const pf2 scale2 = pf_dup(st.scale_c);
      for (int p = J0 * TT / 2 + threadIdx.x; p < np; p += TT_THREADS) {
        pf2 v = pf_mul(pv_load(svc, p), scale2);
        if (2 * p <= c + 1) {
          const ff2 v0 = 2 * p == c + 1 ? ONE : ZERO;
          const ff2 v1 = 2 * p + 1 == c + 1 ? ONE : 2 * p + 1 <= c ? ZERO : pf_odd(v);
          v = pf_join(v0, v1);
          if (2 * p <= c) {
            const bool keep = 2 * p + 1 > c;
            pv_store(svp, p, pf_join(ZERO, keep ? pf_odd(pv_load(svp, p)) : ZERO));
            pv_store(swp, p, pf_join(ZERO, keep ? pf_odd(pv_load(swp, p)) : ZERO));
          }
        }
        pv_store(svc, p, v);
      }
    }
    const int nr = s_nr, nc = s_nc, ni = s_ni;
    __syncthreads();
    tt_halves(Tm, items, 2 * ni * warp / TT_WARPS, 2 * ni * (warp + 1) / TT_WARPS, s_seg[warp],
              c + 1, ct + (size_t)((c + 1) & 1) * npad, svp, swp, svc, rseg, cslot, lane);
    __syncthreads();
    /* the block's sums, in part order: row parts of its tile rows, column parts of its units
     * (tile row kr's k-th unit is part rowb[kr] + k); then one arrival per published sum on its
     * index block's counter */
    if (active) {
      for (int idx = threadIdx.x; idx < nr * TT; idx += TT_THREADS) {
        const int kr = idx / TT, i = idx - kr * TT;
        const double *r = rseg + (size_t)segb[kr] * TT + i;
        ff2 t = ff_load(r);
        for (int k = 1; k < segn[kr]; ++k) t = ff_add(t, ff_load(r + (size_t)k * TT));
        ff_store(prow + ((size_t)rowl[kr] * pc + gb) * TT + i, segn[kr] ? t : ZERO);
      }
      for (int idx = threadIdx.x; idx < nc * TT_U; idx += TT_THREADS) {
        const int kc = idx / TT_U, j = idx - kc * TT_U, J = coll[kc] / TT_UPT;
        ff2 t = ZERO;
        for (int kr = 0; kr < nr; ++kr)
          if (kc < rown[kr] && J != rowl[kr])
            t = ff_add(t, ff_load(cslot + (size_t)(rowb[kr] + kc) * TT_U + j));
        ff_store(pcol + ((size_t)coll[kc] * pr + ga) * TT_U + j, t);
      }
    }
    __syncthreads();
    if (active) {
      for (int k = threadIdx.x; k < nr + nc; k += TT_THREADS)
        red_release_gpu(kcnt + (k < nr ? rowl[k] : coll[k - nr] / TT_UPT), 1u);
    }
    /* index blocks K = b, b + G, ...: wait for their arrivals, then y over the TT indices
     * (pc row parts, then pr column parts of the index's unit, in order: 8 threads per index
     * with four terms each and a fixed shuffle tree) and the partial y.v */
    {
      const unsigned ktarget = arrivals * (unsigned)(c + 1);
      for (int K = b; K < nt; K += G) {
        if (K < J0) continue;
        if (threadIdx.x == 0) {
          int ok = 1;
          volatile int *verr = err;
          const uint64_t t0 = globaltimer_ns();
          for (unsigned it = 1; ld_acquire_gpu(kcnt + K) < ktarget; ++it) {
            if ((it & 63u) == 0) {
              if (*verr) {
                ok = 0;
                break;
              }
              if (globaltimer_ns() - t0 > GP_WAIT_NS) {
                atomicExch(err, TR_ERR_WAIT);
                ok = 0;
                break;
              }
            }
          }
          s_ok = ok;
        }
        __syncthreads();
        if (!s_ok) return;
        const int i = threadIdx.x >> 3, g = threadIdx.x & 7;
        const int nterm = pc + pr;
        /* at most 8 terms a thread (pr, pc <= TT_MAXG), read before any is added */
        ff2 term[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int t = g + 8 * k;
          term[k] = ZERO;
          if (t < nterm)
            term[k] = ff_load(t < pc ? prow + ((size_t)K * pc + t) * TT + i
                                     : pcol + ((size_t)(K * TT_UPT + i / TT_U) * pr + (t - pc)) *
                                                  TT_U + (i & (TT_U - 1)));
        }
        ff2 y = term[0];
#pragma unroll
        for (int k = 1; k < 8; ++k)
          if (8 * k < nterm) y = ff_add(y, term[k]);
        for (int o = 4; o; o >>= 1) y = ff_add(y, ff_shfl_xor(y, o));
        const int q = K * TT + i;
        ff2 dv = ZERO;
        if (g == 0) {
          tag_store(ycur + q, y, (unsigned)c + 1u);
          dv = ff_mul(y, pv_get(svc, q));
        }
        /* the warp's four indices, lanes 0, 8, 16 and 24 */
        dv = ff_add(dv, ff_shfl_xor(dv, 8));
        dv = ff_add(dv, ff_shfl_xor(dv, 16));
        if (lane == 0) s_dot[warp] = dv;
        __syncthreads();
        if (threadIdx.x < 32) {
          ff2 t = lane < TT_WARPS ? s_dot[lane] : ZERO;
          for (int o = 16; o; o >>= 1) t = ff_add(t, ff_shfl_xor(t, o));
          if (threadIdx.x == 0) tag_store(dott + (size_t)(c & 1) * nt + K, t, (unsigned)c + 1u);
        }
        __syncthreads();
      }
    }
    TT_STAMP(c < early ? 2 : 1)
    if (threadIdx.x == 0) { /* read again only after the barrier below */
      s_tau_p = tau_c;
      s_e_p = beta;
    }
    /* a grid barrier only where the tiles change hands, at the end, and where a block might have
     * no sum to publish in the next two steps (it could then fall behind by more than a buffer) */
    if ((c + 2) / TT != J0 || c == cs - 1 || !all || nt - (c + 3) / TT < pr) {
      target += G;
      if (!tr_grid_sync(count, target, err)) return;
    } else {
      __syncthreads(); /* the scalars; the vectors are rewritten from here on */
    }
    TT_STAMP(4)
  }
  /* the trailing block (indices >= cs) of the block's parts into A as float-float pairs, both
   * triangles (the pending update of step cs-1 is applied by the next kernel) */
  const int ni = s_ni;
  for (int64_t idx = threadIdx.x; idx < (int64_t)ni * (TT * TT_U); idx += TT_THREADS) {
    const int u = (int)(idx / (TT * TT_U)), rem = (int)(idx - (int64_t)u * (TT * TT_U));
    const int j = rem / TT, i = rem - j * TT;
    const int4 it = items[u];
    const int J = it.y / TT_UPT, jt = (it.y - J * TT_UPT) * TT_U + j;
    const int r = it.x * TT + i, q = J * TT + jt;
    if (r >= cs && q >= cs && r < n && q < n) {
      const float *f = reinterpret_cast<const float *>(Tm + tt_tile(it.x, J) * (TT * TT)) +
                       4 * ((jt / 2) * TT + i) + (jt & 1);
      const ff2 v = ff_make(f[0], f[2]);
      ff_store(A + (int64_t)q * n + r, v);
      if (it.x != J) ff_store(A + (int64_t)r * n + q, v);
    }
  }
  for (int q = cs + b * TT_THREADS + threadIdx.x; q < n; q += G * TT_THREADS) {
    ff_store(xlast + q, pv_get(svc, q));
    const uint4 y = tag_load(yt + (size_t)((cs + 1) & 1) * npad + q);
    ff_store(ylast + q, ff_make(__uint_as_float(y.x), __uint_as_float(y.z)));
  }
  if (stamp)
    for (int i = 0; i < 5; ++i) phase_ns[i] = s_ph[i];
#undef TT_STAMP
  if (b == 0 && threadIdx.x == 0) *state = {s_tau_p, ONE, s_e_p};
}

/* deterministic start vector entry in (-1, 1) */
__device__ __forceinline__ double start_entry(int j, int i)
{
  uint64_t z = ((uint64_t)(j + 1) << 32) ^ (uint64_t)(i + 1) ^ 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return ((double)(z >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0;
}

/* block sum (fixed order: warp shuffles, then warp 0 over the warps' sums), broadcast to
 * every thread; red holds at least one double per warp */
__device__ double block_sum(double v, double *red)
{
  for (int o = 16; o; o >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    const int nw = blockDim.x >> 5;
    double t = (int)threadIdx.x < nw ? red[threadIdx.x] : 0.0;
    for (int o = 16; o; o >>= 1) t += __shfl_down_sync(0xFFFFFFFFu, t, o);
    if (threadIdx.x == 0) red[32] = t;
  }
  __syncthreads();
  const double r = red[32];
  __syncthreads();
  return r;
}

/* 1/q: rcp_newton and a second Newton step, to the last bits */
__device__ __forceinline__ double rcp_full(double q)
{
  /* rcp_newton's exponent arithmetic holds well inside the normal range only */
  const double a = fabs(q);
  if (!(a > 1e-290 && a < 1e290)) return 1.0 / q;
  const double r = rcp_newton(q);
  return fma(r, fma(-q, r, 1.0), r);
}

/*
 * Inverse iteration, one block per top eigenvalue (vector j belongs to w[n-1-j]): the LU
 * factorisation with partial pivoting of T - lam I and three solves.  The recurrences are
 * sequential, each step a chain of FP64 instructions, so they run from both ends at once (the
 * BABE factorisation, "burn at both ends"): lane 0 of the first warp eliminates columns
 * 0 .. p-1 with rows 0 .. p, lane 0 of the second columns n-1 .. p+2 with rows n-1 .. p+1,
 * p = (n-2)/2; what remains are two rows in the unknowns p and p+1, solved with pivoting, from
 * which both substitute outwards.  The multiplier's reciprocal takes two Newton steps on a
 * 23-bit seed instead of an FP64 division (about 300 clocks of latency against 1,000), and the
 * solves use rows scaled by their pivots' reciprocals, so that a step's chain is one FMA.
 * With in_smem, the factors, the iterate and (during the factorisation) d and e sit in shared
 * memory, 41 n bytes, so that the recurrences wait on shared-memory rather than L2 latency:
 * d is staged where the iterate goes later and e where the second superdiagonal of U is
 * written, each e(i) being read before DU2(i) overwrites it.  Otherwise work holds the
 * factors (per vector 6n doubles) and the iterate stays in Z.
 * n = 5,000: 2.57 ms, of 5.3 from one end; n = 1,000: 0.52 of 1.07.
 * Z [nvec][n] (column-major N x nvec).
 */
__global__ void __launch_bounds__(256)
k_inverse_iteration(const double *__restrict__ d, const double *__restrict__ e, int n,
                    const double *__restrict__ w, int nvec, double tnorm, double *Z, double *work,
                    int in_smem)
{
  __shared__ double red[256];
  __shared__ double mid[2][3]; /* per side: the last row's entries at p, p + 1; its right side */
  extern __shared__ double ii_sm[];
  const int j = blockIdx.x;
  if (j >= nvec) return;
  double *base = in_smem ? ii_sm : work + (int64_t)j * 6 * n;
  double *Dinv = base, *DL = base + n, *DU = base + 2 * n, *DU2 = base + 3 * n;
  double *xg = Z + (int64_t)j * n;
  double *x = in_smem ? base + 4 * n : xg;
  uint8_t *piv = (uint8_t *)(base + 5 * n);
  const double *dd = d, *ee = e;
  if (in_smem) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      x[i] = d[i];
      if (i < n - 1) DU2[i] = e[i];
    }
    __syncthreads();
    dd = x;
    ee = DU2;
  }
  const double lam = w[n - 1 - j];
  const double tiny = DBL_EPSILON * tnorm;
  if (n == 1) {
    if (threadIdx.x == 0) xg[0] = 1.0;
    return;
  }
  const int p = (n - 2) / 2;
  /* this thread's side: row and column k of it are at R(k); E(k) couples k and k + 1 */
  const int side = threadIdx.x >> 5, runs = threadIdx.x == 0 || threadIdx.x == 32;
  const int steps = side ? n - 2 - p : p;
  auto R = [&](int k) { return side ? n - 1 - k : k; };
  auto E = [&](int k) { return ee[side ? n - 2 - k : k]; };
  if (runs) {
    /* dgttrf-style elimination; cur = running diagonal of row k, du = its next entry */
    double cur = dd[R(0)] - lam, du = E(0);
    for (int k = 0; k < steps; ++k) {
      const int i = R(k);
      const double ei = E(k);
      const double dn = dd[R(k + 1)] - lam; /* row k+1: diagonal and next entry */
      const double en = E(k + 1);
      if (fabs(cur) >= fabs(ei)) {
        if (cur == 0.0) cur = tiny;
        const double rc = rcp_full(cur);
        const double f = ei * rc;
        DL[i] = f;
        DU[i] = du;
        DU2[i] = 0.0;
        Dinv[i] = rc;
        piv[i] = 0;
        cur = fma(-f, du, dn);
        du = en;
      } else {
        const double re = rcp_full(ei);
        const double f = cur * re;
        DL[i] = f;
        Dinv[i] = re;
        DU[i] = dn;
        DU2[i] = en;
        piv[i] = 1;
        cur = fma(-f, dn, du);
        du = -f * en;
      }
    }
    mid[side][side] = cur;
    mid[side][1 - side] = du;
  }
  __syncthreads();
  /* rows scaled by their pivots' reciprocals */
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    if (i != p && i != p + 1) {
      DU[i] *= Dinv[i];
      DU2[i] *= Dinv[i];
    }
    x[i] = start_entry(j, i);
  }
  __syncthreads();
  for (int iter = 0; iter < 3; ++iter) {
    double s2 = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s2 += x[i] * x[i];
    s2 = block_sum(s2, red);
    double inv = s2 > 0.0 ? 1.0 / sqrt(s2) : 1.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) x[i] *= inv;
    __syncthreads();
    if (runs) {
      /* inwards: apply the row interchanges and L; the running value in a register */
      double xi = x[R(0)];
      for (int k = 0; k < steps; ++k) {
        const int i = R(k);
        const double xn = x[R(k + 1)];
        if (piv[i] == 0) {
          x[i] = xi;
          xi = fma(-DL[i], xi, xn);
        } else {
          x[i] = xn;
          xi = fma(-DL[i], xn, xi);
        }
      }
      mid[side][2] = xi;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x)
      if (i != p && i != p + 1) x[i] *= Dinv[i];
    if (threadIdx.x == 0) {
      /* the two rows [a b | r], [c d | s] in x(p), x(p+1), with pivoting */
      double a = mid[0][0], b = mid[0][1], r = mid[0][2];
      double c = mid[1][0], dv = mid[1][1], t = mid[1][2];
      if (fabs(c) > fabs(a)) {
        double o = a;
        a = c;
        c = o;
        o = b;
        b = dv;
        dv = o;
        o = r;
        r = t;
        t = o;
      }
      if (a == 0.0) a = tiny;
      const double f = c / a;
      double dd2 = fma(-f, b, dv);
      if (dd2 == 0.0) dd2 = tiny;
      const double x1 = fma(-f, r, t) / dd2;
      x[p + 1] = x1;
      x[p] = fma(-b, x1, r) / a;
    }
    __syncthreads();
    if (runs) {
      /* outwards: x(k) = x'(k) - DU' x(k+1) - DU2' x(k+2) */
      double x1 = x[R(steps)], x2 = x[R(steps + 1)];
      for (int k = steps - 1; k >= 0; --k) {
        const int i = R(k);
        const double v = fma(-DU[i], x1, fma(-DU2[i], x2, x[i]));
        x[i] = v;
        x2 = x1;
        x1 = v;
      }
    }
    __syncthreads();
  }
  double s2 = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s2 += x[i] * x[i];
  s2 = block_sum(s2, red);
  double inv = 1.0 / sqrt(s2);
  for (int i = threadIdx.x; i < n; i += blockDim.x) xg[i] = x[i] * inv;
}

/*
 * Orthonormalisation of the nvec vectors in order.  Inverse iteration leaves them orthogonal to
 * about eps ||T|| / gap; where every product of two is below GS_SMALL, Gram-Schmidt's second-
 * order terms are below rounding, so z_j - sum_{p<j} (z_p . z_j) z_p with the products of the
 * vectors as they are is its result: all products at once (a block each), then every row by
 * itself.  Otherwise one block runs modified Gram-Schmidt, a sum over the block for each pair:
 * 141 us at n = 180 and 1.0 ms at 5,000 (10 and 20 vectors), with the products first 14
 * and 35 us.
 */
#define GS_SMALL 1e-9
#define GS_MAX 64

/* S[p * nvec + j] = z_p . z_j for p <= j: block t for the t-th pair; *far = 1 where one is not
 * small */
__global__ void __launch_bounds__(256)
k_gs_products(const double *__restrict__ Z, int n, int nvec, double *S, int *far)
{
  __shared__ double red[256];
  int j = 0, t = blockIdx.x;
  while (t > j) t -= ++j;
  const double *zp = Z + (int64_t)t * n, *zj = Z + (int64_t)j * n;
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s = fma(zp[i], zj[i], s);
  s = block_sum(s, red);
  if (threadIdx.x == 0) {
    S[t * nvec + j] = s;
    if (!(t == j ? fabs(s - 1.0) < 1e-6 : fabs(s) < GS_SMALL)) *far = 1;
  }
}

__global__ void __launch_bounds__(128)
k_gs_apply(double *Z, int n, int nvec, const double *__restrict__ S, const int *far)
{
  __shared__ double c[GS_MAX * GS_MAX];
  __shared__ double inv[GS_MAX];
  if (*far) return;
  for (int t = threadIdx.x; t < nvec * nvec; t += blockDim.x) c[t] = S[t];
  __syncthreads();
  for (int j = threadIdx.x; j < nvec; j += blockDim.x) inv[j] = 1.0 / sqrt(c[j * nvec + j]);
  __syncthreads();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int j = nvec - 1; j >= 0; --j) { /* the earlier vectors are still as they were */
    double z = Z[(int64_t)j * n + i];
    for (int p = 0; p < j; ++p) z = fma(-c[p * nvec + j], Z[(int64_t)p * n + i], z);
    Z[(int64_t)j * n + i] = z * inv[j];
  }
}

/* modified Gram-Schmidt over the nvec vectors, in order (one block); nothing to do unless *far
 * (NULL: always) */
__global__ void k_mgs(double *Z, int n, int nvec, const int *far)
{
  __shared__ double red[256];
  if (far && !*far) return;
  for (int j = 0; j < nvec; ++j) {
    double *zj = Z + (int64_t)j * n;
    for (int p = 0; p < j; ++p) {
      const double *zp = Z + (int64_t)p * n;
      double s = 0.0;
      for (int i = threadIdx.x; i < n; i += blockDim.x) s += zp[i] * zj[i];
      s = block_sum(s, red);
      for (int i = threadIdx.x; i < n; i += blockDim.x) zj[i] -= s * zp[i];
      __syncthreads();
    }
    double s2 = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s2 += zj[i] * zj[i];
    s2 = block_sum(s2, red);
    double inv = 1.0 / sqrt(s2);
    for (int i = threadIdx.x; i < n; i += blockDim.x) zj[i] *= inv;
    __syncthreads();
  }
}

/*
 * Back-transformation Z := Q Z of the nvec eigenvectors of T (dormtr, side L, lower, no
 * transpose), Q = H(0) H(1) ... H(n-2) with H(i) = I - tau_i v_i v_i^T, v_i(i+1) = 1 and
 * v_i(i+2:n) stored in A(i+2:n, i).  The reflectors are taken WY_B at a time in the compact
 * WY form H(i0)...H(i0+b-1) = I - V T V^T (T upper triangular, LAPACK dlarft's forward
 * recurrence T(j,j) = tau_j, T(0:j,j) = -tau_j T(0:j,0:j) V(:,0:j)^T v_j), last block first,
 * Z := Z - V (T (V^T Z)).  T depends on the reflectors only, so k_wy_tmat builds every
 * block's T at once (one CTA per block) before k_apply_q runs the blocks in order.
 * Float-float arithmetic (about 46 bits) from the FP64 inputs to the FP64 output.
 */
#define WY_B 32
#define WY_THREADS 512
#define WT_THREADS 256
#define WT_ROWS 64

/* entry e of the upper triangle (row-major, k <= c) of a WY_B x WY_B matrix */
__device__ __forceinline__ void wy_upper_entry(int e, int *k, int *c)
{
  int r = 0;
  while (e >= WY_B - r) {
    e -= WY_B - r;
    ++r;
  }
  *k = r;
  *c = r + e;
}

/* Tg [nblk][WY_B][WY_B] (float-float pairs in doubles' storage): block blk's T, from
 * S = V^T V summed over the reflector rows in order (rows staged WT_ROWS at a time) */
__global__ void __launch_bounds__(WT_THREADS)
k_wy_tmat(const double *__restrict__ A, int n, const double *__restrict__ tau, double *Tg)
{
  __shared__ ff2 Vc[WT_ROWS][WY_B + 1];
  __shared__ ff2 Ss[WY_B][WY_B + 1];
  __shared__ ff2 Tm[WY_B][WY_B + 1];
  constexpr int NUP = WY_B * (WY_B + 1) / 2;
  constexpr int SLOTS = (NUP + WT_THREADS - 1) / WT_THREADS;
  const int blk = blockIdx.x, tid = threadIdx.x;
  const int nref = n - 1, i0 = blk * WY_B;
  if (i0 >= nref) return;
  const int nb = nref - i0 < WY_B ? nref - i0 : WY_B;
  const ff2 ZERO = ff_make(0.f, 0.f);
  int ek[SLOTS], ec[SLOTS];
  ff2 acc[SLOTS];
#pragma unroll
  for (int sl = 0; sl < SLOTS; ++sl) {
    const int e = tid + sl * WT_THREADS;
    ek[sl] = ec[sl] = -1;
    if (e < NUP) wy_upper_entry(e, &ek[sl], &ec[sl]);
    acc[sl] = ZERO;
  }
  for (int r0 = i0 + 1; r0 < n; r0 += WT_ROWS) {
    const int nr = n - r0 < WT_ROWS ? n - r0 : WT_ROWS;
    __syncthreads();
    for (int idx = tid; idx < WT_ROWS * WY_B; idx += WT_THREADS) {
      const int k = idx / WT_ROWS, q = idx - k * WT_ROWS, rr = r0 + q, i = i0 + k;
      double v = 0.0;
      if (k < nb && q < nr) v = rr == i + 1 ? 1.0 : (rr > i + 1 ? A[(size_t)i * n + rr] : 0.0);
      Vc[q][k] = ff_from_double(v);
    }
    __syncthreads();
#pragma unroll
    for (int sl = 0; sl < SLOTS; ++sl) {
      if (ek[sl] < 0) continue;
      ff2 t = acc[sl];
      for (int q = 0; q < nr; ++q) t = ff_fma(Vc[q][ek[sl]], Vc[q][ec[sl]], t);
      acc[sl] = t;
    }
  }
#pragma unroll
  for (int sl = 0; sl < SLOTS; ++sl)
    if (ek[sl] >= 0) Ss[ek[sl]][ec[sl]] = acc[sl];
  __syncthreads();
  /* T (dlarft forward, columnwise): one warp, column j after column j-1 */
  if (tid < 32) {
    for (int j = 0; j < WY_B; ++j) {
      const ff2 tj = j < nb ? ff_from_double(tau[i0 + j]) : ZERO;
      ff2 t = ZERO;
      if (tid < j) t = ff_neg(ff_mul(tj, Ss[tid][j]));
      /* T(0:j, j) = T(0:j, 0:j) t: row tid of the upper triangle */
      ff2 a = ZERO;
      for (int l = 0; l < j; ++l) {
        const ff2 tl = ff_make(__shfl_sync(0xFFFFFFFFu, t.h, l), __shfl_sync(0xFFFFFFFFu, t.l, l));
        if (tid <= l) a = ff_fma(Tm[tid][l], tl, a);
      }
      if (tid < j) Tm[tid][j] = a;
      if (tid == j) Tm[j][j] = tj;
      if (tid > j) Tm[tid][j] = ZERO;
      __syncwarp();
    }
  }
  __syncthreads();
  double *T = Tg + (size_t)blk * WY_B * WY_B;
  for (int idx = tid; idx < WY_B * WY_B; idx += WT_THREADS)
    ff_store(T + idx, Tm[idx / WY_B][idx % WY_B]);
}

/*
 * One cooperative launch, one CTA per SM with a fixed slab of rows: per block of reflectors
 * each CTA forms its rows' share of V^T Z (partials), a grid barrier, the partials are summed
 * in fixed order (entries spread over the CTAs), a second barrier, then every CTA forms
 * W = T (V^T Z) with the block's T from k_wy_tmat and updates its own rows.  Bounded grid
 * barriers report through err.
 */
__global__ void __launch_bounds__(WY_THREADS, 1)
k_apply_q(const double *__restrict__ A, int n, const double *__restrict__ Tg, double *Z, int nvec,
          double *part, double *S, unsigned *bar, int *err)
{
  /* all products in float-float on the FP32 pipe (GB300's FP64 pipe issues ~2 FMAs per
   * clock per SM); part and S hold float-float pairs in doubles' storage */
  extern __shared__ double wsm[];
  const int G = gridDim.x, b = blockIdx.x, tid = threadIdx.x;
  const int rpb = (n + G - 1) / G;
  const int R0 = b * rpb < n ? b * rpb : n, R1 = R0 + rpb < n ? R0 + rpb : n;
  const int nent = WY_B * nvec;
  ff2 *Vs = reinterpret_cast<ff2 *>(wsm);    /* [rpb][WY_B]  the CTA's rows of V */
  ff2 *Zs = Vs + (size_t)rpb * WY_B;         /* [rpb][nvec]  its rows of Z */
  ff2 *Ss = Zs + (size_t)rpb * nvec;         /* [WY_B][nvec] V^T Z */
  ff2 *Tm = Ss + (size_t)nent;               /* [WY_B][WY_B] */
  ff2 *Wm = Tm + WY_B * WY_B;                /* [WY_B][nvec] */
  const ff2 ZERO = ff_make(0.f, 0.f);
  unsigned target = 0;
  const int nr = R1 - R0;
  for (int idx = tid; idx < nr * nvec; idx += WY_THREADS) {
    const int c = idx / nr, r = idx - c * nr;
    Zs[r * nvec + c] = ff_from_double(Z[(size_t)c * n + R0 + r]);
  }
  const int nref = n - 1;
  const int nblk = (nref + WY_B - 1) / WY_B;
  for (int blk = nblk - 1; blk >= 0; --blk) {
    const int i0 = blk * WY_B, nb = nref - i0 < WY_B ? nref - i0 : WY_B;
    const int r0 = R0 > i0 + 1 ? R0 : i0 + 1;  /* V is zero above row i0+1 */
    const int m = r0 < R1 ? R1 - r0 : 0;
    __syncthreads();
    for (int idx = tid; idx < m * WY_B; idx += WY_THREADS) {
      const int k = idx / m, rr = r0 + (idx - k * m);
      const int i = i0 + k;
      double v = 0.0;
      if (k < nb) v = rr == i + 1 ? 1.0 : (rr > i + 1 ? A[(size_t)i * n + rr] : 0.0);
      Vs[(rr - R0) * WY_B + k] = ff_from_double(v);
    }
    __syncthreads();
    /* partial V^T Z over the CTA's rows */
    for (int e = tid; e < nent; e += WY_THREADS) {
      const int k = e / nvec, c = e - k * nvec;
      ff2 acc = ZERO;
      for (int rr = r0 - R0; rr < R1 - R0; ++rr)
        acc = ff_fma(Vs[rr * WY_B + k], Zs[rr * nvec + c], acc);
      ff_store(part + (size_t)b * nent + e, acc);
    }
    target += G;
    if (!tr_grid_sync(bar, target, err)) return;
    /* one warp per entry: lanes sum every 32nd partial, then a fixed shuffle tree */
    {
      const int lane = tid & 31, gw = b * (WY_THREADS / 32) + (tid >> 5);
      for (int e = gw; e < nent; e += G * (WY_THREADS / 32)) {
        ff2 acc = ZERO;
        for (int g = lane; g < G; g += 32) acc = ff_add(acc, ff_load(part + (size_t)g * nent + e));
        for (int o = 16; o; o >>= 1) acc = ff_add(acc, ff_shfl_xor(acc, o));
        if (lane == 0) ff_store(S + e, acc);
      }
    }
    target += G;
    if (!tr_grid_sync(bar, target, err)) return;
    if (m == 0) continue;
    for (int e = tid; e < nent; e += WY_THREADS) Ss[e] = ff_load(S + e);
    for (int e = tid; e < WY_B * WY_B; e += WY_THREADS)
      Tm[e] = ff_load(Tg + (size_t)blk * WY_B * WY_B + e);
    __syncthreads();
    /* W = T (V^T Z) */
    for (int e = tid; e < WY_B * nvec; e += WY_THREADS) {
      const int k = e / nvec, c = e - k * nvec;
      ff2 acc = ZERO;
      for (int l = k; l < WY_B; ++l) acc = ff_fma(Tm[k * WY_B + l], Ss[l * nvec + c], acc);
      Wm[e] = acc;
    }
    __syncthreads();
    /* Z(rows) -= V(rows) W */
    for (int idx = tid; idx < m * nvec; idx += WY_THREADS) {
      const int rr = (r0 - R0) + idx / nvec, c = idx % nvec;
      ff2 acc = ZERO;
      for (int k = 0; k < WY_B; ++k) acc = ff_fma(Vs[rr * WY_B + k], Wm[k * nvec + c], acc);
      Zs[rr * nvec + c] = ff_add(Zs[rr * nvec + c], ff_neg(acc));
    }
  }
  __syncthreads();
  for (int idx = tid; idx < nr * nvec; idx += WY_THREADS) {
    const int c = idx / nr, r = idx - c * nr;
    Z[(size_t)c * n + R0 + r] = ff_to_double(Zs[r * nvec + c]);
  }
}

/* evals_desc[i] = w[n-1-i] */
__global__ void k_reverse(const double *w, double *out, int n)
{
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    out[i] = w[n - 1 - i];
}

/* the pr x pc block grid of k_tridiag_tiled: the largest pr * pc <= G with pr <= pc, both at
 * most TT_MAXG (ties: the smaller pr + pc, so that an index block has fewer parts) */
static void tt_grid(int G, int *pr, int *pc)
{
  int best = 0;
  *pr = *pc = 0;
  for (int r = 1; r * r <= G; ++r) {
    const int c = G / r;
    if (r > TT_MAXG || c > TT_MAXG) continue;
    if (r * c > best || (r * c == best && r + c < *pr + *pc)) {
      best = r * c;
      *pr = r;
      *pc = c;
    }
  }
}

/* the assignment tables of k_tridiag_tiled for every first active tile index J0 (row J0 of
 * rgt [nt][nt] and cgt [nt][nt*TT_UPT]): the active tile rows go to the pr row groups longest
 * first, each to the group with the fewest parts so far (ties: the lower group); then the
 * column units, longest first, each to the column group whose largest block part count grows
 * least (ties: the smaller growth of the sum of squares, then the lower group).  Also the
 * bounds of a block's tile rows, column units and parts over all J0. */
static void tt_tables(int nt, int pr, int pc, std::vector<unsigned char> &rgt,
                      std::vector<unsigned char> &cgt, int *maxr, int *maxc, int *maxi)
{
  const int nu = nt * TT_UPT;
  rgt.assign((size_t)nt * nt, 0);
  cgt.assign((size_t)nt * nu, 0);
  std::vector<int> sum((size_t)pr), L((size_t)pr * pc), suf((size_t)(nt + 1) * pr),
      nrow((size_t)pr), ncol((size_t)pc);
  int mr = 1, mc = 1, mi = 1;
  for (int J0 = 0; J0 < nt; ++J0) {
    unsigned char *rg = &rgt[(size_t)J0 * nt], *cg = &cgt[(size_t)J0 * nu];
    std::fill(sum.begin(), sum.end(), 0);
    for (int I = nt - 1; I >= J0; --I) {
      int best = 0;
      for (int g = 1; g < pr; ++g)
        if (sum[g] < sum[best]) best = g;
      rg[I] = (unsigned char)best;
      sum[best] += TT_UPT * (I - J0 + 1);
    }
    /* suf[J][a]: active tile rows I >= J in row group a (the parts of a unit of tile column J) */
    for (int g = 0; g < pr; ++g) suf[(size_t)nt * pr + g] = 0;
    for (int J = nt - 1; J >= J0; --J) {
      for (int g = 0; g < pr; ++g) suf[(size_t)J * pr + g] = suf[(size_t)(J + 1) * pr + g];
      ++suf[(size_t)J * pr + rg[J]];
    }
    std::fill(L.begin(), L.end(), 0);
    std::fill(ncol.begin(), ncol.end(), 0);
    for (int u = J0 * TT_UPT; u < nu; ++u) {
      const int *v = &suf[(size_t)(u / TT_UPT) * pr];
      int best = 0;
      long long bmax = -1, bsq = 0;
      for (int g = 0; g < pc; ++g) {
        long long mx = 0, sq = 0;
        for (int a = 0; a < pr; ++a) {
          const long long l = L[(size_t)a * pc + g];
          mx = std::max(mx, l + v[a]);
          sq += 2 * l * v[a] + (long long)v[a] * v[a];
        }
        if (bmax < 0 || mx < bmax || (mx == bmax && sq < bsq)) {
          bmax = mx;
          bsq = sq;
          best = g;
        }
      }
      cg[u] = (unsigned char)best;
      ++ncol[best];
      for (int a = 0; a < pr; ++a) L[(size_t)a * pc + best] += v[a];
    }
    std::fill(nrow.begin(), nrow.end(), 0);
    for (int I = J0; I < nt; ++I) ++nrow[rg[I]];
    for (int g = 0; g < pr; ++g) mr = std::max(mr, nrow[g]);
    for (int g = 0; g < pc; ++g) mc = std::max(mc, ncol[g]);
    for (size_t k = 0; k < L.size(); ++k) mi = std::max(mi, L[k]);
  }
  *maxr = mr;
  *maxc = mc;
  *maxi = mi;
}

/* dynamic shared memory of tr_smem_steps for trailing order m on G blocks */
static size_t tr_smem_bytes(int m, int G)
{
  return sizeof(double) * (size_t)(3 + (m + G - 1) / G) * (size_t)((m + 1) & ~1);
}
/* blocks for trailing order m: every block reads all of y and the column in each step, which
 * costs more the more blocks ask (about 1,900 clocks for 16 of them, 4,000 for 64, 6,700 for
 * 152 at m = 1,000), so one for 15 columns, but up to ten for small orders, or what shared memory
 * needs (m = 180: 0.515 ms on 12, 0.53 on 18, 0.61 on 6; m = 700: 3.10 on 50, 3.32 on 72; m = 1,000:
 * 5.13 on 64, 5.28 on 100, 5.83 on 40) */
static int tr_smem_blocks(int m, int G)
{
  int Gm = std::min(G, std::max(std::max(m / 15, std::min(m / 8, 10)), (m + 31) / 32));
  while (Gm < G && tr_smem_bytes(m, Gm) > 200 * 1024) ++Gm;
  return Gm;
}
static int tr_smem_order(int G)
{
  int m = std::min(32 * G, TR_SMEM_NT * TR_SMEM_RPT);
  while (m > 1 && tr_smem_bytes(m, G) > 200 * 1024) --m;
  return m;
}

int gp_eig_tridiag(gp_ctx *ctx, int32_t n, int32_t nvec, double *d_evals_desc, double *d_vecs)
{
  return gp_eig_sym(ctx, ctx->d_xtx, n, nvec, d_evals_desc, d_vecs);
}

/*
 * Eigenpairs of the symmetric n x n device matrix A (overwritten): d_evals_desc [n] all
 * eigenvalues descending, d_vecs [nvec][n] top eigenvectors (descending).  Only this
 * library's kernels run unless the matrix is too large for the cooperative kernels' shared
 * memory (order above 8,533, or a back-transformation slab that does not fit), where cuSOLVER's
 * sytrd / ormtr take over.
 */
int gp_eig_sym(gp_ctx *ctx, double *A_in, int32_t n, int32_t nvec, double *d_evals_desc,
               double *d_vecs)
{
  cusolverDnHandle_t h = ctx->solver;
  int lwork = 0, lwork2 = 0;
  /* GP_EIG_TIMING=1 prints the device time of each stage to stderr */
  const char *tenv = getenv("GP_EIG_TIMING");
  const int timing = tenv && tenv[0] == '1';
  cudaEvent_t ev[7];
  if (timing)
    for (int i = 0; i < 7; ++i) cudaEventCreate(&ev[i]);
#define GP_EIG_MARK(i) \
  if (timing) cudaEventRecord(ev[i], ctx->stream)
  /* scratch: d, e, tau, e2, w, work(sytrd), inverse-iteration work, info */
  int nv = nvec > 0 ? nvec : 1;
  size_t nd = (size_t)n;
  const size_t G = (size_t)ctx->num_sms;
  const size_t nwy = (nd + WY_B - 1) / WY_B;
  /* cuSOLVER workspaces only where its fallbacks can run: the tridiagonalisation above the
   * cooperative kernel's shared memory, or a back-transformation slab that does not fit */
  const size_t rpb0 = (nd + G - 1) / G;
  const size_t q_smem0 = sizeof(double) * (rpb0 * (WY_B + (size_t)nv) + (size_t)WY_B * nv +
                                           WY_B * WY_B + (size_t)WY_B * nv);
  const char *sy_env = getenv("GP_EIG_CUSOLVER_SYTRD"), *or_env = getenv("GP_EIG_CUSOLVER_ORMTR");
  const int may_fallback = n < 2 || 24 * nd > 200 * 1024 || (nvec > 0 && q_smem0 > 200 * 1024) ||
                           (sy_env && sy_env[0] == '1') || (or_env && or_env[0] == '1');
  if (may_fallback) {
    if (cusolverDnDsytrd_bufferSize(h, CUBLAS_FILL_MODE_LOWER, n, A_in, n, NULL, NULL, NULL,
                                    &lwork) != CUSOLVER_STATUS_SUCCESS)
      return gp_fail(ctx, GP_ERR_SOLVER, "cusolverDnDsytrd_bufferSize failed");
    if (cusolverDnDormtr_bufferSize(h, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_LOWER, CUBLAS_OP_N, n,
                                    nv, A_in, n, NULL, d_vecs, n, &lwork2) !=
        CUSOLVER_STATUS_SUCCESS)
      return gp_fail(ctx, GP_ERR_SOLVER, "cusolverDnDormtr_bufferSize failed");
  }
  int lw = lwork > lwork2 ? lwork : lwork2;
  /* partials + sums of k_apply_q, then the blocks' T from k_wy_tmat */
  const size_t qpart_n = (G + 1) * (size_t)WY_B * nv + nwy * WY_B * WY_B;
  size_t bytes = sizeof(double) * (18 * nd + 2 * G + (size_t)lw + 6 * nd * nv + 80 + qpart_n) +
                 sizeof(int) * 64;
  double *base;
  int rc = gp_scratch(ctx, bytes, (void **)&base);
  if (rc) return rc;
  double *d = base, *e = d + nd, *tau = e + nd, *e2 = tau + nd, *w = e2 + nd;
  double *wbuf = w + nd, *ybuf = wbuf + nd, *vbuf = ybuf + 2 * nd;
  /* the shared-memory steps' tagged y and columns, [2][n] of 16 bytes each (d.. + 10 nd: 16-byte
   * aligned in the 256-byte aligned scratch) */
  uint4 *ytag = (uint4 *)(base + 10 * nd);
  double *parts = base + 18 * nd;
  unsigned *bar = (unsigned *)(parts + 2 * G);
  double *ws = parts + 2 * G + 16, *iw = ws + lw; /* 16 doubles: barrier words + phase timers */
  int *d_info = (int *)(iw + 6 * nd * nv + 8);
  double *qpart = iw + 6 * nd * nv + 16; /* after d_info's 8 doubles (64 ints) */
  /* the cooperative tridiagonalisation (k_tridiag) unless GP_EIG_CUSOLVER_SYTRD=1, the
   * vectors do not fit shared memory or the device cannot co-schedule one block per SM */
  const char *senv = getenv("GP_EIG_CUSOLVER_SYTRD");
  /* the trailing order from which the matrix stays in shared memory (GP_TRIDIAG_SMEM caps it) */
  const char *m_env = getenv("GP_TRIDIAG_SMEM");
  int m_smem = tr_smem_order((int)G);
  if (m_env && m_env[0]) m_smem = std::max(1, std::min(m_smem, atoi(m_env)));
  const size_t tr_smem = 24 * nd;
  int coop = !(senv && senv[0] == '1') && n >= 2 && tr_smem <= 200 * 1024;
  if (coop) {
    int dev_coop = 0, per_sm = 0;
    cudaDeviceGetAttribute(&dev_coop, cudaDevAttrCooperativeLaunch, ctx->device);
    GP_CUDA(ctx, gp_allow_smem(ctx, (const void *)k_tridiag));
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tridiag, TR_THREADS, tr_smem);
    coop = dev_coop && per_sm >= 1;
  }
  /* the lower-triangle tiled variant (k_tridiag_tiled) where its shared memory fits, unless
   * GP_TRIDIAG_TILED=0; the whole-matrix k_tridiag otherwise */
  const char *tt_env = getenv("GP_TRIDIAG_TILED");
  const int nt = (n + TT - 1) / TT;
  int tt_pr = 0, tt_pc = 0, tt_maxr = 0, tt_maxc = 0, tt_maxi = 0;
  size_t tt_smem = 0;
  /* the tiled steps run until the rest fits the shared memories (GP_TRIDIAG_SWITCH: until the
   * trailing order is at most its value) */
  const char *sw_env = getenv("GP_TRIDIAG_SWITCH");
  const int tt_switch = sw_env && sw_env[0] ? std::max(1, atoi(sw_env)) : n;
  const int tt_cs = std::max(n - m_smem, n - 1 - tt_switch); /* first step after the tiled ones */
  int tiled = !(senv && senv[0] == '1') && !(tt_env && tt_env[0] == '0') && tt_cs >= 1 &&
              tr_smem <= 200 * 1024;
  if (tiled) {
    tt_grid((int)G, &tt_pr, &tt_pc);
    tiled = tt_pr >= 1 && tt_pc >= 1;
  }
  if (tiled && !(ctx->d_tt && ctx->tt_n == n && ctx->tt_G == (int)G)) {
    /* the assignment tables, once per order and grid */
    std::vector<unsigned char> rgt, cgt;
    tt_tables(nt, tt_pr, tt_pc, rgt, cgt, &ctx->tt_maxr, &ctx->tt_maxc, &ctx->tt_maxi);
    ctx->tt_n = 0;
    int rc3 = gp_realloc(ctx, (void **)&ctx->d_tt, rgt.size() + cgt.size());
    if (rc3) return rc3;
    GP_CUDA(ctx, gp_memcpy(ctx, ctx->d_tt, rgt.data(), rgt.size(), cudaMemcpyHostToDevice,
                           ctx->stream));
    GP_CUDA(ctx, gp_memcpy(ctx, ctx->d_tt + rgt.size(), cgt.data(), cgt.size(),
                           cudaMemcpyHostToDevice, ctx->stream));
    GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    ctx->tt_n = n;
    ctx->tt_G = (int)G;
  }
  if (tiled) {
    tt_maxr = ctx->tt_maxr;
    tt_maxc = ctx->tt_maxc;
    tt_maxi = ctx->tt_maxi;
    tt_smem = tt_smem_bytes(nt, tt_maxr, tt_maxc, tt_maxi);
    tiled = tt_smem <= 226 * 1024; /* 227 KB less the static part */
  }
  if (tiled) {
    int dev_coop = 0, per_sm = 0;
    cudaDeviceGetAttribute(&dev_coop, cudaDevAttrCooperativeLaunch, ctx->device);
    tiled = dev_coop && gp_allow_smem(ctx, (const void *)k_tridiag_tiled) == cudaSuccess;
    if (tiled) {
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tridiag_tiled, TT_THREADS,
                                                    tt_smem);
      tiled = per_sm >= 1;
    }
    (void)cudaGetLastError();
  }
  if (tiled) coop = 1;
  if (!coop && !may_fallback)
    return gp_fail(ctx, GP_ERR_CUDA, "eigensolve: the cooperative tridiagonalisation cannot run");
  GP_EIG_MARK(0);
  int info = 0;
  if (coop) {
    int *d_err = ctx->d_err;
    double *A = A_in, *pd2 = parts;
    int nn = n;
    /* the first steps run in tiles or in L2, those of the last m_smem rows in shared memory */
    int c_end = tiled ? tt_cs : std::max(0, n - m_smem);
    tr_state *state = (tr_state *)((char *)bar + 80);
    /* x (of k_tridiag, or v of the tiled steps) and y of step c_end - 1 */
    double *xlast = (c_end & 1) ? vbuf : wbuf, *ylast = ybuf + (int64_t)((c_end + 1) & 1) * n;
    unsigned long long *phase = NULL;
    GP_CUDA(ctx, cudaMemsetAsync(d_err, 0, sizeof(int), ctx->stream));
    GP_CUDA(ctx, cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), ctx->stream));
    GP_CUDA(ctx, cudaMemsetAsync(ytag, 0, sizeof(uint4) * 4 * nd, ctx->stream));
    if (timing) {
      phase = (unsigned long long *)(bar + 8);
      GP_CUDA(ctx, cudaMemsetAsync(phase, 0, 5 * sizeof(unsigned long long), ctx->stream));
    }
    if (tiled) {
      const int64_t ntiles = (int64_t)nt * (nt + 1) / 2;
      const size_t tile_d = (size_t)ntiles * TT * TT;
      const size_t part_d = (size_t)(tt_pr + tt_pc) * nt * TT; /* prow + pcol */
      const size_t tags = 4 * (size_t)nt * TT + 2 * (size_t)nt; /* y, columns, dots, twice */
      const size_t tri_bytes = sizeof(double) * (tile_d + part_d) + sizeof(uint4) * tags +
                               sizeof(unsigned) * (size_t)nt;
      int rc2 = gp_realloc(ctx, (void **)&ctx->d_tri, tri_bytes);
      if (rc2) return rc2;
      double *Tm = ctx->d_tri, *prow = Tm + tile_d, *pcol = prow + (size_t)nt * tt_pc * TT;
      uint4 *yt = (uint4 *)(pcol + (size_t)nt * tt_pr * TT), *ct = yt + 2 * (size_t)nt * TT;
      uint4 *dott = ct + 2 * (size_t)nt * TT;
      unsigned *kcnt = (unsigned *)(dott + 2 * (size_t)nt);
      GP_CUDA(ctx, cudaMemsetAsync(yt, 0, sizeof(uint4) * tags + sizeof(unsigned) * (size_t)nt,
                                   ctx->stream));
      int blocks = (int)std::min<int64_t>(ntiles, (int64_t)ctx->num_sms * 8);
      k_tri_to_tiles<<<blocks, 256, 0, ctx->stream>>>(A_in, n, nt, Tm);
      GP_LAUNCH_CHECK(ctx, "k_tri_to_tiles");
      int nt_ = nt, cs = tt_cs;
      const unsigned char *rgt = ctx->d_tt, *cgt = ctx->d_tt + (size_t)nt * nt;
      void *args[] = {&A,       &Tm,   &nn,    &nt_,   &tt_pr, &tt_pc, &tt_maxr, &tt_maxc,
                      &tt_maxi, &cs,   &rgt,   &cgt,   &d,     &e,     &tau,
                      &yt,      &ct,   &dott,  &xlast, &ylast, &prow,  &pcol,    &kcnt,
                      &bar,     &d_err, &phase, &state};
      GP_CUDA(ctx, cudaEventRecord(ctx->ev_tr0, ctx->stream));
      GP_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)k_tridiag_tiled, dim3((unsigned)G),
                                               dim3(TT_THREADS), args, tt_smem, ctx->stream));
      ctx->launches++;
    } else {
      int64_t tot = (int64_t)n * n;
      int blocks = (int)((tot + 255) / 256);
      if (blocks > ctx->num_sms * 16) blocks = ctx->num_sms * 16;
      k_tri_to_ff<<<blocks, 256, 0, ctx->stream>>>(A, n);
      GP_LAUNCH_CHECK(ctx, "k_tri_to_ff");
      GP_CUDA(ctx, cudaEventRecord(ctx->ev_tr0, ctx->stream));
      if (c_end > 0) {
        void *args[] = {&A,    &nn,   &c_end, &d,     &e,   &tau,   &vbuf,
                        &wbuf, &ybuf, &pd2,   &state, &bar, &d_err, &phase};
        GP_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)k_tridiag, dim3((unsigned)G),
                                                 dim3(TR_THREADS), args, tr_smem, ctx->stream));
        ctx->launches++;
      }
    }
    {
      const int m = n - c_end;
      const void *f = m <= TR_SMALL_ORDER   ? (const void *)k_tridiag_smem<TR_SMEM_NT, 2>
                      : m <= 4 * TR_SMEM_NT ? (const void *)k_tridiag_smem<TR_SMEM_NT, 4>
                                            : (const void *)k_tridiag_smem<TR_SMEM_NT, TR_SMEM_RPT>;
      const int Gm = tr_smem_blocks(m, (int)G);
      const double *xp = xlast, *yp = ylast;
      uint4 *ctag = ytag + 2 * nd;
      unsigned *bar_s = bar + 1;
      void *args[] = {&A,  &nn,   &c_end, &d,     &e,     &tau,  &xp,
                      &yp, &ytag, &ctag,  &state, &bar_s, &d_err};
      GP_CUDA(ctx, gp_allow_smem(ctx, f));
      GP_CUDA(ctx, cudaLaunchCooperativeKernel(f, dim3((unsigned)Gm), dim3(TR_SMEM_NT), args,
                                               tr_smem_bytes(m, Gm), ctx->stream));
      ctx->launches++;
    }
    GP_CUDA(ctx, cudaEventRecord(ctx->ev_tr1, ctx->stream));
    int herr = 0;
    GP_CUDA(ctx, gp_memcpy(ctx, &herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    if (herr == TR_ERR_LISTS)
      return gp_fail(ctx, GP_ERR_CUDA, "tiled tridiagonalisation: a block's tile lists overflowed");
    if (herr == TR_ERR_WAIT)
      return gp_fail(ctx, GP_ERR_TIMEOUT, "tiled tridiagonalisation: an index block's parts "
                                          "did not arrive in time");
    if (herr) return gp_fail(ctx, GP_ERR_TIMEOUT, "tridiagonalisation grid barrier timed out");
    float tms = 0.f;
    GP_CUDA(ctx, cudaEventElapsedTime(&tms, ctx->ev_tr0, ctx->ev_tr1));
    if (A_in == ctx->d_xtx) { /* the Gram's eigensolve: its time is reported */
      ctx->tridiag_ms = tms;
      ctx->tridiag_n = n;
    }
    if (timing) {
      unsigned long long hp[5];
      cudaMemcpy(hp, phase, sizeof hp, cudaMemcpyDeviceToHost);
      fprintf(stderr,
              "tridiagonal n=%d (block 0), steps up to %d: A %.1f ms, B %.1f (first 30%% of "
              "steps %.1f), barrier %.1f\n",
              n, c_end, hp[0] * 1e-6, (hp[1] + hp[2]) * 1e-6, hp[2] * 1e-6, hp[4] * 1e-6);
    }
  } else {
    ctx->tridiag_ms = 0.0;
    ctx->tridiag_n = n;
    if (cusolverDnDsytrd(h, CUBLAS_FILL_MODE_LOWER, n, A_in, n, d, e, tau, ws, lw,
                         d_info) != CUSOLVER_STATUS_SUCCESS)
      return gp_fail(ctx, GP_ERR_SOLVER, "cusolverDnDsytrd failed to launch");
    GP_CUDA(ctx, gp_memcpy(ctx, &info, d_info, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  }
  GP_EIG_MARK(1);
  /* Gershgorin bounds and the pivot guard need d, e on the host (2n doubles) */
  std::vector<double> hd(nd), he(nd > 1 ? nd - 1 : 1);
  GP_CUDA(ctx, gp_memcpy(ctx, hd.data(), d, sizeof(double) * nd, cudaMemcpyDeviceToHost, ctx->stream));
  if (n > 1)
    GP_CUDA(ctx, gp_memcpy(ctx, he.data(), e, sizeof(double) * (nd - 1), cudaMemcpyDeviceToHost,
                           ctx->stream));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (info != 0) return gp_fail(ctx, GP_ERR_SOLVER, "sytrd info = %d", info);
  double gl = hd[0], gu = hd[0], tnorm = 0.0, emax2 = 0.0;
  std::vector<double> he2(nd > 1 ? nd - 1 : 1);
  for (int i = 0; i < n; ++i) {
    double r = (i > 0 ? fabs(he[(size_t)i - 1]) : 0.0) + (i < n - 1 ? fabs(he[(size_t)i]) : 0.0);
    gl = fmin(gl, hd[(size_t)i] - r);
    gu = fmax(gu, hd[(size_t)i] + r);
    tnorm = fmax(tnorm, fabs(hd[(size_t)i]) + r);
    if (i < n - 1) {
      he2[(size_t)i] = he[(size_t)i] * he[(size_t)i];
      emax2 = fmax(emax2, he2[(size_t)i]);
    }
  }
  double span = gu - gl;
  gl -= 2.0 * DBL_EPSILON * tnorm * n + DBL_MIN;
  gu += 2.0 * DBL_EPSILON * tnorm * n + DBL_MIN;
  (void)span;
  /* the pivot guard stays inside FP32's exponent range (the reciprocal starts in FP32) */
  double pivmin = fmax(DBL_MIN * fmax(1.0, emax2), 1e-30 * fmax(tnorm, 1e-300));
  if (n > 1)
    GP_CUDA(ctx, gp_memcpy(ctx, e2, he2.data(), sizeof(double) * (nd - 1), cudaMemcpyHostToDevice,
                           ctx->stream));
  GP_EIG_MARK(2);
  {
    /* GP_EIG_NO_FF=1 selects the path without the float-float phase (as for N > 6,400) */
    const char *ffenv = getenv("GP_EIG_NO_FF");
    size_t smem = (size_t)32 * (size_t)n;
    int use_smem = 2;
    if (smem > 200 * 1024 || (ffenv && ffenv[0] == '1')) {
      smem = (size_t)24 * (size_t)n;
      use_smem = smem <= 200 * 1024 ? 1 : 0;
    }
    const int warps = ctx->num_sms * 4;
    int epw = (n + warps - 1) / warps;
    if (epw > 32) epw = 32;
    const int P = 32 / epw;
    const int nwarps = (n + epw - 1) / epw;
    const int blocks = (nwarps + 3) / 4;
    /* Half of the last FP64 bracket is the error, and how wide it gets depends on the points a step
     * has: with a limit of 1e-13 ||T|| the largest error over all eigenvalues was 3.5e-14 of the norm
     * at 2,500 and 5.1e-14 at 3,600 and 5,000, with 3e-14 it is 0.8e-14, 0.9e-14 and 1.3e-14 for
     * 3.5 ms of 2.9, 5.3 of 4.6 and 9.2 of 8.2 (orders to 1,800 are the same).  With fewer than three
     * points (orders above 6,080) a step costs more, 14.7 ms of 13.4 at 6,200, for less: 1e-13 there,
     * 4.9e-14 */
    const double tol = (P >= 3 ? 3e-14 : 1e-13) * tnorm;
    if (use_smem)
      GP_CUDA(ctx, gp_allow_smem(ctx, (const void *)k_multisect));
    k_multisect<<<blocks, 128, use_smem ? smem : 0, ctx->stream>>>(d, e2, n, gl, gu, tnorm, pivmin,
                                                                   tol, use_smem, epw, P, w);
    GP_LAUNCH_CHECK(ctx, "k_multisect");
  }
  k_reverse<<<(n + 255) / 256, 256, 0, ctx->stream>>>(w, d_evals_desc, n);
  GP_LAUNCH_CHECK(ctx, "k_reverse");
  GP_EIG_MARK(3);
  if (nvec > 0) {
    /* factors, iterate and byte pivots: 41 n bytes */
    const size_t ii_smem = (size_t)n * (5 * sizeof(double) + 1) + 16;
    int smem_optin = 0;
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device);
    /* GP_EIG_II_GLOBAL=1 selects the global-memory path (as for N > 5,600) */
    const char *iienv = getenv("GP_EIG_II_GLOBAL");
    const int ii_in_smem = ii_smem + 2048 <= (size_t)smem_optin && !(iienv && iienv[0] == '1');
    if (ii_in_smem)
      GP_CUDA(ctx, gp_allow_smem(ctx, (const void *)k_inverse_iteration));
    k_inverse_iteration<<<nvec, 256, ii_in_smem ? ii_smem : 0, ctx->stream>>>(
        d, e, n, w, nvec, tnorm, d_vecs, iw, ii_in_smem);
    GP_LAUNCH_CHECK(ctx, "k_inverse_iteration");
    GP_EIG_MARK(5);
    int *far = NULL;
    if (nvec <= GS_MAX) {
      double *S = iw; /* the factors' room: 6 n nvec doubles, nvec <= n */
      far = (int *)(iw + (size_t)nvec * nvec);
      GP_CUDA(ctx, cudaMemsetAsync(far, 0, sizeof(int), ctx->stream));
      k_gs_products<<<nvec * (nvec + 1) / 2, 256, 0, ctx->stream>>>(d_vecs, n, nvec, S, far);
      GP_LAUNCH_CHECK(ctx, "k_gs_products");
      k_gs_apply<<<(n + 127) / 128, 128, 0, ctx->stream>>>(d_vecs, n, nvec, S, far);
      GP_LAUNCH_CHECK(ctx, "k_gs_apply");
    }
    k_mgs<<<1, 1024, 0, ctx->stream>>>(d_vecs, n, nvec, far);
    GP_LAUNCH_CHECK(ctx, "k_mgs");
    GP_EIG_MARK(6);
    /* Z := Q Z: the cooperative WY kernel when its row slab fits shared memory, else
     * cusolverDnDormtr (GP_EIG_CUSOLVER_ORMTR=1 forces the latter) */
    const char *oenv = getenv("GP_EIG_CUSOLVER_ORMTR");
    const int Gq = ctx->num_sms;
    const size_t rpb = ((size_t)n + Gq - 1) / Gq;
    const size_t nent = (size_t)WY_B * nvec;
    const size_t q_smem = sizeof(double) * (rpb * (WY_B + nvec) + nent + WY_B * WY_B + (size_t)WY_B * nvec);
    int qcoop = !(oenv && oenv[0] == '1') && n >= 2 && q_smem <= 200 * 1024 &&
                qpart != NULL;
    if (qcoop) {
      int dev_coop = 0, per_sm = 0;
      cudaDeviceGetAttribute(&dev_coop, cudaDevAttrCooperativeLaunch, ctx->device);
      GP_CUDA(ctx, gp_allow_smem(ctx, (const void *)k_apply_q));
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_apply_q, WY_THREADS, q_smem);
      qcoop = dev_coop && per_sm >= 1;
    }
    if (!qcoop && !may_fallback)
      return gp_fail(ctx, GP_ERR_CUDA, "eigensolve: the cooperative back-transformation cannot run");
    if (qcoop) {
      unsigned *qbar = bar + 4;
      int *d_err = ctx->d_err;
      GP_CUDA(ctx, cudaMemsetAsync(d_err, 0, sizeof(int), ctx->stream));
      GP_CUDA(ctx, cudaMemsetAsync(qbar, 0, sizeof(unsigned), ctx->stream));
      const double *Aq = A_in;
      double *Sq = qpart + (size_t)Gq * nent;
      double *Tg = qpart + (size_t)(Gq + 1) * nent;
      const int nwyb = (n - 1 + WY_B - 1) / WY_B;
      k_wy_tmat<<<nwyb, WT_THREADS, 0, ctx->stream>>>(Aq, n, tau, Tg);
      GP_LAUNCH_CHECK(ctx, "k_wy_tmat");
      const double *Tgc = Tg;
      int nn = n, nv2 = nvec;
      void *qargs[] = {(void *)&Aq, &nn, (void *)&Tgc, &d_vecs, &nv2, &qpart, &Sq, &qbar, &d_err};
      GP_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)k_apply_q, dim3((unsigned)Gq),
                                               dim3(WY_THREADS), qargs, q_smem, ctx->stream));
      ctx->launches++;
      int herr = 0;
      GP_CUDA(ctx, gp_memcpy(ctx, &herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
      GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      if (herr) return gp_fail(ctx, GP_ERR_TIMEOUT, "back-transformation grid barrier timed out");
    } else {
      if (cusolverDnDormtr(h, CUBLAS_SIDE_LEFT, CUBLAS_FILL_MODE_LOWER, CUBLAS_OP_N, n, nvec,
                           A_in, n, tau, d_vecs, n, ws, lw, d_info) != CUSOLVER_STATUS_SUCCESS)
        return gp_fail(ctx, GP_ERR_SOLVER, "cusolverDnDormtr failed to launch");
      GP_CUDA(ctx, gp_memcpy(ctx, &info, d_info, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
      GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
      if (info != 0) return gp_fail(ctx, GP_ERR_SOLVER, "ormtr info = %d", info);
    }
  }
  if (timing) {
    GP_EIG_MARK(4);
    cudaEventSynchronize(ev[4]);
    float t01 = 0, t23 = 0, t34 = 0, t35 = 0, t56 = 0;
    cudaEventElapsedTime(&t01, ev[0], ev[1]);
    cudaEventElapsedTime(&t23, ev[2], ev[3]);
    cudaEventElapsedTime(&t34, ev[3], ev[4]);
    if (nvec > 0) {
      cudaEventElapsedTime(&t35, ev[3], ev[5]);
      cudaEventElapsedTime(&t56, ev[5], ev[6]);
    }
    fprintf(stderr, "eig n=%d: tridiagonal %.1f ms, eigenvalues %.1f ms, vectors %.1f ms "
            "(inverse iteration %.1f, Gram-Schmidt %.1f)\n", n, t01, t23, t34, t35, t56);
    for (int i = 0; i < 7; ++i) cudaEventDestroy(ev[i]);
  }
  return GP_OK;
}
