/*
 * fastmode: randomized block-Krylov PCA (kjg_fpca src/ksrc/kjg_fpca.c:24-102, data table of
 * setgval src/gval.c:31-87).
 *
 *   X (M SNPs x N samples), X[s][i] = ((g - mean_s) fancy_s)/sqrt(2), missing -> 0
 *   G_0 = Omega (N x L);  for i <= I:  Q_i = X G_i,  G_{i+1} = X^T Q_i / M
 *   Q = [Q_0 .. Q_I]  (M x (I+1)L)  ->  orthonormal basis U of its columns
 *   B = X^T U  (N x (I+1)L);  top K left singular vectors of B and S^2/M
 *
 * Omega comes from GSL's default generator exactly as kjg_gsl_rng_init and
 * kjg_gsl_ran_ugaussian_matrix draw it (src/ksrc/kjg_gsl.c:100-190): MT19937 seeded with the
 * parfile's seed (GSL maps seed 0 to 4357), polar Box-Muller pairs along each row from
 * uniform_pos draws (the next 32-bit output / 2^32, zero skipped), the last column of an odd L
 * holding one uniform draw.  MT19937 is the published Matsumoto-Nishimura generator with its
 * 2002 initialisation, which std::mt19937 implements.
 *
 * Products with X use the exact sliced tensor-core products (gp_geno_tc.cu) for the split
 * precisions, written as X = (G fancy - O xmean)/sqrt(2) with G the allele counts and O the
 * observed mask (the FP64 SIMT products with the value table for GP_PREC_FP64).  The code
 * operands are built once per call; with every sample selected the SNP-major device records
 * themselves are the operand of X G.
 *
 * The basis of the Krylov space is orthonormalised block by block as it is built (block
 * classical Gram-Schmidt with reorthogonalisation, BCGS2): each new block Q_i = X G_i (M x L,
 * FP64) loses its components along the earlier orthonormal blocks, then W = Q_i^T Q_i =
 * V diag(s) V^T gives Q_i := Q_i V diag(s^-1/2) over the directions whose remaining norm is
 * above 1e-10 of the block's norm before projection (the others are numerically dependent and
 * become zero columns); the projection and the in-block step run twice.  W's decomposition is
 * a one-block cyclic Jacobi (k_block_orth).  The next block is G_{i+1} = X^T Q_i / M, which
 * spans the same Krylov space as the reference's power step from G_i, and H_i = X^T Q_i is
 * kept: B = X^T U = [H_0 .. H_I] needs no further pass over the genotypes.  B^T B =
 * V_B diag(mu) V_B^T (an FP64 tall-skinny Gram and this library's own eigensolver,
 * gp_eig_sym), eval = mu/M and the top-K left singular vectors B V_B mu^-1/2.  The reference
 * takes U from an SVD of the whole Q (kjg_gsl_SVD, which loses the early blocks once the
 * later ones are 1e16 times larger) and forms B = X^T U with another pass over the
 * genotypes; both are Rayleigh-Ritz on the same space.  All of it is FP64 on the GPU; no
 * vendor solver or BLAS is called.
 */
#include <cuda_runtime.h>
#include <math.h>
#include <stdlib.h>
#include <string.h>

#include <random>
#include <vector>

#include "gp_geno_gemm.h"
#include "gp_geno_tc.h"
#include "gp_internal.h"

static const double INV_SQRT2 = 0.70710678118654752440;

/* gsl_rng_uniform_pos of GSL's mt19937 */
struct gsl_mt19937 {
  std::mt19937 g;
  explicit gsl_mt19937(uint64_t seed)
      : g((std::mt19937::result_type)(seed == 0 ? 4357u : (uint32_t)(seed & 0xffffffffu))) {}
  double uniform_pos()
  {
    double x;
    do {
      x = (double)(uint32_t)g() / 4294967296.0;
    } while (x == 0.0);
    return x;
  }
};

/* Omega (N x L row-major) as kjg_gsl_ran_ugaussian_matrix fills it */
static void make_omega(uint64_t seed, int32_t n, int32_t L, double *om)
{
  gsl_mt19937 r(seed);
  for (int32_t i = 0; i < n; ++i) {
    double *row = om + (size_t)i * L;
    int32_t j = 0;
    for (; j + 1 < L; j += 2) {
      double x, y, r2;
      do {
        x = -1.0 + 2.0 * r.uniform_pos();
        y = -1.0 + 2.0 * r.uniform_pos();
        r2 = x * x + y * y;
      } while (r2 > 1.0 || r2 == 0.0);
      r2 = sqrt(-2.0 * log(r2) / r2);
      row[j] = x * r2;
      row[j + 1] = y * r2;
    }
    if (L % 2) row[j] = r.uniform_pos();
  }
}

/* Q[s][j] (row-major, L) = (fancy_s Yg[s][j] - xmean_s Yo[s][j]) / sqrt2 */
__global__ void k_fast_combine_xg(double *Q, const double *yg, const double *yo,
                                  const int32_t *kept, const double *xfancy, const double *xmean,
                                  int32_t nk, int32_t L, double scale)
{
  int64_t total = (int64_t)nk * L;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int32_t c = kept[idx / L];
    Q[idx] = (xfancy[c] * yg[idx] - xmean[c] * yo[idx]) * scale;
  }
}

/* panels for X^T Q: a[s][j] = fancy_s Q[s][j] / sqrt2, b[s][j] = xmean_s Q[s][j] / sqrt2 */
__global__ void k_fast_panels(double *a, double *b, const double *Q, const int32_t *kept,
                              const double *xfancy, const double *xmean, int32_t nk, int32_t L)
{
  int64_t total = (int64_t)nk * L;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    int32_t c = kept[idx / L];
    double q = Q[idx] * INV_SQRT2;
    a[idx] = xfancy[c] * q;
    b[idx] = xmean[c] * q;
  }
}

/* vtab scaled by 1/sqrt2 for the FP64 products, per kept column */
__global__ void k_fast_vtab(const int32_t *kept, int32_t nk, const int32_t *cols, const double *vtab,
                            int32_t *snprec, double *vt)
{
  for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nk; k += gridDim.x * blockDim.x) {
    int32_t c = kept[k];
    snprec[k] = cols[c];
    for (int t = 0; t < 4; ++t) vt[4 * k + t] = vtab[4 * c + t] * INV_SQRT2;
  }
}

#define TSG_T 32     /* cross-product tile edge at most */
#define TSG_R 64     /* rows staged per step */

/*
 * Partial cross products of two tall-skinny row-major matrices A (n x ca, row stride lda) and
 * B (n x cb, row stride ldb): CTA (p, q) computes the tile p of A^T B over the rows of
 * chunk q and writes it to part[q][i][j] (ca x cb); k_ts_reduce sums the chunks in order
 * (deterministic).  The FP64 pipe bounds it, so a tile is no wider than the matrix: th x tw
 * threads of 2 x 2 outputs, 10 x 10 for blocks of 20 columns (a fixed 16 x 16 spent 2.6 times
 * the multiplications there), and the chunks are short enough for eight CTAs per SM (with
 * chunks of at least 2,048 rows a 20 x 20 product over 100,000 rows had 49 CTAs: 642 us, now
 * 113).  run: NULL, or a device word that is 0 when the call is not needed.
 */
__global__ void __launch_bounds__(256)
k_ts_cross(const double *__restrict__ A, int64_t lda, int32_t ca, const double *__restrict__ B,
           int64_t ldb, int32_t cb, int64_t n, int64_t chunk, int32_t th, int32_t tw, double *part,
           const int *run)
{
  if (run && !*run) return;
  __shared__ double As[TSG_R][TSG_T + 1];
  __shared__ double Bs[TSG_R][TSG_T + 1];
  const int32_t tb = (cb + 2 * tw - 1) / (2 * tw);
  const int32_t ti = (int32_t)blockIdx.x / tb, tj = (int32_t)blockIdx.x - ti * tb;
  const int32_t c0 = ti * 2 * th, d0 = tj * 2 * tw;
  const int64_t r0 = (int64_t)blockIdx.y * chunk;
  const int64_t r1 = r0 + chunk < n ? r0 + chunk : n;
  const int tid = threadIdx.x, ty = tid / tw, tx = tid - ty * tw;
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  for (int64_t rs = r0; rs < r1; rs += TSG_R) {
    for (int e = tid; e < TSG_R * TSG_T; e += blockDim.x) {
      const int rr = e / TSG_T, cc = e - rr * TSG_T;
      const int64_t r = rs + rr;
      double va = 0.0, vb = 0.0;
      if (r < r1) {
        if (cc < 2 * th && c0 + cc < ca) va = A[r * lda + c0 + cc];
        if (cc < 2 * tw && d0 + cc < cb) vb = B[r * ldb + d0 + cc];
      }
      As[rr][cc] = va;
      Bs[rr][cc] = vb;
    }
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < TSG_R; ++k) {
      const double a0 = As[k][ty], a1 = As[k][ty + th];
      const double b0 = Bs[k][tx], b1 = Bs[k][tx + tw];
      acc[0][0] = fma(a0, b0, acc[0][0]);
      acc[0][1] = fma(a0, b1, acc[0][1]);
      acc[1][0] = fma(a1, b0, acc[1][0]);
      acc[1][1] = fma(a1, b1, acc[1][1]);
    }
    __syncthreads();
  }
  double *o = part + (int64_t)blockIdx.y * ca * cb;
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int32_t i = c0 + ty + th * u, j = d0 + tx + tw * v;
      if (i < ca && j < cb) o[(int64_t)i * cb + j] = acc[u][v];
    }
}

/* out[i][j] = sum over the chunks of part[q][i][j] (count = ca * cb): a CTA takes 32 entries,
 * each of its 8 warps an eighth of the chunks in order, then the eighths in order */
__global__ void __launch_bounds__(256)
k_ts_reduce(double *out, const double *part, int32_t nchunk, int64_t count, const int *run)
{
  if (run && !*run) return;
  __shared__ double sp[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t idx = blockIdx.x * (int64_t)32 + lane;
  const int32_t per = (nchunk + 7) / 8, q0 = warp * per;
  const int32_t q1 = q0 + per < nchunk ? q0 + per : nchunk;
  double acc = 0.0;
  if (idx < count)
    for (int32_t q = q0; q < q1; ++q) acc += part[(int64_t)q * count + idx];
  sp[warp][lane] = acc;
  __syncthreads();
  if (warp == 0 && idx < count) {
    for (int w = 1; w < 8; ++w) acc += sp[w][lane];
    out[idx] = acc;
  }
}

/* Q -= Qp C: Q (n x L, row stride L), Qp (n x ca, row stride ldp), C (ca x L) */
__global__ void k_ts_project(double *Q, const double *__restrict__ Qp, int64_t ldp, int32_t ca,
                             const double *__restrict__ C, int64_t n, int32_t L, const int *run)
{
  if (run && !*run) return;
  const int64_t total = n * L;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / L;
    const int32_t j = (int32_t)(idx - r * L);
    double q = 0.0;
    for (int32_t k = 0; k < ca; ++k) q = fma(Qp[r * ldp + k], C[(int64_t)k * L + j], q);
    Q[idx] -= q;
  }
}

#define JAC_MAX 64 /* largest block width of the Jacobi kernel */

/*
 * Partial Q^T Q of a block (n x L, row stride L): CTA q sums over the rows of chunk q into
 * part[q][L][L].  The FP64 pipe bounds it and works for every lane of a warp, so the threads are
 * the th (th + 1) / 2 tiles of 2 x 2 of one triangle, th = ceil(L / 2), packed: 55 threads where
 * k_ts_cross has 100 (100,000 x 20: 114 -> 70 us).
 */
__global__ void __launch_bounds__(544)
k_ts_gram(const double *__restrict__ Q, int32_t L, int64_t n, int64_t chunk, double *part,
          const int *run)
{
  if (run && !*run) return;
  __shared__ double As[TSG_R][JAC_MAX + 1];
  const int32_t th = (L + 1) / 2;
  const int64_t r0 = (int64_t)blockIdx.x * chunk, r1 = r0 + chunk < n ? r0 + chunk : n;
  int32_t ty = 0, tx = threadIdx.x; /* tile (ty, tx), ty <= tx < th */
  while (ty < th && tx >= th - ty) {
    tx -= th - ty;
    ++ty;
  }
  const bool on = ty < th;
  tx = on ? tx + ty : 0;
  if (!on) ty = 0;
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  if (L & 1)
    for (int k = threadIdx.x; k < TSG_R; k += blockDim.x) As[k][L] = 0.0; /* column 2 th - 1 */
  for (int64_t rs = r0; rs < r1; rs += TSG_R) {
    const int32_t rows = (int32_t)(r1 - rs < TSG_R ? r1 - rs : TSG_R);
    for (int e = threadIdx.x; e < TSG_R * L; e += blockDim.x) {
      const int rr = e / L;
      As[rr][e - rr * L] = rr < rows ? Q[rs * L + e] : 0.0;
    }
    __syncthreads();
    if (on) {
#pragma unroll 4
      for (int k = 0; k < TSG_R; ++k) {
        const double a0 = As[k][ty], a1 = As[k][ty + th];
        const double b0 = As[k][tx], b1 = As[k][tx + th];
        acc[0][0] = fma(a0, b0, acc[0][0]);
        acc[0][1] = fma(a0, b1, acc[0][1]);
        acc[1][0] = fma(a1, b0, acc[1][0]);
        acc[1][1] = fma(a1, b1, acc[1][1]);
      }
    }
    __syncthreads();
  }
  if (!on) return;
  double *o = part + (int64_t)blockIdx.x * L * L;
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int32_t i = ty + th * u, j = tx + th * v;
      if (i < L && j < L) {
        o[(int64_t)i * L + j] = acc[u][v];
        if (ty != tx) o[(int64_t)j * L + i] = acc[u][v];
      }
    }
}

/* partial squared column norms of a block (n x L): CTA q over the rows of chunk q into
 * part[q][L]; blockDim.x = L * (rows at a time) */
__global__ void __launch_bounds__(256)
k_ts_norms(const double *__restrict__ Q, int32_t L, int64_t n, int64_t chunk, double *part)
{
  __shared__ double sp[256];
  const int32_t j = threadIdx.x % L, g = threadIdx.x / L, G = blockDim.x / L;
  const int64_t r0 = (int64_t)blockIdx.x * chunk, r1 = r0 + chunk < n ? r0 + chunk : n;
  double acc = 0.0;
  for (int64_t r = r0 + g; r < r1; r += G) {
    const double q = Q[r * L + j];
    acc = fma(q, q, acc);
  }
  sp[threadIdx.x] = acc;
  __syncthreads();
  if (g == 0) {
    for (int k = 1; k < G; ++k) acc += sp[k * L + j];
    part[(int64_t)blockIdx.x * L + j] = acc;
  }
}

/*
 * One block: the L x L matrix W (symmetrised) is diagonalised by Jacobi rotations (Golub & Van
 * Loan, Matrix Computations, 8.5: the symmetric Schur decomposition of each 2 x 2 pivot),
 * W = V diag(s) V^T, and T = V diag(s^-1/2) is written for the directions with
 * s > tol * max(pre) (max(W[j][j]) when pre is NULL; zero columns for the others).  A pivot is
 * rotated while |W_pq| > 1e-15 sqrt(|W_pp W_qq|), the threshold that keeps the small eigenvalues
 * of a positive semidefinite W to high relative accuracy (Demmel & Veselic, 1992); the sweeps
 * stop after one without a rotation, at most 40.  A sweep runs in the rounds of a round-robin
 * tournament (the parallel ordering of Brent & Luk): L/2 disjoint pivots at once, their rotations
 * side by side, then every 2 x 2 block of W by its two pivots' rotations.  The latency of the FP64
 * square roots and divisions of a rotation bounds it, so its tangent is an FP32 value (a rotation
 * need not annihilate its pivot to the last bit, the next sweep does) and only the cosine that
 * belongs to that tangent is FP64, from an FP32 reciprocal root and two Newton steps.  L = 20: one
 * pivot after another 3.3 ms, in rounds with FP64 roots 0.44, now 0.33.
 *
 * info (device): [0] max(pre) and [1] the smallest kept s of the first pass (pre given), written
 * then and read in the later ones: there a direction of s must also have s info[1] > tol info[0],
 * the first pass's rule for what is left of it.  *again (not NULL): 1 when a kept direction lost
 * more than half of its norm.
 */
#define JAC_THREADS 256
__global__ void __launch_bounds__(JAC_THREADS)
k_block_orth(const double *__restrict__ Wg, const double *__restrict__ pre, int32_t L,
             double tol, double *T, double *info, int *again, const int *run)
{
  if (run && !*run) return;
  __shared__ double W[JAC_MAX][JAC_MAX + 1];
  __shared__ double V[JAC_MAX][JAC_MAX + 1];
  __shared__ double sc[JAC_MAX / 2], ss[JAC_MAX / 2];
  __shared__ int sp[JAC_MAX / 2], sq[JAC_MAX / 2];
  const int t = threadIdx.x;
  const int np = (L + 1) / 2, M = 2 * np - 1; /* pairs per round, rounds; index L: a bye */
  for (int e = t; e < L * L; e += blockDim.x) {
    const int i = e / L, j = e - i * L;
    W[i][j] = 0.5 * (Wg[(int64_t)i * L + j] + Wg[(int64_t)j * L + i]);
    V[i][j] = i == j ? 1.0 : 0.0;
  }
  __syncthreads();
  for (int sweep = 0; sweep < 40; ++sweep) {
    int rotated = 0;
    for (int r = 0; r < M; ++r) {
      int rot = 0;
      if (t < np) {
        int p = t == 0 ? M : (r + t) % M, q = t == 0 ? r : (r - t + M) % M;
        if (p > q) {
          const int o = p;
          p = q;
          q = o;
        }
        double c = 1.0, sn = 0.0;
        if (q < L) {
          const double apq = W[p][q];
          const double wpp = W[p][p], wqq = W[q][q];
          if (apq != 0.0 && (apq * 1e15) * (apq * 1e15) > fabs(wpp * wqq)) {
            /* t = sign(tau) / (|tau| + sqrt(1 + tau^2)), tau beyond FP32's squares: 1 / (2 tau) */
            const float tau = (float)((wqq - wpp) / (2.0 * apq)), at = fabsf(tau);
            const float tf = at > 1e9f ? 0.5f / tau : copysignf(1.f, tau) / (at + sqrtf(1.f + at * at));
            const double tt = (double)tf, u = 1.0 + tt * tt, hu = 0.5 * u;
            c = (double)rsqrtf((float)u);
            c *= 1.5 - hu * c * c;
            c *= 1.5 - hu * c * c;
            sn = tt * c;
            rot = 1;
          }
        }
        sc[t] = c;
        ss[t] = sn;
        sp[t] = p;
        sq[t] = q;
      }
      if (!__syncthreads_or(rot)) continue;
      rotated = 1;
      /* W := J^T W J: the block of pairs (a, b) belongs to one thread */
      for (int e = t; e < np * np; e += blockDim.x) {
        const int a = e / np, b = e - a * np;
        const double ca = sc[a], sa = ss[a], cb = sc[b], sb = ss[b];
        if (sa == 0.0 && sb == 0.0) continue;
        const int p = sp[a], q = sq[a], u = sp[b], v = sq[b];
        const bool hq = q < L, hv = v < L;
        double wpu = W[p][u], wpv = hv ? W[p][v] : 0.0;
        double wqu = hq ? W[q][u] : 0.0, wqv = hq && hv ? W[q][v] : 0.0;
        const double pu = ca * wpu - sa * wqu, qu = sa * wpu + ca * wqu;
        const double pv = ca * wpv - sa * wqv, qv = sa * wpv + ca * wqv;
        W[p][u] = cb * pu - sb * pv;
        if (hv) W[p][v] = sb * pu + cb * pv;
        if (hq) W[q][u] = cb * qu - sb * qv;
        if (hq && hv) W[q][v] = sb * qu + cb * qv;
      }
      for (int e = t; e < np * L; e += blockDim.x) { /* V := V J */
        const int i = e / np, a = e - i * np;
        const double sn = ss[a], c = sc[a];
        if (sn == 0.0) continue;
        const double vp = V[i][sp[a]], vq = V[i][sq[a]];
        V[i][sp[a]] = c * vp - sn * vq;
        V[i][sq[a]] = sn * vp + c * vq;
      }
      __syncthreads();
    }
    if (!rotated) break; /* the same for every thread */
  }
  double pmax = 0.0;
  for (int i = 0; i < L; ++i) pmax = fmax(pmax, pre ? pre[i] : Wg[(int64_t)i * L + i]);
  const double p0 = pre ? 0.0 : info[0], s0 = pre ? 0.0 : info[1];
  int lost = 0;
  double kept = INFINITY;
  if (t < L) {
    const double sk = W[t][t];
    const bool keep = sk > tol * pmax && sk > 0.0 && (pre || sk * s0 > tol * p0);
    const double f = keep ? 1.0 / sqrt(sk) : 0.0;
    for (int i = 0; i < L; ++i) T[(int64_t)i * L + t] = V[i][t] * f;
    lost = keep && sk < 0.25;
    if (keep) kept = sk;
    W[t][t] = kept;
  }
  lost = __syncthreads_or(lost);
  if (t == 0) {
    if (pre) {
      for (int i = 0; i < L; ++i) kept = fmin(kept, W[i][i]);
      info[0] = pmax;
      info[1] = kept;
    }
    if (again) *again = lost;
  }
}

/* out (n x L) = Q T; with qp != NULL also qp[:, col0 ..] (row stride ldp) = Q T */
__global__ void k_block_apply(const double *__restrict__ Q, const double *__restrict__ T,
                              double *out, double *qp, int64_t ldp, int32_t col0, int64_t n,
                              int32_t L, const int *run)
{
  if (run && !*run) return;
  const int64_t total = n * L;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / L;
    const int32_t j = (int32_t)(idx - r * L);
    double q = 0.0;
    for (int32_t k = 0; k < L; ++k) q = fma(Q[r * L + k], T[(int64_t)k * L + j], q);
    out[idx] = q;
    if (qp) qp[r * ldp + col0 + j] = q;
  }
}

/* dst := src when *run */
__global__ void k_block_copy(double *dst, const double *src, int64_t count, const int *run)
{
  if (!*run) return;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = src[i];
}

/* G := Hp[:, col0 ..] / M (the next block) */
__global__ void k_block_next(double *G, const double *__restrict__ Hp, int64_t ldp, int32_t col0,
                             int64_t n, int32_t L, double inv_m)
{
  const int64_t total = n * L;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = idx / L;
    const int32_t j = (int32_t)(idx - r * L);
    G[idx] = Hp[r * ldp + col0 + j] * inv_m;
  }
}

/* C := (C + C^T) / 2 (n x n) */
__global__ void k_symmetrize(double *C, int32_t n)
{
  const int64_t total = (int64_t)n * n;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int32_t i = (int32_t)(idx / n), j = (int32_t)(idx - (int64_t)i * n);
    if (i < j) {
      const double v = 0.5 * (C[idx] + C[(int64_t)j * n + i]);
      C[idx] = v;
      C[(int64_t)j * n + i] = v;
    }
  }
}

/* evec[j][i] = sum_c Hp[i][c] U[j][c] / sqrt(mu_j) */
__global__ void k_fast_evecs(double *evecs, const double *__restrict__ Hp, int64_t ldp,
                             const double *__restrict__ U, const double *__restrict__ mu,
                             int64_t n, int32_t c4, int32_t K)
{
  const int64_t total = n * K;
  for (int64_t idx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; idx < total;
       idx += (int64_t)gridDim.x * blockDim.x) {
    const int32_t j = (int32_t)(idx / n);
    const int64_t i = idx - (int64_t)j * n;
    double acc = 0.0;
    for (int32_t c = 0; c < c4; ++c) acc = fma(Hp[i * ldp + c], U[(int64_t)j * c4 + c], acc);
    evecs[idx] = mu[j] > 0.0 ? acc / sqrt(mu[j]) : 0.0;
  }
}

static int grid_for_fast(const gp_ctx *ctx, int64_t work)
{
  int64_t g = (work + 255) / 256;
  if (g > (int64_t)ctx->num_sms * 16) g = (int64_t)ctx->num_sms * 16;
  return (int)(g < 1 ? 1 : g);
}

/* out (ca x cb) = A^T B over n rows, through the chunk partials in part (deterministic) */
static int ts_cross(gp_ctx *ctx, const double *A, int64_t lda, int32_t ca, const double *B,
                    int64_t ldb, int32_t cb, int64_t n, double *part, size_t part_cap,
                    double *out, const int *run)
{
  /* the fewest tiles of at most TSG_T columns, equally wide */
  const int32_t na = (ca + TSG_T - 1) / TSG_T, nb = (cb + TSG_T - 1) / TSG_T;
  const int32_t th = ((ca + na - 1) / na + 1) / 2, tw = ((cb + nb - 1) / nb + 1) / 2;
  const int32_t ntiles = ((ca + 2 * th - 1) / (2 * th)) * ((cb + 2 * tw - 1) / (2 * tw));
  int64_t want = ((int64_t)ctx->num_sms * 8 + ntiles - 1) / ntiles;
  int64_t chunk = ((n + want - 1) / want + TSG_R - 1) / TSG_R * TSG_R;
  int64_t nchunk = (n + chunk - 1) / chunk;
  while ((size_t)(nchunk * ca * cb) > part_cap) { /* fewer, longer chunks when space is short */
    chunk *= 2;
    nchunk = (n + chunk - 1) / chunk;
  }
  dim3 grid((unsigned)ntiles, (unsigned)nchunk);
  k_ts_cross<<<grid, th * tw, 0, ctx->stream>>>(A, lda, ca, B, ldb, cb, n, chunk, th, tw, part,
                                              run);
  GP_LAUNCH_CHECK(ctx, "k_ts_cross");
  k_ts_reduce<<<(unsigned)(((int64_t)ca * cb + 31) / 32), 256, 0, ctx->stream>>>(
      out, part, (int32_t)nchunk, (int64_t)ca * cb, run);
  GP_LAUNCH_CHECK(ctx, "k_ts_reduce");
  return GP_OK;
}

/* out [L][L] = Q^T Q of a block (n x L), or its diagonal [L] */
static int ts_gram(gp_ctx *ctx, const double *Q, int32_t L, int64_t n, bool diag, double *part,
                   size_t part_cap, double *out, const int *run)
{
  const int64_t count = diag ? L : (int64_t)L * L;
  int64_t chunk = (n / (8 * ctx->num_sms) + TSG_R) / TSG_R * TSG_R, nchunk = (n + chunk - 1) / chunk;
  while ((size_t)(nchunk * count) > part_cap) {
    chunk *= 2;
    nchunk = (n + chunk - 1) / chunk;
  }
  if (diag) {
    k_ts_norms<<<(unsigned)nchunk, 256 / L * L, 0, ctx->stream>>>(Q, L, n, chunk, part);
    GP_LAUNCH_CHECK(ctx, "k_ts_norms");
  } else {
    const int32_t th = (L + 1) / 2, nt = th * (th + 1) / 2;
    k_ts_gram<<<(unsigned)nchunk, (nt + 31) / 32 * 32, 0, ctx->stream>>>(Q, L, n, chunk, part, run);
    GP_LAUNCH_CHECK(ctx, "k_ts_gram");
  }
  k_ts_reduce<<<(unsigned)((count + 31) / 32), 256, 0, ctx->stream>>>(out, part, (int32_t)nchunk,
                                                                     count, run);
  GP_LAUNCH_CHECK(ctx, "k_ts_reduce");
  return GP_OK;
}

/* a direction of a new Krylov block is dependent on the earlier blocks when its norm after
 * projection is below 1e-10 of the block's norm before it (s is a squared norm) */
#define GP_FAST_DEP_TOL 1e-20

/* the device buffers of one gp_fastpca call, side by side in the handle's aux scratch (kept
 * there for the next call instead of 17 allocations and releases per call): counted with
 * base == NULL, then placed */
struct fast_bufs {
  uint8_t *base = NULL;
  size_t used = 0;
  template <class T> void get(T **out, size_t count)
  {
    *out = (T *)(base + used);
    used += (count * sizeof(T) + 255) / 256 * 256;
  }
};

extern "C" int gp_fastpca(gp_ctx *ctx, int32_t K, int32_t L, int32_t I, uint64_t seed,
                          const double *omega, const gp_xtx_opts *opts, double *evals,
                          double *evecs)
{
  if (!ctx || !opts) return GP_ERR_ARG;
  const int32_t precision = opts->precision;
  if (!ctx->d_geno || ctx->nrows < 1 || ctx->ncols < 1)
    return gp_fail(ctx, GP_ERR_STATE, "gp_fastpca: genotypes, samples and SNPs must be set first");
  if (K < 1 || L <= K || L > JAC_MAX || I < 1 || (int64_t)(I + 1) * L > 1024)
    return gp_fail(ctx, GP_ERR_ARG,
                   "gp_fastpca: need 0 < K < L <= 64 and 0 < I, (I+1) L <= 1024");
  GP_CUDA(ctx, cudaSetDevice(ctx->device));
  const int32_t n = ctx->nrows, nc = ctx->ncols;
  const int32_t c4 = (I + 1) * L;
  const int use_tc = precision != GP_PREC_FP64;

  /* per-SNP tables over the rows; nothing is killed but the monomorphic SNPs, whose rows of
   * X are zero anyway (setgval) */
  gp_xtx_opts o = {opts->fancynorm, opts->altnormstyle, 0, 0x7fffffff, precision};
  ctx->xtx_valid = ctx->eig_valid = ctx->weights_valid = 0;
  int rc = gp_launch_snp_stats(ctx, &o);
  if (rc) return rc;
  std::vector<uint8_t> hk((size_t)nc);
  GP_CUDA(ctx, gp_memcpy(ctx, hk.data(), ctx->d_killed, (size_t)nc, cudaMemcpyDeviceToHost,
                         ctx->stream));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  std::vector<int32_t> kept;
  for (int32_t c = 0; c < nc; ++c)
    if (!hk[(size_t)c]) kept.push_back(c);
  const int32_t nk = (int32_t)kept.size();
  ctx->nkept = nk;
  ctx->codes4_rows = 0;
  if (nk < 1) return gp_fail(ctx, GP_ERR_NODATA, "gp_fastpca: no polymorphic SNP");
  GP_CUDA(ctx, gp_memcpy(ctx, ctx->d_kept, kept.data(), sizeof(int32_t) * (size_t)nk,
                         cudaMemcpyHostToDevice, ctx->stream));

  /* buffers: the orthonormal blocks Q_i (nk x c4) and H_i = X^T Q_i (n x c4) side by side,
   * the next G (n x L), the current block and two product panels (nk x L), cross-product
   * partials and the small matrices */
  const size_t nG = (size_t)n * L, nQ = (size_t)nk * L;
  const int64_t nmax = n > nk ? n : nk;
  /* chunk partials of about eight CTAs per SM (ts_cross lengthens the chunks when this is
   * short) */
  const size_t part_cap = (size_t)c4 * c4 + ((size_t)nmax / 2048 + 2) * (size_t)c4 * L +
                          (size_t)8 * ctx->num_sms * TSG_T * TSG_T + 4096;
  fast_bufs B;
  double *d_Qp, *d_Hp, *d_G, *d_Q, *d_Y1, *d_Y2, *d_part, *d_C, *d_W, *d_pre, *d_T, *d_mu,
      *d_U, *d_ev, *d_vt;
  int32_t *d_snprec;
  uint8_t *codes_samp = NULL, *codes_snp = NULL;
  int64_t ldc_samp, ldc_snp;
  int32_t pad_samp, pad_snp, *d_inv = NULL;
  gp_tc_code_bytes(1, n, nk, &ldc_samp, &pad_samp);
  gp_tc_code_bytes(0, n, nk, &ldc_snp, &pad_snp);
  for (int pass = 0; pass < 2; ++pass) {
    B.used = 0;
    B.get(&d_Qp, (size_t)nk * c4);
    B.get(&d_Hp, (size_t)n * c4);
    B.get(&d_G, nG);
    B.get(&d_Q, nQ);
    B.get(&d_Y1, nQ);
    B.get(&d_Y2, nQ);
    B.get(&d_part, part_cap);
    B.get(&d_C, (size_t)c4 * c4);
    B.get(&d_W, (size_t)L * L);
    B.get(&d_pre, (size_t)L + 4); /* squared norms, then info and again of k_block_orth */
    B.get(&d_T, (size_t)L * L);
    B.get(&d_mu, (size_t)c4);
    B.get(&d_U, (size_t)K * c4);
    B.get(&d_ev, (size_t)n * K);
    B.get(&d_vt, 4 * (size_t)nk);
    B.get(&d_snprec, (size_t)nk);
    if (use_tc) B.get(&d_inv, (size_t)ctx->nind_all);
    if (use_tc) B.get(&codes_samp, (size_t)pad_samp * ldc_samp);
    if (use_tc && n != ctx->nind_all) B.get(&codes_snp, (size_t)pad_snp * ldc_snp);
    if (pass == 0) {
      rc = gp_scratch_aux(ctx, B.used, (void **)&B.base);
      if (rc) return rc;
    }
  }

  k_fast_vtab<<<grid_for_fast(ctx, nk), 256, 0, ctx->stream>>>(ctx->d_kept, nk, ctx->d_cols,
                                                              ctx->d_vtab, d_snprec, d_vt);
  GP_LAUNCH_CHECK(ctx, "k_fast_vtab");

  /* Omega = G_0 */
  {
    std::vector<double> om(nG);
    if (omega)
      memcpy(om.data(), omega, sizeof(double) * om.size());
    else
      make_omega(seed, n, L, om.data());
    GP_CUDA(ctx, gp_memcpy(ctx, d_G, om.data(), sizeof(double) * om.size(),
                           cudaMemcpyHostToDevice, ctx->stream));
    GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }

  /* code operands: X G reads SNP rows (the device records when every sample is selected, in
   * order), X^T Q reads sample rows */
  gp_tc_codes A_snp, A_samp;
  if (use_tc) {
    rc = gp_tc_build_codes(ctx, 1, ctx->d_rows, n, d_snprec, nk, d_inv, codes_samp, &A_samp);
    if (rc) return rc;
    if (n == ctx->nind_all) {
      A_snp.codes = ctx->d_geno;
      A_snp.ldc = ctx->rlen_dev;
      A_snp.row_map = d_snprec;
      A_snp.nrows = nk;
      A_snp.k0 = n;
    } else {
      rc = gp_tc_build_codes(ctx, 0, ctx->d_rows, n, d_snprec, nk, NULL, codes_snp, &A_snp);
      if (rc) return rc;
    }
  }
  rc = gp_tc_begin(ctx);
  if (rc) return rc;
  /* the Krylov blocks, orthonormalised as they come: Q_i = X G_i, H_i = X^T Q_i */
  for (int32_t it = 0; it <= I; ++it) {
    if (use_tc) {
      gp_tc_panel pg = {d_G, L, 1.0, 1};
      rc = gp_geno_panel_tc_codes(ctx, &A_snp, 1, &pg, L, 4, d_Y1, L);
      if (rc) return rc;
      pg.count = 0;
      rc = gp_geno_panel_tc_codes(ctx, &A_snp, 1, &pg, L, 4, d_Y2, L);
      if (rc) return rc;
      k_fast_combine_xg<<<grid_for_fast(ctx, (int64_t)nQ), 256, 0, ctx->stream>>>(
          d_Q, d_Y1, d_Y2, ctx->d_kept, ctx->d_xfancy, ctx->d_xmean, nk, L, INV_SQRT2);
      GP_LAUNCH_CHECK(ctx, "k_fast_combine_xg");
    } else {
      rc = gp_geno_gemm_f64(ctx, 0, ctx->d_rows, n, d_snprec, d_vt, nk, d_G, L, L, d_Q, L);
      if (rc) return rc;
    }
    /*
     * Project against earlier blocks and orthonormalise within the block, twice: the first time
     * against the last two blocks only, the second against all.  Q_it = A Q_it-1 with A = X X^T
     * symmetric, so Q_j^T A Q_it-1 = (A Q_j)^T Q_it-1 is zero but for rounding when j + 1 < it - 1
     * (A Q_j lies in the blocks up to j + 1), which is what the second time takes away: the
     * three-term recurrence of block Lanczos with one full reorthogonalisation (Golub & Van Loan,
     * Matrix Computations, 10.3).  The first time drops directions below 1e-10 of the block's norm
     * before it.  Should the second time take more than half of a direction's norm, as it can
     * beside dropped ones, a third one follows (decided on the device).  The projections are FP64
     * work of 2 n L columns: all blocks both times took 19.5 ms of
     * 10,007 x 100,003, L = 20, I = 10, now 12.7.
     */
    const int32_t ca = it * L, lo = it > 2 ? ca - 2 * L : 0;
    double *d_info = d_pre + L;
    int *d_again = (int *)(d_pre + L + 2);
    rc = ts_gram(ctx, d_Q, L, nk, true, d_part, part_cap, d_pre, NULL);
    if (rc) return rc;
    for (int pass = 0; pass < 3; ++pass) {
      const int32_t c0 = pass == 0 ? lo : 0;
      const int *run = pass == 2 ? d_again : NULL;
      if (pass == 2 && ca == 0) break;
      if (ca > 0) {
        rc = ts_cross(ctx, d_Qp + c0, c4, ca - c0, d_Q, L, L, nk, d_part, part_cap, d_C, run);
        if (rc) return rc;
        k_ts_project<<<grid_for_fast(ctx, (int64_t)nQ), 256, 0, ctx->stream>>>(
            d_Q, d_Qp + c0, c4, ca - c0, d_C, nk, L, run);
        GP_LAUNCH_CHECK(ctx, "k_ts_project");
      }
      rc = ts_gram(ctx, d_Q, L, nk, false, d_part, part_cap, d_W, run);
      if (rc) return rc;
      k_block_orth<<<1, JAC_THREADS, 0, ctx->stream>>>(d_W, pass == 0 ? d_pre : NULL, L,
                                                      GP_FAST_DEP_TOL, d_T, d_info,
                                                      pass == 1 ? d_again : NULL, run);
      GP_LAUNCH_CHECK(ctx, "k_block_orth");
      k_block_apply<<<grid_for_fast(ctx, (int64_t)nQ), 256, 0, ctx->stream>>>(
          d_Q, d_T, d_Y1, pass > 0 ? d_Qp : NULL, c4, ca, nk, L, run);
      GP_LAUNCH_CHECK(ctx, "k_block_apply");
      if (pass == 2) {
        k_block_copy<<<grid_for_fast(ctx, (int64_t)nQ), 256, 0, ctx->stream>>>(d_Q, d_Y1,
                                                                              (int64_t)nQ, run);
        GP_LAUNCH_CHECK(ctx, "k_block_copy");
      } else {
        double *tq = d_Q;
        d_Q = d_Y1;
        d_Y1 = tq;
      }
    }
    /* H_i = X^T Q_i into its columns of Hp; the next block G = H_i / M */
    if (use_tc) {
      k_fast_panels<<<grid_for_fast(ctx, (int64_t)nQ), 256, 0, ctx->stream>>>(
          d_Y1, d_Y2, d_Q, ctx->d_kept, ctx->d_xfancy, ctx->d_xmean, nk, L);
      GP_LAUNCH_CHECK(ctx, "k_fast_panels");
      gp_tc_panel pp[2] = {{d_Y1, L, 1.0, 1}, {d_Y2, L, -1.0, 0}};
      rc = gp_geno_panel_tc_codes(ctx, &A_samp, 2, pp, L, 4, d_Hp + ca, c4);
      if (rc) return rc;
    } else {
      rc = gp_geno_gemm_f64(ctx, 1, ctx->d_rows, n, d_snprec, d_vt, nk, d_Q, L, L, d_Hp + ca,
                            c4);
      if (rc) return rc;
    }
    if (it < I) {
      k_block_next<<<grid_for_fast(ctx, (int64_t)nG), 256, 0, ctx->stream>>>(
          d_G, d_Hp, c4, ca, n, L, 1.0 / (double)nc);
      GP_LAUNCH_CHECK(ctx, "k_block_next");
    }
  }
  rc = gp_tc_check(ctx);
  if (rc) return rc;
  /* B = X^T U = Hp; B^T B = V diag(mu) V^T; eval = mu / M, evec = B v / sqrt(mu) */
  rc = ts_cross(ctx, d_Hp, c4, c4, d_Hp, c4, c4, n, d_part, part_cap, d_C, NULL);
  if (rc) return rc;
  k_symmetrize<<<grid_for_fast(ctx, (int64_t)c4 * c4), 256, 0, ctx->stream>>>(d_C, c4);
  GP_LAUNCH_CHECK(ctx, "k_symmetrize");
  rc = gp_eig_sym(ctx, d_C, c4, K, d_mu, d_U);
  if (rc) return rc;
  k_fast_evecs<<<grid_for_fast(ctx, (int64_t)n * K), 256, 0, ctx->stream>>>(d_ev, d_Hp, c4, d_U,
                                                                           d_mu, n, c4, K);
  GP_LAUNCH_CHECK(ctx, "k_fast_evecs");
  std::vector<double> hmu((size_t)K);
  GP_CUDA(ctx, gp_memcpy(ctx, hmu.data(), d_mu, sizeof(double) * (size_t)K,
                         cudaMemcpyDeviceToHost, ctx->stream));
  if (evecs)
    GP_CUDA(ctx, gp_memcpy(ctx, evecs, d_ev, sizeof(double) * (size_t)n * K,
                           cudaMemcpyDeviceToHost, ctx->stream));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (evals)
    for (int32_t j = 0; j < K; ++j) evals[j] = hmu[(size_t)j] / (double)nc;
  return GP_OK;
}
