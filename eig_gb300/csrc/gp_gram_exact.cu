/*
 * The FP64 Gram (the drop-in precision) as exact integer sums on the tensor cores, replacing
 * domult_increment_lookup / block_increment_binary (src/eigensrc/smartpca.c:3361-3495) and
 * domult_increment_normal (:3498-3561).
 *
 * A normalised genotype of SNP s is v(g) = (g - m) f, or 0 where it is missing.  With
 * h = g - 1 in {-1, 0, 1} and o = 1 where the genotype is observed (both 0 where it is not),
 * v_i = h_i f + o_i T1 with T1 = (1 - m) f the table's entry of g = 1, so
 *
 *   XTX[i][j] = sum_s h_i(s) R1_j(s) + o_i(s) R2_j(s),   R1 = f v_j,  R2 = T1 v_j.
 *
 * The left factors are small integers.  R1 and R2 are FP64 values with one power-of-two scale
 * 2^E > max |R| for the whole pass, rounded to 59 bits below it (|error| <= 2^(E-60)) and cut
 * into five balanced digits of 12 bits, integers of at most 2048 that fp16 holds exactly.  A
 * tensor-core sum of {-1, 0, 1} times such digits over at most 4,096 SNPs (both terms: at most
 * 4,096 per SNP) is an integer of at most 2^24, which the FP32 accumulator holds exactly.  The
 * digit sums of a chunk are combined into two 64-bit integers (the three upper digits, the
 * lower ones) and added to the tile's sums in global memory with 64-bit integer atomics, whose
 * order does not matter: the Gram is the same whatever the tile shape, split or schedule, and
 * its error is the rounding of R (2^-53 of each value, 2^-60 of the largest) and one rounding
 * of the result.
 *
 * The scale is set by the rarest SNP (|R| up to 4 n where one allele is seen once, about 4 for
 * common ones), so 2^(E-60) can be more than what a sequence of FP64 additions leaves, about
 * 2^-53 sqrt(m) of a sum of m SNPs.  Then (ex_digits) six digits are cut, 71 bits below the scale,
 * and T1 is the entry of the more frequent homozygote plus or minus f, unrounded like the
 * products R, so that the value of most samples enters exactly.  Relative error of the Gram of
 * 5,000 samples x 2,000 SNPs with frequencies down to 1/(2n): 8e-15 with five digits, 1.4e-15 on
 * the FP64 pipe, 6e-17 with six.
 *
 * What bounds it: ten (twelve) fp16 products per genotype pair, i.e. the tensor pipe (GB300's FP64
 * pipe runs at about 1/2,000 of its fp16 rate).  2,003 samples x 120,011 SNPs: 4.4 ms in all, of
 * 485 ms on the FP64 pipe; relative error against 64 bits 1.0e-15, of 9.3e-15.
 *
 *   k_exact_max     the largest |R| of the kept SNPs
 *   k_exact_begin   the kept SNPs' records; the sums cleared
 *   k_exact_slices  the right operand: per block of 48 samples (40 with six digits) and 64 SNPs
 *                   and per term the 240 x 64 tile (digit t of sample jj in row 48 t + jj) in the
 *                   128-byte swizzle of shared memory, stored as one contiguous piece so that a
 *                   stage of the Gram kernel is a single bulk copy
 *   k_gram_exact    256 x 48 (40) tiles of the lower triangle, per 64 SNPs and term two
 *                   128 x 240 x 16 MMAs per k step sharing the right tile (so that it streams
 *                   at half the rate a 128-row tile would need):
 *                     warp 0       bulk copies of right tiles into a 3-stage ring
 *                     warp 1       issues the MMAs
 *                     warps 2-9    decode h and o from the rows' 2-bit codes into the stages,
 *                                  a thread per row
 *                     warps 10-17  after a chunk: tcgen05.ld, combine, atomics
 *   k_exact_finish  XTX (both triangles) from the integer sums
 */
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <math.h>

#include "gp_geno_tc.h"
#include "gp_internal.h"
#include "gp_tc.cuh"

#define EX_ROWS 256                    /* tile rows: two 128-row accumulators */
#define EX_N 240                       /* MMA columns: digits x samples */
#define EX_J(S) (EX_N / (S))           /* tile columns (samples) with S digits: 48 or 40 */
#define EX_BITS(S) (12 * (S) - 1)      /* bits below the scale */
#define EX_K 64                        /* SNPs per k-block */
#define EX_A_BYTES (128 * EX_K * 2)
#define EX_B_BYTES (EX_N * EX_K * 2)   /* 30,720: a multiple of the swizzle's 1,024 */
#define EX_STAGE_BYTES (2 * EX_A_BYTES + EX_B_BYTES)
#define EX_STAGES 3
#define EX_CHUNK_KB 64                 /* 4,096 SNPs per exact FP32 chunk */
#define EX_DEC_WARPS 8
#define EX_EPI_WARPS 8
#define EX_THREADS (64 + 32 * (EX_DEC_WARPS + EX_EPI_WARPS))
#define EX_SMEM (EX_STAGES * EX_STAGE_BYTES + 1024 + 256)
#define EX_PF 4                        /* k-blocks of codes a decoder loads ahead */
#define EX_TILE(S) (EX_ROWS * EX_J(S)) /* elements of a tile's sums */
#define EX_D1 256                      /* TMEM column of the second accumulator */
/* right operand per pass over it: bounds the scratch memory, and a pass of a 5,000-sample
 * panel still has 21,000 SNPs */
#define EX_BUDGET (2ll << 30)

#define EXERR_FULL 31
#define EXERR_EMPTY 32
#define EXERR_ACCF 33
#define EXERR_ACCE 34

/* ---- tiles of the lower triangle ------------------------------------------------------ */

/* J-column tiles of tile row bi: those that start at or before its last row */
__host__ __device__ __forceinline__ int32_t ex_row_tiles(int32_t bi, int32_t n, int32_t J)
{
  int32_t last = (bi + 1) * EX_ROWS < n ? (bi + 1) * EX_ROWS : n;
  return (last + J - 1) / J;
}

template <int S>
__device__ __forceinline__ void ex_tile(int32_t t, int32_t n, int32_t *bi, int32_t *jt)
{
  int32_t b = 0;
  for (;;) {
    const int32_t c = ex_row_tiles(b, n, EX_J(S));
    if (t < c) break;
    t -= c;
    ++b;
  }
  *bi = b;
  *jt = t;
}

/* which 128-row halves of a tile hold an entry of the lower triangle */
template <int S>
__device__ __forceinline__ void ex_halves(int32_t bi, int32_t jt, int32_t n, bool *h0, bool *h1)
{
  *h0 = bi * EX_ROWS + 127 >= jt * EX_J(S);
  *h1 = bi * EX_ROWS + 128 < n;
}

/* ---- digits ---------------------------------------------------------------------------- */

/* per block of the grid the largest |R| of its SNPs (a killed SNP's table is zero) */
__global__ void __launch_bounds__(256)
k_exact_max(int32_t ncols, const double *__restrict__ vtab, const double *__restrict__ xfancy,
            double *part)
{
  __shared__ double sm[8];
  double m = 0.0;
  for (int32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < ncols; c += gridDim.x * blockDim.x) {
    const double f = fmax(fabs(xfancy[c]), fabs(vtab[4 * (int64_t)c + 1]));
    for (int g = 0; g < 3; ++g) m = fmax(m, f * fabs(vtab[4 * (int64_t)c + g]));
  }
  for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) m = fmax(m, sm[w]);
    part[blockIdx.x] = m;
  }
}

/* the record index of each kept SNP; the sums cleared (nsums: an even count) */
__global__ void k_exact_begin(const int32_t *__restrict__ kept, int32_t nkept,
                              const int32_t *__restrict__ cols, int32_t *snprec,
                              unsigned long long *sums, int64_t nsums)
{
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t k = t; k < nkept; k += step) snprec[k] = cols[kept[k]];
  for (int64_t i = t; i < nsums / 2; i += step) ((ulonglong2 *)sums)[i] = make_ulonglong2(0, 0);
}

/* the lower S - 1 of S balanced digits of 12 bits into h[first + 1 ..], the rest of N into h[first] */
template <int S>
__device__ __forceinline__ void ex_cut(long long N, __half *h)
{
#pragma unroll
  for (int t = S - 1; t >= 1; --t) {
    const int d = (int)((N + 2048) & 4095) - 2048;
    h[t] = __int2half_rn(d);
    N = (N - d) >> 12; /* exact */
  }
  h[0] = __int2half_rn((int)N); /* at most 2048: |R| < 2^E */
}

/*
 * One CTA per k-block (blockIdx.x, kept SNPs kb0*64 + 64 x ..) and group of EX_SJT right tiles.
 * The digits of the block's SNPs for every code are cut once into shared memory (per SNP and
 * code S words: term 1's digits and term 2's); a thread then takes 8 SNPs of one sample
 * and writes the 2 S 16-byte pieces of its rows; 8 neighbouring threads complete a 128-byte
 * line.  The octets of SNPs are 164 (196) words apart, 4 banks, so that the 8 threads of a line
 * read different banks.  Writing 4 S bytes per genotype to HBM bounds it.
 */
#define EX_SJT 8
#define EX_OCT(S) (32 * (S) + 4)
template <int S>
__global__ void __launch_bounds__(8 * EX_J(S))
k_exact_slices(const uint8_t *__restrict__ codes, int64_t ldc, int32_t n, int32_t ntj,
               const int32_t *__restrict__ kept, int32_t nkept, const double *__restrict__ vtab,
               const double *__restrict__ xfancy, int e, int32_t kb0, uint8_t *__restrict__ B)
{
  __shared__ uint32_t tab[8 * EX_OCT(S)];
  const int tid = threadIdx.x;
  const int32_t kb = kb0 + (int32_t)blockIdx.x;
  {
    for (int i = tid; i < 8 * EX_OCT(S); i += blockDim.x) tab[i] = 0;
    __syncthreads();
    /* entry (SNP u, term st, code g); code 3 stays zero */
    for (int i = tid; i < 6 * EX_K; i += blockDim.x) {
      const int u = i / 6, st = (i / 3) & 1, g = i % 3;
      const int32_t k = kb * EX_K + u;
      if (k >= nkept) continue;
      const int64_t c = kept[k];
      const double v = vtab[4 * c + g];
      __half *h = (__half *)(tab + (u >> 3) * EX_OCT(S) + (u & 7) * (4 * S) + g * S) + S * st;
      if (S == 5) {
        /* R 2^(59 - E): a power of two within range for any table of this path */
        const double r = (st ? vtab[4 * c + 1] : xfancy[c]) * v;
        ex_cut<5>(__double2ll_rn(scalbn(r, EX_BITS(5) - e)), h);
      } else {
        /* f, or T1 = T0 + f or T2 - f by TwoSum (Knuth), and R by the FMA's exact product, each as
         * a sum a + al; R 2^(35 - E) = N + (the part of R 2^(71 - E) below it), three digits each */
        double a = xfancy[c], al = 0.0;
        if (st) {
          const double t0 = vtab[4 * c], t2 = vtab[4 * c + 2];
          const double x = fabs(t0) <= fabs(t2) ? t0 : t2, y = fabs(t0) <= fabs(t2) ? a : -a;
          a = x + y;
          const double z = a - x;
          al = (x - (a - z)) + (y - z);
        }
        const double r = __dmul_rn(a, v), rl = fma(al, v, fma(a, v, -r));
        const double w = scalbn(r, 35 - e), N = rint(w);
        ex_cut<3>((long long)N, h);
        ex_cut<3>(__double2ll_rn(fma(w - N, 0x1p36, scalbn(rl, 71 - e))), h + 3);
      }
    }
  }
  __syncthreads();
  const int o = tid & 7, jj = tid >> 3;
  const uint32_t *to = tab + o * EX_OCT(S);
  const int32_t jt1 = min(ntj, ((int32_t)blockIdx.y + 1) * EX_SJT);
  for (int32_t jt = (int32_t)blockIdx.y * EX_SJT; jt < jt1; ++jt) {
    const int32_t j = jt * EX_J(S) + jj;
    /* codes 8o..8o+7 of the block: bytes 2o, 2o+1 of the row's 16, MSB first */
    uint32_t cw = 0xFFFFu;
    if (j < n) cw = *(const uint16_t *)(codes + (int64_t)j * ldc + (int64_t)kb * 16 + 2 * o);
    uint32_t out[2 * S][4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int b0 = (p >> 1) * 8 + 6 - 4 * (p & 1);
      const uint32_t *e0 = to + (2 * p) * (4 * S) + ((cw >> b0) & 3u) * S;
      const uint32_t *e1 = to + (2 * p + 1) * (4 * S) + ((cw >> (b0 - 2)) & 3u) * S;
#pragma unroll
      for (int w = 0; w < S; ++w) {
        const uint32_t x = e0[w], y = e1[w];
        out[2 * w][p] = __byte_perm(x, y, 0x5410);
        out[2 * w + 1][p] = __byte_perm(x, y, 0x7632);
      }
    }
    uint8_t *dst = B + ((int64_t)blockIdx.x * ntj + jt) * (2 * EX_B_BYTES);
#pragma unroll
    for (int d = 0; d < 2 * S; ++d) {
      const int r = (d % S) * EX_J(S) + jj;
      *(uint4 *)(dst + (d / S) * EX_B_BYTES + r * 128 + ((o ^ (r & 7)) << 4)) =
          make_uint4(out[d][0], out[d][1], out[d][2], out[d][3]);
    }
  }
}

/* ---- the Gram kernel ------------------------------------------------------------------- */

__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar)
{
  asm volatile(
      "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
      "@e cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      "\n\t}\n" ::"r"(
          smem_u32(dst)),
      "l"((uint64_t)__cvta_generic_to_global(src)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *r)
{
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
}

template <int S>
__global__ void __launch_bounds__(EX_THREADS, 1)
k_gram_exact(const uint8_t *__restrict__ codes, int64_t ldc, int32_t n, int32_t ntiles, int32_t ntj,
             int32_t kb0, int32_t nkb, int32_t ksplit, const uint8_t *__restrict__ B,
             unsigned long long *sums, int *err)
{
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = (uint64_t *)(smem + EX_STAGES * EX_STAGE_BYTES);
  uint64_t *full = bars, *empty = bars + EX_STAGES, *accf = bars + 2 * EX_STAGES,
           *acce = bars + 2 * EX_STAGES + 1, *drain = bars + 2 * EX_STAGES + 2;
  uint32_t *tmem_slot = (uint32_t *)(bars + 2 * EX_STAGES + 3);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  /* items: tile fastest, so that CTAs at work together read the same k range of B */
  const int32_t nitems = ntiles * ksplit, kb_per = (nkb + ksplit - 1) / ksplit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < EX_STAGES; ++s) {
      mbar_init(&full[s], 1 + EX_DEC_WARPS);
      mbar_init(&empty[s], 1);
    }
    mbar_init(accf, 1);
    mbar_init(acce, EX_EPI_WARPS);
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    /* ---------------- right tiles ---------------- */
    uint32_t it = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      int32_t bi, jt;
      ex_tile<S>(w % ntiles, n, &bi, &jt);
      const int32_t a = w / ntiles * kb_per, b = min(nkb, a + kb_per);
      for (int32_t kb = a; kb < b && ok; ++kb) {
        const uint8_t *src = B + ((int64_t)kb * ntj + jt) * (2 * EX_B_BYTES);
        for (int st = 0; st < 2; ++st, ++it) {
          const uint32_t s = it % EX_STAGES, ph = (it / EX_STAGES) & 1u;
          if (!mbar_wait_warp(&empty[s], ph ^ 1u, abort_flag, err, EXERR_EMPTY)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx_warp(&full[s], EX_B_BYTES);
          bulk_load(smem + s * EX_STAGE_BYTES + 2 * EX_A_BYTES, src + st * EX_B_BYTES,
                    EX_B_BYTES, &full[s]);
        }
      }
    }
    if (*abort_flag) {
      /* copies already issued must land before the CTA exits: a stage's barrier completes
       * only if the decoders arrived too, so wait for the time a copy can take at most */
      const uint64_t t0 = globaltimer_ns();
      const uint32_t last = it < EX_STAGES ? it : EX_STAGES;
      for (uint32_t j = it - last; j < it; ++j)
        while (!mbar_try_wait(&full[j % EX_STAGES], (j / EX_STAGES) & 1u) &&
               globaltimer_ns() - t0 < GP_WAIT_NS) {
        }
    }
  } else if (warp == 1) {
    /* ---------------- MMA issuer ---------------- */
    const uint32_t idesc = idesc_f16_f32(128, EX_N);
    uint32_t it = 0, chunk = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      int32_t bi, jt;
      bool h0, h1;
      ex_tile<S>(w % ntiles, n, &bi, &jt);
      ex_halves<S>(bi, jt, n, &h0, &h1);
      const int32_t a = w / ntiles * kb_per, b = min(nkb, a + kb_per);
      for (int32_t c0 = a; c0 < b && ok; c0 += EX_CHUNK_KB, ++chunk) {
        const int32_t c1 = min(b, c0 + EX_CHUNK_KB);
        if (!mbar_wait_warp(acce, (chunk & 1u) ^ 1u, abort_flag, err, EXERR_ACCE)) {
          ok = false;
          break;
        }
        tc_fence_after();
        for (int32_t q = 2 * c0; q < 2 * c1; ++q, ++it) {
          const uint32_t s = it % EX_STAGES, ph = (it / EX_STAGES) & 1u;
          if (!mbar_wait_warp(&full[s], ph, abort_flag, err, EXERR_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t base = smem_u32(smem + s * EX_STAGE_BYTES);
          const uint64_t a0 = sdesc_k128(base), a1 = sdesc_k128(base + EX_A_BYTES),
                         bd = sdesc_k128(base + 2 * EX_A_BYTES);
#pragma unroll
          for (int k = 0; k < EX_K / 16; ++k) {
            const uint32_t acc = (q > 2 * c0 || k > 0) ? 1u : 0u;
            if (h0) umma_bf16(tmem, a0 + 2 * k, bd + 2 * k, idesc, acc);
            if (h1) umma_bf16(tmem + EX_D1, a1 + 2 * k, bd + 2 * k, idesc, acc);
          }
          umma_commit(&empty[s]);
        }
        if (ok) umma_commit(accf);
      }
    }
  } else if (warp < 2 + EX_DEC_WARPS) {
    /* ---------------- decoders: a thread per row of the tile ---------------- */
    const int r = (warp - 2) * 32 + lane;
    uint8_t *rowp = smem + (r >> 7) * EX_A_BYTES + (r & 127) * 128;
    const uint32_t sw = (uint32_t)(r & 7);
    /* high bytes of the fp16 values of codes 0, 1, 2, 3 (byte 0 first) */
    const uint32_t tab[2] = {0x003C00BCu, 0x003C3C3Cu}; /* h: -1, 0, 1, 0; o: 1, 1, 1, 0 */
    uint32_t it = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      int32_t bi, jt;
      bool h0, h1;
      ex_tile<S>(w % ntiles, n, &bi, &jt);
      ex_halves<S>(bi, jt, n, &h0, &h1);
      const int32_t a = w / ntiles * kb_per, b = min(nkb, a + kb_per);
      const int32_t grow = bi * EX_ROWS + r;
      const bool half_on = r < 128 ? h0 : h1, live = half_on && grow < n;
      const uint8_t *crow = codes + (int64_t)(live ? grow : 0) * ldc;
      auto ld_codes = [&](int32_t kb) {
        return live && kb < b ? __ldg((const uint4 *)(crow + (int64_t)(kb0 + kb) * 16))
                              : make_uint4(~0u, ~0u, ~0u, ~0u);
      };
      uint4 pf[EX_PF];
#pragma unroll
      for (int u = 0; u < EX_PF; ++u) pf[u] = ld_codes(a + u);
      for (int32_t kbb = a; kbb < b && ok; kbb += EX_PF) {
#pragma unroll
        for (int u = 0; u < EX_PF; ++u) {
          if (kbb + u >= b) break;
          const uint32_t words[4] = {pf[u].x, pf[u].y, pf[u].z, pf[u].w};
          pf[u] = ld_codes(kbb + u + EX_PF);
#pragma unroll
          for (int st = 0; st < 2; ++st, ++it) {
            const uint32_t s = it % EX_STAGES, ph = (it / EX_STAGES) & 1u;
            const bool got = mbar_wait(&empty[s], ph ^ 1u, abort_flag, err, EXERR_EMPTY);
            if (!__all_sync(0xffffffffu, got)) {
              ok = false;
              break;
            }
            if (half_on) {
              uint8_t *dst = rowp + s * EX_STAGE_BYTES;
#pragma unroll
              for (int o = 0; o < 8; ++o) {
                /* codes 8o..8o+7: bytes 2o, 2o+1 of the row's 16 */
                uint32_t s01, s23, s45, s67;
                const uint32_t hw = words[o >> 1] >> ((o & 1) * 16);
                code_selectors(hw & 0xFFu, &s01, &s23);
                code_selectors((hw >> 8) & 0xFFu, &s45, &s67);
                *(uint4 *)(dst + (((uint32_t)o ^ sw) << 4)) =
                    make_uint4(__byte_perm(tab[st], 0, s01), __byte_perm(tab[st], 0, s23),
                               __byte_perm(tab[st], 0, s45), __byte_perm(tab[st], 0, s67));
              }
              fence_proxy_async_smem();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&full[s]);
          }
          if (!ok) break;
        }
      }
    }
  } else {
    /* ---------------- epilogue ---------------- */
    const int q = warp & 3, half = (warp - 2 - EX_DEC_WARPS) >> 2;
    const uint32_t t_acc = tmem + ((uint32_t)(q * 32) << 16) + half * EX_D1;
    uint32_t chunk = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      int32_t bi, jt;
      bool h0, h1;
      const int32_t tile = w % ntiles;
      ex_tile<S>(tile, n, &bi, &jt);
      ex_halves<S>(bi, jt, n, &h0, &h1);
      const int32_t a = w / ntiles * kb_per, b = min(nkb, a + kb_per);
      /* column u of this warp's 32 rows, all lanes together; upper sums, then lower */
      unsigned long long *out =
          sums + (int64_t)tile * (2 * EX_TILE(S)) + (half * 4 + q) * (EX_J(S) * 32) + lane;
      for (int32_t c0 = a; c0 < b; c0 += EX_CHUNK_KB, ++chunk) {
        const bool got = mbar_wait(accf, chunk & 1u, abort_flag, err, EXERR_ACCF);
        if (!__all_sync(0xffffffffu, got)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (half ? h1 : h0) {
#pragma unroll
          for (int g = 0; g < EX_J(S) / 8; ++g) {
            uint32_t d[S][8];
#pragma unroll
            for (int t = 0; t < S; ++t) tmem_ld8(t_acc + t * EX_J(S) + 8 * g, d[t]);
            tmem_wait_ld();
#pragma unroll
            for (int v = 0; v < 8; ++v) {
              long long hi = 0, lo = 0;
#pragma unroll
              for (int t = 0; t < 3; ++t) hi = (hi << 12) + __float2int_rn(__uint_as_float(d[t][v]));
#pragma unroll
              for (int t = 3; t < S; ++t) lo = (lo << 12) + __float2int_rn(__uint_as_float(d[t][v]));
              const int at = (8 * g + v) * 32;
              atomicAdd(out + at, (unsigned long long)hi);
              atomicAdd(out + EX_TILE(S) + at, (unsigned long long)lo);
            }
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(acce);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) {
    if (*abort_flag) {
      umma_commit(drain);
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try_wait(drain, 0) && globaltimer_ns() - t0 < GP_WAIT_NS) {
      }
    }
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

/*
 * XTX[i][j] = XTX[j][i] = 2^(E-59) (2^24 hi + lo), or 2^(E-71) (2^36 hi + lo) with six digits,
 * for the tile's entries of the lower triangle; a CTA per 128 rows x half of the columns, transposed through shared memory so that both the row
 * pieces (24 or 20 doubles) and the column pieces (128 doubles) are written contiguously.
 */
template <int S>
__global__ void __launch_bounds__(256)
k_exact_finish(const unsigned long long *__restrict__ sums, int e, int32_t n, double *x)
{
  constexpr int EX_FC = EX_J(S) / 2;
  __shared__ double sm[128][EX_FC + 1];
  int32_t bi, jt;
  ex_tile<S>((int32_t)blockIdx.x, n, &bi, &jt);
  const int half = (int)blockIdx.y, jh = (int)blockIdx.z;
  const int32_t i0 = bi * EX_ROWS + 128 * half, j0 = jt * EX_J(S) + jh * EX_FC;
  bool h0, h1;
  ex_halves<S>(bi, jt, n, &h0, &h1);
  if (!(half ? h1 : h0)) return;
  for (int p = threadIdx.x; p < 128 * EX_FC; p += blockDim.x) {
    const int lane = p & 31, c = (p >> 5) % EX_FC, q = (p >> 5) / EX_FC;
    const unsigned long long *src = sums + (int64_t)blockIdx.x * (2 * EX_TILE(S)) +
                                    (half * 4 + q) * (EX_J(S) * 32) + (jh * EX_FC + c) * 32 + lane;
    const double hi = (double)(long long)src[0], lo = (double)(long long)src[EX_TILE(S)];
    sm[q * 32 + lane][c] = scalbn(fma(hi, S == 5 ? 0x1p24 : 0x1p36, lo), e - EX_BITS(S));
  }
  __syncthreads();
  for (int p = threadIdx.x; p < 128 * EX_FC; p += blockDim.x) {
    const int r = p / EX_FC, c = p - r * EX_FC;
    const int32_t i = i0 + r, j = j0 + c;
    if (i < n && j <= i) x[(int64_t)i * n + j] = sm[r][c];
  }
  for (int p = threadIdx.x; p < 128 * EX_FC; p += blockDim.x) {
    const int c = p >> 7, r = p & 127;
    const int32_t i = i0 + r, j = j0 + c;
    if (i < n && j < i) x[(int64_t)j * n + i] = sm[r][c];
  }
}

/* ---- host ------------------------------------------------------------------------------ */

/* splits of the k range: the count (at most 32, each at least 4 k-blocks) whose busiest CTA
 * does least, a work item costing its k-blocks and about 3 more (ring fill, TMEM read, atomics) */
static int32_t ex_split(int32_t ntiles, int32_t nkb, int32_t sms)
{
  int32_t best = 1;
  int64_t best_cost = INT64_MAX;
  for (int32_t s = 1; s <= 32; ++s) {
    const int32_t per = (nkb + s - 1) / s;
    if (s > 1 && per < 4) break;
    const int64_t cost = (((int64_t)ntiles * s + sms - 1) / sms) * (per + 3);
    if (cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

/*
 * Digits for a largest |R| below 2^e over nk SNPs.  The rounding of R leaves an entry an error of
 * about 2^(e-61) sqrt(nk), a sequence of FP64 additions 2^-55 nk (their partial sums are about
 * sqrt(nk) with the SNPs' signs mixed): five digits where the first is at most half of the second.
 * Panels of common SNPs (e = 6 or 7) take five from 16 SNPs on.  Six cost 1.2 times the MMAs: 5,003
 * samples x 20,000 SNPs with frequencies from 2e-4 on 4.66 ms, of 3.97, and 2,003 x 20,011 0.91, of
 * 0.78.
 */
static int ex_digits(int e, int32_t nk) { return 2 * (e - 5) <= ilogb((double)nk) ? 5 : 6; }

int gp_gram_exact_max(gp_ctx *ctx, double *d_part)
{
  k_exact_max<<<GP_EXACT_PARTS, 256, 0, ctx->stream>>>(ctx->ncols, ctx->d_vtab, ctx->d_xfancy, d_part);
  GP_LAUNCH_CHECK(ctx, "k_exact_max");
  return GP_OK;
}

template <int S>
static int gram_exact(gp_ctx *ctx, int e)
{
  const int32_t n = ctx->nrows, nk = ctx->nkept;
  const int32_t ntj = (n + EX_J(S) - 1) / EX_J(S), nkb = (nk + EX_K - 1) / EX_K;
  int32_t ntiles = 0;
  for (int32_t b = 0; b * EX_ROWS < n; ++b) ntiles += ex_row_tiles(b, n, EX_J(S));
  uint8_t *B;
  unsigned long long *sums;
  int32_t *snprec;
  int rc = gp_scratch(ctx, sizeof(int32_t) * (size_t)nk, (void **)&snprec);
  if (rc) return rc;
  const size_t sum_bytes = sizeof(*sums) * 2 * EX_TILE(S) * (size_t)ntiles;
  rc = gp_scratch5(ctx, sum_bytes, (void **)&sums);
  if (rc) return rc;
  /* the right operand of as many k-blocks as fit the budget, fewer where memory is short */
  const size_t per_kb = 2 * EX_B_BYTES * (size_t)ntj;
  int32_t kbp = (int32_t)(EX_BUDGET / (int64_t)per_kb);
  {
    const char *env = getenv("GP_EXACT_BUDGET_BYTES"); /* tests: several passes on a small panel */
    if (env && atoll(env) > 0) kbp = (int32_t)(atoll(env) / (int64_t)per_kb);
  }
  if (kbp < 1) kbp = 1;
  if (kbp > nkb) kbp = nkb;
  const int32_t npass = (nkb + kbp - 1) / kbp;
  kbp = (nkb + npass - 1) / npass;
  while ((rc = gp_scratch2(ctx, per_kb * kbp, (void **)&B)) == GP_ERR_NOMEM && kbp > 1) {
    cudaGetLastError();
    kbp = (kbp + 1) / 2;
  }
  if (rc) return rc;

  rc = gp_tc_begin(ctx);
  if (rc) return rc;
  const int64_t nsums = (int64_t)(sum_bytes / sizeof(*sums));
  const int64_t work = nsums / 2 > nk ? nsums / 2 : nk;
  const int64_t blocks = (work + 255) / 256 < ctx->num_sms * 16 ? (work + 255) / 256 : ctx->num_sms * 16;
  k_exact_begin<<<(unsigned)blocks, 256, 0, ctx->stream>>>(ctx->d_kept, nk, ctx->d_cols, snprec, sums,
                                                          nsums);
  GP_LAUNCH_CHECK(ctx, "k_exact_begin");
  gp_tc_codes A;
  rc = gp_tc_codes_for(ctx, 1, ctx->d_rows, n, snprec, nk, 1, &A);
  if (rc) return rc;
  GP_CUDA(ctx, cudaFuncSetAttribute(k_gram_exact<S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    EX_SMEM));
  for (int32_t kb0 = 0; kb0 < nkb; kb0 += kbp) {
    const int32_t cur = nkb - kb0 < kbp ? nkb - kb0 : kbp;
    dim3 sg((unsigned)cur, (unsigned)((ntj + EX_SJT - 1) / EX_SJT));
    k_exact_slices<S><<<sg, 8 * EX_J(S), 0, ctx->stream>>>(A.codes, A.ldc, n, ntj, ctx->d_kept, nk,
                                                          ctx->d_vtab, ctx->d_xfancy, e, kb0, B);
    GP_LAUNCH_CHECK(ctx, "k_exact_slices");
    const int32_t ks = ex_split(ntiles, cur, ctx->num_sms);
    const int32_t items = ntiles * ks;
    k_gram_exact<S><<<items < ctx->num_sms ? items : ctx->num_sms, EX_THREADS, EX_SMEM,
                      ctx->stream>>>(
        A.codes, A.ldc, n, ntiles, ntj, kb0, cur, ks, B, sums, ctx->d_err);
    GP_LAUNCH_CHECK(ctx, "k_gram_exact");
    ctx->gram_launches++;
  }
  k_exact_finish<S><<<dim3((unsigned)ntiles, 2, 2), 256, 0, ctx->stream>>>(sums, e, n, ctx->d_xtx);
  GP_LAUNCH_CHECK(ctx, "k_exact_finish");
  return GP_OK;
}

int gp_gram_exact(gp_ctx *ctx, const double *part)
{
  double big = 0.0;
  for (int i = 0; i < GP_EXACT_PARTS; ++i) big = part[i] > big ? part[i] : big;
  int e = 0;
  if (big > 0.0) frexp(big, &e); /* big < 2^e */
  return ex_digits(e, ctx->nkept) == 5 ? gram_exact<5>(ctx, e) : gram_exact<6>(ctx, e);
}
