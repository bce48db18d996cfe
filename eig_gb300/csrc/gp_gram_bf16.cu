/*
 * Split-BF16 Gram on the 5th-generation tensor cores (tcgen05), replacing the reference's
 * XTX accumulation (domult_increment_lookup / block_increment_binary,
 * src/eigensrc/smartpca.c:3361-3495) for GP_PREC_SPLIT_BF16.
 *
 * Each normalised value v (the FP64 table entry of its SNP and genotype code) is split into
 * hi = r(v) and lo = r(v - hi) in a 16-bit format (bf16 or fp16).  XTX = Xhi Xhi^T +
 * Xhi Xlo^T + Xlo Xhi^T (+ Xlo Xlo^T with 4 MMAs): tcgen05 MMAs with FP32 accumulation in
 * TMEM over a short SNP chunk (128 SNPs by default: the tensor core's FP32 accumulation
 * truncates, so its error grows with the chunk depth), chunk sums added in FP32 registers
 * (round to nearest) for a few chunks, then folded into a per-element running sum held in
 * TMEM as an FP32 (hi, lo) pair with TwoSum (~48 bits), which stands in for FP64
 * accumulation at FP32 speed (GB300's FP64 rate is a small fraction of its FP32 rate); the
 * tile is written out in FP64.
 *
 * Data layout in HBM: Xhi and Xlo as [Kc / 64][Npad][64] (for each k-block of 64 kept SNPs of
 * the current super-chunk, the samples' 128-byte rows one after the other), written by
 * k_split_transpose from the packed records; the Gram kernel reads them with TMA as boxes of
 * 128 such rows, 16 KB in a piece, in the 128-byte swizzle.
 *
 * Kernel structure (persistent, one CTA per SM, 18 warps):
 *   warp 0      TMA producer: per k-block of 64 SNPs four 16 KB boxes (A hi/lo, B hi/lo)
 *               into a 3-stage shared-memory ring;
 *   warp 1      allocates 512 TMEM columns; issues 12 (or 16) tcgen05.mma (128x128x16) per
 *               k-block, converged, one elected lane each, into FP32 accumulator buffer
 *               (chunk & 1), columns 0-255;
 *   warps 2-17  epilogue: at the end of each chunk read the FP32 buffer (tcgen05.ld),
 *               release it and add it into registers; every GP_FOLD chunks fold those into
 *               the (hi, lo) running sums in TMEM columns 256-511; after the last chunk of a
 *               tile write the tile to the Gram in FP64.
 * Tiles are the 128x128 blocks of the lower triangle, distributed round-robin over the CTAs;
 * the tiles of a last wave that would leave half of the CTAs or more without work are cut along
 * the SNPs into as many parts as there are CTAs for (at fold boundaries, so that every FP32 sum
 * is the same), and k_gram_parts adds the parts.
 *
 * What bounds it is the shared memory's 128 bytes a clock: a 128x128x16 MMA reads 8 KB, so the 12
 * MMAs of a k-block read 96 KB and its boxes' 64 KB come in: 1,250 clocks, against 768 of tensor
 * work; measured 1,285 (5,000 x 600,000 in split fp16: 35.0 ms with the transpose, 43.4 before the
 * warp-wide issue, the k-block layout and the parts).  The pieces of the running sums fill the
 * TMEM, so a CTA's tile cannot be larger.  Tried and not kept: pairs of CTAs (cta_group::2,
 * 256x128, 120 KB a k-block) wait for one another's barriers, 1,430 clocks (1,000 with the loads
 * left out); clusters of four CTAs that share their boxes by multicast halve the L2 reads, which
 * are not the limit: the same 38.2 ms without the parts, and 2 x 2 blocks of tiles fill the last
 * wave worse (3,001 samples: 2.04 against 1.46 ms).
 */
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>

#include <stdlib.h>

#include "gp_internal.h"
#include "gp_tc.cuh"

#define BT 128          /* tile edge (rows of A and B) */
#define BK 64           /* SNPs per k-block (128 bytes of bf16) */
#define NSTAGE 3
#define BOX_BYTES (BT * BK * 2)
#define STAGE_BYTES (4 * BOX_BYTES)
#ifndef EPI_COLS
#define EPI_COLS 32 /* tile columns per epilogue thread */
#endif
#ifndef GP_FOLD
#define GP_FOLD 8   /* chunks summed in FP32 registers before the TwoSum fold */
#endif
#define GRAM_THREADS (64 + 32 * 4 * (128 / EPI_COLS)) /* producer + MMA + epilogue warps */
#define GRAM_SMEM (NSTAGE * STAGE_BYTES + 1024 + 256)

/* error codes recorded by the kernel */
#define GP_KERR_TIMEOUT_FULL 1
#define GP_KERR_TIMEOUT_EMPTY 2
#define GP_KERR_TIMEOUT_ACCF 3
#define GP_KERR_TIMEOUT_ACCE 4
#define GP_KERR_TIMEOUT_SYNC 5
#define GRAM_SYNC_KB 64 /* k-blocks between the producers' lockstep points */
#define GRAM_PART_FOLDS 4 /* folds of the smallest part (4,096 SNPs: 40 us) */

__device__ __forceinline__ int32_t tri_root(int32_t t)
{
  int32_t i = (int32_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
  while ((i + 1) * (i + 2) / 2 <= t) ++i;
  while (i * (i + 1) / 2 > t) --i;
  return i;
}

/*
 * Tile t of the lower triangle of nt x nt tiles, in groups: the tile grid is cut into
 * GRAM_GROUP x GRAM_GROUP blocks (lower triangle of blocks, row by row), tiles row by row
 * inside a block.  The CTAs that run at the same time then hold tiles of a few row blocks
 * and walk the SNPs at the same pace, so the operand boxes they load are shared in L2
 * instead of being read from HBM once per tile.
 */
#define GRAM_GROUP 12
__device__ __forceinline__ void tri_tile(int32_t t, int32_t nt, int32_t *bi, int32_t *bj)
{
  const int32_t ng = (nt + GRAM_GROUP - 1) / GRAM_GROUP;
  for (int32_t gi = 0; gi < ng; ++gi) {
    const int32_t r0 = gi * GRAM_GROUP, nr = min(nt, r0 + GRAM_GROUP) - r0;
    for (int32_t gj = 0; gj <= gi; ++gj) {
      const int32_t c0 = gj * GRAM_GROUP, nc = min(nt, c0 + GRAM_GROUP) - c0;
      const int32_t cnt = gi == gj ? nr * (nr + 1) / 2 : nr * nc;
      if (t < cnt) {
        if (gi == gj) {
          const int32_t i = tri_root(t);
          *bi = r0 + i;
          *bj = c0 + t - i * (i + 1) / 2;
        } else {
          *bi = r0 + t / nc;
          *bj = c0 + t % nc;
        }
        return;
      }
      t -= cnt;
    }
  }
  *bi = *bj = 0; /* not reached for t < ntiles */
}

/* a CTA's work: nfull whole tiles, then the other tiles in nsplit parts each */
struct gram_plan {
  int32_t nt;       /* tile rows */
  int32_t nfull;    /* tiles done whole: the first ones */
  int32_t nsplit;   /* parts of each further tile */
  int32_t nitems;   /* nfull + nsplit (ntiles - nfull) */
  int32_t nkb;      /* k-blocks */
  int32_t chunk_kb; /* k-blocks per FP32 accumulation chunk */
};

/* item w: its tile and its k-blocks [*kb0, *kb1), whole folds unless the last */
__device__ __forceinline__ void gram_item(const gram_plan &p, int32_t w, int32_t *bi, int32_t *bj,
                                          int32_t *kb0, int32_t *kb1)
{
  const int32_t u = w - p.nfull;
  tri_tile(u < 0 ? w : p.nfull + u / p.nsplit, p.nt, bi, bj);
  *kb0 = 0;
  *kb1 = p.nkb;
  if (u >= 0) {
    const int32_t fold_kb = GP_FOLD * p.chunk_kb, nf = (p.nkb + fold_kb - 1) / fold_kb;
    const int32_t q = u % p.nsplit;
    *kb0 = (int32_t)((int64_t)nf * q / p.nsplit) * fold_kb;
    *kb1 = min(p.nkb, (int32_t)((int64_t)nf * (q + 1) / p.nsplit) * fold_kb);
  }
}

/*
 * grams: XTX (n x n row-major FP64); accumulate != 0 adds to the values already there
 * (super-chunks after the first).  The items after the whole tiles go to parts, [item][128][128].
 */
template <int FP16, int NMMA>
__global__ void __launch_bounds__(GRAM_THREADS, 1)
k_gram_split(const __grid_constant__ CUtensorMap tm_hi, const __grid_constant__ CUtensorMap tm_lo,
             gram_plan p, double *xtx, int32_t n, int32_t accumulate, double *parts,
             unsigned *sync_ctr, int *err)
{
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = (uint64_t *)(smem + NSTAGE * STAGE_BYTES);
  uint64_t *full = bars;                 /* [NSTAGE] */
  uint64_t *empty = bars + NSTAGE;       /* [NSTAGE] */
  uint64_t *accf = bars + 2 * NSTAGE;    /* [2] */
  uint64_t *acce = bars + 2 * NSTAGE + 2;/* [2] */
  uint64_t *drain = bars + 2 * NSTAGE + 4; /* abort path: wait for issued MMAs */
  uint32_t *tmem_slot = (uint32_t *)(bars + 2 * NSTAGE + 5);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGE; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], 4 * (128 / EPI_COLS));
    }
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tm_hi);
    tma_prefetch_desc(&tm_lo);
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    /* ---------------- TMA producer ---------------- */
    uint32_t it = 0;
    bool ok = true;
    const int32_t nsync = (p.nkb + GRAM_SYNC_KB - 1) / GRAM_SYNC_KB;
    for (int32_t w = blockIdx.x; w < p.nitems && ok; w += gridDim.x) {
      int32_t bi, bj, kb0, kb1;
      gram_item(p, w, &bi, &bj, &kb0, &kb1);
      /* the CTAs of one wave of whole tiles meet every GRAM_SYNC_KB k-blocks, so that the boxes
       * one of them loads are still in L2 when the others need them */
      const int32_t wave = w / (int32_t)gridDim.x;
      const unsigned wave_n = (unsigned)min((int32_t)gridDim.x, p.nfull - wave * (int32_t)gridDim.x);
      for (int32_t kb = kb0; kb < kb1; ++kb, ++it) {
        if (w < p.nfull && kb > 0 && kb % GRAM_SYNC_KB == 0) {
          unsigned *ctr = sync_ctr + (int64_t)wave * nsync + kb / GRAM_SYNC_KB;
          bool met = true;
          if (lane == 0) {
            atomicAdd(ctr, 1u);
            volatile unsigned *vc = ctr;
            const uint64_t t0 = globaltimer_ns();
            while (met && *vc < wave_n) {
              if (*abort_flag) {
                met = false;
              } else if (globaltimer_ns() - t0 > GP_WAIT_NS) {
                atomicExch(err, GP_KERR_TIMEOUT_SYNC);
                *abort_flag = 1;
                met = false;
              }
            }
          }
          ok = __all_sync(0xffffffffu, met);
          if (!ok) break;
        }
        const uint32_t s = it % NSTAGE, ph = (it / NSTAGE) & 1u;
        ok = mbar_wait_warp(&empty[s], ph ^ 1u, abort_flag, err, GP_KERR_TIMEOUT_EMPTY);
        if (!ok) break;
        uint8_t *st = smem + s * STAGE_BYTES;
        const int32_t ya = (kb * p.nt + bi) * BT, yb = (kb * p.nt + bj) * BT;
        mbar_arrive_expect_tx_warp(&full[s], STAGE_BYTES);
        tma_load_2d(st, &tm_hi, &full[s], 0, ya);
        tma_load_2d(st + BOX_BYTES, &tm_lo, &full[s], 0, ya);
        tma_load_2d(st + 2 * BOX_BYTES, &tm_hi, &full[s], 0, yb);
        tma_load_2d(st + 3 * BOX_BYTES, &tm_lo, &full[s], 0, yb);
      }
    }
    if (*abort_flag) {
      /* copies already issued must land before the CTA exits (bounded) */
      const uint32_t last = it < NSTAGE ? it : NSTAGE;
      for (uint32_t j = it - last; j < it; ++j) {
        const uint64_t t0 = globaltimer_ns();
        while (!mbar_try_wait(&full[j % NSTAGE], (j / NSTAGE) & 1u) &&
               globaltimer_ns() - t0 < GP_WAIT_NS) {
        }
      }
    }
  } else if (warp == 1) {
    /* ---------------- MMA issuer ---------------- */
    const uint32_t idesc = FP16 ? idesc_f16_f32(BT, BT) : idesc_bf16_f32(BT, BT);
    uint32_t it = 0, chunk = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < p.nitems && ok; w += gridDim.x) {
      int32_t bi, bj, kb0, kb1;
      gram_item(p, w, &bi, &bj, &kb0, &kb1);
      for (int32_t c0 = kb0; c0 < kb1 && ok; c0 += p.chunk_kb, ++chunk) {
        const uint32_t buf = chunk & 1u, use = chunk >> 1;
        ok = mbar_wait_warp(&acce[buf], (use & 1u) ^ 1u, abort_flag, err, GP_KERR_TIMEOUT_ACCE);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d = tmem + buf * BT;
        const int32_t c1 = min(kb1, c0 + p.chunk_kb);
        for (int32_t kb = c0; kb < c1; ++kb, ++it) {
          const uint32_t s = it % NSTAGE, ph = (it / NSTAGE) & 1u;
          ok = mbar_wait_warp(&full[s], ph, abort_flag, err, GP_KERR_TIMEOUT_FULL);
          if (!ok) break;
          tc_fence_after();
          const uint32_t base = smem_u32(smem + s * STAGE_BYTES);
          const uint64_t ahi = sdesc_k128(base), alo = sdesc_k128(base + BOX_BYTES);
          const uint64_t bhi = sdesc_k128(base + 2 * BOX_BYTES);
          const uint64_t blo = sdesc_k128(base + 3 * BOX_BYTES);
#pragma unroll
          for (int k = 0; k < BK / 16; ++k) {
            /* +32 bytes along K per 16 bf16 = +2 in the 16-byte address field */
            const uint64_t o = (uint64_t)(2 * k);
            const uint32_t acc0 = (kb > c0 || k > 0) ? 1u : 0u;
            umma_bf16(d, ahi + o, bhi + o, idesc, acc0);
            umma_bf16(d, ahi + o, blo + o, idesc, 1u);
            umma_bf16(d, alo + o, bhi + o, idesc, 1u);
            if (NMMA == 4) umma_bf16(d, alo + o, blo + o, idesc, 1u);
          }
          umma_commit(&empty[s]);
        }
        if (ok) umma_commit(&accf[buf]);
      }
    }
  } else {
    /* ---------------- epilogue (warps 2..17) ----------------
     * Warp w reads TMEM lanes 32*(w%4)..+31 (its row quarter); the four warps of a quarter
     * take EPI_COLS columns each.  Three levels of accumulation:
     *   tensor core  FP32 over one chunk (chunk_kb k-blocks) in TMEM buffer (chunk & 1);
     *   registers    FP32 (round-to-nearest) sum of GP_FOLD chunks, A[];
     *   TMEM         running sum as an FP32 (hi, lo) pair updated with TwoSum (~48 bits),
     *                columns 256+col (hi) and 384+col (lo), written out in FP64 per tile.
     * No FP64 arithmetic on the per-chunk path (GB300's FP64 rate is low). */
    const int q = warp & 3;
    const int row = q * 32 + lane;
    const int col0 = ((warp - 2) >> 2) * EPI_COLS;
    const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
    const uint32_t t_acc = tmem + lane_addr;
    uint32_t chunk = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < p.nitems && ok; w += gridDim.x) {
      int32_t bi, bj, kb0, kb1;
      gram_item(p, w, &bi, &bj, &kb0, &kb1);
      const int32_t nchunk = (kb1 - kb0 + p.chunk_kb - 1) / p.chunk_kb;
      const int32_t gi = bi * BT + row;
      const int32_t gj0 = bj * BT + col0;
      float A[EPI_COLS];
      {
        uint32_t z[16];
#pragma unroll
        for (int v = 0; v < 16; ++v) z[v] = 0u;
#pragma unroll
        for (int g = 0; g < EPI_COLS / 16; ++g) {
          tmem_st16(t_acc + 256 + col0 + 16 * g, z);
          tmem_st16(t_acc + 384 + col0 + 16 * g, z);
        }
        tmem_wait_st();
      }
#pragma unroll
      for (int u = 0; u < EPI_COLS; ++u) A[u] = 0.f;
      for (int32_t c = 0; c < nchunk; ++c, ++chunk) {
        uint32_t buf = chunk & 1u, use = chunk >> 1;
        bool got = mbar_wait(&accf[buf], use & 1u, abort_flag, err, GP_KERR_TIMEOUT_ACCF);
        if (!__all_sync(0xffffffffu, got)) {
          ok = false;
          break;
        }
        tc_fence_after();
#pragma unroll
        for (int g = 0; g < EPI_COLS / 16; ++g) {
          uint32_t f[16];
          tmem_ld16(t_acc + buf * BT + col0 + 16 * g, f);
          tmem_wait_ld();
#pragma unroll
          for (int v = 0; v < 16; ++v) A[16 * g + v] = __fadd_rn(A[16 * g + v], __uint_as_float(f[v]));
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acce[buf]); /* buffer free: the MMA may reuse it */
        if ((c + 1) % GP_FOLD == 0 || c + 1 == nchunk) {
          /* fold A into the (hi, lo) running sum with TwoSum */
#pragma unroll
          for (int g = 0; g < EPI_COLS / 16; ++g) {
            uint32_t hs[16], ls[16];
            tmem_ld16(t_acc + 256 + col0 + 16 * g, hs);
            tmem_ld16(t_acc + 384 + col0 + 16 * g, ls);
            tmem_wait_ld();
#pragma unroll
            for (int v = 0; v < 16; ++v) {
              float Sv = __uint_as_float(hs[v]), x = A[16 * g + v];
              float s1 = __fadd_rn(Sv, x);
              float bp = __fsub_rn(s1, Sv);
              float e = __fadd_rn(__fsub_rn(Sv, __fsub_rn(s1, bp)), __fsub_rn(x, bp));
              hs[v] = __float_as_uint(s1);
              ls[v] = __float_as_uint(__fadd_rn(__uint_as_float(ls[v]), e));
              A[16 * g + v] = 0.f;
            }
            tmem_st16(t_acc + 256 + col0 + 16 * g, hs);
            tmem_st16(t_acc + 384 + col0 + 16 * g, ls);
          }
          tmem_wait_st();
        }
      }
      if (!ok) break;
      /* the tile -> Gram rows in FP64 (super-chunks after the first add to what is there), or
       * the part -> its place */
      double *orow = w < p.nfull ? xtx + (int64_t)gi * n + gj0
                                 : parts + ((int64_t)(w - p.nfull) * BT + row) * BT + col0;
      const int32_t ncol = w >= p.nfull ? EPI_COLS : gi < n ? n - gj0 : 0;
      const bool add = accumulate && w < p.nfull;
#pragma unroll
      for (int g = 0; g < EPI_COLS / 16; ++g) {
        uint32_t hs[16], ls[16];
        tmem_ld16(t_acc + 256 + col0 + 16 * g, hs);
        tmem_ld16(t_acc + 384 + col0 + 16 * g, ls);
        tmem_wait_ld();
        for (int v = 0; v < 16; ++v) {
          if (16 * g + v < ncol) {
            double x = (double)__uint_as_float(hs[v]) + (double)__uint_as_float(ls[v]);
            orow[16 * g + v] = add ? orow[16 * g + v] + x : x;
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) {
    if (*abort_flag) {
      /* let MMAs already issued finish before the columns are released and the CTA leaves */
      umma_commit(drain);
      const uint64_t t0 = globaltimer_ns();
      while (!mbar_try_wait(drain, 0) && globaltimer_ns() - t0 < GP_WAIT_NS) {
      }
    }
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

/* the parts of the tiles after the whole ones, in order, into the Gram: a thread per entry */
__global__ void __launch_bounds__(256)
k_gram_parts(gram_plan p, const double *__restrict__ parts, double *xtx, int32_t n,
             int32_t accumulate)
{
  int32_t bi, bj;
  tri_tile(p.nfull + blockIdx.x, p.nt, &bi, &bj);
  const double *src = parts + (int64_t)blockIdx.x * p.nsplit * (BT * BT);
  for (int e = blockIdx.y * blockDim.x + threadIdx.x; e < BT * BT; e += gridDim.y * blockDim.x) {
    const int32_t gi = bi * BT + e / BT, gj = bj * BT + e % BT;
    if (gi >= n || gj >= n) continue;
    double *dst = xtx + (int64_t)gi * n + gj;
    double x = accumulate ? *dst : 0.0;
    for (int32_t q = 0; q < p.nsplit; ++q) x += src[(int64_t)q * (BT * BT) + e];
    *dst = x;
  }
}

/* ------------------------------------------------------------------------------------ */
/* split materialisation                                                                  */

/* per kept column: (hi, lo) 16-bit pairs (bf16 or fp16) for codes 0..3 packed as
 * 4 x uint32 (lo << 16 | hi); hi = round(v), lo = round(v - hi) */
template <int FP16>
__global__ void k_split_tables(const int32_t *kept, int32_t nkept, const double *vtab,
                               uint32_t *split)
{
  for (int32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < nkept; k += gridDim.x * blockDim.x) {
    int32_t c = kept[k];
    for (int g = 0; g < 4; ++g) {
      double v = vtab[4 * c + g];
      uint32_t h, l;
      if (FP16) {
        __half hi = __double2half(v);
        __half lo = __double2half(v - (double)__half2float(hi));
        h = (uint32_t)__half_as_ushort(hi);
        l = (uint32_t)__half_as_ushort(lo);
      } else {
        __nv_bfloat16 hi = __double2bfloat16(v);
        __nv_bfloat16 lo = __double2bfloat16(v - (double)__bfloat162float(hi));
        h = (uint32_t)__bfloat16_as_ushort(hi);
        l = (uint32_t)__bfloat16_as_ushort(lo);
      }
      split[4 * k + g] = h | (l << 16);
    }
  }
}

/*
 * Xhi/Xlo [kc / 64][npad][64] for kept columns [k0, k0 + kc), rows >= nrows and columns >= nkept
 * zero, tile by tile through shared memory (a transpose of the SNP-major records):
 * CTA (kt, rt) covers 64 kept SNPs x 256 output rows.  When the tile's samples span at most
 * 256 record bytes (always when the rows are all samples or a subset with few gaps) the 64
 * records' byte ranges are read once, coalesced, into shared memory; each thread then writes
 * whole 16-byte groups so that a warp stores four 128-byte row segments.  Wider spans (sparse
 * sample subsets) read the bytes from global memory per thread.
 */
#define MT_SNP 64
#define MT_ROWS 256
#define MT_SPAN 256
/* shared-memory words of SNP u: a warp's lanes ask for the SNPs 8 g + k, g = 0 .. 7, and four rows;
 * with 65 words and 4 table entries a SNP two of them shared a bank in the records and all eight
 * in the table (5,000 x 150,000: 0.89 ms, now 0.62, 5 TB/s) */
#define MT_REC(u) ((u) * (MT_SPAN / 4 + 1) + ((u) >> 5) * 4)
#define MT_TAB(u) ((u) * 4 + ((u) >> 3) * 4)
__global__ void __launch_bounds__(256)
k_split_transpose(const uint8_t *__restrict__ geno, int64_t rlen, const int32_t *__restrict__ rows,
                  int32_t nrows, const int32_t *__restrict__ cols, const int32_t *__restrict__ kept,
                  int32_t nkept, const uint32_t *__restrict__ split, int32_t k0, int32_t npad,
                  __nv_bfloat16 *xhi, __nv_bfloat16 *xlo)
{
  __shared__ uint32_t srec[MT_REC(MT_SNP)];
  __shared__ uint32_t stab[MT_TAB(MT_SNP)];
  __shared__ int64_t srecoff[MT_SNP];
  const int tid = threadIdx.x;
  const int32_t kt = blockIdx.x, r0 = blockIdx.y * MT_ROWS;
  const int32_t kbase = k0 + kt * MT_SNP;
  int32_t base = 0, span = 0;
  if (r0 < nrows) {
    const int32_t rl = (r0 + MT_ROWS < nrows ? r0 + MT_ROWS : nrows) - 1;
    base = (rows[r0] >> 2) & ~15;
    span = (rows[rl] >> 2) - base + 1;
  }
  const bool fast = span <= MT_SPAN;
  if (tid < MT_SNP) {
    const int32_t k = kbase + tid;
    srecoff[tid] = k < nkept ? (int64_t)cols[kept[k]] * rlen : -1;
  }
  {
    const int u = tid >> 2, g = tid & 3;
    const int32_t k = kbase + u;
    stab[MT_TAB(u) + g] = k < nkept ? __ldg(split + 4 * k + g) : 0u;
  }
  __syncthreads();
  if (fast && span > 0) {
    const int nvec = (span + 15) >> 4;
    for (int i = tid; i < MT_SNP * nvec; i += blockDim.x) {
      const int u = i / nvec, v = i - u * nvec;
      uint4 val = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
      if (srecoff[u] >= 0) val = __ldg((const uint4 *)(geno + srecoff[u] + base + 16 * v));
      uint32_t *dst = srec + MT_REC(u) + 4 * v;
      dst[0] = val.x;
      dst[1] = val.y;
      dst[2] = val.z;
      dst[3] = val.w;
    }
  }
  __syncthreads();
  const int g8 = tid & 7, rsub = tid >> 3;
#pragma unroll 1
  for (int i = 0; i < MT_ROWS / 32; ++i) {
    const int32_t r = r0 + rsub + 32 * i;
    if (r >= npad) break;
    uint32_t hv[4] = {0, 0, 0, 0}, lv[4] = {0, 0, 0, 0};
    if (r < nrows) {
      const int32_t sidx = rows[r];
      const int32_t b = (sidx >> 2) - base, sh = (3 - (sidx & 3)) * 2;
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int uu = g8 * 8 + u;
        uint32_t byte;
        if (fast)
          byte = (srec[MT_REC(uu) + (b >> 2)] >> ((b & 3) * 8)) & 0xFFu;
        else
          byte = srecoff[uu] >= 0 ? __ldg(geno + srecoff[uu] + (sidx >> 2)) : 0xFFu;
        const uint32_t pair = stab[MT_TAB(uu) + ((byte >> sh) & 3u)];
        hv[u >> 1] |= (pair & 0xFFFFu) << ((u & 1) * 16);
        lv[u >> 1] |= (pair >> 16) << ((u & 1) * 16);
      }
    }
    const int64_t off = ((int64_t)kt * npad + r) * MT_SNP + g8 * 8;
    *(uint4 *)(xhi + off) = make_uint4(hv[0], hv[1], hv[2], hv[3]);
    *(uint4 *)(xlo + off) = make_uint4(lv[0], lv[1], lv[2], lv[3]);
  }
}

/* ------------------------------------------------------------------------------------ */

static PFN_cuTensorMapEncodeTiled_v12000 get_encode(gp_ctx *ctx)
{
  static PFN_cuTensorMapEncodeTiled_v12000 fn = NULL;
  if (fn) return fn;
  cudaDriverEntryPointQueryResult q;
  void *p = NULL;
  cudaError_t e = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                                                   cudaEnableDefault, &q);
  if (e != cudaSuccess || q != cudaDriverEntryPointSuccess || !p) {
    gp_fail(ctx, GP_ERR_CUDA, "cuTensorMapEncodeTiled entry point not found");
    return NULL;
  }
  fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
  return fn;
}

static int make_map(gp_ctx *ctx, CUtensorMap *m, void *base, int64_t rows, CUtensorMapDataType dt)
{
  PFN_cuTensorMapEncodeTiled_v12000 enc = get_encode(ctx);
  if (!enc) return GP_ERR_CUDA;
  cuuint64_t dims[2] = {BK, (cuuint64_t)rows};
  cuuint64_t strides[1] = {BK * 2};
  cuuint32_t box[2] = {BK, BT};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(m, dt, 2, base, dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return gp_fail(ctx, GP_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return GP_OK;
}

/* FP32 accumulation depth in k-blocks of 64 SNPs before the (hi, lo) add; split budget in bytes */
#define GP_BF16_CHUNK_KB 2
#define GP_BF16_BUDGET (24ll << 30)

/*
 * Whole tiles for the full waves; a last wave that would fill at most half of the nsm CTAs is cut
 * along the SNPs (5,000 samples x 600,000 SNPs: 60 tiles in two parts, 38.4 -> 35.7 ms; 1,000 x
 * 60,000: 36 tiles in four, 0.70 -> 0.29), into parts of GRAM_PART_FOLDS folds at least.  nsm = 0:
 * no parts.
 */
static gram_plan gram_make_plan(int32_t nt, int32_t nkb, int32_t chunk_kb, int32_t nsm)
{
  const int32_t ntiles = nt * (nt + 1) / 2, rest = nsm ? ntiles % nsm : 0;
  const int32_t nfold = (nkb + GP_FOLD * chunk_kb - 1) / (GP_FOLD * chunk_kb);
  gram_plan p = {nt, ntiles, 1, ntiles, nkb, chunk_kb};
  if (rest > 0) {
    const int32_t ns = nsm / rest < nfold / GRAM_PART_FOLDS ? nsm / rest : nfold / GRAM_PART_FOLDS;
    if (ns > 1) {
      p.nfull = ntiles - rest;
      p.nsplit = ns;
      p.nitems = p.nfull + rest * ns;
    }
  }
  return p;
}

int gp_gram_split(gp_ctx *ctx, int precision)
{
  const int fp16 = precision == GP_PREC_SPLIT_FP16;
  const int nmma = precision == GP_PREC_SPLIT_BF16X4 ? 4 : 3;
  const int32_t n = ctx->nrows, nk = ctx->nkept;
  const int32_t npad = (n + BT - 1) / BT * BT;
  const int32_t nt = npad / BT, ntiles = nt * (nt + 1) / 2;
  GP_CUDA(ctx, cudaMemsetAsync(ctx->d_xtx, 0, sizeof(double) * (size_t)n * n, ctx->stream));
  if (nk == 0) return GP_OK;
  const int32_t kpad = (nk + BK - 1) / BK * BK;
  /* super-chunk of kept SNPs so that Xhi + Xlo fit the budget; the budget and the FP32
   * chunk depth can be overridden (GP_BF16_BUDGET_BYTES, GP_BF16_CHUNK_SNPS) for tests and
   * accuracy sweeps */
  int64_t budget = GP_BF16_BUDGET;
  int32_t chunk_kb = GP_BF16_CHUNK_KB;
  {
    const char *e = getenv("GP_BF16_BUDGET_BYTES");
    if (e && atoll(e) > 0) budget = atoll(e);
    e = getenv("GP_BF16_CHUNK_SNPS");
    if (e && atoi(e) >= BK) chunk_kb = atoi(e) / BK;
  }
  int64_t per_col = (int64_t)npad * 4;
  int64_t kc_max = budget / per_col / BK * BK;
  if (kc_max < BK) kc_max = BK;
  int32_t kc = (int32_t)(kpad < kc_max ? kpad : kc_max);
  size_t xbytes = (size_t)npad * kc * 2;
  size_t tab_bytes = (size_t)nk * 16 + 256;
  gram_plan plan;
  size_t part_bytes = 0, sync_bytes = 0;
  int grid = 0, rc = GP_OK;
  uint8_t *base = NULL;
  for (int split = 1; split >= 0; --split) { /* without parts if there is no memory for them */
    plan = gram_make_plan(nt, kc / BK, chunk_kb, split ? ctx->num_sms : 0);
    part_bytes = sizeof(double) * BT * BT * (size_t)(plan.nitems - plan.nfull);
    grid = ctx->num_sms < plan.nitems ? ctx->num_sms : plan.nitems;
    sync_bytes = sizeof(unsigned) * (size_t)((kc / BK + GRAM_SYNC_KB - 1) / GRAM_SYNC_KB) *
                 (size_t)((plan.nitems + grid - 1) / grid);
    rc = gp_scratch2(ctx, 2 * xbytes + part_bytes + tab_bytes + sync_bytes + 512, (void **)&base);
    if (rc != GP_ERR_NOMEM || !part_bytes) break;
  }
  if (rc) return rc;
  const int32_t nsplit_tiles = ntiles - plan.nfull;
  __nv_bfloat16 *xhi = (__nv_bfloat16 *)base;
  __nv_bfloat16 *xlo = (__nv_bfloat16 *)(base + xbytes);
  double *parts = (double *)(base + 2 * xbytes);
  uint32_t *split = (uint32_t *)(base + 2 * xbytes + part_bytes);
  unsigned *sync_ctr =
      (unsigned *)(base + ((2 * xbytes + part_bytes + tab_bytes + 255) / 256) * 256);
  int *d_err = ctx->d_err;
  GP_CUDA(ctx, cudaMemsetAsync(d_err, 0, sizeof(int), ctx->stream));
  {
    int blocks = (nk + 255) / 256;
    if (blocks > ctx->num_sms * 8) blocks = ctx->num_sms * 8;
    if (fp16)
      k_split_tables<1><<<blocks, 256, 0, ctx->stream>>>(ctx->d_kept, nk, ctx->d_vtab, split);
    else
      k_split_tables<0><<<blocks, 256, 0, ctx->stream>>>(ctx->d_kept, nk, ctx->d_vtab, split);
    GP_LAUNCH_CHECK(ctx, "k_split_tables");
  }
  typedef void (*gram_kern_t)(const CUtensorMap, const CUtensorMap, gram_plan, double *, int32_t,
                              int32_t, double *, unsigned *, int *);
  gram_kern_t kern = fp16 ? k_gram_split<1, 3> : (nmma == 4 ? k_gram_split<0, 4> : k_gram_split<0, 3>);
  GP_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GRAM_SMEM));
  CUtensorMap mhi, mlo;
  CUtensorMapDataType dt = fp16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
  const int64_t xrows = (int64_t)kc / BK * npad;
  rc = make_map(ctx, &mhi, xhi, xrows, dt);
  if (!rc) rc = make_map(ctx, &mlo, xlo, xrows, dt);
  if (rc) return rc;
  for (int32_t k0 = 0; k0 < kpad; k0 += kc) {
    int32_t kcur = kpad - k0 < kc ? kpad - k0 : kc;
    /* columns beyond kcur in this super-chunk are zero (k >= nkept guard covers the tail) */
    dim3 tgrid((unsigned)(kc / MT_SNP), (unsigned)((npad + MT_ROWS - 1) / MT_ROWS));
    k_split_transpose<<<tgrid, 256, 0, ctx->stream>>>(ctx->d_geno, ctx->rlen_dev, ctx->d_rows, n,
                                                      ctx->d_cols, ctx->d_kept, nk, split, k0,
                                                      npad, xhi, xlo);
    GP_LAUNCH_CHECK(ctx, "k_split_transpose");
    int32_t nkb = kcur / BK;
    GP_CUDA(ctx, cudaMemsetAsync(sync_ctr, 0, sync_bytes, ctx->stream));
    /* cooperative launch: the producers' lockstep points need every CTA resident */
    plan.nkb = nkb;
    int32_t a_n = n, a_acc = k0 > 0 ? 1 : 0;
    double *a_xtx = ctx->d_xtx;
    void *args[] = {&mhi, &mlo, &plan, &a_xtx, &a_n, &a_acc, &parts, &sync_ctr, &d_err};
    GP_CUDA(ctx, cudaLaunchCooperativeKernel((const void *)kern, dim3(grid), dim3(GRAM_THREADS),
                                             args, GRAM_SMEM, ctx->stream));
    if (nsplit_tiles > 0) {
      k_gram_parts<<<dim3((unsigned)nsplit_tiles, 8), 256, 0, ctx->stream>>>(plan, parts, ctx->d_xtx,
                                                                             n, a_acc);
      GP_LAUNCH_CHECK(ctx, "k_gram_parts");
    }
    ctx->launches++;
    ctx->gram_launches++;
  }
  int herr = 0;
  GP_CUDA(ctx, gp_memcpy(ctx, &herr, d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (herr) return gp_fail(ctx, GP_ERR_TIMEOUT, "split-BF16 Gram kernel wait timed out (code %d)", herr);
  return GP_OK;
}
