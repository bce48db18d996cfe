/*
 * Exact genotype x FP64-panel products on the tensor cores.
 *
 *   Y[r][c] = sum_k A_r(k) P[k][c]
 *
 * A_r(k) is a small integer decoded from a 2-bit genotype code (observed mask {1,1,1,0} or
 * allele count {0,1,2,0}); P is an FP64 panel.  Each column of
 * P is scaled by a power of two 2^e_c >= max|P[.][c]| and cut into 4 fixed-point slices,
 * x = P/2^e_c = sum_t q_t 1024^-(t+1) with |q_0| <= 1024 and |q_t| <= 512 (t > 0): integers
 * that fp16 holds exactly.  A tensor-core MMA of {0,1,2} by such integers over at most 8,192
 * k values sums to an integer below 2^24, which FP32 holds exactly, so the FP32 accumulation
 * of the MMA loses nothing; chunk sums are added with 64-bit integer atomics
 * (order-independent, hence deterministic).  The only error left
 * is the slicing, about 2^-41 of the column maximum: the split precisions' products.
 *
 * The FP64 precision's products take 5 slices of 12 bits (x = sum_t q_t 2^-(11 + 12 t),
 * |q_t| <= 2048, at most 4,096 k values per chunk): an error of 2^-60 of the column maximum,
 * below what FP64 additions in sequence leave, for 5/4 of the MMAs.  They replace the FP64
 * pipe's products (1,501 x 80,003, K = 10, weights and lsqproject: 59.4 ms there, 1.56 here).
 *
 * This is how the masked per-sample normal equations of lsqproject (regressit
 * src/regsubs.c:19-26, lsqproj src/eigensrc/smartpca.c:4690-4712), the sample scores fxvecs
 * and the SNP weights ffvecs (smartpca.c:1485-1525) reach FP64 accuracy at tensor-core
 * speed.  Both orientations use the same kernel; only the operand layout differs:
 *   sum over SNPs     rows = samples, k = kept SNPs (codes in sample-major order)
 *   sum over samples  rows = kept SNPs, k = samples (codes in SNP-major order)
 *
 * Kernel structure (grid-stride over work items = 256-row tile x column tile of up to 256
 * slice columns x k-split, the row tile fastest, so that the CTAs running at one time share the
 * B tile and k range they stream and B is read from DRAM about once per wave instead of once
 * per row tile):
 *   warp 0      TMA of the B tile (slice columns x 64 k, fp16, 128-byte swizzle), 3 stages;
 *   warp 1      issues 2 x 4 tcgen05.mma (128 x N x 16, f16 -> f32) per k-block, converged, one
 *               elected lane each: the tile's two 128-row halves share the B tile;
 *   warps 2-9   decode the A tile, a thread per row: 16 bytes of codes (the next four
 *               k-blocks' loads in flight) become 64 fp16 values in the same swizzled layout;
 *               then fence.proxy.async and one arrival per warp;
 *   warps 10-17 epilogue: per chunk tcgen05.ld the exact FP32 sums and add them to the tile's
 *               64-bit integer sums in global memory (atomics, 32 rows side by side).
 * The decode is a mask per two values.  Missing codes are cleared in a word of 16 (or the word
 * made observed bits), and its bit pairs f and f + 8 are, as the low bits of two fp16 numbers, the
 * subnormals c 4^j 2^-24, j = f mod 5 or so (x_field): the factor 4^j is taken out of the other
 * operand, whose slices are multiplied by 4^-j (exact) and lie in the fields' order.  Every product
 * is an integer times 2^-24.  Byte permutes through a
 * table, as before, took 200 instructions a row and k-block where this takes 75: with 256 x 256
 * tiles the normal equations of 5,000 samples x 200,000 SNPs, K = 20, 1.41 -> 1.15 ms (128 x 128
 * tiles, decoded again for every 128 columns: 2.98), the weights' two products 0.33 -> 0.26 each.
 */
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <cudaTypedefs.h>
#include <limits.h>
#include <math.h>

#include "gp_geno_tc.h"
#include "gp_tc.cuh"

#define XT 128              /* rows of a half tile; code operands are padded to it */
#define XR 256              /* rows per tile: two 128-row accumulators */
#define XN 256              /* slice columns per tile at most */
#define XK 64               /* k per k-block */
#define XSTAGES 3
#define XA_BYTES (XT * XK * 2)
#define XB_BYTES (XN * XK * 2)
#define XSTAGE_BYTES (2 * XA_BYTES + XB_BYTES)
#define X_DEC_WARPS 8       /* decoder warps: a thread per row of the A tile */
#define X_EPI_WARPS 8
#define X_THREADS (64 + 32 * (X_DEC_WARPS + X_EPI_WARPS))
#define X_SMEM (XSTAGES * XSTAGE_BYTES + 1024 + 256)
#define XPF 4               /* k-blocks of codes a decoder thread loads ahead */

#define XERR_FULL 11
#define XERR_EMPTY 12
#define XERR_ACCF 13
#define XERR_ACCE 14

/* where the code at position kk of a k-block goes among its 64 values, and its power j of four: the
 * code is the bit pair f of its 32-bit word (the first code of a byte in the byte's high bits) */
__device__ __forceinline__ void x_field(int kk, int *pos, int *j)
{
  const int f = (kk & 12) + 3 - (kk & 3);
  *pos = (kk & ~15) + 2 * (f & 7) + (f >> 3);
  *j = (f & 7) < 5 ? f & 7 : (f & 7) - 5;
}
/* k-blocks per exact FP32 chunk: 8,192 k with 10-bit slices, 4,096 with 12-bit ones */
#define X_CHUNK_KB(digits) ((digits) == 5 ? 64 : 128)
/* columns of a panel cut and multiplied at a time with 5 slices */
#define X_GROUP5 256

/* slice columns per tile: the fewest tiles of at most XN, equally wide, a multiple of the
 * MMA's 16 */
static int32_t x_tile_cols(int32_t slice_cols)
{
  const int32_t nct = (slice_cols + XN - 1) / XN;
  return ((slice_cols + nct - 1) / nct + 15) / 16 * 16;
}

/* k splits: a work item costs its k-blocks and about 3 more (ring fill, TMEM read, atomics);
 * of the splits that fill one to four waves of the grid the one whose busiest CTA does least */
__host__ __device__ __forceinline__ int32_t x_split(int32_t tiles, int32_t nkb, int32_t grid)
{
  int32_t best = 1, best_cost = ((tiles + grid - 1) / grid) * (nkb + 3);
  for (int32_t w = 1; w <= 4; ++w) {
    int32_t s = w * grid / tiles;
    if (s > nkb / 4) s = nkb / 4;
    if (s < 2) continue;
    const int32_t cost = ((tiles * s + grid - 1) / grid) * ((nkb + s - 1) / s + 3);
    if (cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

/* exponent e_c with max|P| < 2^e_c (frexp) from the bits of a column's largest magnitude, 0 for an
 * all-zero column; with 5 slices X_NONFINITE for one with an infinity or NaN (its products are NaN,
 * as FP64 products of 0 and it are) */
#define X_NONFINITE (-(1 << 30))
template <int S>
__device__ __forceinline__ int x_exponent(unsigned long long mx)
{
  if (S == 5 && mx >= 0x7FF0000000000000ull) return X_NONFINITE;
  int e = 0;
  if (mx) frexp(__longlong_as_double((long long)mx), &e); /* v = f 2^e, f in [0.5, 1) */
  return e;
}

/* z 2^(e - 40), rounded once: what k_panel_combine<4> makes of the slices' sums */
__device__ __forceinline__ double x_scaled(long long z, int e)
{
  const double v = __ll2double_rn(z);
  if (e > -900 && e < 900) return v * __longlong_as_double((long long)(e - 40 + 1023) << 52);
  return ldexp(v, e - 40);
}

/*
 * codes: rows of ldc bytes (2-bit codes, MSB first, 3 = missing -> 0); output row r reads
 * code row row_map[r] (r itself when row_map is NULL); its k-block kb is the 16 bytes at
 * (kb % kb_period)*16, taken as allele counts or as the observed mask by count_lo for kb <
 * kb_period and count_hi otherwise (the concatenated-k form [G | O]).  tn: slice columns per tile; nct column tiles.
 * sums: per row tile, slice column (nct * tn of them) and row of the tile the exact integer
 * sum, added atomically.  With Y (ksplit 1, 4 slices, gp_tc_sums_fit) the item that has all of a
 * row's sums writes the products themselves, Y[row][column] by mx, the columns' largest magnitudes:
 * the slices' sums make one 64-bit integer, kept in Y's place between chunks.  No buffer of sums
 * is cleared, added to and read again (200,000 x 20 products over 5,000 samples: 0.40 -> 0.30 ms).
 */
__global__ void __launch_bounds__(X_THREADS, 1)
k_geno_panel_tc(const __grid_constant__ CUtensorMap tm_b, const uint8_t *__restrict__ codes,
                int64_t ldc, const int32_t *__restrict__ row_map, int32_t nrows, int32_t tn,
                int32_t nct, int32_t nkb, int32_t kb_period, int count_lo, int count_hi,
                int32_t ksplit, int32_t chunk_kb, unsigned long long *sums,
                const unsigned long long *__restrict__ mx, double *Y, int64_t ldy, int32_t ncols,
                int *err, const gp_tc_batch *db)
{
  if (db) {
    /* a device-resident loop's batch: rows and their count are read at run time */
    codes = db->codes;
    nrows = db->nrows;
    if (nrows < 1) return;
    ksplit = x_split(((nrows + XR - 1) / XR) * nct, nkb, (int32_t)gridDim.x);
  }
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t *bars = (uint64_t *)(smem + XSTAGES * XSTAGE_BYTES);
  uint64_t *full = bars, *empty = bars + XSTAGES, *accf = bars + 2 * XSTAGES,
           *acce = bars + 2 * XSTAGES + 1, *drain = bars + 2 * XSTAGES + 2;
  uint32_t *tmem_slot = (uint32_t *)(bars + 2 * XSTAGES + 3);
  volatile int *abort_flag = (volatile int *)(tmem_slot + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  const int32_t nrt = (nrows + XR - 1) / XR;
  const int32_t nitems = nrt * nct * ksplit;
  const int32_t kb_per = (nkb + ksplit - 1) / ksplit;

  if (threadIdx.x == 0) {
    for (int s = 0; s < XSTAGES; ++s) {
      mbar_init(&full[s], 1 + X_DEC_WARPS);
      mbar_init(&empty[s], 1);
    }
    mbar_init(accf, 1);
    mbar_init(acce, X_EPI_WARPS);
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) tma_prefetch_desc(&tm_b);
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    /* ---------------- B producer (TMA) ---------------- */
    uint32_t it = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      const int32_t ks = (w / nrt) % ksplit, ct = w / (nrt * ksplit);
      const int32_t kb0 = ks * kb_per, kb1 = min(nkb, kb0 + kb_per);
      for (int32_t kb = kb0; kb < kb1; ++kb, ++it) {
        const uint32_t s = it % XSTAGES, ph = (it / XSTAGES) & 1u;
        if (!mbar_wait_warp(&empty[s], ph ^ 1u, abort_flag, err, XERR_EMPTY)) {
          ok = false;
          break;
        }
        mbar_arrive_expect_tx_warp(&full[s], (uint32_t)tn * (XK * 2));
        tma_load_2d(smem + s * XSTAGE_BYTES + 2 * XA_BYTES, &tm_b, &full[s], kb * XK, ct * tn);
      }
    }
    if (*abort_flag) {
      /* copies already issued must land before the CTA exits (bounded) */
      const uint64_t t0 = globaltimer_ns();
      const uint32_t last = it < XSTAGES ? it : XSTAGES;
      for (uint32_t j = it - last; j < it; ++j)
        while (!mbar_try_wait(&full[j % XSTAGES], (j / XSTAGES) & 1u) &&
               globaltimer_ns() - t0 < GP_WAIT_NS) {
        }
    }
  } else if (warp == 1) {
    /* ---------------- MMA issuer ---------------- */
    const uint32_t idesc = idesc_f16_f32(XT, (uint32_t)tn);
    uint32_t it = 0, chunk = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      const int32_t ks = (w / nrt) % ksplit, rt = w % nrt;
      const int32_t kb0 = ks * kb_per, kb1 = min(nkb, kb0 + kb_per);
      const bool h1 = rt * XR + XT < nrows;
      for (int32_t c0 = kb0; c0 < kb1 && ok; c0 += chunk_kb, ++chunk) {
        const int32_t c1 = min(kb1, c0 + chunk_kb);
        if (!mbar_wait_warp(acce, (chunk & 1u) ^ 1u, abort_flag, err, XERR_ACCE)) {
          ok = false;
          break;
        }
        tc_fence_after();
        for (int32_t kb = c0; kb < c1; ++kb, ++it) {
          const uint32_t s = it % XSTAGES, ph = (it / XSTAGES) & 1u;
          if (!mbar_wait_warp(&full[s], ph, abort_flag, err, XERR_FULL)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t base = smem_u32(smem + s * XSTAGE_BYTES);
          const uint64_t a0 = sdesc_k128(base), a1 = sdesc_k128(base + XA_BYTES),
                         bd = sdesc_k128(base + 2 * XA_BYTES);
#pragma unroll
          for (int k = 0; k < XK / 16; ++k) {
            const uint32_t acc = (kb > c0 || k > 0) ? 1u : 0u;
            umma_bf16(tmem, a0 + 2 * k, bd + 2 * k, idesc, acc);
            if (h1) umma_bf16(tmem + XN, a1 + 2 * k, bd + 2 * k, idesc, acc);
          }
          umma_commit(&empty[s]);
        }
        if (ok) umma_commit(accf);
      }
    }
  } else if (warp < 2 + X_DEC_WARPS) {
    /* ---------------- A decoders: a thread per row of the tile ---------------- */
    const int r = (warp - 2) * 32 + lane;
    uint8_t *rowp = smem + (r >> 7) * XA_BYTES + (r & 127) * 128;
    const uint32_t sw = (uint32_t)(r & 7);
    uint32_t it = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      const int32_t ks = (w / nrt) % ksplit, rt = w % nrt;
      const int32_t kb0 = ks * kb_per, kb1 = min(nkb, kb0 + kb_per);
      const int32_t grow = rt * XR + r;
      /* a half with no row at all is not multiplied and needs no decode */
      const bool live = grow < nrows, half_on = rt * XR + (r & ~127) < nrows;
      const uint8_t *crow =
          codes + (live ? (row_map ? (int64_t)row_map[grow] : (int64_t)grow) : 0) * ldc;
      auto ld_codes = [&](int32_t kb) {
        return live && kb < kb1
                   ? __ldg((const uint4 *)(crow + (int64_t)(kb < kb_period ? kb : kb - kb_period) * 16))
                   : make_uint4(~0u, ~0u, ~0u, ~0u);
      };
      uint4 pf[XPF];
#pragma unroll
      for (int u = 0; u < XPF; ++u) pf[u] = ld_codes(kb0 + u);
      for (int32_t kbb = kb0; kbb < kb1 && ok; kbb += XPF) {
#pragma unroll
        for (int u = 0; u < XPF; ++u) {
          const int32_t kb = kbb + u;
          if (kb >= kb1) break;
          const uint32_t words[4] = {pf[u].x, pf[u].y, pf[u].z, pf[u].w};
          pf[u] = ld_codes(kb + XPF);
          const uint32_t s = it % XSTAGES, ph = (it / XSTAGES) & 1u;
          ++it;
          const bool got = mbar_wait(&empty[s], ph ^ 1u, abort_flag, err, XERR_EMPTY);
          if (!__all_sync(0xffffffffu, got)) {
            ok = false;
            break;
          }
          if (half_on) {
            const bool count = kb < kb_period ? count_lo : count_hi;
            uint8_t *dst = rowp + s * XSTAGE_BYTES;
#pragma unroll
            for (int o = 0; o < 8; o += 2) {
              uint32_t x = words[o >> 1];
              const uint32_t gone = x & (x >> 1) & 0x55555555u; /* missing */
              x = count ? x & ~(gone | gone << 1) : gone ^ 0x55555555u;
              const uint32_t y = x >> 10;
              *(uint4 *)(dst + (((uint32_t)o ^ sw) << 4)) = make_uint4(
                  x & 0x00030003u, x & 0x000C000Cu, x & 0x00300030u, x & 0x00C000C0u);
              *(uint4 *)(dst + (((uint32_t)(o + 1) ^ sw) << 4)) = make_uint4(
                  x & 0x03000300u, y & 0x00030003u, y & 0x000C000Cu, y & 0x00300030u);
            }
            fence_proxy_async_smem();
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&full[s]);
        }
      }
    }
  } else {
    /* ---------------- epilogue: warps 2 + X_DEC_WARPS .. ---------------- */
    const int q = warp & 3, half = (warp - 2 - X_DEC_WARPS) >> 2;
    const uint32_t t_acc = tmem + ((uint32_t)(q * 32) << 16) + half * XN;
    uint32_t chunk = 0;
    bool ok = true;
    for (int32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
      const int32_t ks = (w / nrt) % ksplit, ct = w / (nrt * ksplit), rt = w % nrt;
      const int32_t kb0 = ks * kb_per, kb1 = min(nkb, kb0 + kb_per);
      const int32_t row = half * XT + q * 32 + lane;
      const bool live = rt * XR + row < nrows, any = rt * XR + half * XT + q * 32 < nrows;
      unsigned long long *out = sums + ((int64_t)rt * nct * tn + (int64_t)ct * tn) * XR + row;
      for (int32_t c0 = kb0; c0 < kb1; c0 += chunk_kb, ++chunk) {
        const bool got = mbar_wait(accf, chunk & 1u, abort_flag, err, XERR_ACCF);
        if (!__all_sync(0xffffffffu, got)) {
          ok = false;
          break;
        }
        tc_fence_after();
        if (any && Y) {
          const bool first = c0 == kb0, last = c0 + chunk_kb >= kb1;
          double *yr = Y + (int64_t)(rt * XR + row) * ldy;
          for (int g = 0; g < tn; g += 16) {
            uint32_t f[16];
            tmem_ld16(t_acc + g, f);
            tmem_wait_ld();
#pragma unroll
            for (int v = 0; v < 16; v += 4) {
              const int32_t c = (ct * tn + g + v) >> 2;
              if (!live || c >= ncols) continue;
              long long z = 0;
#pragma unroll
              for (int t = 0; t < 4; ++t)
                z = (z << 10) + __float2int_rn(__uint_as_float(f[v + t]) * 0x1p24f);
              if (!first) z += __double_as_longlong(yr[c]);
              yr[c] = last ? x_scaled(z, x_exponent<4>(__ldg(mx + c))) : __longlong_as_double(z);
            }
          }
        } else if (any)
          for (int g = 0; g < tn; g += 16) {
            uint32_t f[16];
            tmem_ld16(t_acc + g, f);
            tmem_wait_ld();
#pragma unroll
            for (int v = 0; v < 16; ++v) {
              const long long z = __float2int_rn(__uint_as_float(f[v]) * 0x1p24f);
              if (live) atomicAdd(out + (int64_t)(g + v) * XR, (unsigned long long)z);
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

/* ------------------------------------------------------------------------------------ */
/* operand preparation                                                                    */

/*
 * sum over SNPs: codes[r][k] = code of sample samp[r] at kept SNP k (record snprec[k]);
 * row stride ldc bytes; pad k (>= nk) and pad rows are 3.  A transpose through shared
 * memory: CTA (kt, rt) covers 128 kept SNPs x 128 rows; when the rows' samples span at most
 * CB_SPAN record bytes, the 128 records' byte ranges are read once (coalesced), and two
 * threads build each row's 32 output bytes; wider spans read per thread.  The samples may come
 * in any order and repeat, so the span is that of the least and the greatest of them.
 */
#define CB_SNP 128
#define CB_ROWS 128
#define CB_SPAN 64
#define CB_PITCH_W (CB_SPAN / 4 + 1)
__global__ void __launch_bounds__(256)
k_codes_by_sample(const uint8_t *__restrict__ geno, int64_t rlen, const int32_t *__restrict__ samp,
                  int32_t nsamp, int32_t nrows_pad, const int32_t *__restrict__ snprec, int32_t nk,
                  int64_t ldc, uint8_t *codes)
{
  __shared__ uint32_t srec[CB_SNP][CB_PITCH_W];
  __shared__ int64_t soff[CB_SNP];
  __shared__ int32_t win[2]; /* the rows' first and last record byte */
  const int tid = threadIdx.x;
  const int32_t r0 = blockIdx.y * CB_ROWS;
  const int rl = tid >> 1, half = tid & 1;
  const int32_t r = r0 + rl;
  const int32_t sidx = r < nsamp ? samp[r] : 0;
  if (tid == 0) {
    win[0] = INT_MAX;
    win[1] = -1;
  }
  __syncthreads();
  const int32_t first = __reduce_min_sync(0xffffffffu, r < nsamp ? sidx >> 2 : INT_MAX);
  const int32_t last = __reduce_max_sync(0xffffffffu, r < nsamp ? sidx >> 2 : -1);
  if ((tid & 31) == 0) {
    atomicMin(&win[0], first);
    atomicMax(&win[1], last);
  }
  __syncthreads();
  const int32_t base = win[1] < 0 ? 0 : win[0] & ~15, span = win[1] < 0 ? 0 : win[1] - base + 1;
  const bool fast = span <= CB_SPAN;
  /* the CTA walks the SNP tiles of its row block (grid-stride over x) */
  const int32_t nkt = (int32_t)((ldc * 4 + CB_SNP - 1) / CB_SNP);
  for (int32_t kt = blockIdx.x; kt < nkt; kt += gridDim.x) {
    const int32_t k0 = kt * CB_SNP;
    if (tid < CB_SNP) soff[tid] = (k0 + tid < nk) ? (int64_t)snprec[k0 + tid] * rlen : -1;
    __syncthreads();
    if (fast && span > 0) {
      const int nvec = (span + 15) >> 4;
      for (int i = tid; i < CB_SNP * nvec; i += blockDim.x) {
        const int u = i / nvec, v = i - u * nvec;
        uint4 val = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        if (soff[u] >= 0) val = __ldg((const uint4 *)(geno + soff[u] + base + 16 * v));
        srec[u][4 * v] = val.x;
        srec[u][4 * v + 1] = val.y;
        srec[u][4 * v + 2] = val.z;
        srec[u][4 * v + 3] = val.w;
      }
    }
    __syncthreads();
    if (r < nrows_pad && (int64_t)k0 + 64 * half < ldc * 4) {
      uint32_t out[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
      if (r < nsamp) {
        const int32_t bb = (sidx >> 2) - base, sh = (3 - (sidx & 3)) * 2;
#pragma unroll 8
        for (int j = 0; j < 64; ++j) {
          const int u = 64 * half + j;
          uint32_t byte = 0xFFu;
          if (soff[u] >= 0)
            byte = fast ? (srec[u][bb >> 2] >> ((bb & 3) * 8)) & 0xFFu
                        : __ldg(geno + soff[u] + (sidx >> 2));
          const uint32_t c = (byte >> sh) & 3u;
          /* code j of the group: byte j>>2 (word j>>4), bits (3-(j&3))*2 within the byte */
          const uint32_t wpos = (uint32_t)((j >> 2) & 3) * 8u + (3u - (uint32_t)(j & 3)) * 2u;
          out[j >> 4] = (out[j >> 4] & ~(3u << wpos)) | (c << wpos);
        }
      }
      *(uint4 *)(codes + (int64_t)r * ldc + (k0 >> 2) + 16 * half) =
          make_uint4(out[0], out[1], out[2], out[3]);
    }
    __syncthreads(); /* srec and soff are rewritten by the next tile */
  }
}

/* inv[samp[r]] = r (inv preset to -1) */
__global__ void k_invert_rows(const int32_t *samp, int32_t nsamp, int32_t *inv)
{
  for (int32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < nsamp; r += gridDim.x * blockDim.x)
    inv[samp[r]] = r;
}

/*
 * The same operand for rows that are distinct samples: all samples are transposed, the selected
 * ones written to their rows (inv; NULL: every sample in order).  A CTA covers 512 samples x 128 SNPs; a thread holds a word
 * (16 samples) of 16 SNPs and transposes the 16 x 16 codes in registers: the 4 x 4 bytes of
 * words 4 apart by byte permutes, then the 4 x 4 codes of neighbouring words by masked swaps,
 * about half an instruction per code; pieces of 32 bytes per row leave through shared memory.
 * HBM bounds it (5,000 x 200,000: 120 us for 500 MB; a code at a time as below: 734).
 */
#define CT_W 32
__global__ void __launch_bounds__(256)
k_codes_transpose(const uint8_t *__restrict__ geno, int64_t rlen, int32_t nind,
                  const int32_t *__restrict__ inv, const int32_t *__restrict__ snprec, int32_t nk,
                  int64_t ldc, uint8_t *codes)
{
  __shared__ uint32_t so[16 * CT_W][9];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int32_t k0 = (int32_t)blockIdx.x * 128;
  const int64_t w = (int64_t)blockIdx.y * CT_W + lane;
  const bool in = w < (rlen >> 2);
  uint32_t a[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int32_t k = k0 + 16 * g + i;
    a[i] = in && k < nk ? __ldg((const uint32_t *)(geno + (int64_t)snprec[k] * rlen) + w)
                        : 0xFFFFFFFFu;
  }
  /* x[J][ii]: byte I = byte J of word 4 I + ii */
  uint32_t x[4][4];
#pragma unroll
  for (int ii = 0; ii < 4; ++ii) {
    const uint32_t p0 = __byte_perm(a[ii], a[4 + ii], 0x5140), p1 = __byte_perm(a[8 + ii], a[12 + ii], 0x5140);
    const uint32_t q0 = __byte_perm(a[ii], a[4 + ii], 0x7362), q1 = __byte_perm(a[8 + ii], a[12 + ii], 0x7362);
    x[0][ii] = __byte_perm(p0, p1, 0x5410);
    x[1][ii] = __byte_perm(p0, p1, 0x7632);
    x[2][ii] = __byte_perm(q0, q1, 0x5410);
    x[3][ii] = __byte_perm(q0, q1, 0x7632);
  }
#pragma unroll
  for (int J = 0; J < 4; ++J) {
#pragma unroll
    for (int ii = 0; ii < 2; ++ii) { /* codes 2, 3 of word ii and 0, 1 of word ii + 2 */
      const uint32_t t = ((x[J][ii + 2] >> 4) ^ x[J][ii]) & 0x0F0F0F0Fu;
      x[J][ii] ^= t;
      x[J][ii + 2] ^= t << 4;
    }
#pragma unroll
    for (int ii = 0; ii < 4; ii += 2) { /* codes 1, 3 of word ii and 0, 2 of word ii + 1 */
      const uint32_t t = ((x[J][ii + 1] >> 2) ^ x[J][ii]) & 0x33333333u;
      x[J][ii] ^= t;
      x[J][ii + 1] ^= t << 2;
    }
#pragma unroll
    for (int jj = 0; jj < 4; ++jj) so[(4 * J + jj) * CT_W + lane][g] = x[J][jj];
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * 16 * CT_W; i += blockDim.x) {
    const int idx = i >> 1, half = i & 1;
    const int64_t q = ((int64_t)blockIdx.y * CT_W + (idx & (CT_W - 1))) * 16 + idx / CT_W;
    const int64_t at = (k0 >> 2) + 16 * half;
    if (q >= nind || at >= ldc) continue;
    const int64_t r = inv ? inv[q] : q;
    if (r < 0) continue;
    const uint32_t *o = so[idx] + 4 * half;
    *(uint4 *)(codes + (int64_t)r * ldc + at) = make_uint4(o[0], o[1], o[2], o[3]);
  }
}

/*
 * sum over samples: codes[k][j] = code of sample samp[j] at kept SNP k; one row per kept
 * SNP, j over the nsamp samples; pad j and pad rows are 3.  One warp per SNP row: the
 * record is staged in shared memory (coalesced), then each lane gathers its 64-sample
 * groups from it.  Dynamic shared memory: warps x rlen bytes.
 */
__global__ void __launch_bounds__(256)
k_codes_by_snp(const uint8_t *__restrict__ geno, int64_t rlen, const int32_t *__restrict__ samp,
               int32_t nsamp, const int32_t *__restrict__ snprec, int32_t nk, int32_t nrows_pad,
               int64_t ldc, uint8_t *codes)
{
  extern __shared__ uint4 srec4[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  uint8_t *rec_s = (uint8_t *)(srec4 + (int64_t)warp * (rlen / 16));
  const int64_t groups = ldc / 16;
  for (int64_t k = (int64_t)blockIdx.x * nw + warp; k < nrows_pad; k += (int64_t)gridDim.x * nw) {
    if (k < nk) {
      const uint4 *src = (const uint4 *)(geno + (int64_t)snprec[k] * rlen);
      for (int64_t v = lane; v < rlen / 16; v += 32) ((uint4 *)rec_s)[v] = __ldg(src + v);
    }
    __syncwarp();
    for (int64_t gq = lane; gq < groups; gq += 32) {
      uint32_t out[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
      if (k < nk) {
#pragma unroll 8
        for (int j = 0; j < 64; ++j) {
          const int64_t q = gq * 64 + j;
          uint32_t c = 3u;
          if (q < nsamp) {
            const int32_t sidx = samp[q];
            c = (rec_s[sidx >> 2] >> ((3 - (sidx & 3)) * 2)) & 3u;
          }
          const uint32_t wpos = (uint32_t)((j >> 2) & 3) * 8u + (3u - (uint32_t)(j & 3)) * 2u;
          out[j >> 4] = (out[j >> 4] & ~(3u << wpos)) | (c << wpos);
        }
      }
      *(uint4 *)(codes + k * ldc + gq * 16) = make_uint4(out[0], out[1], out[2], out[3]);
    }
    __syncwarp();
  }
}

/* one or two panels as the kernels take them */
struct x_panels {
  const double *P[2];
  int64_t ldp[2];
  double sign[2];
};

/*
 * per column c of the panels P [nk][ldp] (FP64, blockIdx.y): max of |P[k][c]| as its bit pattern
 * (the order of non-negative doubles), folded into mx[c] with atomicMax: the panels' joint
 * scale.  Threads keep a fixed column so that a warp reads rows of P contiguously.
 */
__global__ void k_panel_absmax(const x_panels pan, int32_t nk, int32_t ncols,
                               unsigned long long *mx)
{
  __shared__ unsigned long long smx[1024];
  for (int c = threadIdx.x; c < ncols; c += blockDim.x) smx[c] = 0ull;
  __syncthreads();
  const double *__restrict__ P = pan.P[blockIdx.y];
  const int64_t ldp = pan.ldp[blockIdx.y];
  const int32_t rows = (int32_t)((int64_t)gridDim.x * blockDim.x / ncols); /* per round */
  const int32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  const int32_t k0 = t / ncols, c = t - k0 * ncols;
  if (k0 < rows) {
    unsigned long long m = 0ull;
#pragma unroll 4
    for (int64_t k = k0; k < nk; k += rows) {
      const unsigned long long bits =
          (unsigned long long)__double_as_longlong(P[k * ldp + c]) & 0x7FFFFFFFFFFFFFFFull;
      m = bits > m ? bits : m;
    }
    if (m) atomicMax(smx + c, m);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ncols; i += blockDim.x)
    if (smx[i]) atomicMax(mx + i, smx[i]);
}

/*
 * The slices of x = sign P / 2^e_c (|x| < 1) in integer arithmetic (GB300's FP64 pipe is
 * narrow): N = rint(x 2^F) from the double's mantissa and exponent (round half to even), F = 40
 * with S = 4 slices of 10 bits, 59 with 5 of 12, then balanced digits from the bottom: all but
 * the first in [-2^(b-1), 2^(b-1) - 1], d_0 = the rest (at most 1024 = 2^(40-30) or
 * 2048 = 2^(59-48) since |N| <= 2^F), so that x = sum_t d_t 2^(b(S-1-t) - F) + O(2^-F-1).
 */
template <int S>
__device__ __forceinline__ void slice(double v, int e, bool neg, int d[S])
{
  constexpr int b = S == 5 ? 12 : 10, F = S == 5 ? 59 : 40;
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
  const int E = (int)((bits >> 52) & 0x7FF);
  unsigned long long M = bits & 0xFFFFFFFFFFFFFull;
  /* |v| = M 2^(E' - 1075) with E' = max(E, 1); x 2^F = M / 2^sh, sh >= 53 - F when |v| < 2^e */
  if (E) M |= 1ull << 52;
  const int sh = 1075 - F + e - (E ? E : 1);
  long long N = 0;
  if (M != 0 && sh < 64) {
    if (sh < 1) {
      N = (long long)(M << -sh);
    } else {
      unsigned long long q = M >> sh;
      const unsigned long long rem = M & ((1ull << sh) - 1), half = 1ull << (sh - 1);
      if (rem > half || (rem == half && (q & 1ull))) ++q;
      N = (long long)q;
    }
  }
  if (neg != (bool)(bits >> 63)) N = -N;
#pragma unroll
  for (int t = S - 1; t >= 1; --t) {
    int r = (int)(N & ((1 << b) - 1));
    if (r >= 1 << (b - 1)) r -= 1 << b;
    d[t] = r;
    N = (N - r) >> b; /* exact: N - r is a multiple of 2^b */
  }
  d[0] = (int)N;
}

/*
 * B[(Sc+t)][p kpad + k] (fp16, row stride ldb elements, rows of them) = slice t of sign P[k][c] /
 * 2^e_c of panel p = blockIdx.z for k < nk; pad k and pad rows zero.  A tile of 64 k x 32
 * columns is read row-wise (coalesced) into shared memory and written as 128-byte rows of B.
 */
#define SL_K 64
#define SL_C 32
template <int S>
__global__ void __launch_bounds__(256)
k_panel_slices(const x_panels pan, int32_t nk, int32_t ncols,
               const unsigned long long *__restrict__ mx, __half *B, int64_t ldb, int32_t kpad,
               int32_t rows)
{
  __shared__ double sp[SL_K][SL_C + 1];
  __shared__ __align__(16) __half ss[SL_C * S][SL_K + 8];
  __shared__ int sexp[SL_C];
  const double *__restrict__ P = pan.P[blockIdx.z];
  const int64_t ldp = pan.ldp[blockIdx.z];
  const bool neg = pan.sign[blockIdx.z] < 0.0;
  const int tid = threadIdx.x;
  const int32_t kt0 = blockIdx.x * SL_K, ct0 = blockIdx.y * SL_C;
  if (tid < SL_C) {
    const int32_t c = ct0 + tid;
    sexp[tid] = c < ncols ? x_exponent<S>(mx[c]) : 0;
  }
  for (int i = tid; i < SL_K * SL_C; i += blockDim.x) {
    const int kk = i / SL_C, cc = i - kk * SL_C;
    const int32_t k = kt0 + kk, c = ct0 + cc;
    sp[kk][cc] = (k < nk && c < ncols) ? P[(int64_t)k * ldp + c] : 0.0;
  }
  __syncthreads();
  for (int i = tid; i < SL_K * SL_C; i += blockDim.x) {
    const int cc = i / SL_K, kk = i - cc * SL_K;
    int d[S], pos, j;
    x_field(kk, &pos, &j);
    const float scale = 1.f / (float)(1 << (2 * j));
    const bool bad = S == 5 && sexp[cc] == X_NONFINITE;
    slice<S>(bad ? 0.0 : sp[kk][cc], bad ? 0 : sexp[cc], neg, d);
#pragma unroll
    for (int t = 0; t < S; ++t) ss[S * cc + t][pos] = __float2half_rn((float)d[t] * scale);
  }
  __syncthreads();
  /* 32 S output rows x 64 halves: 8 threads write one row's 128 bytes */
  for (int i = tid; i < SL_C * S * 8; i += blockDim.x) {
    const int o = i >> 3, seg = i & 7;
    const int32_t r = S * ct0 + o;
    if (r >= rows) continue;
    __half *dst = B + (int64_t)r * ldb + (int64_t)blockIdx.z * kpad + kt0 + seg * 8;
    *(uint4 *)dst = *(const uint4 *)&ss[o][seg * 8];
  }
}

/*
 * Y[r][c] = 2^e_c sum_t Z_t 2^(b(S-1-t) - F) with Z_t the integer sum of row r and slice column
 * Sc + t (sums as k_geno_panel_tc leaves them: rows contiguous; wcols slice columns per row
 * tile).  A CTA takes 32 rows x 32 columns through shared memory so that sums are read and Y
 * written contiguously.
 */
template <int S>
__global__ void __launch_bounds__(256)
k_panel_combine(const unsigned long long *__restrict__ sums, int32_t wcols, int32_t nrows,
                int32_t ncols, const unsigned long long *__restrict__ mx, double *Y, int64_t ldy,
                const gp_tc_batch *db)
{
  __shared__ double sy[32][33];
  if (db) nrows = db->nrows;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t nrb = (nrows + 31) / 32, ncb = (ncols + 31) / 32;
  for (int64_t blk = blockIdx.x; blk < nrb * ncb; blk += gridDim.x) {
    const int64_t r0 = (blk / ncb) * 32;
    const int32_t c0 = (int32_t)(blk % ncb) * 32;
    const unsigned long long *src =
        sums + (r0 / XR * wcols + (int64_t)S * c0) * XR + r0 % XR + lane;
    if (r0 + lane < nrows) {
      for (int cc = warp; cc < 32 && c0 + cc < ncols; cc += 8) {
        double z[S];
#pragma unroll
        for (int t = 0; t < S; ++t) z[t] = (double)(long long)src[(int64_t)(S * cc + t) * XR];
        const int e = x_exponent<S>(mx[c0 + cc]);
        if (S == 4) {
          const double v = ((z[0] * 0x1p-10 + z[1] * 0x1p-20) + z[2] * 0x1p-30) + z[3] * 0x1p-40;
          sy[cc][lane] = ldexp(v, e);
        } else {
          double v = z[S - 1];
#pragma unroll
          for (int t = S - 2; t >= 0; --t) v = fma(v, 0x1p-12, z[t]);
          sy[cc][lane] = e == X_NONFINITE ? nan("") : ldexp(v, e - 11);
        }
      }
    }
    __syncthreads();
    if (c0 + lane < ncols)
      for (int rr = warp; rr < 32 && r0 + rr < nrows; rr += 8)
        Y[(r0 + rr) * ldy + c0 + lane] = sy[lane][rr];
    __syncthreads();
  }
}

/* ------------------------------------------------------------------------------------ */

static PFN_cuTensorMapEncodeTiled_v12000 tc_encode(gp_ctx *ctx)
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

static int grid_cap(const gp_ctx *ctx, int64_t work, int per_block, int mult)
{
  int64_t g = (work + per_block - 1) / per_block;
  int64_t cap = (int64_t)ctx->num_sms * mult;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

static size_t align256(size_t b) { return (b + 255) / 256 * 256; }

int gp_tc_code_bytes(int sum_over_snps, int32_t nsamp, int32_t nk, int64_t *ldc, int32_t *rows_pad)
{
  const int32_t nrows = sum_over_snps ? nsamp : nk;
  const int32_t k0 = sum_over_snps ? nk : nsamp;
  *rows_pad = (nrows + XT - 1) / XT * XT;
  *ldc = (int64_t)((k0 + XK - 1) / XK) * XK / 4;
  return GP_OK;
}

int gp_tc_build_codes(gp_ctx *ctx, int sum_over_snps, const int32_t *d_samp, int32_t nsamp,
                      const int32_t *d_snprec, int32_t nk, int32_t *inv, uint8_t *codes,
                      gp_tc_codes *out)
{
  int64_t ldc;
  int32_t nrows_pad;
  gp_tc_code_bytes(sum_over_snps, nsamp, nk, &ldc, &nrows_pad);
  /* transposing every sample reads and shuffles nind_all / nsamp times the codes that are kept;
   * measured six times as fast per code as gathering them (all of 5,000 x 200,000: 120 us and
   * 734) */
  if (sum_over_snps && inv && ctx->nind_all <= 4 * (int64_t)nsamp) {
    if (nsamp == ctx->nind_all && d_samp == ctx->d_rows) {
      inv = NULL; /* every sample, in order */
    } else {
      GP_CUDA(ctx, cudaMemsetAsync(inv, 0xFF, sizeof(int32_t) * (size_t)ctx->nind_all, ctx->stream));
      k_invert_rows<<<grid_cap(ctx, nsamp, 256, 4), 256, 0, ctx->stream>>>(d_samp, nsamp, inv);
      GP_LAUNCH_CHECK(ctx, "k_invert_rows");
    }
    dim3 grid((unsigned)((ldc * 4 + 127) / 128),
              (unsigned)((ctx->rlen_dev / 4 + CT_W - 1) / CT_W));
    k_codes_transpose<<<grid, 256, 0, ctx->stream>>>(ctx->d_geno, ctx->rlen_dev, ctx->nind_all, inv,
                                                     d_snprec, nk, ldc, codes);
  } else if (sum_over_snps) {
    /* about 16 CTAs per SM in all; each walks the SNP tiles of its row block */
    const int64_t nkt = (ldc * 4 + CB_SNP - 1) / CB_SNP, nrb = (nrows_pad + CB_ROWS - 1) / CB_ROWS;
    int64_t gx = ((int64_t)ctx->num_sms * 16 + nrb - 1) / nrb;
    if (gx > nkt) gx = nkt;
    if (gx < 1) gx = 1;
    dim3 grid((unsigned)gx, (unsigned)nrb);
    k_codes_by_sample<<<grid, 256, 0, ctx->stream>>>(ctx->d_geno, ctx->rlen_dev, d_samp, nsamp,
                                                     nrows_pad, d_snprec, nk, ldc, codes);
  } else {
    int warps = (int)((200 * 1024) / ctx->rlen_dev);
    if (warps > 8) warps = 8;
    if (warps < 1)
      return gp_fail(ctx, GP_ERR_ARG, "gp_tc_build_codes: records of %lld bytes are too long",
                     (long long)ctx->rlen_dev);
    const size_t smem = (size_t)warps * ctx->rlen_dev;
    GP_CUDA(ctx, gp_allow_smem(ctx, (const void *)k_codes_by_snp));
    int blocks = (int)((nrows_pad + warps - 1) / warps);
    if (blocks > ctx->num_sms * 16) blocks = ctx->num_sms * 16;
    k_codes_by_snp<<<blocks, 32 * warps, smem, ctx->stream>>>(ctx->d_geno, ctx->rlen_dev, d_samp,
                                                              nsamp, d_snprec, nk, nrows_pad, ldc,
                                                              codes);
  }
  GP_LAUNCH_CHECK(ctx, "k_codes");
  out->codes = codes;
  out->ldc = ldc;
  out->row_map = NULL;
  out->nrows = sum_over_snps ? nsamp : nk;
  out->k0 = sum_over_snps ? nk : nsamp;
  return GP_OK;
}

size_t gp_tc_prepared_bytes(int npanels, int32_t ncols, int32_t k0, int digits)
{
  const int32_t kpad0 = (k0 + XK - 1) / XK * XK;
  const int32_t tn = x_tile_cols(digits * ncols), nct = (digits * ncols + tn - 1) / tn;
  const int32_t ncols4_pad = nct * tn;
  return align256((size_t)ncols4_pad * kpad0 * npanels * 2) + align256((size_t)ncols * 8) + 256;
}

int gp_tc_prepare(gp_ctx *ctx, int npanels, const gp_tc_panel *pp, int32_t ncols, int32_t k0,
                  int digits, void *storage, gp_tc_prepared *out)
{
  if ((digits != 4 && digits != 5) || npanels < 1 || npanels > 2 || ncols < 1 || ncols > 1024 || k0 < 1)
    return gp_fail(ctx, GP_ERR_ARG, "gp_tc_prepare: bad panel shape");
  const int32_t kb0 = (k0 + XK - 1) / XK, kpad0 = kb0 * XK;
  const int32_t ncols4 = digits * ncols, tn = x_tile_cols(ncols4);
  const int32_t nct = (ncols4 + tn - 1) / tn, ncols4_pad = nct * tn;
  const int64_t ldb = (int64_t)kpad0 * npanels;
  uint8_t *base = (uint8_t *)storage;
  __half *B = (__half *)base;
  /* [ncols] joint max |P| bits */
  unsigned long long *mx = (unsigned long long *)(base + align256((size_t)ncols4_pad * ldb * 2));
  x_panels pan = {};
  for (int p = 0; p < npanels; ++p) {
    pan.P[p] = pp[p].P;
    pan.ldp[p] = pp[p].ldp;
    pan.sign[p] = pp[p].sign;
  }
  GP_CUDA(ctx, cudaMemsetAsync(mx, 0, 8 * (size_t)ncols, ctx->stream));
  int blocks = grid_cap(ctx, (int64_t)k0 * ncols, 256 * 16, 8);
  const int need = (ncols + 255) / 256;
  if (blocks < need) blocks = need;
  k_panel_absmax<<<dim3((unsigned)blocks, (unsigned)npanels), 256, 0, ctx->stream>>>(pan, k0, ncols,
                                                                                    mx);
  GP_LAUNCH_CHECK(ctx, "k_panel_absmax");
  dim3 sgrid((unsigned)(kpad0 / SL_K), (unsigned)((ncols4_pad + digits * SL_C - 1) / (digits * SL_C)),
             (unsigned)npanels);
  (digits == 5 ? k_panel_slices<5> : k_panel_slices<4>)<<<sgrid, 256, 0, ctx->stream>>>(
      pan, k0, ncols, mx, B, ldb, kpad0, ncols4_pad);
  GP_LAUNCH_CHECK(ctx, "k_panel_slices");
  PFN_cuTensorMapEncodeTiled_v12000 enc = tc_encode(ctx);
  if (!enc) return GP_ERR_CUDA;
  {
    cuuint64_t dims[2] = {(cuuint64_t)ldb, (cuuint64_t)ncols4_pad};
    cuuint64_t strides[1] = {(cuuint64_t)ldb * 2};
    cuuint32_t box[2] = {XK, (cuuint32_t)tn};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(&out->tmb, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, B, dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return gp_fail(ctx, GP_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  }
  out->B = B;
  out->mx = mx;
  out->ncols = ncols;
  out->tn = tn;
  out->nct = nct;
  out->npanels = npanels;
  out->digits = digits;
  out->kb0 = kb0;
  out->k0 = k0;
  out->ldb = ldb;
  out->count_lo = pp[0].count != 0;
  out->count_hi = npanels > 1 ? pp[1].count != 0 : out->count_lo;
  return GP_OK;
}

size_t gp_tc_sum_bytes(int32_t slice_cols, int32_t nrows)
{
  const size_t tn = (size_t)x_tile_cols(slice_cols), nct = ((size_t)slice_cols + tn - 1) / tn;
  return sizeof(unsigned long long) * (((size_t)nrows + XR - 1) / XR * XR) * nct * tn;
}

static int combine_grid(const gp_ctx *ctx, int64_t nrows, int32_t ncols)
{
  return grid_cap(ctx, (nrows + 31) / 32 * ((ncols + 31) / 32), 1, 32);
}

int gp_tc_begin(gp_ctx *ctx)
{
  GP_CUDA(ctx, cudaMemsetAsync(ctx->d_err, 0, sizeof(int), ctx->stream));
  return GP_OK;
}

int gp_tc_check(gp_ctx *ctx)
{
  int herr = 0;
  GP_CUDA(ctx, gp_memcpy(ctx, &herr, ctx->d_err, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  GP_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  if (herr) return gp_fail(ctx, GP_ERR_TIMEOUT, "tensor-core product wait timed out (code %d)", herr);
  return GP_OK;
}

int gp_tc_apply(gp_ctx *ctx, const gp_tc_codes *A, const gp_tc_prepared *P, double *d_Y,
                int64_t ldy)
{
  const int32_t nrows = A->nrows;
  if (nrows < 1) return GP_OK;
  if (A->k0 != P->k0 || A->ldc < (int64_t)P->kb0 * XK / 4)
    return gp_fail(ctx, GP_ERR_ARG, "gp_tc_apply: code operand and panel disagree");
  const int32_t nkb = P->kb0 * P->npanels;
  const int32_t tiles = (nrows + XR - 1) / XR * P->nct;
  const int32_t ksplit = x_split(tiles, nkb, ctx->num_sms);
  const bool whole = ksplit == 1 && P->digits == 4 && gp_tc_sums_fit((int64_t)nkb * XK);
  unsigned long long *sums = NULL;
  if (!whole) {
    const size_t sum_bytes = gp_tc_sum_bytes(P->digits * P->ncols, nrows);
    int rc = gp_scratch5(ctx, sum_bytes + 256, (void **)&sums);
    if (rc) return rc;
    GP_CUDA(ctx, cudaMemsetAsync(sums, 0, sum_bytes, ctx->stream));
  }
  GP_CUDA(ctx, cudaFuncSetAttribute(k_geno_panel_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    X_SMEM));
  const int32_t nitems = tiles * ksplit;
  const int grid = nitems < ctx->num_sms ? nitems : ctx->num_sms;
  k_geno_panel_tc<<<grid, X_THREADS, X_SMEM, ctx->stream>>>(
      P->tmb, A->codes, A->ldc, A->row_map, nrows, P->tn, P->nct, nkb, P->kb0, P->count_lo,
      P->count_hi, ksplit, X_CHUNK_KB(P->digits), sums, P->mx, whole ? d_Y : NULL, ldy, P->ncols,
      ctx->d_err, NULL);
  GP_LAUNCH_CHECK(ctx, "k_geno_panel_tc");
  if (whole) return GP_OK;
  (P->digits == 5 ? k_panel_combine<5> : k_panel_combine<4>)
      <<<combine_grid(ctx, nrows, P->ncols), 256, 0, ctx->stream>>>(
          sums, P->nct * P->tn, nrows, P->ncols, P->mx, d_Y, ldy, NULL);
  GP_LAUNCH_CHECK(ctx, "k_panel_combine");
  return GP_OK;
}

/* the sums of the batch's row tiles = 0 */
__global__ void k_zero_batch_sums(unsigned long long *sums, int32_t wcols, const gp_tc_batch *db)
{
  const int64_t total = (int64_t)((db->nrows + XR - 1) / XR) * wcols * (XR / 2);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x)
    ((ulonglong2 *)sums)[i] = make_ulonglong2(0, 0);
}

int gp_tc_apply_dev(gp_ctx *ctx, const gp_tc_batch *db, int32_t max_rows, int64_t ldc,
                    const gp_tc_prepared *P, void *sums, double *d_Y, int64_t ldy)
{
  if (max_rows < 1) return GP_OK;
  if (P->digits != 4 || ldc < (int64_t)P->kb0 * XK / 4)
    return gp_fail(ctx, GP_ERR_ARG, "gp_tc_apply_dev: code rows shorter than the panel");
  unsigned long long *z = (unsigned long long *)sums;
  const int32_t wcols = P->nct * P->tn;
  k_zero_batch_sums<<<grid_cap(ctx, ((int64_t)max_rows + XR) * wcols / 2, 256, 8), 256, 0,
                      ctx->stream>>>(z, wcols, db);
  GP_LAUNCH_CHECK(ctx, "k_zero_batch_sums");
  GP_CUDA(ctx, cudaFuncSetAttribute(k_geno_panel_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    X_SMEM));
  /* every SM: the kernel takes the batch's row count, and with it its work items, from db */
  k_geno_panel_tc<<<ctx->num_sms, X_THREADS, X_SMEM, ctx->stream>>>(
      P->tmb, NULL, ldc, NULL, 0, P->tn, P->nct, P->kb0 * P->npanels, P->kb0, P->count_lo,
      P->count_hi, 1, X_CHUNK_KB(4), z, NULL, NULL, 0, 0, ctx->d_err, db);
  GP_LAUNCH_CHECK(ctx, "k_geno_panel_tc");
  k_panel_combine<4><<<combine_grid(ctx, max_rows, P->ncols), 256, 0, ctx->stream>>>(
      z, wcols, 0, P->ncols, P->mx, d_Y, ldy, db);
  GP_LAUNCH_CHECK(ctx, "k_panel_combine");
  return GP_OK;
}

int gp_geno_panel_tc_codes(gp_ctx *ctx, const gp_tc_codes *A, int npanels, const gp_tc_panel *pp,
                           int32_t ncols, int digits, double *d_Y, int64_t ldy)
{
  if (A->nrows < 1 || A->k0 < 1) return GP_OK;
  /* 5 slices: any number of columns, a group at a time, which bounds the slices and sums */
  const int32_t step = digits == 5 && ncols > X_GROUP5 ? X_GROUP5 : ncols;
  for (int32_t c0 = 0; c0 < ncols; c0 += step) {
    const int32_t nc = ncols - c0 < step ? ncols - c0 : step;
    gp_tc_panel pg[2];
    for (int p = 0; p < npanels && p < 2; ++p) {
      pg[p] = pp[p];
      pg[p].P += c0;
    }
    uint8_t *storage;
    int rc = gp_scratch2(ctx, gp_tc_prepared_bytes(npanels, nc, A->k0, digits), (void **)&storage);
    if (rc) return rc;
    gp_tc_prepared P;
    rc = gp_tc_prepare(ctx, npanels, pg, nc, A->k0, digits, storage, &P);
    if (!rc) rc = gp_tc_apply(ctx, A, &P, d_Y + c0, ldy);
    if (rc) return rc;
  }
  return GP_OK;
}

int gp_tc_codes_for(gp_ctx *ctx, int sum_over_snps, const int32_t *d_samp, int32_t nsamp,
                    const int32_t *d_snprec, int32_t nk, int distinct, gp_tc_codes *out)
{
  const int current_rows = sum_over_snps && d_samp == ctx->d_rows && nsamp == ctx->nrows &&
                           nk == ctx->nkept;
  if (current_rows && ctx->codes4_rows) {
    /* the sample-major codes of the current rows are still in place */
    int64_t ldc;
    int32_t rows_pad;
    gp_tc_code_bytes(1, nsamp, nk, &ldc, &rows_pad);
    out->codes = (uint8_t *)ctx->d_scratch4;
    out->ldc = ldc;
    out->row_map = NULL;
    out->nrows = nsamp;
    out->k0 = nk;
    return GP_OK;
  }
  if (!sum_over_snps && nsamp == ctx->nind_all) {
    /* every sample in order: the resident records are the SNP-major operand */
    out->codes = ctx->d_geno;
    out->ldc = ctx->rlen_dev;
    out->row_map = d_snprec;
    out->nrows = nk;
    out->k0 = nsamp;
    return GP_OK;
  }
  int64_t ldc;
  int32_t rows_pad;
  gp_tc_code_bytes(sum_over_snps, nsamp, nk, &ldc, &rows_pad);
  uint8_t *codes;
  const size_t cb = align256((size_t)rows_pad * ldc + 256);
  int rc = gp_scratch4(ctx, cb + sizeof(int32_t) * (size_t)ctx->nind_all, (void **)&codes);
  if (rc) return rc;
  rc = gp_tc_build_codes(ctx, sum_over_snps, d_samp, nsamp, d_snprec, nk,
                         distinct ? (int32_t *)(codes + cb) : NULL, codes, out);
  if (!rc && current_rows) ctx->codes4_rows = 1;
  return rc;
}
