/* Exact genotype x FP64-panel products on the tensor cores (gp_geno_tc.cu). */
#ifndef GP_GENO_TC_H
#define GP_GENO_TC_H
#include <cuda.h>
#include <cuda_fp16.h>
#include <vector>

#include "gp_internal.h"

/* one FP64 panel P [k][ldp] (device); count = 1: the genotype operand is the allele count
 * {0,1,2}, else the observed mask {0,1}; sign multiplies the panel */
struct gp_tc_panel {
  const double *P;
  int64_t ldp;
  double sign;
  int count;
};

/* A genotype code operand: rows of ldc bytes of 2-bit codes (MSB first, 3 -> 0); output
 * row r reads code row row_map[r] (or r); k0 = the k extent of one panel. */
struct gp_tc_codes {
  const uint8_t *codes;
  int64_t ldc;
  const int32_t *row_map;
  int32_t nrows;
  int32_t k0;
};

/* bytes of the code operand built by gp_tc_build_codes: rows_pad * ldc */
int gp_tc_code_bytes(int sum_over_snps, int32_t nsamp, int32_t nk, int64_t *ldc, int32_t *rows_pad);
/* the code operand of the samples d_samp, in any order, into codes.  inv: room for nind_all integers
 * when the samples of a sum over SNPs are distinct (the faster transpose then applies), or NULL */
int gp_tc_build_codes(gp_ctx *ctx, int sum_over_snps, const int32_t *d_samp, int32_t nsamp,
                      const int32_t *d_snprec, int32_t nk, int32_t *inv, uint8_t *codes,
                      gp_tc_codes *out);
/* a panel cut into fp16 slices once (B operand + column exponents + its tensor map): `digits`
 * slices, 4 of 10 bits (the split precisions) or 5 of 12 bits (FP64) */
struct gp_tc_prepared {
  __half *B;
  unsigned long long *mx; /* per column the bits of its largest magnitude: its exponent */
  int32_t ncols, npanels, digits, kb0, k0;
  int32_t tn, nct; /* slice columns per tile, column tiles */
  int64_t ldb;
  int count_lo, count_hi; /* the panels multiply counts (1) or observed masks (0) */
  CUtensorMap tmb;
};
size_t gp_tc_prepared_bytes(int npanels, int32_t ncols, int32_t k0, int digits);
/* slice the panels into caller storage of gp_tc_prepared_bytes bytes (device) */
int gp_tc_prepare(gp_ctx *ctx, int npanels, const gp_tc_panel *pp, int32_t ncols, int32_t k0,
                  int digits, void *storage, gp_tc_prepared *out);
/* whether a row's four slice sums over k values (of all panels) fit one 64-bit integer: a term is at
 * most a count of 2 times 2^40 */
static inline bool gp_tc_sums_fit(int64_t k) { return k <= (int64_t)1 << 21; }
/* Y[r][c] = products of the code operand with a prepared panel, queued on ctx->stream.  Its
 * bounded waits report through ctx->d_err: gp_tc_begin clears it ahead of any number of
 * products, gp_tc_check waits for them and returns the error */
int gp_tc_apply(gp_ctx *ctx, const gp_tc_codes *A, const gp_tc_prepared *P, double *d_Y,
                int64_t ldy);
int gp_tc_begin(gp_ctx *ctx);
int gp_tc_check(gp_ctx *ctx);

/* The batch a device-resident loop works on: nrows code rows at codes (ring position row0
 * of the pool), requests [req_begin, req_end) of the loop's queue.  Written on the device
 * by the loop's batch former and read by the kernels at run time, so that one captured
 * launch serves every batch. */
struct gp_tc_batch {
  const uint8_t *codes;
  int32_t nrows;
  int32_t pad;
  int64_t row0, req_begin, req_end;
};
/* gp_tc_apply inside a loop body: the rows come from db at run time (at most max_rows, row
 * stride ldc); sums: gp_tc_sum_bytes(digits * ncols, max_rows) bytes of the caller's;
 * errors of the bounded waits go to ctx->d_err */
size_t gp_tc_sum_bytes(int32_t slice_cols, int32_t nrows);
int gp_tc_apply_dev(gp_ctx *ctx, const gp_tc_batch *db, int32_t max_rows, int64_t ldc,
                    const gp_tc_prepared *P, void *sums, double *d_Y, int64_t ldy);

/* the code operand of a sum over SNPs (rows = samples d_samp) or over samples (rows = SNPs),
 * built into scratch4, or the resident records when a SNP-major operand covers every sample in
 * order; distinct: no sample occurs twice in d_samp */
int gp_tc_codes_for(gp_ctx *ctx, int sum_over_snps, const int32_t *d_samp, int32_t nsamp,
                    const int32_t *d_snprec, int32_t nk, int distinct, gp_tc_codes *out);
/* Y[r][c] = sum_p sum_k A_p(r, k) sign_p P_p[k][c] with a prepared code operand: npanels (1 or
 * 2) panels share the k extent and are concatenated along k with one joint column scale; Y is
 * device FP64 with row stride ldy; ncols <= 1024 with 4 digits, any number with 5.  Uses
 * scratch2 and scratch5. */
int gp_geno_panel_tc_codes(gp_ctx *ctx, const gp_tc_codes *A, int npanels, const gp_tc_panel *pp,
                           int32_t ncols, int digits, double *d_Y, int64_t ldy);

#endif
