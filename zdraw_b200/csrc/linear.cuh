// Launch interface of the projection GEMM (internal to the library).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace zdraw {

constexpr int kEpiloguePlain = 0;   // C = A W^T (rows divided by the sum of row_sum when given)
constexpr int kEpilogueQk = 1;      // q/k prologue applied to the accumulator
constexpr int kEpilogueRowMax = 2;  // no C: row_key[row] = max over the row, as an ordered key
constexpr int kEpilogueExp = 3;     // C = half(exp2((A W^T - max[row]) * exp_scale)), partial row sums

// Largest score (in exp2 units) up to which row maxima are taken from a sample, see LinearArgs::norms. N(0, 1) operands
// of 512 channels are at 42. Beyond it rows are peaked, and under its exact maximum a row's largest weight is 1 and
// not rounded: error 2.3e-4 against 2.8e-4 from the sample (operands times 1.7, 4096 tokens). That costs a product
// with all keys: with operands times 3, 69 against 64 us at 4096 x 512, 690 against 590 at 16384.
constexpr float kMaxSampledScore = 80.0f;

constexpr int kMaxLinearParts = 3;

// One output of a launch: C_p[m, n] = A[m, k] * W_p[n, k]^T with its own epilogue.
struct LinearPart {
  int epilogue;  // kEpilogue*
  int c_f32;     // plain: 1 = f32 C, 0 = f16 C (exp: f16)
  void* c;       // plain, exp: [m][ld_c]; qk: f16 head-major [image][head][token][128]
  long long ld_c;
  const float *w_txt, *w_img;  // qk: norm weights [128]
  // row max: out, one ordered key per row (see float_key), zeroed by the caller. exp: in, the same keys;
  // row_sum receives [m][n_partial] partial sums of the exponentials (f32, before rounding to half), one
  // per 128 columns. plain: with row_sum the rows are divided by the sum of their partial sums (added in
  // a fixed order). n_partial is even.
  unsigned int* row_key;
  float* row_sum;
  int n_partial;
  float exp_scale;
  // exp, when row_key may lie below a row's maximum (nullptr: it does not): 128 columns of a row whose largest
  // exponential leaves the half range are stored times 2^-d, the whole number d in shift[row][128-column block], their
  // partial sum (times 2^-d as well) negated; row_missed[row] and *any_missed are set to 1 (both zeroed by the caller).
  float* shift;
  unsigned int* row_missed;
  unsigned int* any_missed;
  // row max / exp: columns at and beyond n_valid are padding of the last column block (W has no
  // such rows): they do not count for the maximum and are stored as zeros.
  int n_valid;
};

// Up to three products that share A (the Q, K and V projections of one activation) run as one
// launch over n_parts * (n / 256) column blocks. A and every W are reached through tensor maps
// (f16, 128-byte swizzle, boxes of 64 columns x 128 rows). Tiles are 256 columns x 64 of K; partial
// tiles read zeros beyond the matrices.
struct LinearArgs {
  int m, n, k;
  // 1, or 2 (f32 plain C that holds zeros before the launch, k > 64): each tile's K is walked in two halves by
  // two CTA pairs that add their results to C. Two additions to zero give the same sum in either order.
  int k_splits;
  int n_parts;
  LinearPart part[kMaxLinearParts];
  // qk epilogue (n == heads * 128, m == images * tokens)
  int tokens, heads, txt_tokens;
  float norm_eps;
  const float *rope_cos, *rope_sin;  // [tokens][128]
  long long rope_batch_stride;
  uint32_t* status;
  // Row max over a sample of the rows of W (the wide attention): norms holds the largest |row|^2 of A and of the whole W
  // as float bits, and where |row of A| |row of W| norm_scale can exceed kMaxSampledScore (or is not a number) the
  // launch takes all of W instead: n_all columns, n_valid_all of them real, through maps.w[1]; *all_rows is set to 1.
  const unsigned int* norms;
  float norm_scale;
  int n_all, n_valid_all;
  unsigned int* all_rows;
  unsigned int* norms_done;  // exp: two words that the launch leaves at zero (the norms, for the call after this one)
  float4* zero;  // optional: zero_n4 pieces set to zero by warps that have no part in the product
  long long zero_n4;
  int early_dependents;  // 1: the next launch in the stream may be set up before this one ends
  // Tile order: 0 = down the rows of one column block (W stays in L2), 1 = across the column blocks
  // of one row block (A stays in L2).
  int rows_first;
};

struct LinearMaps {
  CUtensorMap a;
  CUtensorMap w[kMaxLinearParts];  // unused entries repeat w[0]; with LinearArgs::norms w[1] is all of W
  // Plain and exp parts: C as a 2-D map (columns, rows) with a box of 128 bytes (32 columns of f32, 64 of
  // f16) x 32 rows and 128-byte swizzle, for the epilogue's tile stores. Unused entries hold any valid map.
  CUtensorMap c[kMaxLinearParts];
};

cudaError_t linear_configure();
// CTA pairs that the current device holds at once.
cudaError_t linear_pairs(int sm_count, int* pairs);
// Tiles of 256 x 256 of a launch, and whether splitting their K in two lets it end sooner: each pair takes whole
// work items, so a launch lasts as long as its busiest pair's items. (4096 x 512 x 4096: 32 tiles on 74 pairs,
// 64 half-length items when split.)
inline int linear_tiles(int m, int n, int n_parts) { return ((m + 255) / 256) * ((n + 255) / 256) * n_parts; }
inline bool linear_split_pays(int tiles, int pairs) {
  return (2 * tiles + pairs - 1) / pairs < 2 * ((tiles + pairs - 1) / pairs);
}
cudaError_t launch_linear(cudaStream_t stream, const LinearMaps& maps, const LinearArgs& args, int pairs);

}  // namespace zdraw
