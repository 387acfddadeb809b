// Launch interface of the wide-attention helper kernels (internal to the library).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace zdraw {

// Words of the wide attention's state in device memory, zeroed when the context is made: the largest |row|^2 of Q and of
// K as float bits (zero again once the exp product has run, so that what a call leaves behind goes no further than
// the next one), whether the call took its row maxima from all keys, and whether its sample missed a row's.
constexpr int kWideNorms = 0, kWideAllKeys = 2, kWideMissed = 3, kWideStateWords = 4;

// The operands of one call: [tokens][ch] f32 -> q16, k16 [tokens][ch] and vt16 [ch][tokens] in half (clamped);
// row_key[tokens] and row_missed[tokens] zeroed; the norms of state raised to this call's, its other words zeroed.
// tokens and ch are multiples of 32.
struct WideCast {
  const float *q, *k, *v;
  void *q16, *k16, *vt16;
  int tokens, ch;
  unsigned int* row_key;
  unsigned int* row_missed;
  unsigned int* state;
};
cudaError_t launch_wide_cast(cudaStream_t stream, const WideCast& args);

// exp(scores) p [tokens][ld_p] in half, n_partial * 128 columns, with the partial sums, offsets and flags that the exp
// epilogue leaves (LinearPart): rows that are flagged are brought to one scale. Leaves at once when *any_missed is 0.
struct WideRescale {
  void* p;
  long long ld_p;
  int tokens, n_partial;
  float* row_sum;
  const float* shift;
  const unsigned int* row_missed;
  const unsigned int* any_missed;
};
cudaError_t launch_wide_rescale(cudaStream_t stream, const WideRescale& args, int sm_count);

}  // namespace zdraw
