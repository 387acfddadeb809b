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
// row_key[tokens] and block_flags[ceil(tokens / 256)] zeroed; the norms of state raised to this call's, its other words zeroed.
// tokens and ch are multiples of 32.
struct WideCast {
  const float *q, *k, *v;
  void *q16, *k16, *vt16;
  int tokens, ch;
  unsigned int* row_key;
  unsigned int* block_flags;
  unsigned int* state;
  float* zero;  // optional: [tokens][ch] set to zero
};
cudaError_t launch_wide_cast(cudaStream_t stream, const WideCast& args);

}  // namespace zdraw
