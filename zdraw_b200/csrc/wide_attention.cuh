// Launch interface of the helper kernels of the wide-head attention (internal to the library).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace zdraw {

// Words of WideCast::state (zeroed once when the context is made): running maxima of the launch (the last
// block leaves them at zero again), a block counter, and the route of the row maxima (see linear.cuh).
constexpr int kWideStatQ = 0, kWideStatK = 2, kWideCounter = 4, kWideRoute = 5, kWideStateWords = 8;

// The operands of one call: [tokens][ch] f32 -> q16, k16 [tokens][ch] and vt16 [ch][tokens] in half (clamped);
// row_key[tokens] and block_flags[ceil(tokens / 256)] zeroed; state[kWideRoute] = 0 or 1. tokens and ch are
// multiples of 32.
struct WideCast {
  const float *q, *k, *v;
  void *q16, *k16, *vt16;
  int tokens, ch;
  float exp_scale;
  unsigned int* row_key;
  unsigned int* block_flags;
  unsigned int* state;
  float* zero;  // optional: [tokens][ch] set to zero
};
cudaError_t launch_wide_cast(cudaStream_t stream, const WideCast& args);

}  // namespace zdraw
