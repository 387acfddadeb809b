// First kernel of the wide-head attention (one head, head_dim 512: the VAE mid-block shape), which
// follows the reference's decomposition into GEMMs (src/metal/mvattn_owned.zig:283-330, product tier:
// half Q, K and V^T, S = Q K^T with f32 output, a row softmax writing half P, O = P (V^T)^T), with
// the softmax (krow_softmax_h, :95-128) folded into the epilogues of linear_kernel so that the f32
// scores never reach memory. This file holds the casts of Q and K (kf32_to_h), the transpose-and-cast
// of V (kvt_transpose_h, :84-94) and the operands' norms, by which the row maxima are taken.
#include "wide_attention.cuh"

#include <cuda_fp16.h>

#include "ptx.cuh"

namespace zdraw {

namespace {

constexpr float kHalfMax = 65504.0f;
constexpr int kRowsPerBlock = 8;  // Q, K: one warp per row
constexpr int kVTile = 64;        // V: 64 tokens x 64 channels per block

__device__ __forceinline__ float clamp_half(float x) { return fminf(fmaxf(x, -kHalfMax), kHalfMax); }

// V: float4 reads along the channels, 128-byte writes along the tokens (two halves per lane).
__device__ __forceinline__ void transpose_block(const WideCast& a, int block, __half (*tile)[kVTile + 2]) {
  const int blocks_t = (a.tokens + kVTile - 1) / kVTile;
  const int t0 = (block % blocks_t) * kVTile, c0 = (block / blocks_t) * kVTile;
  const int piece = static_cast<int>(threadIdx.x) & 15, row = static_cast<int>(threadIdx.x) >> 4;
#pragma unroll
  for (int r = 0; r < kVTile; r += 16) {
    const int t = t0 + r + row, c = c0 + 4 * piece;
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (t < a.tokens && c < a.ch) v = __ldg(reinterpret_cast<const float4*>(a.v + static_cast<long long>(t) * a.ch + c));
    tile[4 * piece + 0][r + row] = __float2half_rn(clamp_half(v.x));
    tile[4 * piece + 1][r + row] = __float2half_rn(clamp_half(v.y));
    tile[4 * piece + 2][r + row] = __float2half_rn(clamp_half(v.z));
    tile[4 * piece + 3][r + row] = __float2half_rn(clamp_half(v.w));
  }
  __syncthreads();
  const int lane = static_cast<int>(threadIdx.x) & 31, warp = static_cast<int>(threadIdx.x) >> 5;
  __half* out = static_cast<__half*>(a.vt16);
#pragma unroll
  for (int i = 0; i < kVTile / 8; ++i) {
    const int c = 8 * i + warp, t = t0 + 2 * lane;
    if (c0 + c < a.ch && t < a.tokens)
      *reinterpret_cast<__half2*>(out + static_cast<long long>(c0 + c) * a.tokens + t) =
          *reinterpret_cast<const __half2*>(&tile[c][2 * lane]);
  }
}

// Q or K: one warp per row, four floats per lane and step -> four halves (clamped). The block's largest row sum of
// squares raises *norm as float bits (which order like unsigned integers; a NaN lies above them all), so the
// result does not depend on the order of the updates.
__device__ __forceinline__ void cast_block(const WideCast& a, const float* in, __half* out16, int block, bool zero_rows,
                                           unsigned int* block_norm, unsigned int* norm) {
  const int row_raw = block * kRowsPerBlock + (static_cast<int>(threadIdx.x) >> 5);
  const bool live = row_raw < a.tokens;
  const long long row = live ? row_raw : a.tokens - 1;  // a repeated row changes no maximum and is not stored
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const float4* src = reinterpret_cast<const float4*>(in + row * a.ch);
  uint2* dst16 = reinterpret_cast<uint2*>(out16 + row * a.ch);
  float4* zero = zero_rows ? reinterpret_cast<float4*>(a.zero + row * a.ch) : nullptr;
  float ss = 0.0f;
  const int n4 = a.ch / 4;
  // Four loads in flight per lane (512 floats per pass of the warp): the row of the VAE shape in one pass.
  for (int i0 = lane; i0 < n4; i0 += 128) {
    float4 vv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + 32 * u < n4) vv[u] = __ldg(src + i0 + 32 * u);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = i0 + 32 * u;
      if (i >= n4) break;
      const float4 v = vv[u];
      ss = fmaf(v.x, v.x, ss);
      ss = fmaf(v.y, v.y, ss);
      ss = fmaf(v.z, v.z, ss);
      ss = fmaf(v.w, v.w, ss);
      const __half2 h0 = __floats2half2_rn(clamp_half(v.x), clamp_half(v.y));
      const __half2 h1 = __floats2half2_rn(clamp_half(v.z), clamp_half(v.w));
      uint2 o;
      o.x = *reinterpret_cast<const uint32_t*>(&h0);
      o.y = *reinterpret_cast<const uint32_t*>(&h1);
      if (live) dst16[i] = o;
      if (zero && live) zero[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  if (threadIdx.x == 0) *block_norm = 0u;
  __syncthreads();
  if (lane == 0) atomicMax(block_norm, __float_as_uint(ss));
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(norm, *block_norm);
}

// One launch for the three operands (three launches, two memsets and a one-thread kernel took about 25 us of a
// call at 4096 x 512, this takes 8). Memory-bound: 6 bytes per element, 26 us at 16384 x 512.
__global__ void __launch_bounds__(256) wide_cast_kernel(const WideCast a, int row_blocks) {
  __shared__ __half tile[kVTile][kVTile + 2];
  __shared__ unsigned int block_norm;
  // The launches before this one may still read what it writes.
  grid_dependency_wait();
  grid_launch_dependents();
  const int block = static_cast<int>(blockIdx.x);
  if (block >= 2 * row_blocks) {
    transpose_block(a, block - 2 * row_blocks, tile);
  } else if (block >= row_blocks) {
    cast_block(a, a.k, static_cast<__half*>(a.k16), block - row_blocks, false, &block_norm,
               a.state + kWideNorms + 1);
  } else {
    cast_block(a, a.q, static_cast<__half*>(a.q16), block, a.zero != nullptr, &block_norm, a.state + kWideNorms);
    const int row = block * kRowsPerBlock + static_cast<int>(threadIdx.x);
    if (threadIdx.x < kRowsPerBlock && row < a.tokens) {
      a.row_key[row] = 0u;  // lies below the key of every float
      if (row % 256 == 0) a.block_flags[row / 256] = 0u;
      if (row == 0) a.state[kWideAllKeys] = a.state[kWideMissed] = 0u;
    }
  }
}

}  // namespace

cudaError_t launch_wide_cast(cudaStream_t stream, const WideCast& args) {
  const int row_blocks = (args.tokens + kRowsPerBlock - 1) / kRowsPerBlock;
  const int v_blocks = ((args.tokens + kVTile - 1) / kVTile) * ((args.ch + kVTile - 1) / kVTile);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * row_blocks + v_blocks);
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, wide_cast_kernel, args, row_blocks);
}

}  // namespace zdraw
