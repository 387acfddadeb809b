// First kernel of the wide-head attention (one head, head_dim 512: the VAE mid-block shape), which
// follows the reference's decomposition into GEMMs (src/metal/mvattn_owned.zig:283-330, product tier:
// half Q, K and V^T, S = Q K^T with f32 output, a row softmax writing half P, O = P (V^T)^T), with
// the softmax (krow_softmax_h, :95-128) folded into the epilogues of linear_kernel so that the f32
// scores never reach memory. This file holds the casts of Q and K (kf32_to_h), the transpose-and-cast
// of V (kvt_transpose_h, :84-94), and the pass over the rows whose subtracted maximum was too small.
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
__device__ __forceinline__ void cast_block(const WideCast& a, const float* in, __half* out16, int block,
                                           unsigned int* block_norm, unsigned int* norm) {
  const int row_raw = block * kRowsPerBlock + (static_cast<int>(threadIdx.x) >> 5);
  const bool live = row_raw < a.tokens;
  const long long row = live ? row_raw : a.tokens - 1;  // a repeated row changes no maximum and is not stored
  const int lane = static_cast<int>(threadIdx.x) & 31;
  const float4* src = reinterpret_cast<const float4*>(in + row * a.ch);
  uint2* dst16 = reinterpret_cast<uint2*>(out16 + row * a.ch);
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
// call at 4096 x 512, this takes 8). Memory-bound: 6 bytes per element, 23 us at 16384 x 512.
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
    cast_block(a, a.k, static_cast<__half*>(a.k16), block - row_blocks, &block_norm, a.state + kWideNorms + 1);
  } else {
    cast_block(a, a.q, static_cast<__half*>(a.q16), block, &block_norm, a.state + kWideNorms);
    const int row = block * kRowsPerBlock + static_cast<int>(threadIdx.x);
    if (threadIdx.x < kRowsPerBlock && row < a.tokens) {
      a.row_key[row] = 0u;  // lies below the key of every float
      a.row_missed[row] = 0u;
      if (row == 0) a.state[kWideAllKeys] = a.state[kWideMissed] = 0u;
    }
  }
}

// Brings the rows that the sample of the keys missed to one scale. The exp product has stored each 128 columns of
// such a row times 2^-d, with a d of their own (0 where the sample served); they become times 2^-D, D the row's
// largest d, and so do their partial sums. The factors are powers of two: nothing but what falls below the half
// range is rounded, as it would be under the exact maximum. A piece whose sum shows that all of it rounds to zero
// is only written.
// One warp per row and step: a row is a chain of memory latencies (flag, sums, offsets, its elements), so many rows
// are kept in flight. 16384 x 512 with every row missed: 85 to 164 us (the latter reads and writes all of P, 1.02 GB
// at 6.2 TB/s); one block per row took 126 to 176, but 18 instead of 21 where 64 rows are missed.
constexpr int kMaxPartial = 512;  // 65536 tokens
constexpr int kRescaleWarps = 8;
__device__ __forceinline__ bool shifted(float sum) { return __float_as_int(sum) < 0 && sum == sum; }
__global__ void __launch_bounds__(32 * kRescaleWarps) wide_rescale_kernel(const WideRescale a) {
  __shared__ float factors[kRescaleWarps][kMaxPartial];  // of each 128 columns; 0 = all of them round to zero
  grid_dependency_wait();
  if (ld_volatile_u32(a.any_missed) == 0u) return;
  const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
  float* factor = factors[warp];
  // From the last row to the first: what is rescaled last is still in L2 when P V begins with the first rows.
  const int n_warps = kRescaleWarps * static_cast<int>(gridDim.x);
  for (int back = kRescaleWarps * static_cast<int>(blockIdx.x) + warp; back < a.tokens; back += n_warps) {
    const int row = a.tokens - 1 - back;
    if (a.row_missed[row] == 0u) continue;
    float* sums = a.row_sum + static_cast<long long>(row) * a.n_partial;
    const float* shifts = a.shift + static_cast<long long>(row) * a.n_partial;
    float top = 0.0f;
    for (int t = lane; t < a.n_partial; t += 32)
      if (shifted(sums[t])) top = fmaxf(top, shifts[t]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
    for (int t = lane; t < a.n_partial; t += 32) {
      const float sum = sums[t];
      const float d = shifted(sum) ? shifts[t] : 0.0f;
      const int e = static_cast<int>(fmaxf(d - top, -200.0f));
      const float f = e < -126 ? 0.0f : __uint_as_float(static_cast<uint32_t>(127 + e) << 23);  // 2^e
      const float scaled = fabsf(sum) * f;  // no element is larger: at 2^-25 and below all of them round to zero
      sums[t] = scaled;
      factor[t] = scaled <= 0x1p-25f ? 0.0f : (scaled == scaled ? f : 1.0f);  // NaN stays
    }
    __syncwarp();
    uint4* p = reinterpret_cast<uint4*>(static_cast<__half*>(a.p) + static_cast<long long>(row) * a.ld_p);
    const int n8 = a.n_partial * 16;  // 8 halves each; a multiple of 32
    for (int i0 = lane; i0 < n8; i0 += 8 * 32) {
      uint4 x[8];
      float f[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = i0 + 32 * u;
        f[u] = i < n8 ? factor[i >> 4] : 1.0f;
        x[u] = make_uint4(0u, 0u, 0u, 0u);
        if (f[u] != 0.0f && f[u] != 1.0f) x[u] = p[i];
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        if (f[u] == 1.0f) continue;
        uint32_t* h = reinterpret_cast<uint32_t*>(&x[u]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 v = __half22float2(*reinterpret_cast<const __half2*>(h + j));
          h[j] = pack_f16x2(v.x * f[u], v.y * f[u]);
        }
        p[i0 + 32 * u] = x[u];
      }
    }
    __syncwarp();  // the factors are used again
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

cudaError_t launch_wide_rescale(cudaStream_t stream, const WideRescale& args, int sm_count) {
  if (args.n_partial > kMaxPartial) return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg = {};
  const int blocks = 8 * sm_count, needed = (args.tokens + kRescaleWarps - 1) / kRescaleWarps;
  cfg.gridDim = dim3(needed < blocks ? needed : blocks);
  cfg.blockDim = dim3(32 * kRescaleWarps);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, wide_rescale_kernel, args);
}

}  // namespace zdraw
