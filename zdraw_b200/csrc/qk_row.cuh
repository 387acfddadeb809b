// The q/k prologue of one row of 128 elements, spread over 16 lanes with 8 consecutive elements each: shared
// by the prologue kernel and by the attention kernels that carry the prologue themselves, so that both give
// the same bytes.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "ptx.cuh"

namespace zdraw {

// f16 q and k are read once: the loads bypass L1 allocation (measured 21.1 us against 21.4 with plain
// read-only loads; an L2 evict-first policy on top made it slower, 22.4).
__device__ __forceinline__ uint4 ld_stream16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void load8(const __half* p, float* x) {
  const uint4 raw = ld_stream16(p);
  const __half2* h = reinterpret_cast<const __half2*>(&raw);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 f = __half22float2(h[i]);
    x[2 * i] = f.x;
    x[2 * i + 1] = f.y;
  }
}
__device__ __forceinline__ void load8(const float* p, float* x) {
  // (also the weight and table slices, which every head of a token reuses: through L1)
  const float4 a = __ldg(reinterpret_cast<const float4*>(p));
  const float4 b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
  x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}

constexpr float kHalfMax = 65504.0f;

// Rounds to f16 and clamps to +-65504 (an overflow rounds to +-inf first, then clamps).
__device__ __forceinline__ uint32_t pack_clamped(float lo, float hi) {
  const __half2 lim = __float2half2_rn(kHalfMax);
  __half2 h = __floats2half2_rn(lo, hi);
  h = __hmin2(__hmax2(h, __hneg2(lim)), lim);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint4 pack8_clamped(const float* x) {
  return make_uint4(pack_clamped(x[0], x[1]), pack_clamped(x[2], x[3]), pack_clamped(x[4], x[5]), pack_clamped(x[6], x[7]));
}

// y0 = (x0 inv w0) c0 - (x1 inv w1) s0 = inv (x0 (w0 c0) - x1 (w1 s0)), likewise y1: the weight
// is folded into the rotation coefficients once per token, not once per head. The arithmetic
// runs on packed f32 pairs: the even elements of two rotation pairs in one register pair, the
// odd ones in another, so a rotation is two packed multiplies and two packed FMAs per four
// elements. ca0/nsb0 give y_even = x_even ca0 + x_odd nsb0, ca1/sb1 give y_odd = x_odd ca1 +
// x_even sb1.
struct RopeCoef {
  uint64_t ca0[2], nsb0[2], ca1[2], sb1[2];
};
__device__ __forceinline__ RopeCoef rope_coef(const float* wv, const float* cv, const float* sv) {
  RopeCoef c;
#pragma unroll
  for (int j = 0; j < 2; ++j) {  // elements 4j .. 4j+3: pairs (4j, 4j+1) and (4j+2, 4j+3)
    const int e = 4 * j;
    c.ca0[j] = f2_pack(wv[e] * cv[e], wv[e + 2] * cv[e + 2]);
    c.nsb0[j] = f2_pack(-(wv[e + 1] * sv[e]), -(wv[e + 3] * sv[e + 2]));
    c.ca1[j] = f2_pack(wv[e + 1] * cv[e + 1], wv[e + 3] * cv[e + 3]);
    c.sb1[j] = f2_pack(wv[e] * sv[e + 1], wv[e + 2] * sv[e + 3]);
  }
  return c;
}

// The lane's 8 elements, normalised over the row's 16 lanes (all 32 lanes of the warp call this: lanes 0-15
// and 16-31 hold different rows), rotated and rounded to half.
__device__ __forceinline__ uint4 norm_rope_row(const float* x, const RopeCoef& c, float eps) {
  uint64_t xe[2], xo[2];  // even / odd elements of the two rotation pairs of each half
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    xe[j] = f2_pack(x[4 * j], x[4 * j + 2]);
    xo[j] = f2_pack(x[4 * j + 1], x[4 * j + 3]);
  }
  uint64_t ss2 = f2_mul(xe[0], xe[0]);
  ss2 = f2_fma(xo[0], xo[0], ss2);
  ss2 = f2_fma(xe[1], xe[1], ss2);
  ss2 = f2_fma(xo[1], xo[1], ss2);
  float s_lo, s_hi;
  f2_unpack(ss2, s_lo, s_hi);
  float ss = s_lo + s_hi;
  // Offsets < 16 keep the two rows of a warp apart.
#pragma unroll
  for (int off = 8; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
  // rsqrt.approx is within 2 units in the last place of f32, far below the half rounding of the result.
  const float inv = rsqrtf(fmaf(ss, 1.0f / 128.0f, eps));
  const uint64_t inv2 = f2_pack(inv, inv);
  uint32_t out[4];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint64_t ye = f2_mul(f2_fma(xo[j], c.nsb0[j], f2_mul(xe[j], c.ca0[j])), inv2);
    const uint64_t yo = f2_mul(f2_fma(xe[j], c.sb1[j], f2_mul(xo[j], c.ca1[j])), inv2);
    float e0, e1, o0, o1;
    f2_unpack(ye, e0, e1);
    f2_unpack(yo, o0, o1);
    out[2 * j] = pack_f16x2_sat(e0, o0);      // elements 4j, 4j+1, clamped to +-65504 by the conversion
    out[2 * j + 1] = pack_f16x2_sat(e1, o1);  // elements 4j+2, 4j+3
  }
  return make_uint4(out[0], out[1], out[2], out[3]);
}

}  // namespace zdraw
