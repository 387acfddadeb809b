// Classification of the K/V tiles of one image under an additive key mask (internal to the library):
// shared by the prologue launch of the joint call, which carries it as extra blocks, and by the
// stand-alone kernel of the attention-only calls.
#pragma once
#include <cuda_runtime.h>

namespace zdraw {

// Tile-list entries: K/V tile index, plus a flag for tiles the key mask covers partly.
constexpr int kTileMixedFlag = 0x40000000;
constexpr int kTileIndexMask = 0x3FFFFFFF;

constexpr int kMaskThreads = 256;  // threads of the block that classifies one image

// One block of kMaskThreads threads writes list[0] = count, list[1..] = entries in ascending order (so
// the reduction order over keys does not depend on the mask). A tile of 128 keys is left out when every
// one of them is masked (-inf or beyond the sequence), listed plain when all 128 exist and carry mask 0,
// else listed with the mixed flag.
//
// Latency-bound: a warp reads a whole tile as one 16-byte load per lane and the warps take the tiles in
// turn, so 256 tiles cost a few memory latencies. (One tile per block step with two block-wide votes took
// 39 us for the 68 tiles of an 8704-token image; as a block of the prologue launch this adds nothing to it.)
// `mask` is 16-byte aligned (the entry points check pointer and image stride).
__device__ __forceinline__ void classify_mask_tiles(const float* __restrict__ mask, int tokens, int n_kv_tiles,
                                                    int* __restrict__ list) {
  __shared__ int entry[kMaskThreads];            // one chunk of tiles: list entry, or -1
  __shared__ int warp_count[kMaskThreads / 32];
  const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
  constexpr int kWarps = kMaskThreads / 32;
  const float neg_inf = __int_as_float(0xff800000);
  int base = 0;  // entries written by the chunks before
  for (int chunk = 0; chunk < n_kv_tiles; chunk += kMaskThreads) {
    const int n = min(kMaskThreads, n_kv_tiles - chunk);
#pragma unroll 4
    for (int i = warp; i < n; i += kWarps) {
      const int key = (chunk + i) * 128 + 4 * lane;
      float4 v = make_float4(neg_inf, neg_inf, neg_inf, neg_inf);
      if (key + 4 <= tokens) {
        v = __ldg(reinterpret_cast<const float4*>(mask + key));
      } else {  // the ragged end of the sequence
        if (key < tokens) v.x = __ldg(mask + key);
        if (key + 1 < tokens) v.y = __ldg(mask + key + 1);
        if (key + 2 < tokens) v.z = __ldg(mask + key + 2);
      }
      const bool closed = v.x == neg_inf && v.y == neg_inf && v.z == neg_inf && v.w == neg_inf;
      const bool open = v.x == 0.0f && v.y == 0.0f && v.z == 0.0f && v.w == 0.0f;
      const bool all_closed = __all_sync(0xffffffffu, closed), all_open = __all_sync(0xffffffffu, open);
      if (lane == 0) entry[i] = all_closed ? -1 : (all_open ? (chunk + i) : ((chunk + i) | kTileMixedFlag));
    }
    __syncthreads();
    const int mine = static_cast<int>(threadIdx.x) < n ? entry[threadIdx.x] : -1;
    const unsigned live = __ballot_sync(0xffffffffu, mine >= 0);
    if (lane == 0) warp_count[warp] = __popc(live);
    __syncthreads();
    int before = base, total = 0;
    for (int w = 0; w < kWarps; ++w) {
      if (w < warp) before += warp_count[w];
      total += warp_count[w];
    }
    if (mine >= 0) list[1 + before + __popc(live & ((1u << lane) - 1u))] = mine;
    base += total;
    __syncthreads();  // entry and warp_count are reused by the next chunk
  }
  if (threadIdx.x == 0) list[0] = base;
}

}  // namespace zdraw
