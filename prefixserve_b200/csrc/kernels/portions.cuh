// Which of a step's portions, or of the chunks they are cut into, a block works on: a warp looks at 32 requests at a time.
// All lanes of a warp call these together.
#pragma once
#include "common.cuh"

namespace portions {

__device__ __forceinline__ int sums_upto(int mine, int lane) {  // of the lanes up to this one
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, mine, off);
    if (lane >= off) mine += v;
  }
  return mine;
}

// Chunk ``at`` of the portions of at least ``min_tokens`` (1 or more) tokens, in order: its first token and how many it has.
template <int CHUNK>
__device__ __forceinline__ bool find_chunk(const int32_t* __restrict__ item_start, int items, int min_tokens, int at, int& t0, int& n) {
  const int lane = threadIdx.x & 31;
  for (int i0 = 0; i0 < items; i0 += 32) {
    const int i = i0 + lane, a = i < items ? item_start[i] : 0, len = i < items ? item_start[i + 1] - a : 0;
    const int mine = len >= min_tokens ? (len + CHUNK - 1) / CHUNK : 0, upto = sums_upto(mine, lane);
    const unsigned behind = __ballot_sync(0xffffffffu, at < upto);
    if (behind) {
      const int who = __ffs(behind) - 1, in = at - __shfl_sync(0xffffffffu, upto - mine, who);
      t0 = __shfl_sync(0xffffffffu, a, who) + in * CHUNK;
      n = min(CHUNK, __shfl_sync(0xffffffffu, len, who) - in * CHUNK);
      return true;
    }
    at -= __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

// Portion ``nth`` of those: its request, and how many chunks lie before its first.
template <int CHUNK>
__device__ __forceinline__ bool find_portion(const int32_t* __restrict__ item_start, int items, int min_tokens, int nth, int& item, int& chunks_before) {
  const int lane = threadIdx.x & 31;
  chunks_before = 0;
  for (int i0 = 0; i0 < items; i0 += 32) {
    const int i = i0 + lane, len = i < items ? item_start[i + 1] - item_start[i] : 0;
    const bool counts = len >= min_tokens;
    const int mine = counts ? (len + CHUNK - 1) / CHUNK : 0, upto = sums_upto(mine, lane), rank = sums_upto(counts ? 1 : 0, lane);
    const unsigned behind = __ballot_sync(0xffffffffu, nth < rank);
    if (behind) {
      const int who = __ffs(behind) - 1;
      item = i0 + who;
      chunks_before += __shfl_sync(0xffffffffu, upto - mine, who);
      return true;
    }
    nth -= __shfl_sync(0xffffffffu, rank, 31);
    chunks_before += __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

}  // namespace portions
