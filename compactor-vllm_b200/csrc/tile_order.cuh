// Order of the query tiles of a prefill launch, shared by the tcgen05 prefill kernels (prefill_attn2.cu,
// prefill_attn_bias.cu): one CTA per (query tile, head pair, sequence), each holding its SM.
//
// Two things pull in opposite directions.  A causal tile costs as much as its index, so a launch of few waves ends
// well only if the longest tiles of ALL head pairs and sequences start first; with the pairs outside, each of them
// begins again with its longest tile, the last one included.  But CTAs that run side by side read K and V at about
// the rate that L2 can give, and tiles of one head at adjacent places share those reads.
// So the order by tiles (all pairs and sequences inside) is taken for launches of at most twelve waves of CTAs that have
// work and a short past; the order by pairs otherwise.  Short is, in prefill_attn2.cu, a longest past (the caller's bound) of
// at most three quarters of the longest prompt, and in prefill_attn_bias.cu, whose callers bring no bound, a mean past (over
// sequences, whatever their order; read by every CTA) of at most half of it.
// Measured in turn in one process, by pairs -> by tiles (whatever the rule says of the case), us, 32 / 8 heads of 128 unless
// said:
//   prompts of 1000: 25 -> 25     2048: 56 -> 42     4096: 141 -> 121     8192: 513 -> 465     12000: 1053 -> 999
//   4096 with 16 / 2 heads: 119 -> 83     2 x 2000: 88 -> 79     16 x 500: 92 -> 90     2048 after 1000: 80 -> 68
//   32768 (28 waves): 7210 -> 7170, and 1.8 % slower in a run of its own; 3000 after 8000 tokens with 16 / 4
//   heads, all tiles about equal: 161 -> 190
//   portions with slopes, 4096: 206 -> 177; with a window: 156 -> 148; 2000 + 700 + 3000 after 9000: 1053 -> 1092
//   4000 + 2077 + 911 + 3301: 269 -> 257     one of 4000 among three of 100: 150 -> 140     twelve of 500, the first
//   without a past, the others after 4000: 328 -> 342
//   4000 + 2077 + 911 + 3301 after up to 1440 tokens a head 446 -> 438, 3480 608 -> 630, 7200 943 -> 1031; 4096 after up to
//   3000 255 -> 249, 5400 329 -> 331; 2000 + 700 + 3000 after up to 2400 274 -> 266; 3000 (16 / 4 heads) after 3000 94 -> 93
#pragma once
#include <algorithm>

#include "common.cuh"

namespace cvllm {

// CTAs of a launch that have a tile, at most.  Tiles of shorter sequences that lie past their end cost nothing: those of `tokens` new
// tokens in all are one partial tile per sequence more than whole ones.
inline int64_t ctas_with_work(dim3 grid, int tokens, int tile_rows) {
  const int64_t padded = (int64_t)grid.x * grid.y * grid.z;
  return std::min(padded, ((int64_t)tokens / tile_rows + grid.z) * grid.y);
}

// Launches of one wave start all their tiles at once: no order to choose, and no past to read first.
inline bool order_by_tile(dim3 grid, int tokens, int tile_rows) {
  const int64_t live = ctas_with_work(grid, tokens, tile_rows);
  return live > sm_count() && live <= 12 * (int64_t)sm_count();
}

// A caller without a bound says -1.
inline bool past_is_short(int max_past, int longest) { return max_past >= 0 && 4 * (int64_t)max_past <= 3 * (int64_t)longest; }

struct TileOrder {
  int qt, pair, b;  // query tile (may lie beyond the sequence's tiles), head pair, sequence
};

// Grid (tiles, pairs, sequences) for which order_by_tile() holds; past [n]: tokens before the new ones, of every sequence or
// of every (sequence, head).  If they are short on the mean, the order is by tiles.  Called by whole warps.
__device__ __forceinline__ bool pasts_are_short(const int32_t* past, int n, int tile_rows) {
  // a sum that the compiler knows to be the warp's own: with shuffles, what follows from the order (the sequence, its
  // addresses) is kept per lane, and the whole kernel runs 13 to 17 % slower.  No overflow: n is at most 12 CTAs an SM
  unsigned own = 0;
  for (int i = threadIdx.x & 31; i < n; i += 32) own += (unsigned)min(past[i], 1 << 20);
  const unsigned sum = __reduce_add_sync(0xffffffffu, own);
  return 2 * (long long)sum <= (long long)gridDim.x * tile_rows * n;
}

// This CTA's place in the order by tiles.
__device__ __forceinline__ TileOrder tile_order() {
  const unsigned idx = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  const unsigned h = idx / gridDim.y;
  return {(int)(gridDim.x - 1 - h / gridDim.z), (int)(idx % gridDim.y), (int)(h % gridDim.z)};
}

}  // namespace cvllm
