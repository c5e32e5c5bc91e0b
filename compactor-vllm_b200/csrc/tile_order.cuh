// Order of the query tiles of a prefill launch, shared by the tcgen05 prefill kernels (prefill_attn2.cu,
// prefill_attn_bias.cu): one CTA per (query tile, head pair, sequence), each holding its SM.
//
// Two things pull in opposite directions.  A causal tile costs as much as its index, so a launch of few waves ends
// well only if the longest tiles of ALL head pairs and sequences start first; with the pairs outside, each of them
// begins again with its longest tile, the last one included.  But CTAs that run side by side read K and V at about
// the rate that L2 can give, and tiles of one head at adjacent places share those reads.
// So the order by tiles (all pairs and sequences inside) is taken for launches of up to kOrderCtas CTAs whose first
// sequence has a past of at most half the longest prompt; the order by pairs otherwise.
// Measured in turn in one process, by pairs -> by tiles, us, 32 / 8 heads of 128 unless said:
//   prompts of 1000: 25 -> 25     2048: 56 -> 42     4096: 141 -> 121     8192: 513 -> 465     12000: 1053 -> 999
//   4096 with 16 / 2 heads: 119 -> 83     2 x 2000: 88 -> 79     16 x 500: 92 -> 90     2048 after 1000: 80 -> 68
//   32768 (28 waves): 7210 -> 7170, and 1.8 % slower in a run of its own; 3000 after 8000 tokens with 16 / 4
//   heads, all tiles about equal: 161 -> 190
//   portions with slopes, 4096: 206 -> 177; with a window: 156 -> 148; 2000 + 700 + 3000 after 9000: 1053 -> 1092
#pragma once

namespace cvllm {

// Launches of one wave start all their tiles at once: no order to choose, and no past to read first.
constexpr int64_t kOneWave = 148, kOrderCtas = 12 * kOneWave;

__host__ __device__ __forceinline__ bool order_by_tile(unsigned tiles, unsigned pairs, unsigned seqs) {
  const int64_t ctas = (int64_t)tiles * pairs * seqs;
  return ctas > kOneWave && ctas <= kOrderCtas;
}

struct TileOrder {
  int qt, pair, b;  // query tile (may lie beyond the sequence's tiles), head pair, sequence
};

// Grid (tiles, pairs, sequences) for which order_by_tile() holds; `past`: the first sequence's.
__device__ __forceinline__ TileOrder tile_order(const int32_t* past, int tile_rows) {
  if (2 * (int64_t)*past > (int64_t)gridDim.x * tile_rows)
    return {(int)(gridDim.x - 1 - blockIdx.x), (int)blockIdx.y, (int)blockIdx.z};
  const unsigned idx = (blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
  const unsigned h = idx / gridDim.y;
  return {(int)(gridDim.x - 1 - h / gridDim.z), (int)(idx % gridDim.y), (int)(h % gridDim.z)};
}

}  // namespace cvllm
