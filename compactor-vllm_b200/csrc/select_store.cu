// Fused top-k eviction + paged-cache compaction, multi-CTA.
//
// Reference: compression/common.py:126-168 (scores -> torch.topk full sort -> K4 atomic-slot store
// -> K5 serial pad walk, kv_cache/store_kv_cache.py:9-248).  The closed form:
// after the per-sequence global top-`retain`, head h holds c_h pairs; it is padded to
// n_h = min(c_h + pad, len) and its kept set is exactly the top-n_h tokens OF THAT HEAD.  So:
//
//   phase 1  4 radix passes (8 bits each) over all len*H keys of a sequence  -> threshold T, ties
//   phase 2  count per head: keys > T, ties at T taken in ascending flat index  -> c_h -> n_h
//   phase 3  4 radix passes per (sequence, head)                              -> T_h, ties_h
//   phase 4  per tile / head: #keys > T_h and #keys == T_h
//   phase 5  ordered compaction: rank inside the head = (kept before this tile) + (kept before
//            this token inside the tile); rows copied straight into the paged cache
//
// Every phase is a grid of (token tiles x sequences) CTAs: the keys of a 32K-token sequence are
// 1 MB and live in L2, each pass is a few microseconds instead of a single-SM walk.  The CTA that
// takes the last ticket of a sequence folds the global histogram into the next digit.
// Phases 1 to 4 are ONE kernel (sel_cluster_kernel) where the keys of the longest sequence fit the shared memory of a cluster
// of up to eight CTAs (160 tiles at 8 heads: 40960 tokens, 327680 keys): twelve short launches of 4 to 12 us each, one
// waiting for the other, were three quarters of an eviction.  Calls with a longer sequence take the launches.
// Order everywhere: key descending, ties by ascending flat index tok*H + head, NaN above +inf.
// Rows land in ascending token order per head (the reference's order is atomic-nondeterministic).
#include <cooperative_groups.h>

#include "common.cuh"
#include "select_common.cuh"

namespace cvllm {

constexpr int kTileTok = 256;   // tokens per tile (one thread per token in phase 5)
constexpr int kPassThreads = 256;
constexpr int kMaxH = 16;

struct SegState {
  uint32_t prefix;     // decided high digits of the threshold key
  uint32_t remaining;  // rank still to resolve inside the prefix bucket (after 4 passes: ties)
  uint32_t active;     // 0: nothing is selected in this segment
  uint32_t pad_;
};

struct SelWs {
  uint32_t* hist_g;    // [B][256]
  uint32_t* hist_h;    // [B][H][256]
  uint32_t* ticket;    // [B][2]
  uint32_t* gt_h;      // [B][H]   keys > T per head
  SegState* state_g;   // [B]
  SegState* state_h;   // [B][H]
  int32_t* n_keep;     // [B][H]
  int32_t* len0;       // [B][H]   bh_lens before this call
  uint32_t* tile_tie;  // [B][tiles][H]
  uint2* tile_cnt;     // [B][tiles][H]  (gt, tie) w.r.t. T_h
  int tiles;           // tile slots per sequence
};

// ---------------------------------------------------------------------------
// init: k per sequence, copy of the starting lengths
// ---------------------------------------------------------------------------
__global__ void sel_init_kernel(const int32_t* __restrict__ cu, const int32_t* __restrict__ num_retain,
                                const int32_t* __restrict__ batch_mapping,
                                const int32_t* __restrict__ bh_lens, int B, int H, int reserved_batch,
                                SelWs w) {
  pdl_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < B) {
    const int cnt = (cu[i + 1] - cu[i]) * H;
    const int k = max(0, min(num_retain[i], cnt));
    SegState s;
    s.prefix = 0;
    s.remaining = (uint32_t)k;
    s.active = (batch_mapping[i] != reserved_batch && k > 0) ? 1u : 0u;
    s.pad_ = 0;
    w.state_g[i] = s;
  }
  if (i < B * H) w.len0[i] = bh_lens[i];
}

// digit pick: 256-bin histogram (descending) -> digit holding the `remaining`-th entry.
// Executed by one full warp; returns through lane-uniform refs.  bin(i): count of digit i.
// `held`: how many entries that digit holds.
template <typename Bin>
__device__ __forceinline__ void pick_digit(Bin bin, uint32_t remaining, uint32_t& digit, uint32_t& new_remaining,
                                           uint32_t& held) {
  const int lane = threadIdx.x & 31;
  uint32_t h8[8];
  uint32_t own = 0;
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    h8[t] = bin(255 - 8 * lane - t);
    own += h8[t];
  }
  uint32_t incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  const uint32_t above = incl - own;
  const bool mine = (above < remaining) && (remaining <= incl);
  uint32_t d = 0, rem = 0, n = 0;
  if (mine) {
    uint32_t acc = above;
    int t = 0;
    for (; t < 8; ++t) {
      if (remaining <= acc + h8[t]) break;
      acc += h8[t];
    }
    d = (uint32_t)(255 - 8 * lane - t);
    rem = remaining - acc;
#pragma unroll
    for (int u = 0; u < 8; ++u) n = u == t ? h8[u] : n;
  }
  const uint32_t who = __ballot_sync(0xffffffffu, mine);
  const int src = who ? (__ffs(who) - 1) : 0;
  digit = __shfl_sync(0xffffffffu, d, src);
  new_remaining = __shfl_sync(0xffffffffu, rem, src);
  held = __shfl_sync(0xffffffffu, n, src);
}

// ---------------------------------------------------------------------------
// one radix pass.  PER_HEAD == false: segment = sequence; true: segment = (sequence, head)
// grid (tiles, B)
// ---------------------------------------------------------------------------
template <bool PER_HEAD>
__global__ void __launch_bounds__(kPassThreads) sel_pass_kernel(const float* __restrict__ scores,
                                                                int64_t stride_n,
                                                                const int32_t* __restrict__ cu, int H,
                                                                int pass, SelWs w) {
  pdl_begin();
  __shared__ uint32_t s_hist[PER_HEAD ? kMaxH * 256 : 256];
  __shared__ uint32_t s_prefix[kMaxH];
  __shared__ uint32_t s_active[kMaxH];
  __shared__ int s_last;
  const int b = blockIdx.y, tile = blockIdx.x;
  const int beg = cu[b], len = cu[b + 1] - beg;
  const int tiles_b = cdiv(len, kTileTok);
  if (tile >= tiles_b) return;
  const int nseg = PER_HEAD ? H : 1;
  SegState* st = PER_HEAD ? (w.state_h + (int64_t)b * H) : (w.state_g + b);
  uint32_t* hist = PER_HEAD ? (w.hist_h + (int64_t)b * H * 256) : (w.hist_g + (int64_t)b * 256);
  const int tid = threadIdx.x;
  if (tid < nseg) {
    s_prefix[tid] = st[tid].prefix;
    s_active[tid] = st[tid].active;
  }
  for (int i = tid; i < nseg * 256; i += kPassThreads) s_hist[i] = 0;
  __syncthreads();
  bool any_active = false;
  for (int s = 0; s < nseg; ++s) any_active |= (s_active[s] != 0);
  if (!any_active) return;  // uniform over the sequence's CTAs: no ticket needed

  const int shift = 24 - 8 * pass;
  const uint32_t mask = pass == 0 ? 0u : (0xffffffffu << (32 - 8 * pass));
  const int t0 = tile * kTileTok;
  const int nk = min(kTileTok, len - t0) * H;
  const float* src = scores + (int64_t)(beg + t0) * stride_n;
  for (int i = tid; i < nk; i += kPassThreads) {
    const int tok = i / H, h = i - tok * H;
    const int seg = PER_HEAD ? h : 0;
    if (!s_active[seg]) continue;
    const uint32_t key = score_key(__float_as_uint(__ldg(src + (int64_t)tok * stride_n + h)));
    if ((key & mask) == s_prefix[seg]) atomicAdd(&s_hist[seg * 256 + ((key >> shift) & 255u)], 1u);
  }
  __syncthreads();
  for (int i = tid; i < nseg * 256; i += kPassThreads) {
    const uint32_t c = s_hist[i];
    if (c) atomicAdd(hist + i, c);
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const uint32_t t = atomicAdd(w.ticket + 2 * b + (PER_HEAD ? 1 : 0), 1u);
    s_last = (t == (uint32_t)(tiles_b - 1));
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // last CTA of the sequence: fold the histogram(s) into the next digit
  const int warp = tid >> 5, lane = tid & 31;
  for (int s = warp; s < nseg; s += kPassThreads / 32) {
    if (s_active[s]) {
      uint32_t digit, rem, held;
      pick_digit([&](int i) { return __ldcg(hist + s * 256 + i); }, st[s].remaining, digit, rem, held);
      if (lane == 0) {
        st[s].prefix = s_prefix[s] | (digit << shift);
        st[s].remaining = rem;
      }
    }
    __syncwarp();
    for (int i = lane; i < 256; i += 32) hist[s * 256 + i] = 0;
  }
  if (tid == 0) w.ticket[2 * b + (PER_HEAD ? 1 : 0)] = 0;
}

// ---------------------------------------------------------------------------
// phase 2a: per tile, per head: keys > T (-> global per-head counters), ties at T (-> per tile)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kPassThreads) sel_count_global_kernel(const float* __restrict__ scores,
                                                                        int64_t stride_n,
                                                                        const int32_t* __restrict__ cu,
                                                                        int H, SelWs w) {
  pdl_begin();
  __shared__ uint32_t s_gt[kMaxH], s_tie[kMaxH];
  const int b = blockIdx.y, tile = blockIdx.x;
  const int beg = cu[b], len = cu[b + 1] - beg;
  if (tile >= cdiv(len, kTileTok)) return;
  const SegState sg = w.state_g[b];
  const int tid = threadIdx.x;
  if (tid < H) s_gt[tid] = s_tie[tid] = 0;
  __syncthreads();
  if (sg.active) {
    const int t0 = tile * kTileTok;
    const int nk = min(kTileTok, len - t0) * H;
    const float* src = scores + (int64_t)(beg + t0) * stride_n;
    for (int i = tid; i < nk; i += kPassThreads) {
      const int tok = i / H, h = i - tok * H;
      const uint32_t key = score_key(__float_as_uint(__ldg(src + (int64_t)tok * stride_n + h)));
      if (key > sg.prefix) atomicAdd(&s_gt[h], 1u);
      else if (key == sg.prefix) atomicAdd(&s_tie[h], 1u);
    }
  }
  __syncthreads();
  if (tid < H) {
    if (s_gt[tid]) atomicAdd(w.gt_h + b * H + tid, s_gt[tid]);
    w.tile_tie[((int64_t)b * w.tiles + tile) * H + tid] = s_tie[tid];
  }
}

// ---------------------------------------------------------------------------
// phase 2b: one CTA per sequence: allocate the ties in flat-index order, c_h -> n_h, seed phase 3
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kPassThreads) sel_resolve_kernel(const float* __restrict__ scores,
                                                                   int64_t stride_n,
                                                                   const int32_t* __restrict__ cu,
                                                                   const int32_t* __restrict__ batch_mapping,
                                                                   int H, int PS, int pad_to_page,
                                                                   int reserved_batch, SelWs w) {
  pdl_begin();
  __shared__ uint32_t s_tiesel[kMaxH];
  __shared__ int s_warp[32];
  __shared__ int s_btile;
  __shared__ uint32_t s_before;
  const int b = blockIdx.x, tid = threadIdx.x;
  const int beg = cu[b], len = cu[b + 1] - beg;
  const int tiles_b = cdiv(len, kTileTok);
  const SegState sg = w.state_g[b];
  const uint32_t* tt = w.tile_tie + (int64_t)b * w.tiles * H;
  if (tid < H) s_tiesel[tid] = 0;
  if (tid == 0) { s_btile = -1; s_before = 0; }
  __syncthreads();
  if (sg.active) {
    // boundary tile: the first one whose cumulative tie count (flat order) exceeds `remaining`
    {
      const int lane = tid & 31, warp = tid >> 5;
      uint32_t carry = 0;
      if (tid == 0) s_btile = tiles_b;  // default: every tie is taken
      __syncthreads();
      for (int base = 0; base < tiles_b; base += kPassThreads) {
        const int t = base + tid;
        uint32_t c = 0;
        if (t < tiles_b)
          for (int h = 0; h < H; ++h) c += tt[t * H + h];
        // block-wide exclusive prefix of c
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t x = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += x;
        }
        if (lane == 31) s_warp[warp] = (int)incl;
        __syncthreads();
        uint32_t wbase = 0, total = 0;
        for (int wv = 0; wv < kPassThreads / 32; ++wv) {
          if (wv < warp) wbase += (uint32_t)s_warp[wv];
          total += (uint32_t)s_warp[wv];
        }
        const uint32_t run = carry + wbase + incl - c;
        if (t < tiles_b && run <= sg.remaining && run + c > sg.remaining) {
          s_btile = t;  // unique: the prefix is monotone
          s_before = run;
        }
        carry += total;
        __syncthreads();
      }
      if (tid == 0 && s_btile == tiles_b) s_before = carry;
      __syncthreads();
    }
    const int bt = s_btile;
    // whole tiles before the boundary: all their ties are taken
    for (int i = tid; i < min(bt, tiles_b) * H; i += kPassThreads) {
      const uint32_t c = tt[i];
      if (c) atomicAdd(&s_tiesel[i % H], c);
    }
    __syncthreads();
    if (bt < tiles_b) {
      // ordered pass inside the boundary tile (flat order = token major, head minor)
      const int need = (int)(sg.remaining - s_before);
      const int t0 = bt * kTileTok;
      const int nk = min(kTileTok, len - t0) * H;
      const float* src = scores + (int64_t)(beg + t0) * stride_n;
      int seen = 0;
      for (int base = 0; base < nk && seen < need; base += kPassThreads) {
        const int i = base + tid;
        bool tie = false;
        int h = 0;
        if (i < nk) {
          const int tok = i / H;
          h = i - tok * H;
          tie = score_key(__float_as_uint(__ldg(src + (int64_t)tok * stride_n + h))) == sg.prefix;
        }
        int tot;
        const int rank = seen + block_excl_count(tie, s_warp, tot);
        if (tie && rank < need) atomicAdd(&s_tiesel[h], 1u);
        seen += tot;
      }
      __syncthreads();
    }
  }
  if (tid < H) {
    const int h = tid;
    int n = 0;
    if (sg.active) {
      const int c = (int)(w.gt_h[b * H + h] + s_tiesel[h]);
      n = c;
      if (pad_to_page) n += pad_amount(w.len0[b * H + h] + c, len, PS);
      n = min(n, len);
    }
    w.n_keep[b * H + h] = n;
    SegState s;
    s.prefix = 0;
    s.remaining = (uint32_t)n;
    s.active = (n > 0 && batch_mapping[b] != reserved_batch) ? 1u : 0u;
    s.pad_ = 0;
    w.state_h[b * H + h] = s;
    w.gt_h[b * H + h] = 0;  // leave the workspace clean for the next call on this stream
  }
}

// ---------------------------------------------------------------------------
// phase 4: per tile / head: (#keys > T_h, #keys == T_h)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kPassThreads) sel_count_heads_kernel(const float* __restrict__ scores,
                                                                       int64_t stride_n,
                                                                       const int32_t* __restrict__ cu,
                                                                       int H, SelWs w) {
  pdl_begin();
  __shared__ uint32_t s_gt[kMaxH], s_tie[kMaxH], s_thr[kMaxH], s_act[kMaxH];
  const int b = blockIdx.y, tile = blockIdx.x;
  const int beg = cu[b], len = cu[b + 1] - beg;
  if (tile >= cdiv(len, kTileTok)) return;
  const int tid = threadIdx.x;
  if (tid < H) {
    s_gt[tid] = s_tie[tid] = 0;
    s_thr[tid] = w.state_h[b * H + tid].prefix;
    s_act[tid] = w.state_h[b * H + tid].active;
  }
  __syncthreads();
  const int t0 = tile * kTileTok;
  const int nk = min(kTileTok, len - t0) * H;
  const float* src = scores + (int64_t)(beg + t0) * stride_n;
  for (int i = tid; i < nk; i += kPassThreads) {
    const int tok = i / H, h = i - tok * H;
    if (!s_act[h]) continue;
    const uint32_t key = score_key(__float_as_uint(__ldg(src + (int64_t)tok * stride_n + h)));
    if (key > s_thr[h]) atomicAdd(&s_gt[h], 1u);
    else if (key == s_thr[h]) atomicAdd(&s_tie[h], 1u);
  }
  __syncthreads();
  if (tid < H) w.tile_cnt[((int64_t)b * w.tiles + tile) * H + tid] = make_uint2(s_gt[tid], s_tie[tid]);
}

// ---------------------------------------------------------------------------
// Phases 1 to 4 in one launch: a cluster of CS CTAs per sequence, each with a run of whole tiles whose keys stay in its shared
// memory.  A pass counts digits in its own histogram (256 x 32 words: a column per head and neighbouring token, so that the
// lanes of a warp never meet in a word or a bank), the cluster's CTAs add up each other's sums through distributed shared
// memory, each for itself, behind one cluster barrier (two buffers: whoever writes a buffer again has passed a barrier that
// all readers have reached).  The first digit of the per-head passes is counted together with the first of the whole
// sequence.  A pass is the last one when its digit's entries are all taken: the low bits then make no difference (keys from
// the prefix up are kept, "ties" with it all).  Bound by latency: up to seven rounds of a pass over the CTA's keys and an
// exchange, 5 to 8 k cycles a round.  Whole evictions in a graph, chain of launches / one launch: 700 tokens of 8 heads
// 83 / 41 us, 5000 87 / 46 us, 32768 99 / 72 us (half of it the copy), six of 6000 148 / 103 us.
// ---------------------------------------------------------------------------
constexpr int kClThreads = 1024;

inline size_t sel_cluster_smem(int tiles_per_cta, int H) {
  return sizeof(uint32_t) * ((size_t)tiles_per_cta * kTileTok * H + 256 * 32 + 2 * 256 + 4 * (size_t)H * 256);
}

__global__ void __launch_bounds__(kClThreads) sel_cluster_kernel(
    const float* __restrict__ scores, int64_t stride_n, const int32_t* __restrict__ cu, const int32_t* __restrict__ num_retain,
    const int32_t* __restrict__ batch_mapping, const int32_t* __restrict__ bh_lens, int H, int PS, int pad_to_page,
    int reserved_batch, int keys_cap, SelWs w) {
  namespace cg = cooperative_groups;
  extern __shared__ uint32_t sm[];
  uint32_t* keys = sm;                    // [keys_cap] token major, head minor
  uint32_t* col = keys + keys_cap;        // [256][32] the pass's counts, zero between passes
  uint32_t* g = col + 256 * 32;           // [2][256] this CTA's counts over all heads
  uint32_t* hh = g + 2 * 256;             // [3][H][256] ... per head: first digit | two buffers
  uint32_t* tot = hh + 3 * H * 256;       // [H][256] the cluster's sums
  __shared__ uint32_t s_gt[kMaxH], s_tie[kMaxH], s_sel[kMaxH];
  __shared__ uint32_t s_prefix[kMaxH], s_remaining[kMaxH], s_active[kMaxH], s_open[kMaxH];
  __shared__ uint32_t s_all_gt[kMaxH], s_all_tie[kMaxH], s_all_sel[kMaxH], s_before;
  __shared__ uint32_t s_pick[3];   // digit, remaining, whether its entries are all taken
  __shared__ int s_warp[32];
  cg::cluster_group cl = cg::this_cluster();
  const int CS = (int)cl.num_blocks(), rank = (int)cl.block_rank();
  const int b = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int beg = cu[b], len = cu[b + 1] - beg;
  const uint32_t k = (uint32_t)max(0, min(num_retain[b], len * H));
  const bool active = batch_mapping[b] != reserved_batch && k > 0;
  if (rank == 0 && tid < H) w.len0[b * H + tid] = bh_lens[b * H + tid];
  if (!active) {   // the same for every CTA of the cluster
    if (rank == 0 && tid < H) w.state_h[b * H + tid] = SegState{0, 0, 0, 0};
    return;
  }
  const int tiles_b = cdiv(len, kTileTok), tpc = cdiv(tiles_b, CS);
  const int tile0 = min(rank * tpc, tiles_b), tile1 = min(tile0 + tpc, tiles_b);
  const int tok0 = tile0 * kTileTok, ntok = max(0, min(len, tile1 * kTileTok) - tok0), nkeys = ntok * H;
  // keys in shared memory: whole tiles, all of them unless the sequence is longer than the caller's bound; the others are
  // read again from `scores` in every pass
  const int held = min(nkeys, keys_cap);
  // a thread keeps to one head: it takes every (stride / H)-th token
  const int stride = kClThreads / H * H, my_h = tid % H, my_tok = tid / H;
  const bool on = tid < stride;
  int lg = 5;   // columns per head (log2)
  while (lg > 0 && (H << lg) > 32) --lg;
  const int copies = 1 << lg, col_head = lane >> lg;
  const bool col_first = (lane & (copies - 1)) == 0 && col_head < H;
  // sum over the cluster of word i of a shared array: all loads in flight together (a cluster has at most eight CTAs)
  auto cluster_sum = [&](uint32_t* array, int i) {
    uint32_t v[8], t = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = r < CS ? cl.map_shared_rank(array, r)[i] : 0;
#pragma unroll
    for (int r = 0; r < 8; ++r) t += v[r];
    return t;
  };
  const int my_col = my_h * copies + (my_tok & (copies - 1));
  if (on) {
    const float* src = scores + (int64_t)(beg + tok0 + my_tok) * stride_n + my_h;
    const int64_t step = (int64_t)(stride / H) * stride_n;
#pragma unroll 4
    for (int i = tid; i < held; i += stride, src += step) keys[i] = score_key(__float_as_uint(__ldg(src)));
  }
  auto far_key = [&](int i) {
    return score_key(__float_as_uint(__ldg(scores + (int64_t)(beg + tok0 + i / H) * stride_n + i % H)));
  };
  auto each_key = [&](auto use) {   // all keys of this thread
    int i = tid;
#pragma unroll 4
    for (; i < held; i += stride) use(keys[i]);
    if (nkeys > held)
#pragma unroll 1
      for (; i < nkeys; i += stride) use(far_key(i));
  };
  for (int i = tid; i < 256 * 32; i += kClThreads) col[i] = 0;
  __syncthreads();
  // counts of digit `shift` of the keys that match (prefix, mask); pre: this thread's head's prefix
  auto count = [&](uint32_t pre, uint32_t mask, int shift, bool want) {
    if (on && want)
      each_key([&](uint32_t key) {
        if ((key & mask) == pre) atomicAdd(&col[((key >> shift) & 255u) * 32 + my_col], 1u);
      });
    __syncthreads();
  };
  // columns -> per-head counts (dst) and, where asked, counts over all heads (all); the columns are zero afterwards
  auto collect = [&](uint32_t* dst, uint32_t* all) {
    constexpr int ROWS = 256 / (kClThreads / 32);
    uint32_t v[ROWS];
    uint32_t* mine = col + warp * ROWS * 32 + lane;
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
      v[r] = mine[r * 32];
      mine[r * 32] = 0;
    }
    if (all) {
#pragma unroll
      for (int r = 0; r < ROWS; ++r) {
        const uint32_t t = __reduce_add_sync(0xffffffffu, v[r]);
        if (lane == 0) all[warp * ROWS + r] = t;
      }
    }
    if (dst) {
      for (int o = 1; o < copies; o <<= 1) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) v[r] += __shfl_xor_sync(0xffffffffu, v[r], o);
      }
      if (col_first) {
#pragma unroll
        for (int r = 0; r < ROWS; ++r) dst[col_head * 256 + warp * ROWS + r] = v[r];
      }
    }
  };
  // ---- phase 1: the sequence's threshold ----
  uint32_t prefix = 0, remaining = k;
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    count(prefix, pass == 0 ? 0u : 0xffffffffu << (32 - 8 * pass), shift, true);
    uint32_t* mine = g + (pass & 1) * 256;
    collect(pass == 0 ? hh : nullptr, mine);
    cl.sync();
    if (tid < 256) tot[tid] = cluster_sum(mine, tid);
    __syncthreads();
    if (warp == 0) {
      uint32_t digit, rem, held;
      pick_digit([&](int i) { return tot[i]; }, remaining, digit, rem, held);
      if (lane == 0) s_pick[0] = digit, s_pick[1] = rem, s_pick[2] = held == rem;
    }
    __syncthreads();
    prefix |= s_pick[0] << shift;
    remaining = s_pick[1];
    if (s_pick[2]) {   // (the same in every CTA)
      remaining = 0xffffffffu;
      break;
    }
  }
  // ---- phase 2: keys above it per head, ties in flat order ----
  if (tid < H) s_gt[tid] = s_tie[tid] = s_sel[tid] = 0;
  __syncthreads();
  {
    uint32_t gt = 0, tie = 0;
    if (on)
      each_key([&](uint32_t key) {
        gt += key > prefix;
        tie += key == prefix;
      });
    if (gt) atomicAdd(&s_gt[my_h], gt);
    if (tie) atomicAdd(&s_tie[my_h], tie);
  }
  cl.sync();
  if (tid < H) {
    s_all_gt[tid] = cluster_sum(s_gt, tid);
    s_all_tie[tid] = cluster_sum(s_tie, tid);
  }
  if (warp == 1) {   // ties of the CTAs before this one
    uint32_t t = 0;
    for (int i = lane; i < rank * H; i += 32) t += cl.map_shared_rank(s_tie, i / H)[i % H];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) s_before = t;
  }
  __syncthreads();
  uint32_t ties = 0, own_ties = 0;
  for (int h = 0; h < H; ++h) {
    ties += s_all_tie[h];
    own_ties += s_tie[h];
  }
  if (remaining < ties) {   // (the same in every CTA) some are left out: the first `remaining` in flat order are taken
    const uint32_t before = s_before;
    if (before + own_ties <= remaining) {
      if (tid < H) s_sel[tid] = s_tie[tid];
    } else if (before < remaining) {
      const uint32_t need = remaining - before;
      uint32_t seen = 0;
      for (int base = 0; base < nkeys && seen < need; base += kClThreads) {
        const int i = base + tid;
        const bool tie = i < nkeys && (i < held ? keys[i] : far_key(i)) == prefix;
        int tot;
        const uint32_t at = seen + block_excl_count(tie, s_warp, tot);
        if (tie && at < need) atomicAdd(&s_sel[i % H], 1u);
        seen += tot;
      }
    }
    cl.sync();
    if (tid < H) s_all_sel[tid] = cluster_sum(s_sel, tid);
  } else if (tid < H) {
    s_all_sel[tid] = s_all_tie[tid];
  }
  if (tid < H) {
    const int c = (int)(s_all_gt[tid] + s_all_sel[tid]);
    int n = c;
    if (pad_to_page) n += pad_amount(bh_lens[b * H + tid] + c, len, PS);
    n = min(n, len);
    s_prefix[tid] = 0;
    s_remaining[tid] = (uint32_t)n;
    s_active[tid] = s_open[tid] = n > 0;
  }
  cl.sync();   // from here on the heads' states are written by the CTAs that own the heads
  // ---- phase 3: every head's own threshold ----
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    uint32_t* mine = hh;
    if (pass > 0) {
      mine = hh + (1 + (pass & 1)) * H * 256;
      count(s_prefix[my_h], 0xffffffffu << (32 - 8 * pass), shift, s_open[my_h] != 0);
      collect(mine, nullptr);
      cl.sync();
    }
    // head h belongs to CTA h mod CS: each sums and picks its heads' digits and tells all (every CTA summing every head's
    // bins moved 64 KB into each CTA, 6 k cycles a pass)
    for (int i = tid; i < (H - rank + CS - 1) / CS * 256; i += kClThreads) {
      const int at = (rank + (i >> 8) * CS) * 256 + (i & 255);
      tot[at] = cluster_sum(mine, at);
    }
    __syncthreads();
    const int head = rank + warp * CS;
    if (head < H && s_open[head]) {
      uint32_t digit, rem, held;
      pick_digit([&](int i) { return tot[head * 256 + i]; }, s_remaining[head], digit, rem, held);
      const uint32_t pre = s_prefix[head] | (digit << shift);
      __syncwarp();
      if (lane < CS) {
        cl.map_shared_rank(s_prefix, lane)[head] = pre;
        cl.map_shared_rank(s_remaining, lane)[head] = held == rem ? 0xffffffffu : rem;
        cl.map_shared_rank(s_open, lane)[head] = held != rem;
      }
    }
    cl.sync();
    bool open = false;
    for (int h = 0; h < H; ++h) open |= s_open[h] != 0;
    if (!open) break;   // (the same in every CTA)
  }
  if (rank == 0 && tid < H)
    w.state_h[b * H + tid] = SegState{s_prefix[tid], s_remaining[tid], s_active[tid], 0};
  pdl_trigger();   // late: the copy's CTAs wait on the SMs that the clusters leave free, and keep others from them
  // ---- phase 4: per tile / head: (#keys > T_h, #keys == T_h), a warp per tile ----
  const int subs = 32 / H;
  for (int t = tile0 + warp; t < tile1; t += kClThreads / 32) {
    const int h = lane % H, sub = lane / H;
    uint32_t gt = 0, tie = 0;
    if (sub < subs) {
      const uint32_t thr = s_prefix[h];
      const int first = (t - tile0) * kTileTok * H + h, n = min(kTileTok, len - t * kTileTok);
      if (first < held) {   // whole tiles are held
        for (int i = sub; i < n; i += subs) {
          const uint32_t key = keys[first + i * H];
          gt += key > thr;
          tie += key == thr;
        }
      } else {
#pragma unroll 1
        for (int i = sub; i < n; i += subs) {
          const uint32_t key = far_key(first + i * H);
          gt += key > thr;
          tie += key == thr;
        }
      }
    }
    uint32_t gs = gt, ts = tie;   // lanes h, h + H, ..: the tile's counts of head h
    for (int j = 1; j < subs; ++j) {
      gs += __shfl_down_sync(0xffffffffu, gt, j * H);
      ts += __shfl_down_sync(0xffffffffu, tie, j * H);
    }
    if (lane < H) w.tile_cnt[((int64_t)b * w.tiles + t) * H + lane] = make_uint2(gs, ts);
  }
  cl.sync();   // nobody leaves while its counts may still be read
}

// ---------------------------------------------------------------------------
// phase 5: ordered compaction + row copy.  One thread per token of the tile; gridDim.z CTAs share a tile's kept rows, each
// finding all of them.  Bound by the copy (the rows' bytes twice) and by what precedes it: scores, counts and thresholds are
// loaded together, the kept rows become a list in the order of their places (head, rank), which all lanes copy from - a lane per
// row of the tile had nothing to do for the dropped ones - and a row's page is looked up beside its load.  Tokens 9000, 3500, 12000,
// 511 of 8 heads, half kept (102 MB): 30.3 -> 22.1 us (cold, ncu).
// ---------------------------------------------------------------------------
template <int VEC_PER_ROW>
__global__ void __launch_bounds__(kTileTok, 4) sel_gather_kernel(
    const float* __restrict__ scores, int64_t stride_n, const uint4* __restrict__ keys,
    const uint4* __restrict__ vals, int64_t sk_n, int64_t sk_h, int64_t sv_n, int64_t sv_h,
    const int32_t* __restrict__ cu, const int32_t* __restrict__ batch_mapping,
    const int32_t* __restrict__ page_table, int32_t* __restrict__ bh_lens, uint4* __restrict__ k_cache,
    uint4* __restrict__ v_cache, int H, int PS, int NLP, SelWs w) {
  pdl_begin();
  constexpr int kWarps = kTileTok / 32;
  __shared__ uint32_t s_gt_before[kMaxH], s_tie_before[kMaxH], s_gt_all[kMaxH], s_tie_all[kMaxH];
  __shared__ uint32_t s_thr[kMaxH], s_ties[kMaxH], s_act[kMaxH];
  __shared__ uint32_t s_wsel[kMaxH][kWarps], s_wtie[kMaxH][kWarps];
  __shared__ int32_t s_place[kMaxH], s_first[kMaxH + 1];     // cache position and list index of a head's first kept row
  __shared__ int32_t s_pos[kTileTok * kMaxH];                // list: position in the head's cache
  __shared__ uint16_t s_src[kTileTok * kMaxH];               // and token of the tile * H + head
  const int b = blockIdx.y, tile = blockIdx.x;
  const int beg = cu[b], len = cu[b + 1] - beg;
  const int tiles_b = cdiv(len, kTileTok);
  if (tile >= tiles_b) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tok = tile * kTileTok + tid;
  const bool valid = tok < len;
  const float* srow = scores + (int64_t)(beg + tok) * stride_n;
  float sc[kMaxH];
#pragma unroll
  for (int h = 0; h < kMaxH; ++h) sc[h] = valid && h < H ? __ldg(srow + h) : 0.f;
  const int32_t* pt = page_table + (int64_t)batch_mapping[b] * H * NLP;
  SegState st = {};
  int len0 = 0;
  if (tid < H) {
    st = w.state_h[b * H + tid];
    len0 = w.len0[b * H + tid];
    s_gt_before[tid] = s_tie_before[tid] = s_gt_all[tid] = s_tie_all[tid] = 0;
  }
  __syncthreads();
  // prefix of the per-tile counts over the tiles before this one (and totals, for bh_lens); those of a sequence that keeps
  // nothing are not written, and not used
  {
    const uint2* tc = w.tile_cnt + (int64_t)b * w.tiles * H;
    for (int i = tid; i < (tile == 0 ? tiles_b : tile) * H; i += kTileTok) {
      const int t = i / H, h = i - t * H;
      const uint2 c = tc[i];
      if (t < tile) {
        if (c.x) atomicAdd(&s_gt_before[h], c.x);
        if (c.y) atomicAdd(&s_tie_before[h], c.y);
      }
      if (tile == 0) {
        if (c.x) atomicAdd(&s_gt_all[h], c.x);
        if (c.y) atomicAdd(&s_tie_all[h], c.y);
      }
    }
  }
  if (tid < H) {
    s_thr[tid] = st.prefix;
    s_ties[tid] = st.remaining;
    s_act[tid] = st.active;
  }
  __syncthreads();
  // per-head flags of this token
  uint32_t gt_mask = 0, tie_mask = 0;
#pragma unroll
  for (int h = 0; h < kMaxH; ++h) {
    if (h < H && valid && s_act[h]) {
      const uint32_t key = score_key(__float_as_uint(sc[h]));
      if (key > s_thr[h]) gt_mask |= 1u << h;
      else if (key == s_thr[h]) tie_mask |= 1u << h;
    }
  }
  // ties first (their rank decides whether they are kept)
  const uint32_t lt_mask = (1u << lane) - 1u;
  uint32_t sel_mask = gt_mask;
  if (__syncthreads_or(tie_mask != 0)) {
    uint32_t tie_lane[kMaxH];
#pragma unroll
    for (int h = 0; h < kMaxH; ++h) {
      if (h < H) {
        const uint32_t m = __ballot_sync(0xffffffffu, (tie_mask >> h) & 1u);
        tie_lane[h] = __popc(m & lt_mask);
        if (lane == 0) s_wtie[h][warp] = __popc(m);
      }
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < kMaxH; ++h) {
      if (h < H && ((tie_mask >> h) & 1u)) {
        uint32_t before = s_tie_before[h] + tie_lane[h];
        for (int wv = 0; wv < warp; ++wv) before += s_wtie[h][wv];
        if (before < s_ties[h]) sel_mask |= 1u << h;
      }
    }
  }
  uint32_t sel_lane[kMaxH];
#pragma unroll
  for (int h = 0; h < kMaxH; ++h) {
    if (h < H) {
      const uint32_t m = __ballot_sync(0xffffffffu, (sel_mask >> h) & 1u);
      sel_lane[h] = __popc(m & lt_mask);
      if (lane == 0) s_wsel[h][warp] = __popc(m);
    }
  }
  __syncthreads();
  if (warp == 0) {   // lane h: head h
    int n = 0;
    if (lane < H) {
      for (int wv = 0; wv < kWarps; ++wv) {   // counts -> rows of the warps before
        const uint32_t c = s_wsel[lane][wv];
        s_wsel[lane][wv] = n;
        n += c;
      }
      s_place[lane] = len0 + (int)(s_gt_before[lane] + min(s_tie_before[lane], s_ties[lane]));
    }
    int incl = n;
#pragma unroll
    for (int o = 1; o < kMaxH; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane < H) s_first[lane + 1] = incl;
    if (lane == 0) s_first[0] = 0;
    if (tile == 0 && blockIdx.z == 0 && lane < H && s_act[lane])
      bh_lens[b * H + lane] = len0 + (int)(s_gt_all[lane] + min(s_tie_all[lane], s_ties[lane]));
  }
  __syncthreads();
#pragma unroll
  for (int h = 0; h < kMaxH; ++h) {
    if (h < H && ((sel_mask >> h) & 1u)) {
      const int r = s_wsel[h][warp] + sel_lane[h];
      s_pos[s_first[h] + r] = s_place[h] + r;
      s_src[s_first[h] + r] = (uint16_t)(tid * H + h);
    }
  }
  __syncthreads();
  // cooperative row copy: VEC_PER_ROW lanes per (token, head) row
  constexpr int ROWS_PER_IT = kTileTok / VEC_PER_ROW, kAhead = 4;
  const int vec = tid % VEC_PER_ROW, rin = tid / VEC_PER_ROW;
  const int n_rows = s_first[H], r_end = n_rows * (blockIdx.z + 1) / gridDim.z;
  const int64_t tok0 = beg + tile * kTileTok;
  for (int r0 = n_rows * blockIdx.z / gridDim.z + rin; r0 < r_end; r0 += kAhead * ROWS_PER_IT) {
    uint4 kk[kAhead], vv[kAhead];
    int64_t d[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int r = r0 + u * ROWS_PER_IT;
      if (r < r_end) {
        const int src = s_src[r], t = src / H, h = src - t * H, p = s_pos[r], lp = p / PS;
        kk[u] = ldg_nc_v4(keys + (tok0 + t) * sk_n + h * sk_h + vec);
        vv[u] = ldg_nc_v4(vals + (tok0 + t) * sv_n + h * sv_h + vec);
        d[u] = (int64_t)__ldg(pt + h * NLP + lp) * PS + (p - lp * PS);
      }
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (r0 + u * ROWS_PER_IT < r_end) {
        stg_na_v4(k_cache + d[u] * VEC_PER_ROW + vec, kk[u]);
        stg_na_v4(v_cache + d[u] * VEC_PER_ROW + vec, vv[u]);
      }
    }
  }
}

}  // namespace cvllm

using namespace cvllm;

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct SelLayout {
  size_t hist_g, hist_h, ticket, gt_h, zero_end, state_g, state_h, n_keep, len0, tile_tie, tile_cnt, total;
  int tiles;
};

static SelLayout sel_layout(int B, int H, int N) {
  SelLayout l;
  l.tiles = (N + kTileTok - 1) / kTileTok + 1;
  size_t o = 0;
  l.hist_g = o; o += align256((size_t)B * 256 * 4);
  l.hist_h = o; o += align256((size_t)B * H * 256 * 4);
  l.ticket = o; o += align256((size_t)B * 2 * 4);
  l.gt_h = o; o += align256((size_t)B * H * 4);
  l.zero_end = o;
  l.state_g = o; o += align256((size_t)B * sizeof(SegState));
  l.state_h = o; o += align256((size_t)B * H * sizeof(SegState));
  l.n_keep = o; o += align256((size_t)B * H * 4);
  l.len0 = o; o += align256((size_t)B * H * 4);
  l.tile_tie = o; o += align256((size_t)B * l.tiles * H * 4);
  l.tile_cnt = o; o += align256((size_t)B * l.tiles * H * 8);
  l.total = o;
  return l;
}

extern "C" size_t cvllm_select_store_workspace_bytes(int B, int H, int N) {
  if (B <= 0 || H <= 0 || N < 0) return 0;
  return sel_layout(B, H, N).total;
}

template <int V>
static void launch_sel_gather(bool behind, dim3 grid, cudaStream_t st, const float* scores, int64_t s_stride_n,
                              const void* keys, const void* vals, int64_t sk_n, int64_t sk_h,
                              int64_t sv_n, int64_t sv_h, const int32_t* cu, const int32_t* bm,
                              const int32_t* pt, int32_t* bh_lens, void* kc, void* vc, int H, int PS,
                              int NLP, const SelWs& w) {
  auto go = [&](auto launch) {
    launch(sel_gather_kernel<V>, grid, dim3(kTileTok), 0, st, scores, s_stride_n, (const uint4*)keys, (const uint4*)vals, sk_n, sk_h,
           sv_n, sv_h, cu, bm, pt, bh_lens, (uint4*)kc, (uint4*)vc, H, PS, NLP, w);
  };
  if (behind) go([](auto... a) { return launch_behind(a...); });
  else go([](auto... a) { return launch_pdl(a...); });
}

extern "C" int cvllm_select_store_topk_bounded(const float* scores, int64_t s_stride_n, const void* keys,
                                       const void* vals, int64_t sk_n, int64_t sk_h, int64_t sv_n,
                                       int64_t sv_h, const int32_t* num_retain,
                                       const int32_t* cu_seqlens_k, const int32_t* batch_mapping,
                                       int32_t* bh_lens, const int32_t* page_table, void* k_cache,
                                       void* v_cache, int B, int N, int HKV, int D, int PS, int NLP,
                                       int elem_bytes, int pad_to_page, int reserved_batch, int max_len,
                                       void* workspace, size_t workspace_bytes, cvllm_stream_t stream) {
  CVLLM_CHECK_ARG(B > 0 && N >= 0 && HKV > 0 && D > 0 && PS > 0 && NLP > 0);
  CVLLM_CHECK_ARG(scores && keys && vals && num_retain && cu_seqlens_k && batch_mapping && bh_lens &&
                  page_table && k_cache && v_cache && workspace);
  if (N == 0) return CVLLM_OK;
  int vpr;
  int64_t per16;
  const int rc = cvllm_check_store_args(keys, vals, sk_n, sk_h, sv_n, sv_h, k_cache, v_cache, D,
                                        elem_bytes, HKV, &vpr, &per16);
  if (rc != CVLLM_OK) return rc;
  CVLLM_CHECK_SUPPORTED(HKV <= kMaxH);
  const SelLayout l = sel_layout(B, HKV, N);
  CVLLM_CHECK_ARG(workspace_bytes >= l.total);
  CVLLM_CHECK_ALIGN(aligned16(workspace));
  char* base = reinterpret_cast<char*>(workspace);
  SelWs w;
  w.hist_g = reinterpret_cast<uint32_t*>(base + l.hist_g);
  w.hist_h = reinterpret_cast<uint32_t*>(base + l.hist_h);
  w.ticket = reinterpret_cast<uint32_t*>(base + l.ticket);
  w.gt_h = reinterpret_cast<uint32_t*>(base + l.gt_h);
  w.state_g = reinterpret_cast<SegState*>(base + l.state_g);
  w.state_h = reinterpret_cast<SegState*>(base + l.state_h);
  w.n_keep = reinterpret_cast<int32_t*>(base + l.n_keep);
  w.len0 = reinterpret_cast<int32_t*>(base + l.len0);
  w.tile_tie = reinterpret_cast<uint32_t*>(base + l.tile_tie);
  w.tile_cnt = reinterpret_cast<uint2*>(base + l.tile_cnt);
  w.tiles = l.tiles;
  auto st = static_cast<cudaStream_t>(stream);
  const dim3 grid((N + kTileTok - 1) / kTileTok, B);
  // One cluster per sequence while its share of the longest sequence's keys fits a CTA's shared memory; smaller clusters
  // for fewer keys: an exchange costs more than 16 K keys less per CTA save.  While all CTAs take up to 0.7 of the SMs,
  // which the others would only leave idle, twice as many for half the keys is the better trade; beyond that a CTA,
  // which fills its SM, waits for another (clusters of eight for each of many short sequences ran in waves).  Whole
  // evictions in a graph, 8 heads, chain of launches / clusters by N alone / this, us:
  // 128 of 100 tokens 166 / 230 / 71, 64 of 500 217 / 196 / 102, 25 of 1000 162 / 121 / 96, 16 of 3000 180 / 180 / 109,
  // 12 of 6000 190 / 190 / 119, 8 of 4000 146 / 98 / 96, one of 32768 118 / 88 / 88.
  const int longest = min(max(max_len, 1), N);
  auto room = [&](int c) { return c < 8 && 20 * (int64_t)B * c <= 7 * (int64_t)sm_count(); };
  int cluster = 1;
  while (cluster < 8 && (int64_t)longest * HKV > (int64_t)cluster * 16384) cluster *= 2;
  while (room(cluster) && (int64_t)N * HKV > (int64_t)cluster * 16384) cluster *= 2;
  const int tiles_per_cta = cdiv(cdiv(longest, kTileTok), cluster);
  const size_t cl_smem = sel_cluster_smem(tiles_per_cta, HKV);
  constexpr size_t kClSmemMax = 226 * 1024;   // beside the static arrays
  const bool one_launch = cl_smem <= kClSmemMax && test_options().select_passes.load() == 0;
  if (one_launch) {
    static std::atomic<uint64_t> attr{0};
    CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)sel_cluster_kernel, (int)kClSmemMax, attr));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster, B);
    cfg.blockDim = dim3(kClThreads);
    cfg.dynamicSmemBytes = cl_smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CVLLM_CHECK_CUDA(cudaLaunchKernelEx(&cfg, sel_cluster_kernel, scores, s_stride_n, cu_seqlens_k, num_retain, batch_mapping,
                                        (const int32_t*)bh_lens, HKV, PS, pad_to_page, reserved_batch,
                                        tiles_per_cta * kTileTok * HKV, w));
    CVLLM_CHECK_LAUNCH();
  } else {
    CVLLM_CHECK_CUDA(cudaMemsetAsync(base, 0, l.zero_end, st));
    sel_init_kernel<<<(B * HKV + 255) / 256, 256, 0, st>>>(cu_seqlens_k, num_retain, batch_mapping, bh_lens,
                                                           B, HKV, reserved_batch, w);
    // eleven short kernels in a row, each dependent on the one before; launch_pdl is a plain launch unless the test
    // option "pdl" is set (common.cuh has the measurements)
    const dim3 pb(kPassThreads);
    for (int pass = 0; pass < 4; ++pass)
      CVLLM_CHECK_CUDA(launch_pdl(sel_pass_kernel<false>, grid, pb, 0, st, scores, s_stride_n, cu_seqlens_k, HKV, pass, w));
    CVLLM_CHECK_CUDA(launch_pdl(sel_count_global_kernel, grid, pb, 0, st, scores, s_stride_n, cu_seqlens_k, HKV, w));
    CVLLM_CHECK_CUDA(launch_pdl(sel_resolve_kernel, dim3(B), pb, 0, st, scores, s_stride_n, cu_seqlens_k, batch_mapping,
                                HKV, PS, pad_to_page, reserved_batch, w));
    for (int pass = 0; pass < 4; ++pass)
      CVLLM_CHECK_CUDA(launch_pdl(sel_pass_kernel<true>, grid, pb, 0, st, scores, s_stride_n, cu_seqlens_k, HKV, pass, w));
    CVLLM_CHECK_CUDA(launch_pdl(sel_count_heads_kernel, grid, pb, 0, st, scores, s_stride_n, cu_seqlens_k, HKV, w));
    CVLLM_CHECK_LAUNCHES(12);
  }
  // as many copy CTAs per tile as the chip holds at once (four an SM), one where the tiles alone fill it
  const int tiles = cdiv(N, kTileTok) + (B - 1);   // at most: each sequence may end inside one
  const dim3 ggrid(grid.x, grid.y, max(1, min(8, 4 * sm_count() / tiles)));
#define G(V)                                                                                            \
  launch_sel_gather<V>(one_launch, ggrid, st, scores, s_stride_n, keys, vals, sk_n / per16, sk_h / per16, sv_n / per16, \
                       sv_h / per16, cu_seqlens_k, batch_mapping, page_table, bh_lens, k_cache, v_cache,   \
                       HKV, PS, NLP, w)
  switch (vpr) {
    case 1: G(1); break;
    case 2: G(2); break;
    case 4: G(4); break;
    case 8: G(8); break;
    case 16: G(16); break;
    case 32: G(32); break;
    default: return CVLLM_E_UNSUPPORTED;
  }
#undef G
  CVLLM_CHECK_LAUNCH();
  return CVLLM_OK;
}

extern "C" int cvllm_select_store_topk(const float* scores, int64_t s_stride_n, const void* keys,
                                       const void* vals, int64_t sk_n, int64_t sk_h, int64_t sv_n,
                                       int64_t sv_h, const int32_t* num_retain,
                                       const int32_t* cu_seqlens_k, const int32_t* batch_mapping,
                                       int32_t* bh_lens, const int32_t* page_table, void* k_cache,
                                       void* v_cache, int B, int N, int HKV, int D, int PS, int NLP,
                                       int elem_bytes, int pad_to_page, int reserved_batch,
                                       void* workspace, size_t workspace_bytes, cvllm_stream_t stream) {
  return cvllm_select_store_topk_bounded(scores, s_stride_n, keys, vals, sk_n, sk_h, sv_n, sv_h, num_retain, cu_seqlens_k,
                                         batch_mapping, bh_lens, page_table, k_cache, v_cache, B, N, HKV, D, PS, NLP,
                                         elem_bytes, pad_to_page, reserved_batch, N, workspace, workspace_bytes, stream);
}
