// Head-sparse split-KV decode attention over the paged cache.
//
// Replaces attention/sparse_decode_kernel.py:10-165 (stage 1 :247-388, stage 2
// :392-435) with ONE persistent launch, one CTA per SM:
//   * work = 128-token units of every (b, kv-head); the flattened unit list
//     is cut into gridDim.x equal ranges (stream-K style), so ragged per-head
//     lengths after compression are balanced exactly — the reference gives
//     every head the same KEY_SPLIT regardless of its length (:303-306).  Ranges
//     over short heads end at heads' ends instead (heads_whole)
//   * warp 8 is the TMA producer: it resolves (head, page) for 32 units at a
//     time (one lane per unit/page piece), then streams K and V units through
//     a ring of kSlots x 32 KB shared-memory slots (cp.async.bulk.tensor, 128B
//     swizzle, mbarrier full/empty pairs).  Up to 160 KB per SM are in flight,
//     which is what HBM3e needs (Little: 6.5 TB/s x ~1 us / 148 SMs ~ 45 KB)
//     with a wide margin; the previous register-staged version peaked at 64 KB
//     and measured 4.5 TB/s
//   * warps 0-7 consume: a warp owns 16 keys of a unit, reads its K rows and V
//     rows from the swizzled slot as conflict-free 16-byte vectors laid out
//     directly in mma.sync m16n8k16 fragment order (the contraction dim is
//     permuted identically on both operands, so no ldmatrix is needed)
//   * S^T = K.Q^T (keys on M, the G<=8 query heads on N), softmax stats per
//     column with warp shuffles, P^T goes through movmatrix to the B-operand
//     layout, O^T += V^T.P^T
//   * partial (m, l, O) of a range that does not cover its whole head goes to
//     a scratch slot; the CTA that completes a head merges (atomic ticket),
//     every warp folding every eighth of the states with independent loads
//   * the launch is scheduled beside the kernel in front of it where that one lets it (the norm and store of a step, another
//     decode step): barriers and descriptors are ready when it ends.  One sequence of 8192 rows 17.9 -> 15.5 us a call back to
//     back, 8 x 384 rows 12.3 -> 10.1, a biased step of 8 x 4096 rows, whose fold is scheduled beside it, 40.7 -> 37.3
// HBM-bound: 4*D bytes per cached (token, head).
//
// BIAS: the same streaming for the biased attention's decode steps (cvllm_launch_bias_decode, called by
// cvllm_bias_attn_decode_stream): heads of 128 or 64, keys 0 .. position of a sequence cut by its chunk or window (the unit list
// starts at the first visible key's unit, behind the units of kept first tokens), a distance bias and a sink in the softmax.
// What that path computes in 32 bits stays so: P is the sum of two 16-bit numbers (2^-17 relative), whose low parts take
// the query columns 4 .. 7 that groups of up to four heads leave free.  Partial states are folded by a second kernel
// (its workspace needs no zeroed tickets).
#include <stdlib.h>
#include <type_traits>

#include <algorithm>

#include "common.cuh"
#include "mma.cuh"
#include "tma.cuh"

namespace cvllm {

constexpr int kUnit = 128;        // tokens per work unit
constexpr int kDecWarps = 8;      // consumer warps: 8 x 16 keys = one unit
constexpr int kDecCons = kDecWarps * 32;
constexpr int kDecThreads = kDecCons + 32;  // + producer warp
constexpr int kMaxSlots = 6;      // ring slots (one K unit or one V unit each): 6 when G <= 4, else 5
constexpr int kDecMaxSmem = 224 * 1024;     // 227 KB opt-in limit minus static smem
constexpr int kSlotBytes = kUnit * 256;     // 32 KB at D = 128, 16-bit (half of it used at D = 64)
constexpr int kHalfBytes = kUnit * 128;     // one 64-column half of a slot

// Whether the ranges of the C CTAs end at heads' ends (`most` units in the longest head, U in all).  A cut costs 3 to 4 us at the
// end where units outnumber the CTAs, 1 where they don't (a partial state through memory, a ticket, the fold); a head left whole
// costs what its CTA has more than the even share, where a unit takes 0.7 us on a chip that has few and 1.4 on a full one.
// Measured in a graph, cut / whole, us, 32 / 8 heads, longest head up to 1.4 times the rows given: 8 x 384 13.1 / 9.0, 8 x 600
// 14.0 / 10.8, 16 x 600 15.2 / 12.5, 32 x 200 15.7 / 11.9, 64 x 400 32.3 / 29.7, 1 x 300 9.0 / 7.8, 4 x 300 9.1 / 8.1, but 24 x 650
// 19.4 / 19.6, 48 x 600 33.4 / 34.9, 32 x 800 29.8 / 32.7 (shares above 6 units), 1 x 500 8.9 / 9.5, 4 x 500 9.2 / 10.0, 4 x 1000
// 12.2 / 14.5 (long beside the share).
__device__ __forceinline__ bool heads_whole(int most, int64_t U, int C) {
  if (U > 6 * (int64_t)C) return most <= 5;
  return most <= 8 && (int64_t)C * (most - (U >= C ? 6 : 4)) <= U;
}

struct DecodeParams {
  const void* q;
  void* out;
  const int32_t* seq_lens_bh;
  const int32_t* page_table;
  const int32_t* batch_mapping;
  float* scratch;     // [(BH + C)] slots of G*(D+2) floats
  int32_t* counters;  // [BH], zero on entry, left zero on exit
  int B, HQ, HKV, G, PS, NLP;
  int box_rows;       // min(PS, 128): rows of one TMA box (a box never crosses a page)
  int slots;          // ring depth (<= kMaxSlots)
  int lens_by_slot;   // seq_lens_bh is the cache's [Bmax+1, HKV] table, indexed through batch_mapping
  int mode;           // 0 = normal; 1 = consumers only drain the ring (load ceiling, profiling only)
  int map_in_smem;    // batch_mapping has a copy in shared memory (decode_smem)
  float scale_log2;
#ifdef CVLLM_DECODE_TRACE
  unsigned long long* trace;  // profiling build only (tools/trace_decode.py): 8 globaltimer stamps per CTA
#endif
};

struct BiasDecodeParams : DecodeParams {   // what the biased attention adds
  const int32_t* positions;   // [B] position of every sequence's token
  int64_t pt_slot, pt_head;   // page table strides
  int64_t o_stride;           // output row stride (elements)
  const float* slopes;        // [HQ] or NULL
  const float* dist_bias;     // [dist_rows][HQ] or NULL
  int dist_rows, chunk, window, keep, reserved_slot;
  float sink;                 // 1 = a sink in the denominator
  const float* sink_logits;   // [HQ] or NULL (score 0)
};

__device__ __forceinline__ unsigned long long gtime() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// The stamps cost ~2 us at B = 1 (measured), so they exist only in the -DCVLLM_DECODE_TRACE variant build.
#ifdef CVLLM_DECODE_TRACE
#define DEC_TRACE(slot) do { if (p.trace) p.trace[blockIdx.x * 8 + (slot)] = gtime(); } while (0)
#else
#define DEC_TRACE(slot) do { } while (0)
#endif

// One warp's 16-key slice: K rows r / r+8 (D / 32 chunks each), V for 4 keys x D / 64 chunks.
template <int D>
struct Slice {
  uint4 k_lo[D / 32], k_hi[D / 32];  // rows r, r+8; 16-byte chunk kchunk(j, c)
  uint4 v[4][D / 64];                // keys {2j,2j+1,2j+8,2j+9}; chunks r (d 8r..8r+7), 8+r
};

// The keys that a sequence's token sees, as a list of kUnit-key units: the units that hold kept first tokens and lie
// before the unit of the first key inside chunk and window, then the units from that one to the token's own.
struct UnitList {
  int pi, lo, begin, kept, count;
  UnitList() = default;
  __device__ __forceinline__ UnitList(const BiasDecodeParams& p, int b) {
    const bool live = p.batch_mapping[b] != p.reserved_slot;
    pi = p.positions[b];
    lo = p.chunk > 0 ? pi / p.chunk * p.chunk : 0;
    if (p.window > 0) lo = max(lo, pi - p.window + 1);
    begin = lo / kUnit;
    kept = min(cdiv(min(p.keep, lo), kUnit), begin);
    count = live ? kept + pi / kUnit - begin + 1 : 0;
  }
  __device__ __forceinline__ int base(int u) const { return (u < kept ? u : u - kept + begin) * kUnit; }
};

// Lane j owns the 16-byte chunks {2j, 2j+1} of each 128-byte half of a row; c = 0..3 walks them.
// With the 128B swizzle (chunk ^= row & 7) the eight lanes of a quarter-warp (rows r0, r0+1 x
// j = 0..3) then hit eight distinct bank groups.  Q uses the same chunk order, so the
// contraction is unchanged.
__device__ __forceinline__ int kchunk(int j, int c) { return ((c >> 1) << 3) + 2 * j + (c & 1); }

__device__ __forceinline__ uint4 lds_v4(uint32_t addr) {
  uint4 r;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
               : "r"(addr));
  return r;
}
// address of 16-byte chunk `ch` (0..15) of row t (0..127) inside a swizzled slot
__device__ __forceinline__ uint32_t slot_addr(uint32_t slot, int t, int ch) {
  return slot + (uint32_t)((ch >> 3) * kHalfBytes + t * 128 + (((ch & 7) ^ (t & 7)) << 4));
}

// 1 / denominator of a biased head's row whose running maximum is m (log2 units) and whose sum is l, sink included: the
// row's values are relative to m, and so is what the sink adds
__device__ __forceinline__ float bias_inv(const BiasDecodeParams& p, int hq, float m, float l) {
  if (p.sink > 0.f) {
    const float sm = (p.sink_logits ? p.sink_logits[hq] : 0.f) * 1.4426950408889634f;
    if (sm - m > 120.f) return 0.f;   // a sink far above every key takes all the weight
    l += ex2(sm - m);
  }
  return l > 0.f ? 1.f / l : 0.f;
}

__device__ __forceinline__ void cons_bar() { asm volatile("bar.sync 1, %0;" ::"n"(kDecCons) : "memory"); }

// (a division of 64 bits takes 0.1 us, and some stand in front of all else)
__device__ __forceinline__ int quotient(int64_t x, int d) {   // x >= 0, d > 0
  return x >> 32 ? (int)(x / d) : (int)((uint32_t)x / (uint32_t)d);
}
// First unit of CTA t's equal share of U
__device__ __forceinline__ int share(int U, int t, int C) { return quotient((int64_t)U * t, C); }

// Where the partial states of a cut head lie: state k = 0 .. n - 1 in the slot of CTA cta(k).  With at least as many units as CTAs every
// CTA from the head's first to its last has one; with fewer a unit is a state, and most CTAs between have none.  Going through
// those too, with the two divisions that tell, was most of a fold.  One sequence of 700 rows, a head with a group of eight:
// 19.0 -> 9.5 us back to back, a biased step over 1500 rows of it 24.7 -> 12.1; 5 x 60 rows of 8 heads 6.8 -> 6.1 (no searches).
struct HeadStates {
  int h_beg, U, C, c_first, n;
  __device__ __forceinline__ HeadStates(int h_beg, int h_end, int U, int C) : h_beg(h_beg), U(U), C(C) {
    c_first = holder(h_beg);
    n = U < C ? h_end - h_beg : holder(h_end - 1) - c_first + 1;
  }
  __device__ __forceinline__ int holder(int u) const { return quotient((int64_t)(u + 1) * C - 1, U); }   // the CTA of unit u
  __device__ __forceinline__ int cta(int k) const { return U < C ? holder(h_beg + k) : c_first + k; }
};

// The partial states of a cut head (units h_beg .. h_end - 1) into s_merge's rows: each consumer warp folds every eighth of them into a
// running (m, l, O), the loads of AHEAD states in flight together; lane owns d = 2*lane, 2*lane+1, 64 + 2*lane, 65 + 2*lane.
// A function of its own: its registers beside the streaming loop's would make that loop spill.
template <int NQ, int AHEAD>
__device__ __noinline__ void fold_slots(const float* scratch, float* s_merge, int head, int G, int h_beg, int h_end, int U, int C) {
  constexpr int ROW = 128 + 2;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* mw = s_merge + warp * G * ROW;
  float M[NQ], ls[NQ];
  float2 oa[NQ], ob[NQ];
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    M[q] = -INFINITY; ls[q] = 0.f;
    oa[q] = make_float2(0.f, 0.f); ob[q] = make_float2(0.f, 0.f);
  }
  const HeadStates states(h_beg, h_end, U, C);
  for (int k = warp; k < states.n; k += AHEAD * kDecWarps) {
    float2 va[AHEAD][NQ], vb[AHEAD][NQ], ml[AHEAD][NQ];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int ki = k + i * kDecWarps;
      const bool used = ki < states.n;
      const float* sl = scratch + (int64_t)(head + states.cta(ki)) * G * ROW;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        ml[i][q] = make_float2(-INFINITY, 0.f);
        va[i][q] = vb[i][q] = make_float2(0.f, 0.f);
        if (used && q < G) {
          va[i][q] = __ldcg(reinterpret_cast<const float2*>(sl + q * ROW + 2 * lane));
          vb[i][q] = __ldcg(reinterpret_cast<const float2*>(sl + q * ROW + 64 + 2 * lane));
          ml[i][q] = __ldcg(reinterpret_cast<const float2*>(sl + q * ROW + 128));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const float Mn = fmaxf(M[q], ml[i][q].x);
        const float so = (M[q] > -INFINITY) ? ex2(M[q] - Mn) : 0.f;
        const float sn = (ml[i][q].x > -INFINITY) ? ex2(ml[i][q].x - Mn) : 0.f;
        oa[q].x = oa[q].x * so + va[i][q].x * sn; oa[q].y = oa[q].y * so + va[i][q].y * sn;
        ob[q].x = ob[q].x * so + vb[i][q].x * sn; ob[q].y = ob[q].y * so + vb[i][q].y * sn;
        ls[q] = ls[q] * so + ml[i][q].y * sn;
        M[q] = Mn;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < NQ; ++q) {
    if (q < G) {
      *reinterpret_cast<float2*>(mw + q * ROW + 2 * lane) = oa[q];
      *reinterpret_cast<float2*>(mw + q * ROW + 64 + 2 * lane) = ob[q];
      if (lane == 0) *reinterpret_cast<float2*>(mw + q * ROW + 128) = make_float2(M[q], ls[q]);
    }
  }
}

template <bool BF16, int D, bool BIAS = false>
__global__ void __launch_bounds__(kDecThreads, 1)
decode_attn_kernel(const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                   const std::conditional_t<BIAS, BiasDecodeParams, DecodeParams> p) {
  static_assert(D == 128 || (BIAS && D == 64), "head sizes");
  constexpr int KSTEPS = D / 16;  // 8
  constexpr int MT = D / 16;      // 8 output m-tiles (16 d each)
  constexpr int KC = D / 32;      // 16-byte chunks of a row per lane
  constexpr int ROW = D + 2;      // merged row: O[D], m, l
  constexpr int NW = kDecThreads / 32;

  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem_raw =
      reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~(uintptr_t)1023);
  const int BH = p.B * p.HKV;
  unsigned char* ring = smem_raw;
  const int kSlots = p.slots;
  uint64_t* bar_full = reinterpret_cast<uint64_t*>(smem_raw + kSlots * kSlotBytes);
  uint64_t* bar_empty = bar_full + kMaxSlots;
  float* s_merge = reinterpret_cast<float*>(bar_empty + kMaxSlots);   // [kDecWarps][G][ROW]
  int32_t* s_prefix = reinterpret_cast<int32_t*>(s_merge + kDecWarps * p.G * ROW);  // [BH + 1]
  int32_t* s_map = s_prefix + BH + 1;                                 // [B] batch_mapping, where there is room
  // (as one pointer: chosen at every look-up, 16 x 10240 rows took 0.5 % longer)
  const int32_t* slot_of = p.map_in_smem ? s_map : p.batch_mapping;
  __shared__ int32_t s_warp_tot[NW], s_warp_max[NW];
  __shared__ int s_near[2], s_last;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int C = gridDim.x, c = blockIdx.x;
  const int G = p.G;
  // rows cached for flattened head i = b * HKV + h
  auto len_of = [&](int i) -> int {
    if constexpr (BIAS) return p.positions[i / p.HKV] + 1;
    if (!p.lens_by_slot) return p.seq_lens_bh[i];
    const int b = i / p.HKV;
    return p.seq_lens_bh[p.batch_mapping[b] * p.HKV + (i - b * p.HKV)];
  };
  auto units_of = [&](int i) -> int {
    if constexpr (BIAS) return UnitList(p, i / p.HKV).count;
    else return cdiv(len_of(i), kUnit);
  };
  auto out_row = [&](int b, int h) -> uint32_t* {   // the G heads of (b, h), as pairs
    if constexpr (BIAS) return reinterpret_cast<uint32_t*>(p.out) + b * (p.o_stride / 2) + h * G * (D / 2);
    else return reinterpret_cast<uint32_t*>(p.out) + ((int64_t)b * p.HQ + h * G) * (D / 2);
  };

  if (tid == 0) DEC_TRACE(0);
  if (tid == kDecCons) {  // producer warp: descriptor fetch overlaps the prologue
    tma_prefetch_desc(&tm_k);
    tma_prefetch_desc(&tm_v);
  }
  if (tid == 0) {
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(&bar_full[s], 1);
      mbar_init(&bar_empty[s], kDecWarps);
    }
    mbar_fence_init();
  }
  pdl_wait();      // what came before wrote the query, the cache's new rows and the lengths
  pdl_trigger();   // the fold may start (behind the wait: what it reads ahead is then as this kernel finds it)

  // ---- phase 0: units per head, exclusive prefix over the BH heads ---------
  int x0, x1, most = 0;   // an equal share of the units begins and ends here; units of the longest head
  {
    const int per = cdiv(BH, kDecThreads);
    const int beg = min(BH, tid * per), end = min(BH, beg + per);
    int local = 0;
    if (p.map_in_smem)
      for (int i = tid; i < p.B; i += kDecThreads) s_map[i] = p.batch_mapping[i];   // in flight with the lengths
    for (int i = beg; i < end; ++i) {
      const int n = units_of(i);
      local += n;
      most = max(most, n);
    }
    most = __reduce_max_sync(0xffffffffu, most);
    int incl = local;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) {
      s_warp_tot[warp] = incl;
      s_warp_max[warp] = most;
    }
    __syncthreads();
    int base = 0, all = 0;
    most = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
      base += w < warp ? s_warp_tot[w] : 0;
      all += s_warp_tot[w];
      most = max(most, s_warp_max[w]);
    }
    int run = base + incl - local;
    x0 = share(all, c, C);
    x1 = share(all, c + 1, C);
    for (int i = beg; i < end; ++i) {
      const int next = run + units_of(i);
      s_prefix[i] = run;
      // the heads' ends next to the share's: the thread that has the head knows; a search of the prefix for each was 0.5 us of
      // a step over 128 heads of one unit, 6.9 us
      if (run <= x0 && x0 < next) s_near[0] = x0 - run < next - x0 ? run : next;
      if (run <= x1 && x1 < next) s_near[1] = x1 - run < next - x1 ? run : next;
      run = next;
    }
    if (tid == kDecThreads - 1) s_prefix[BH] = run;
    __syncthreads();
  }
  const int U = s_prefix[BH];
  if (tid == 0) DEC_TRACE(1);

  // zero rows for empty heads (reference leaves them uninitialised)
  for (int i = c; i < BH; i += C) {
    if (s_prefix[i + 1] == s_prefix[i]) {
      const int b = i / p.HKV, h = i % p.HKV;
      uint32_t* o = out_row(b, h);
      for (int e = tid; e < G * D / 2; e += kDecThreads) o[e] = 0u;
    }
  }
  if (U == 0) return;

  // largest i with s_prefix[i] <= u
  auto find_head = [&](int u) {
    int lo = 0, hi = BH;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_prefix[mid] <= u) lo = mid; else hi = mid;
    }
    return lo;
  };
  const bool uncut = (BIAS || G <= 4) && heads_whole(most, U, C);
  const int u_begin = uncut ? s_near[0] : x0, u_end = uncut && c + 1 < C ? s_near[1] : x1;
  if (u_begin >= u_end) return;

  // =========================== producer warp ================================
  if (warp == kDecWarps) {
    const int BR = p.box_rows;
    const int pieces = kUnit / BR;      // TMA boxes per (unit, half): 1 when PS % 128 == 0
    const int upb = 32 / pieces;        // units resolved per batch (one lane per piece)
    int p_slot = 0;                     // ring position of the next item (K and V units alternate)
    uint32_t p_par = 0;                 // and its phase parity
    // first cache row of this lane's (unit, piece) of the batch starting at unit ub
    auto resolve = [&](int ub, int& row, int& nvp) {
      const int my_unit = ub + lane / pieces, my_piece = lane % pieces;
      row = 0;
      nvp = 0;
      if (my_unit < u_end) {
        const int head = find_head(my_unit);
        int t0 = (my_unit - s_prefix[head]) * kUnit;
        if constexpr (BIAS) t0 = UnitList(p, head / p.HKV).base(my_unit - s_prefix[head]);
        const int L = len_of(head);
        nvp = min(pieces, cdiv(L - t0, BR));  // pages past the head's length are not mapped
        if (my_piece < nvp) {
          const int b = head / p.HKV, h = head % p.HKV;
          const int tok = t0 + my_piece * BR;
          const int pg = tok / p.PS;
          const int32_t* pt;
          if constexpr (BIAS) pt = p.page_table + p.batch_mapping[b] * p.pt_slot + h * p.pt_head;
          else pt = p.page_table + ((int64_t)slot_of[b] * p.HKV + h) * p.NLP;
          row = pt[pg] * p.PS + (tok - pg * p.PS);
        }
      }
    };
    int row, nvp;
    resolve(u_begin, row, nvp);
    for (int ub = u_begin; ub < u_end; ub += upb) {
      // the next batch's page-table loads are in flight while this batch is issued
      int row_next = 0, nvp_next = 0;
      if (ub + upb < u_end) resolve(ub + upb, row_next, nvp_next);
      const int cnt = min(upb, u_end - ub);
      for (int i = 0; i < cnt; ++i) {
        const int nv = __shfl_sync(0xffffffffu, nvp, i * pieces);
#pragma unroll
        for (int kv = 0; kv < 2; ++kv) {
          const int slot = p_slot;
          const uint32_t par = p_par;
          if (++p_slot == kSlots) { p_slot = 0; p_par ^= 1u; }
          unsigned char* dst = ring + slot * kSlotBytes;
          const CUtensorMap* tm = kv ? &tm_v : &tm_k;
          if (lane == 0) {
            mbar_wait(&bar_empty[slot], par ^ 1u);
            mbar_expect_tx(&bar_full[slot], (uint32_t)(nv * BR * D * 2));
          }
          for (int pc = 0; pc < nv; ++pc) {
            const int r0 = __shfl_sync(0xffffffffu, row, i * pieces + pc);
            if (lane == 0) {
              tma_load_2d(dst + pc * BR * 128, tm, &bar_full[slot], 0, r0);
              if constexpr (D == 128) tma_load_2d(dst + kHalfBytes + pc * BR * 128, tm, &bar_full[slot], 64, r0);
            }
          }
        }
      }
      row = row_next;
      nvp = nvp_next;
    }
    return;
  }

  // =========================== consumer warps ===============================
  const int r = lane >> 2, j = lane & 3;
  // P as the sum of two 16-bit numbers (see the top): biased attention, and heads left whole.  Their one running maximum
  // leaves fewer keys with the exact probability 1 than the cut ones' many, 2 % more error at 384 keys a head; so, it is 16 %
  // less in fp16 (2.07e-4 for 2.46e-4 of the result, twelve seeds) and 17 % in bf16 (1.66e-3 for 2.00e-3).
  const bool low_parts = G <= 4 && (BIAS || uncut);
  const uint32_t ring_u32 = smem_u32(ring);
  int c_slot = 0;        // ring position of the next item to consume
  uint32_t c_par = 0;    // and its mbarrier phase parity
  int head = find_head(u_begin);
  int u = u_begin;
  while (u < u_end) {
    while (s_prefix[head + 1] <= u) ++head;  // skip finished / empty heads
    const int h_beg = s_prefix[head], h_end = s_prefix[head + 1];
    const int seg_end = min(u_end, h_end);
    const int ua = u - h_beg, ub = seg_end - h_beg;  // units of this head
    const int b = head / p.HKV, h = head % p.HKV;
    const int L = len_of(head);
    const UnitList list = [&]() {
      if constexpr (BIAS) return UnitList(p, b);
      else return UnitList{};
    }();
    // this lane's query columns 2j, 2j + 1 (columns 4 .. 7 of a small group carry the low parts of P)
    const bool low_cols = low_parts && j >= 2;
    const int qc = low_cols ? 2 * j - 4 : 2 * j;
    float slope0 = 0.f, slope1 = 0.f;
    if constexpr (BIAS) {
      if (p.slopes) {
        slope0 = qc < G ? p.slopes[h * G + qc] * 1.4426950408889634f : 0.f;
        slope1 = qc + 1 < G ? p.slopes[h * G + qc + 1] * 1.4426950408889634f : 0.f;
      }
    }

    // ---- Q^T as B operand (n = query r, k = permuted d) ----
    uint32_t qb[KSTEPS][2];
    {
      const uint4 z = make_uint4(0, 0, 0, 0);
      const char* qrow = reinterpret_cast<const char*>(p.q) + ((int64_t)b * p.HQ + h * G + r) * (D * 2);
#pragma unroll
      for (int cc = 0; cc < KC; ++cc) {
        const uint4 v = (r < G) ? *reinterpret_cast<const uint4*>(qrow + kchunk(j, cc) * 16) : z;
        qb[2 * cc][0] = v.x; qb[2 * cc][1] = v.y;
        qb[2 * cc + 1][0] = v.z; qb[2 * cc + 1][1] = v.w;
      }
    }

    float acc[MT][4];
#pragma unroll
    for (int t = 0; t < MT; ++t) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
    float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;

    auto stream_units = [&](auto parts) {
      constexpr bool LOW = decltype(parts)::value;
      for (int uu = ua; uu < ub; ++uu) {
        // ring positions of this unit's K and V items (advanced without divisions)
        const int ks_slot = c_slot;
        const uint32_t k_par = c_par;
        if (++c_slot == kSlots) { c_slot = 0; c_par ^= 1u; }
        const int vs_slot = c_slot;
        const uint32_t v_par = c_par;
        if (++c_slot == kSlots) { c_slot = 0; c_par ^= 1u; }
        const uint32_t k_base = ring_u32 + ks_slot * kSlotBytes, v_base = ring_u32 + vs_slot * kSlotBytes;
        const int t0 = warp * 16;                               // this warp's rows inside the unit
        const int unit0 = BIAS ? list.base(uu) : uu * kUnit;    // position of the unit's first key
        const int n_valid = min(16, L - (unit0 + t0));          // <= 0: nothing for this warp
        // what distance and head add to this lane's four logits, requested before the unit's data is waited for
        float bias0 = 0.f, bias1 = 0.f, bias2 = 0.f, bias3 = 0.f;
        if constexpr (BIAS) {
          const int n_lo = list.pi - (unit0 + t0 + r), n_hi = n_lo - 8;
          bias0 = -slope0 * (float)n_lo; bias1 = -slope1 * (float)n_lo;
          bias2 = -slope0 * (float)n_hi; bias3 = -slope1 * (float)n_hi;
          if (p.dist_bias && qc < G) {
            const float* t_lo = p.dist_bias + (int64_t)min(max(n_lo, 0), p.dist_rows - 1) * p.HQ + h * G + qc;
            const float* t_hi = p.dist_bias + (int64_t)min(max(n_hi, 0), p.dist_rows - 1) * p.HQ + h * G + qc;
            bias0 = fmaf(t_lo[0], 1.4426950408889634f, bias0);
            bias2 = fmaf(t_hi[0], 1.4426950408889634f, bias2);
            if (qc + 1 < G) {
              bias1 = fmaf(t_lo[1], 1.4426950408889634f, bias1);
              bias3 = fmaf(t_hi[1], 1.4426950408889634f, bias3);
            }
          }
        }

        // every warp waits (so nobody can run a full ring ahead) and releases the slots
        mbar_wait(&bar_full[ks_slot], k_par);
        if (tid == 0 && u == u_begin && uu == ua) DEC_TRACE(2);
        if (n_valid > 0 && p.mode == 0) {
          Slice<D> cur;
#pragma unroll
          for (int cc = 0; cc < KC; ++cc) {
            cur.k_lo[cc] = lds_v4(slot_addr(k_base, t0 + r, kchunk(j, cc)));
            cur.k_hi[cc] = lds_v4(slot_addr(k_base, t0 + r + 8, kchunk(j, cc)));
          }
          // V rows of keys past the head's length are uninitialised memory: P is 0 there but
          // 0 * NaN would poison O, so those rows are read as zeros.  V is fetched before the
          // S chain so its shared-memory latency hides behind the mma / softmax dependency chain.
          mbar_wait(&bar_full[vs_slot], v_par);
          {
            const uint4 z = make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int key = 2 * j + (i & 1) + ((i >> 1) << 3);
              bool ok = key < n_valid;
              if constexpr (BIAS) ok = ok && (unit0 + t0 + key >= list.lo || unit0 + t0 + key < p.keep);
              cur.v[i][0] = ok ? lds_v4(slot_addr(v_base, t0 + key, r)) : z;
              if constexpr (D == 128) cur.v[i][D / 64 - 1] = ok ? lds_v4(slot_addr(v_base, t0 + key, 8 + r)) : z;
            }
          }
          // ---- S^T[16 keys x 8 queries]: two accumulators halve the dependent mma chain ----
          float s[4] = {0.f, 0.f, 0.f, 0.f}, s_b[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int ks = 0; ks < KSTEPS; ++ks) {
            const int cc = ks >> 1;
            const uint32_t a0 = (ks & 1) ? cur.k_lo[cc].z : cur.k_lo[cc].x;
            const uint32_t a1 = (ks & 1) ? cur.k_hi[cc].z : cur.k_hi[cc].x;
            const uint32_t a2 = (ks & 1) ? cur.k_lo[cc].w : cur.k_lo[cc].y;
            const uint32_t a3 = (ks & 1) ? cur.k_hi[cc].w : cur.k_hi[cc].y;
            if (ks & 1) mma16816<BF16>(s_b, a0, a1, a2, a3, qb[ks][0], qb[ks][1]);
            else mma16816<BF16>(s, a0, a1, a2, a3, qb[ks][0], qb[ks][1]);
          }
#pragma unroll
          for (int e = 0; e < 4; ++e) s[e] += s_b[e];
          __syncwarp();
          if (lane == 0) mbar_arrive(&bar_empty[ks_slot]);  // K rows are in registers: free the slot now
          bool ok_lo = r < n_valid, ok_hi = r + 8 < n_valid;
          if constexpr (BIAS) {
            const int kp = unit0 + t0 + r;
            ok_lo = ok_lo && (kp >= list.lo || kp < p.keep);
            ok_hi = ok_hi && (kp + 8 >= list.lo || kp + 8 < p.keep);
          }
          if constexpr (LOW) {   // columns 4 .. 7 repeat the scores of columns 0 .. 3: same maximum, same probabilities
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float other = __shfl_xor_sync(0xffffffffu, s[e], 2);
              if (low_cols) s[e] = other;
            }
          }
          const float x0 = ok_lo ? (BIAS ? fmaf(s[0], p.scale_log2, bias0) : s[0] * p.scale_log2) : -INFINITY;
          const float x1 = ok_lo ? (BIAS ? fmaf(s[1], p.scale_log2, bias1) : s[1] * p.scale_log2) : -INFINITY;
          const float x2 = ok_hi ? (BIAS ? fmaf(s[2], p.scale_log2, bias2) : s[2] * p.scale_log2) : -INFINITY;
          const float x3 = ok_hi ? (BIAS ? fmaf(s[3], p.scale_log2, bias3) : s[3] * p.scale_log2) : -INFINITY;
          float mx0 = fmaxf(x0, x2), mx1 = fmaxf(x1, x3);
#pragma unroll
          for (int o = 4; o < 32; o <<= 1) {
            mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, o));
            mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
          }
          if constexpr (BIAS) {   // a first unit may be all masked: the lowest finite reference, so that every score can pass it
            m0 = fmaxf(m0, -3.402823466e38f);
            m1 = fmaxf(m1, -3.402823466e38f);
          }
          float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
          // a NaN/-inf column max (garbage q) must not poison the rest
          if (!(mn0 > -INFINITY)) mn0 = 0.f;
          if (!(mn1 > -INFINITY)) mn1 = 0.f;
          const float al0 = ex2(m0 - mn0), al1 = ex2(m1 - mn1);
          m0 = mn0; m1 = mn1;
          const float p0 = ex2(x0 - mn0), p1 = ex2(x1 - mn1), p2 = ex2(x2 - mn0), p3 = ex2(x3 - mn1);
          l0 = l0 * al0 + p0 + p2;
          l1 = l1 * al1 + p1 + p3;
          if (__any_sync(0xffffffffu, (al0 != 1.f) | (al1 != 1.f))) {
#pragma unroll
            for (int t = 0; t < MT; ++t) {
              acc[t][0] *= al0; acc[t][1] *= al1; acc[t][2] *= al0; acc[t][3] *= al1;
            }
          }
          uint32_t hi01 = pack2<BF16>(p0, p1), hi23 = pack2<BF16>(p2, p3), lo01 = 0u, lo23 = 0u;
          if constexpr (BIAS || LOW) {
            const float2 h01 = unpack2<BF16>(hi01), h23 = unpack2<BF16>(hi23);
            lo01 = pack2<BF16>(p0 - h01.x, p1 - h01.y);
            lo23 = pack2<BF16>(p2 - h23.x, p3 - h23.y);
            if (low_cols) { hi01 = lo01; hi23 = lo23; }
          }
          const uint32_t pb0 = movmatrix_trans(hi01);
          const uint32_t pb1 = movmatrix_trans(hi23);

          // ---- O^T[D x 8] += V^T[D x 16] . P^T[16 x 8] ----
          // tile t: rows r and r + 8 are numbers 8 r + t and 64 + 8 r + t (D = 64: 8 r + t and 8 r + 4 + t) of the value rows
          auto add_pv = [&](uint32_t b0, uint32_t b1) {
#pragma unroll
            for (int t = 0; t < MT; ++t) {
              const uint32_t sel = (t & 1) ? 0x7632u : 0x5410u;
              const int w = t >> 1, c2 = D / 64 - 1, w2 = D == 128 ? w : w + 2;
              const uint32_t a0 = __byte_perm(u4_get(cur.v[0][0], w), u4_get(cur.v[1][0], w), sel);
              const uint32_t a1 = __byte_perm(u4_get(cur.v[0][c2], w2), u4_get(cur.v[1][c2], w2), sel);
              const uint32_t a2 = __byte_perm(u4_get(cur.v[2][0], w), u4_get(cur.v[3][0], w), sel);
              const uint32_t a3 = __byte_perm(u4_get(cur.v[2][c2], w2), u4_get(cur.v[3][c2], w2), sel);
              mma16816<BF16>(acc[t], a0, a1, a2, a3, b0, b1);
            }
          };
          add_pv(pb0, pb1);
          if constexpr (BIAS) {
            if (G > 4) add_pv(movmatrix_trans(lo01), movmatrix_trans(lo23));   // no free columns: a second product
          }
        } else {
          if (lane == 0) mbar_arrive(&bar_empty[ks_slot]);
          mbar_wait(&bar_full[vs_slot], v_par);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_empty[vs_slot]);
      }
    };
    // two loops, the long heads' first: 16 x 10240 rows take 114.1 us so, 115.3 with the other one first, 115.7 with one loop and
    // branches in it
    if (__builtin_expect(!low_parts, 1)) stream_units(std::false_type{});
    else stream_units(std::true_type{});

    if (tid == 0) DEC_TRACE(3);
    // ---- per-warp state -> smem ----
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      l0 += __shfl_xor_sync(0xffffffffu, l0, o);
      l1 += __shfl_xor_sync(0xffffffffu, l1, o);
    }
    if (low_parts) {   // the low parts' products join their columns
#pragma unroll
      for (int t = 0; t < MT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float low = __shfl_xor_sync(0xffffffffu, acc[t][e], 2);
          // the sum over an infinite value is infinite; its low part may be of the other sign, or 0 times infinity
          if (BIAS || fabsf(acc[t][e]) < INFINITY) acc[t][e] += low;
        }
    }
    {
      float* mw = s_merge + warp * G * ROW;
      const int q0 = 2 * j, q1 = 2 * j + 1;  // query columns of this lane; only q < G exist
      constexpr int kRow2 = D == 128 ? 64 : 4;   // where a tile's second eight rows lie (see add_pv)
      if (q0 < G) {
#pragma unroll
        for (int t = 0; t < MT; t += 2) {
          *reinterpret_cast<float2*>(mw + q0 * ROW + 8 * r + t) = make_float2(acc[t][0], acc[t + 1][0]);
          *reinterpret_cast<float2*>(mw + q0 * ROW + kRow2 + 8 * r + t) = make_float2(acc[t][2], acc[t + 1][2]);
        }
        if (r == 0) { mw[q0 * ROW + D] = m0; mw[q0 * ROW + D + 1] = l0; }
      }
      if (q1 < G) {
#pragma unroll
        for (int t = 0; t < MT; t += 2) {
          *reinterpret_cast<float2*>(mw + q1 * ROW + 8 * r + t) = make_float2(acc[t][1], acc[t + 1][1]);
          *reinterpret_cast<float2*>(mw + q1 * ROW + kRow2 + 8 * r + t) = make_float2(acc[t][3], acc[t + 1][3]);
        }
        if (r == 0) { mw[q1 * ROW + D] = m1; mw[q1 * ROW + D + 1] = l1; }
      }
    }
    cons_bar();

    // ---- merge the 8 warps' rows: put(q, pair, O (unnormalised), m, l) ----
    auto fold_warps = [&](auto put) {
      for (int e = tid; e < G * (D / 2); e += kDecCons) {
        const int q = e / (D / 2), d2 = e - q * (D / 2);
        float2 ml[kDecWarps], o = make_float2(0.f, 0.f);
        float M = -INFINITY, l = 0.f;
#pragma unroll
        for (int w = 0; w < kDecWarps; ++w) {
          ml[w] = *reinterpret_cast<const float2*>(s_merge + (w * G + q) * ROW + D);
          M = fmaxf(M, ml[w].x);
        }
#pragma unroll
        for (int w = 0; w < kDecWarps; ++w) {
          const float2 v = *reinterpret_cast<const float2*>(s_merge + (w * G + q) * ROW + 2 * d2);
          const float sc = (ml[w].x > -INFINITY) ? ex2(ml[w].x - M) : 0.f;
          l += ml[w].y * sc;
          o.x += v.x * sc;
          o.y += v.y * sc;
        }
        put(q, d2, o, M, l);
      }
    };
    auto write_out = [&](int q, int d2, float2 o, float M, float l) {
      float inv = l > 0.f ? 1.f / l : 0.f;
      if constexpr (BIAS) inv = bias_inv(p, h * G + q, M, l);
      out_row(b, h)[q * (D / 2) + d2] = pack2<BF16>(o.x * inv, o.y * inv);
    };

    const bool whole = (ua == 0) && (ub == h_end - h_beg);
    if (whole) {
      fold_warps(write_out);
    } else {
      // publish the partial, then take a ticket; the CTA completing the head merges
      float* slot = p.scratch + (int64_t)(head + c) * G * ROW;
      fold_warps([&](int q, int d2, float2 o, float M, float l) {
        __stcg(reinterpret_cast<float2*>(slot + q * ROW + 2 * d2), o);
        if (d2 == 0) __stcg(reinterpret_cast<float2*>(slot + q * ROW + D), make_float2(M, l));
      });
      cons_bar();
      if constexpr (BIAS) {   // s_merge reused by the next segment; bias_decode_fold_kernel merges
        u = seg_end;
        continue;
      }
      if (tid == 0) {
        __threadfence();      // the CTA's partial (behind the barrier) before its ticket
        const int done = atomicAdd(p.counters + head, ub - ua) + (ub - ua);
        __threadfence();
        s_last = (done == h_end - h_beg);
      }
      cons_bar();
      if (tid == 0) DEC_TRACE(6);
      if (s_last) {
        if (G <= 4) fold_slots<4, 3>(p.scratch, s_merge, head, G, h_beg, h_end, U, C);
        else fold_slots<8, 1>(p.scratch, s_merge, head, G, h_beg, h_end, U, C);
        cons_bar();
        if (tid == 0) DEC_TRACE(7);
        fold_warps(write_out);
        if (tid == 0) p.counters[head] = 0;
      }
    }
    cons_bar();  // s_merge reused by the next segment
#ifdef CVLLM_DECODE_TRACE
    if (tid == 0 && p.trace) {
      DEC_TRACE(4);
      p.trace[blockIdx.x * 8 + 5] = (unsigned long long)(whole ? 0 : (s_last ? 2 : 1));
    }
#endif
    u = seg_end;
  }
}

// Folds the partial states of the heads that the split cut (BIAS): a CTA per query head, which recomputes the split; a warp
// per every eighth slot, whose loads are all independent (a single KV head's rows may lie in as many slots as there are
// CTAs: with a CTA per KV head and the slots one after the other 1 x 16000 keys of
// 8 / 1 heads took 122 us with norms and cache write, 26 us so).
template <int D>
__global__ void __launch_bounds__(256) bias_decode_fold_kernel(const BiasDecodeParams p, int C) {
  constexpr int ROW = D + 2, PER = D / 32;
  const int hq = blockIdx.x % p.HQ, b = blockIdx.x / p.HQ, G = p.G, h = hq / G, q = hq - h * G, head = b * p.HKV + h;
  __shared__ float s_o[8][D];
  __shared__ float s_l[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int before = 0, all = 0, most = 0;   // units of the sequences before, of all, of the longest
  for (int i = lane; i < p.B; i += 32) {
    const int n = UnitList(p, i).count;
    most = max(most, n);
    all += n;
    if (i < b) before += n;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    before += __shfl_xor_sync(0xffffffffu, before, o);
    all += __shfl_xor_sync(0xffffffffu, all, o);
  }
  const int n = UnitList(p, b).count;
  pdl_wait();   // for the states (what is read above was there when the kernel in front let this one start)
  if (n == 0) return;
  const int U = all * p.HKV, h_beg = before * p.HKV + h * n;
  if (heads_whole(__reduce_max_sync(0xffffffffu, most), U, C)) return;
  const HeadStates states(h_beg, h_beg + n, U, C);
  if (states.n == 1) return;   // one CTA had the whole head and has written it
  auto row = [&](int k) { return p.scratch + ((int64_t)(head + states.cta(k)) * G + q) * ROW; };
  float M = -INFINITY;
  for (int k = lane; k < states.n; k += 32) M = fmaxf(M, __ldcg(row(k) + D));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xffffffffu, M, o));
  float acc[PER], l = 0.f;
#pragma unroll
  for (int i = 0; i < PER; ++i) acc[i] = 0.f;
#pragma unroll 4
  for (int k = warp; k < states.n; k += 8) {
    const float* x = row(k);
    const float w = ex2(__ldcg(x + D) - M);
    l = fmaf(__ldcg(x + D + 1), w, l);
#pragma unroll
    for (int i = 0; i < PER; i += 2) {
      const float2 v = __ldcg(reinterpret_cast<const float2*>(x + i * 32 + 2 * lane));
      acc[i] = fmaf(v.x, w, acc[i]);
      acc[i + 1] = fmaf(v.y, w, acc[i + 1]);
    }
  }
#pragma unroll
  for (int i = 0; i < PER; i += 2) {
    s_o[warp][i * 32 + 2 * lane] = acc[i];
    s_o[warp][i * 32 + 2 * lane + 1] = acc[i + 1];
  }
  if (lane == 0) s_l[warp] = l;
  __syncthreads();
  if (threadIdx.x < D / 2) {
    float x = 0.f, y = 0.f, sum = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      x += s_o[w][2 * threadIdx.x];
      y += s_o[w][2 * threadIdx.x + 1];
      sum += s_l[w];
    }
    const float inv = bias_inv(p, hq, M, sum);
    reinterpret_cast<uint32_t*>(p.out)[b * (p.o_stride / 2) + hq * (D / 2) + threadIdx.x] = pack2<true>(x * inv, y * inv);
  }
}

}  // namespace cvllm

using namespace cvllm;

static unsigned long long* g_decode_trace = nullptr;
// profiling only: device buffer of 8 x #CTAs uint64 that the next decode launches stamp (nullptr: off).
// Returns 0 when the library was built with -DCVLLM_DECODE_TRACE, -1 when the stamps are compiled out.
extern "C" int cvllm_debug_decode_trace(void* dev_buf) {
  g_decode_trace = reinterpret_cast<unsigned long long*>(dev_buf);
#ifdef CVLLM_DECODE_TRACE
  return 0;
#else
  return -1;
#endif
}

static int decode_ctas(int num_ctas) { return num_ctas > 0 ? num_ctas : sm_count(); }
static size_t decode_counter_bytes(size_t BH) { return (BH * 4 + 255) & ~(size_t)255; }

extern "C" size_t cvllm_decode_attention_workspace_bytes(int B, int HQ, int HKV, int D, int num_ctas) {
  if (B <= 0 || HKV <= 0 || HQ <= 0) return 0;
  const int G = HQ / HKV;
  const size_t BH = (size_t)B * HKV;
  const size_t slots = BH + (size_t)decode_ctas(num_ctas);
  return decode_counter_bytes(BH) + slots * G * (D + 2) * sizeof(float);
}

// Shared memory of a launch: the merge rows, the prefix of the heads' units, as many 32 KB slots as fit beside them (6 for G <= 4, else 5;
// fewer for thousands of heads), and the table of slot numbers where it costs no ring slot.  False: not even two slots fit.
static bool decode_smem(DecodeParams& p, int D, bool want_map, size_t& bytes) {
  const size_t fixed = 1024 + 2 * kMaxSlots * 8 + (size_t)kDecWarps * p.G * (D + 2) * 4 + ((size_t)p.B * p.HKV + 1) * 4;
  const size_t map = want_map ? (size_t)p.B * 4 : 0;
  if (fixed + 2 * (size_t)kSlotBytes > (size_t)kDecMaxSmem) return false;
  p.slots = (int)std::min<size_t>(kMaxSlots, (kDecMaxSmem - fixed) / kSlotBytes);
  bytes = fixed + (size_t)p.slots * kSlotBytes;
  p.map_in_smem = want_map && bytes + map <= (size_t)kDecMaxSmem;
  if (p.map_in_smem) bytes += map;
  return true;
}

static int launch_decode_attn(const void* q, void* out, const void* k_cache, const void* v_cache,
                              const int32_t* seq_lens_bh, const int32_t* page_table,
                              const int32_t* batch_mapping, void* workspace, size_t workspace_bytes, int B,
                              int HQ, int HKV, int D, int PS, int NLP, float sm_scale, int dtype,
                              int num_ctas, int lens_by_slot, cvllm_stream_t stream) {
  CVLLM_CHECK_ARG(B >= 0 && HQ > 0 && HKV > 0 && PS > 0 && NLP > 0);
  if (B == 0) return CVLLM_OK;
  CVLLM_CHECK_ARG(q && out && k_cache && v_cache && seq_lens_bh && page_table && batch_mapping &&
                  workspace);
  CVLLM_CHECK_ARG(HQ % HKV == 0);
  CVLLM_CHECK_ARG(dtype == CVLLM_F16 || dtype == CVLLM_BF16);
  const int G = HQ / HKV;
  CVLLM_CHECK_SUPPORTED(D == 128);
  CVLLM_CHECK_SUPPORTED(G <= 8);
  // a TMA box (min(PS,128) rows) must tile the 128-token unit and never cross a page
  CVLLM_CHECK_SUPPORTED(PS % kUnit == 0 || PS == 64 || PS == 32 || PS == 16);
  CVLLM_CHECK_ALIGN(aligned16(q) && aligned16(out) && aligned16(k_cache) && aligned16(v_cache) &&
                    aligned16(workspace));
  const int C = decode_ctas(num_ctas);
  CVLLM_CHECK_ARG(workspace_bytes >= cvllm_decode_attention_workspace_bytes(B, HQ, HKV, D, num_ctas));
  const size_t BH = (size_t)B * HKV;
  const size_t counters_bytes = decode_counter_bytes(BH);
  auto st = static_cast<cudaStream_t>(stream);

  DecodeParams p;
  p.q = q; p.out = out;
  p.seq_lens_bh = seq_lens_bh; p.page_table = page_table; p.batch_mapping = batch_mapping;
  p.counters = reinterpret_cast<int32_t*>(workspace);
  p.scratch = reinterpret_cast<float*>(reinterpret_cast<char*>(workspace) + counters_bytes);
  p.B = B; p.HQ = HQ; p.HKV = HKV; p.G = G; p.PS = PS; p.NLP = NLP;
  p.box_rows = PS < kUnit ? PS : kUnit;
  p.lens_by_slot = lens_by_slot;
  p.scale_log2 = sm_scale * 1.4426950408889634f;
#ifdef CVLLM_DECODE_TRACE
  p.trace = g_decode_trace;
#endif
  p.mode = test_options().decode_mode.load(std::memory_order_relaxed);

  // 2-D maps over the flat [rows, D] caches; the row bound is not known to this ABI (only
  // mapped pages are ever addressed), so it is the largest int32 coordinate
  const bool bf16 = dtype == CVLLM_BF16;
  CUtensorMap tm_k, tm_v;
  {
    const uint32_t box[2] = {64, (uint32_t)p.box_rows};
    const uint64_t dims[2] = {(uint64_t)D, (uint64_t)0x7fffffff};
    const uint64_t strides[1] = {(uint64_t)D * 2};
    int rc = make_tmap_16b(&tm_k, k_cache, 2, dims, strides, box, bf16);
    if (rc) return rc;
    rc = make_tmap_16b(&tm_v, v_cache, 2, dims, strides, box, bf16);
    if (rc) return rc;
  }

  size_t smem = 0;
  CVLLM_CHECK_SUPPORTED(decode_smem(p, D, true, smem));
  {
    const int cap = test_options().decode_slots.load(std::memory_order_relaxed);  // profiling knob
    if (cap >= 2 && cap < p.slots) p.slots = cap;
  }
  // raise the dynamic-smem cap once per (kernel, device)
  static std::atomic<uint64_t> attr_bf{0}, attr_h{0};
  if (bf16) CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)decode_attn_kernel<true, 128>, kDecMaxSmem, attr_bf));
  else CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)decode_attn_kernel<false, 128>, kDecMaxSmem, attr_h));
  if (bf16) {
    CVLLM_CHECK_CUDA(launch_behind(decode_attn_kernel<true, 128>, dim3(C), dim3(kDecThreads), smem, st, tm_k, tm_v, p));
  } else {
    CVLLM_CHECK_CUDA(launch_behind(decode_attn_kernel<false, 128>, dim3(C), dim3(kDecThreads), smem, st, tm_k, tm_v, p));
  }
  CVLLM_CHECK_LAUNCH();
  return CVLLM_OK;
}

// What the streaming kernel serves of the biased attention's decode steps (bfloat16, contiguous 16-byte aligned rows), and
// the scratch that it needs there.
bool cvllm_bias_decode_serves(int B, int H, int G, int D, int page_size, int64_t o_stride) {
  return (D == 128 || D == 64) && H / G <= 8 && (int64_t)B * G <= 4096 && o_stride % 2 == 0 &&
         (page_size % kUnit == 0 || page_size == 64 || page_size == 32 || page_size == 16);
}
extern "C" size_t cvllm_bias_decode_workspace_bytes(int B, int H, int G, int D) {
  if (B <= 0 || H <= 0 || G <= 0) return 0;
  return ((size_t)B * G + (size_t)sm_count()) * (H / G) * (D + 2) * sizeof(float);
}

int cvllm_launch_bias_decode(const void* q, const void* k_cache, const void* v_cache, int64_t cache_rows, void* out,
                             int64_t o_stride, const int32_t* positions, const int32_t* batch_mapping,
                             const int32_t* page_table, int64_t pt_slot, int64_t pt_head, int B, int H, int G, int D, int PS,
                             float scale, const float* slopes, int chunk, int window, int keep, const float* dist_bias,
                             int dist_rows, int sink, const float* sink_logits, int reserved_slot, float* workspace,
                             cudaStream_t st) {
  BiasDecodeParams p = {};
  p.q = q; p.out = out;
  p.page_table = page_table; p.batch_mapping = batch_mapping;
  p.scratch = workspace;
  p.B = B; p.HQ = H; p.HKV = G; p.G = H / G; p.PS = PS;
  p.box_rows = PS < kUnit ? PS : kUnit;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.positions = positions; p.pt_slot = pt_slot; p.pt_head = pt_head; p.o_stride = o_stride;
  p.slopes = slopes; p.dist_bias = dist_bias; p.dist_rows = dist_rows;
  p.chunk = chunk; p.window = window; p.keep = keep; p.reserved_slot = reserved_slot;
  p.sink = sink ? 1.f : 0.f; p.sink_logits = sink ? sink_logits : nullptr;
  CUtensorMap tm_k, tm_v;
  {
    const uint32_t box[2] = {64, (uint32_t)p.box_rows};
    const uint64_t dims[2] = {(uint64_t)D, (uint64_t)cache_rows};
    const uint64_t strides[1] = {(uint64_t)D * 2};
    int rc = make_tmap_16b(&tm_k, k_cache, 2, dims, strides, box, true);
    if (rc) return rc;
    rc = make_tmap_16b(&tm_v, v_cache, 2, dims, strides, box, true);
    if (rc) return rc;
  }
  const int C = sm_count();
  size_t smem = 0;
  CVLLM_CHECK_SUPPORTED(decode_smem(p, D, false, smem));   // (the producer reads the slot numbers from memory)
  static std::atomic<uint64_t> attr_128{0}, attr_64{0};
  if (D == 128) {
    CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)decode_attn_kernel<true, 128, true>, kDecMaxSmem, attr_128));
    CVLLM_CHECK_CUDA(launch_behind(decode_attn_kernel<true, 128, true>, dim3(C), dim3(kDecThreads), smem, st, tm_k, tm_v, p));
    CVLLM_CHECK_LAUNCH();
    CVLLM_CHECK_CUDA(launch_behind(bias_decode_fold_kernel<128>, dim3(B * H), dim3(256), 0, st, p, C));
  } else {
    CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)decode_attn_kernel<true, 64, true>, kDecMaxSmem, attr_64));
    CVLLM_CHECK_CUDA(launch_behind(decode_attn_kernel<true, 64, true>, dim3(C), dim3(kDecThreads), smem, st, tm_k, tm_v, p));
    CVLLM_CHECK_LAUNCH();
    CVLLM_CHECK_CUDA(launch_behind(bias_decode_fold_kernel<64>, dim3(B * H), dim3(256), 0, st, p, C));
  }
  CVLLM_CHECK_LAUNCH();
  return CVLLM_OK;
}

extern "C" int cvllm_decode_attention(const void* q, void* out, const void* k_cache,
                                      const void* v_cache, const int32_t* seq_lens_bh,
                                      const int32_t* page_table, const int32_t* batch_mapping,
                                      void* workspace, size_t workspace_bytes, int B, int HQ, int HKV,
                                      int D, int PS, int NLP, float sm_scale, int dtype, int num_ctas,
                                      cvllm_stream_t stream) {
  return launch_decode_attn(q, out, k_cache, v_cache, seq_lens_bh, page_table, batch_mapping, workspace,
                            workspace_bytes, B, HQ, HKV, D, PS, NLP, sm_scale, dtype, num_ctas, 0, stream);
}

// One decode step of Attention.forward (layers/attention.py:133-160): append the new (b, h) rows, then attend,
// both indexing the cache's own bh_seq_lens table [Bmax+1, HKV] through batch_mapping — the reference's
// index_select / clone / index_copy_ of a gathered length copy around the two kernels disappear.
extern "C" int cvllm_decode_step(const void* key, const void* value, int64_t sk_b, int64_t sk_h,
                                 int64_t sv_b, int64_t sv_h, const void* q, void* out, void* k_cache,
                                 void* v_cache, int32_t* bh_seq_lens, const int32_t* page_table,
                                 const int32_t* batch_mapping, void* workspace, size_t workspace_bytes,
                                 int B, int HQ, int HKV, int D, int PS, int NLP, float sm_scale, int dtype,
                                 int reserved_batch, int num_ctas, cvllm_stream_t stream) {
  int rc = launch_decode_store(key, value, sk_b, sk_h, sv_b, sv_h, batch_mapping, bh_seq_lens, page_table,
                               k_cache, v_cache, B, HKV, D, PS, NLP, 2, reserved_batch, 1, stream);
  if (rc) return rc;
  return launch_decode_attn(q, out, k_cache, v_cache, bh_seq_lens, page_table, batch_mapping, workspace,
                            workspace_bytes, B, HQ, HKV, D, PS, NLP, sm_scale, dtype, num_ctas, 1, stream);
}
