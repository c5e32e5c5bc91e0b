// Attention with a distance bias, a chunk mask and a softmax sink on the tcgen05 pipeline of prefill_attn2.cu: bfloat16
// storage, key and value size 128 or 64, pages of 16, 32, 64 or a multiple of 128 rows, an even number of query heads per
// KV head.  Same roles (warps 0-7 softmax of two heads, warp 8 TMA producer, warp 9 UMMA
// issuer), same ring of five 32 KB slots, same TMEM layout and hand-offs; what differs:
//   * every key - the step's own tokens included - is already in the paged cache, so all K / V tiles are cache tiles
//     [128 j, 128 j + 127] of the sequence and the causal mask is positional: key position <= query position;
//   * tiles before the chunk (or the sliding window) of the query tile's first row are never loaded: the tile list is
//     the tiles that hold kept first tokens, if any, then the tiles from j_begin on;
//   * the softmax adds slope * (key position - query position) in log2 units to the scaled logits, masks keys outside
//     the row's chunk or window (the kept first tokens stay visible), and starts from (max 0, sum 1) when there is a sink;
//   * a learned bias per distance (DIST) comes out of shared memory: the two heads' columns of the table lie there in
//     log2 units with the slope's part added, so a row reads its 128 biases of a tile at consecutive addresses (and
//     the 32 rows of a warp 32 neighbouring words); tiles wholly beyond the table add one constant.  With heads of 128 the
//     ring gives up one of its five slots for the table.  One 4096-token portion, 32 / 8 heads of 128, window 1024, a table
//     of 1024 rows, with the q / k norms and the cache write: 725 us on mma.sync, 170 us here;
//   * EXACT: bias tables, heads of 64 and short pages came from bias_attn_varlen_mma_kernel, and must not be further from the
//     formula than there.  Every exponential is ex2, and P is the sum of two bfloat16 numbers (2^-17 relative), whose low
//     parts lie behind the high ones in the score's TMEM columns and take a second product with V.  With P in one part, a
//     polynomial for 3 of 8 pairs and a reference up to 2^8 below the row's maximum (which then is not an exact 1 in P)
//     these rows were 2.5 to 19 % further from 64 bits than on mma.sync; now they are 12 to 23 % nearer (the result's own
//     rounding is left).  P in one part with the reference at every new maximum takes as long and is 0.3 to 0.7 % further.
//     With the polynomial it is slower (the extra instructions are what bounds the tile).  Heads of 128 in whole pages without
//     a table have always run here with the polynomial and one part;
//   * pages shorter than a tile arrive in pieces of a page each; pieces past the last query's page are not loaded (the same
//     portion without a window: pages of 64 1293 -> 217 us, heads of 64 599 -> 174 us).
#include <stdlib.h>

#include "common.cuh"
#include "tile_order.cuh"
#include "tma.cuh"

namespace cvllm {

namespace pb {
constexpr int kBM = 128, kBN = 128;
constexpr int kBoxBytes = kBN * 64 * 2;    // one [128 x 64] swizzled box
// distances -kTabFront .. rows - 1 + kTabBack of a bias table lie in shared memory: a tile's rows and columns reach 254
// before distance 0 (masked) and, unless the whole tile is past the table, 254 beyond its last row (which they repeat)
constexpr int kTabFront = 256, kTabBack = 256, kTab = 4096;
constexpr int kMaxDistRows = kTab - kTabFront - kTabBack;
constexpr int kThreads = 384;              // 3 warpgroups
constexpr int kRegsSoftmax = 224, kRegsOther = 56;  // 2*128*224 + 128*56 = 64512 <= 65536
}  // namespace pb

struct PrefillBiasParams {
  void* out;
  const int32_t* seq_start;   // [B] position of each sequence's first query of this step
  const float* slopes;        // [HQ] or NULL
  const int32_t* page_table;
  const int32_t* batch_mapping;
  const int32_t* cu_seqlens_q;
  int B, HQ, HKV, G, PS, NLP;
  int64_t o_stride_n;
  float scale_log2;
  float rescale_threshold;
  int chunk;                  // 0 = no chunking
  int window;                 // keys at distances 0 .. window - 1 (0 = no limit)
  int keep;                   // the sequence's first positions that stay visible whatever window and chunk say
  float sink;                 // 1 = a sink in the denominator, 0 = none
  const float* sink_logits;   // [HQ] the sink's score per head, or NULL (score 0)
  const float* dist_bias;     // [dist_rows][HQ] added to the score by distance (the last row beyond), DIST only
  int dist_rows;
  bool by_tile;               // the order of the query tiles (tile_order.cuh)
};

template <int HD, bool DIST>
struct PrefillBiasSmem {
  static constexpr int kTileBytes = pb::kBN * HD * 2;
  static constexpr int kSlots = HD == 128 && DIST ? 4 : 5;
  unsigned char q[2][kTileBytes];
  unsigned char kv[kSlots][kTileBytes];
  float table[DIST ? 2 : 1][DIST ? pb::kTab : 4];
  uint64_t q_full;
  uint64_t full[kSlots], empty[kSlots];
  uint64_t s_full[2], p_full[2];
  uint64_t p_half[2];   // P of the tile's first 64 keys is in TMEM: the PV UMMAs of those keys may start
  uint64_t o_done[2];   // one phase per PV_t(i)
  uint64_t o_final[2];  // last PV_t complete
  uint32_t tmem_base;
};

// kPolyPairsB = e: e of every 8 logit PAIRS take their exponentials on the FMA pipe (ex2_poly2_b) instead of the MUFU.
// An exponential occupies its scheduler's special-function unit for 8 cycles (16 per clock and SM); a few packed fp32x2
// operations do a PAIR on the FMA pipe instead.  Measured with the in-kernel trace
// (cycles per KV tile, together with the converged-warp UMMA issue below, P handed over at once): e = 0: 3161, 1: 3050,
// 2: 2881, 3: 2887, 4: 3218 — beyond a third the FMA-pipe work outweighs the MUFU time it frees.
#ifndef CVLLM_PREFILL_POLY_PAIRS
#define CVLLM_PREFILL_POLY_PAIRS 3
#endif
// P is handed to the issuer in two parts (the first kPSplitB 32-key pieces, then the rest): the first PV UMMAs run while
// the softmax group is still on the second part.  With the first, slower issuer this LOST 3 % (the issuer stalled in the
// middle of a group); with the converged-warp issue it takes another 230 cycles off the tile: trace, cycles per KV tile,
// polynomial pairs 3 of 8: split 0: 2887, 1: 2678, 2: 2647, 3: 2668 (and 3021 with 4 of 8 pairs).
#ifndef CVLLM_PREFILL_P_SPLIT
#define CVLLM_PREFILL_P_SPLIT 2
#endif
constexpr int kPSplitB = CVLLM_PREFILL_P_SPLIT;  // 32-key pieces of P handed to the issuer ahead of the rest (0: all at once)
constexpr int kPolyPairsB = CVLLM_PREFILL_POLY_PAIRS;
// 2^x for two values x <= ~8 with packed fp32x2 arithmetic: round-to-nearest split x = n + f (|f| <= 0.5), degree-3
// polynomial in f (relative error ~1e-4, far below the 2^-9 rounding of P to 16 bits), exponent added as an integer.
// Inputs below -125 (masked logits are -inf) flush to 2^-125, which the 16-bit P and the fp32 row sum take as 0.
__device__ __forceinline__ float2 ex2_poly2_b(float2 x) {
  x.x = fmaxf(x.x, -125.f);
  x.y = fmaxf(x.y, -125.f);
  const float2 magic = make_float2(12582912.f, 12582912.f);
  const float2 t = __fadd2_rn(x, magic);
  const float2 n = __fadd2_rn(t, make_float2(-12582912.f, -12582912.f));
  const float2 f = __ffma2_rn(n, make_float2(-1.f, -1.f), x);
  float2 p = __ffma2_rn(f, make_float2(0.05550357f, 0.05550357f), make_float2(0.24022652f, 0.24022652f));
  p = __ffma2_rn(p, f, make_float2(0.69314575f, 0.69314575f));
  p = __ffma2_rn(p, f, make_float2(1.f, 1.f));
  return make_float2(__int_as_float(__float_as_int(p.x) + (__float_as_int(t.x) << 23)),
                     __int_as_float(__float_as_int(p.y) + (__float_as_int(t.y) << 23)));
}

// What rounding two probabilities to bfloat16 has left over, itself as bfloat16.
__device__ __forceinline__ uint32_t rounded_off(float2 e, uint32_t hi) {
  const float2 r = __fadd2_rn(e, make_float2(-__uint_as_float(hi << 16), -__uint_as_float(hi & 0xffff0000u)));
  return pack2<true>(r.x, r.y);
}

#ifdef CVLLM_PREFILL_TRACE  // profiling build only (tools/trace_prefill.py): clock64 stamps of CTA (0,0,0), first 256 KV tiles
__device__ long long g_pb_trace[8][256];
#define P2_TRACE(rowi, jj)                                                                              \
  do {                                                                                                  \
    if (blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0 && lane == 0 && (jj) < 256) g_pb_trace[rowi][jj] = clock64(); \
  } while (0)
#else
#define P2_TRACE(rowi, jj) do { } while (0)
#endif

template <int kHD, bool DIST, bool EXACT>
__global__ void __launch_bounds__(pb::kThreads, 1)
prefill_attn_bias_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kc,
                         const __grid_constant__ CUtensorMap tm_vc, const PrefillBiasParams p) {
  using namespace pb;
  using Smem = PrefillBiasSmem<kHD, DIST>;
  constexpr bool BF16 = true;
  constexpr int kPoly = EXACT ? 0 : kPolyPairsB;
  constexpr int kSlots = Smem::kSlots, kTileBytes = Smem::kTileBytes, kBoxes = kHD / 64;
  extern __shared__ unsigned char smem_raw[];
  Smem& sm = *reinterpret_cast<Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_wait();      // the launch is scheduled beside the norm and store in front
  TileOrder at = {(int)(gridDim.x - 1 - blockIdx.x), (int)blockIdx.y, (int)blockIdx.z};
  int q_beg = p.cu_seqlens_q[at.b], q_end = p.cu_seqlens_q[at.b + 1], start = p.seq_start[at.b];
  if (p.by_tile && pasts_are_short(p.seq_start, p.B, kBM)) {   // (behind the loads above: see prefill_attn2.cu)
    at = tile_order();
    q_beg = p.cu_seqlens_q[at.b], q_end = p.cu_seqlens_q[at.b + 1], start = p.seq_start[at.b];
  }
  const int b = at.b;
  const int hq0 = 2 * at.pair;  // heads hq0, hq0 + 1 share KV head hkv (G even)
  const int hkv = hq0 / p.G;
  const int La = q_end - q_beg;
  const int n_qt = (La + kBM - 1) / kBM;
  const int qt = at.qt;  // heaviest (latest) tiles first
  if (qt >= n_qt) return;
  const int q0 = qt * kBM;
  const int p0 = start + q0;                               // position of the tile's first query
  const int p_last = p0 + min(kBM, La - q0) - 1;           // ... and of its last valid one
  auto first_key = [&](int pi) {                           // first position a query at pi sees through chunk and window
    int lo = p.chunk > 0 ? (pi / p.chunk) * p.chunk : 0;
    if (p.window > 0) lo = max(lo, pi - p.window + 1);
    return lo;
  };
  const int lo0 = first_key(p0);
  const int j_begin = lo0 / kBN;
  const int n_kept = min((min(p.keep, lo0) + kBN - 1) / kBN, j_begin);   // tiles of kept first tokens before j_begin
  const int n_tiles = n_kept + p_last / kBN - j_begin + 1;               // then the tiles j_begin .. p_last / 128
  const int j_skip = j_begin - n_kept;
  auto tile_base = [&](int j) { return (j < n_kept ? j : j + j_skip) * kBN; };   // first position of the list's tile j
  const int last_valid = p_last + 1 - (p_last / kBN) * kBN;  // keys of the last tile at or before p_last

  // ---------------- setup ----------------
  if (threadIdx.x == 0) {
    mbar_init(&sm.q_full, 1);
    for (int s = 0; s < kSlots; ++s) {
      mbar_init(&sm.full[s], 1);
      mbar_init(&sm.empty[s], 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(&sm.s_full[t], 1);
      mbar_init(&sm.p_full[t], 128);
      mbar_init(&sm.p_half[t], 128);
      mbar_init(&sm.o_done[t], 1);
      mbar_init(&sm.o_final[t], 1);
    }
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  if (warp == 8 && lane == 0) {
    tma_prefetch_desc(&tm_q);
    tma_prefetch_desc(&tm_kc);
    tma_prefetch_desc(&tm_vc);
  }
  if constexpr (DIST) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const float slope = p.slopes ? p.slopes[hq0 + t] : 0.f;
      for (int i = threadIdx.x; i < p.dist_rows + kTabFront + kTabBack; i += kThreads) {
        const int n = i - kTabFront;
        const float r = p.dist_bias[(int64_t)min(max(n, 0), p.dist_rows - 1) * p.HQ + hq0 + t];
        sm.table[t][i] = (r - slope * (float)n) * 1.4426950408889634f;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp == 8) {
    // =========================== TMA producer ===========================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
    if (lane == 0) {
      mbar_expect_tx(&sm.q_full, 2 * kTileBytes);
#pragma unroll
      for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int x = 0; x < kBoxes; ++x)
          tma_load_3d(sm.q[t] + x * kBoxBytes, &tm_q, &sm.q_full, 64 * x, hq0 + t, q_beg + q0);
      const int piece = min(p.PS, kBN), last_page = p_last / p.PS;   // rows of a box
      const int32_t* pt = p.page_table + ((int64_t)p.batch_mapping[b] * p.HKV + hkv) * p.NLP;
      for (int n = 0; n < 2 * n_tiles; ++n) {
        const int j = n >> 1;
        const bool is_v = n & 1;
        const int slot = n % kSlots;
        const uint32_t ph = (n / kSlots) & 1;
        const int t0 = tile_base(j);
        const int pg = t0 / p.PS;
        mbar_wait(&sm.empty[slot], ph ^ 1);
#ifdef CVLLM_PROBE_NO_TMA  // timing probe only (wrong results): K / V tiles are never fetched
        mbar_arrive(&sm.full[slot]);
        continue;
#endif
        unsigned char* dst = sm.kv[slot];
        const CUtensorMap* m = is_v ? &tm_vc : &tm_kc;
        const int pieces = min(kBN / piece, last_page - pg + 1);
        mbar_expect_tx(&sm.full[slot], pieces * piece * kHD * 2);
        for (int i = 0; i < pieces; ++i) {
          const int row = pt[pg + i] * p.PS + (t0 - pg * p.PS);   // the offset is 0 in pages shorter than a tile
#pragma unroll
          for (int x = 0; x < kBoxes; ++x)
            tma_load_2d(dst + x * kBoxBytes + i * piece * 128, m, &sm.full[slot], 64 * x, row);
        }
      }
    }
  } else if (warp == 9) {
    // ============================ UMMA issuer ============================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
    constexpr uint32_t idesc_qk = umma_idesc(BF16, kBM, kBN, false, false);
    constexpr uint32_t idesc_pv = umma_idesc(BF16, kBM, kHD, false, true);

    auto slot_of = [](int n) { return n % kSlots; };
    auto phase_of = [](int n) { return (uint32_t)((n / kSlots) & 1); };

    // The issuing thread is on the critical path of every hand-off (tools/trace_prefill.py: 86 cycles per UMMA in the
    // loop against 64 on the pipe).  Two things keep its per-UMMA work small (measured with that trace): the TMEM base is
    // made provably warp-uniform (a shuffle from lane 0), and a descriptor is its tile's base descriptor plus a constant
    // (the 14-bit start-address field cannot carry: shared memory ends below 256 KB) instead of a shift and two masks.
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);
    auto desc_at = [](uint64_t base, uint32_t byte_off) {
      return (base & 0xffffffff00000000ull) | (uint64_t)((uint32_t)base + (byte_off >> 4));
    };
    const uint64_t q_desc[2] = {umma_smem_desc(smem_u32(sm.q[0]), 16, 1024), umma_smem_desc(smem_u32(sm.q[1]), 16, 1024)};

    // S_t = Q_t . K_j^T  (K_j in ring entry 2j, already waited for)
    auto issue_qk = [&](int t, int j) {
      const uint64_t k_desc = umma_smem_desc(smem_u32(sm.kv[slot_of(2 * j)]), 16, 1024);
      const uint32_t s_tmem = tmem_u + t * kBN;
#pragma unroll
      for (int kk = 0; kk < kHD / 16; ++kk) {
        const uint32_t off = (kk >> 2) * kBoxBytes + (kk & 3) * 32;
        umma_ss_warp(s_tmem, desc_at(q_desc[t], off), desc_at(k_desc, off), idesc_qk, kk > 0 ? 1u : 0u);
      }
      umma_commit_warp(&sm.s_full[t]);
      if (t == 1) umma_commit_warp(&sm.empty[slot_of(2 * j)]);
    };
    auto issue_pv = [&](int t, int j) {
      const uint64_t v_desc = umma_smem_desc(smem_u32(sm.kv[slot_of(2 * j + 1)]), kBoxBytes, 1024);
      const uint32_t p_tmem = tmem_u + t * kBN;
      const uint32_t o_tmem = tmem_u + 256 + t * kHD;
      auto pv = [&](int kk, bool first) {   // 16 keys
        umma_ts_warp(o_tmem, p_tmem + kk * 8, desc_at(v_desc, kk * 2048), idesc_pv, first ? 0u : 1u);
        if constexpr (EXACT) umma_ts_warp(o_tmem, p_tmem + kBN / 2 + kk * 8, desc_at(v_desc, kk * 2048), idesc_pv, 1u);
      };
#if CVLLM_PREFILL_P_SPLIT > 0
      mbar_wait(&sm.p_half[t], j & 1);
      P2_TRACE(2 * t, j);
      tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < 2 * kPSplitB; ++kk) pv(kk, j == 0 && kk == 0);
      mbar_wait(&sm.p_full[t], j & 1);
      tc_fence_after();
#pragma unroll
      for (int kk = 2 * kPSplitB; kk < kBN / 16; ++kk) pv(kk, false);
#else
      mbar_wait(&sm.p_full[t], j & 1);
      P2_TRACE(2 * t, j);
      tc_fence_after();
#pragma unroll
      for (int kk = 0; kk < kBN / 16; ++kk) pv(kk, j == 0 && kk == 0);
#endif
      if (t == 1) umma_commit_warp(&sm.empty[slot_of(2 * j + 1)]);
      umma_commit_warp(&sm.o_done[t]);
      if (j == n_tiles - 1) umma_commit_warp(&sm.o_final[t]);
    };
    auto wait_v = [&](int j) {
      const int n = 2 * j + 1;
      mbar_wait(&sm.full[slot_of(n)], phase_of(n));
      if (j == n_tiles - 1 && last_valid < kBN) {
        // last tile: rows after the tile's last query position may be uninitialised memory; P is
        // exactly 0 there but 0 * NaN would poison O, so zero those V rows.
        const int valid = last_valid;
        uint4* v4 = reinterpret_cast<uint4*>(sm.kv[slot_of(n)]);
        const uint4 z = make_uint4(0, 0, 0, 0);
        for (int idx = lane; idx < (kBN - valid) * 8 * kBoxes; idx += 32) {
          const int r = valid + idx / (8 * kBoxes), c = idx % (8 * kBoxes);  // 8 x 16B per row and box
          v4[(c >> 3) * (kBoxBytes / 16) + r * 8 + (c & 7)] = z;
        }
        fence_proxy_async_smem();
        __syncwarp();
      }
      if constexpr (EXACT) {
        // nor do keys before the first row's chunk or window, which share its tile, reach any row of this CTA: their
        // values may be infinite or NaN
        const int base = tile_base(j), hidden = min(lo0 - base, kBN), shown = max(p.keep - base, 0);   // rows shown .. hidden - 1
        if (hidden > shown) {
          uint4* v4 = reinterpret_cast<uint4*>(sm.kv[slot_of(n)]);
          for (int idx = lane; idx < (hidden - shown) * 8 * kBoxes; idx += 32) {
            const int r = shown + idx / (8 * kBoxes), c = idx % (8 * kBoxes);
            v4[(c >> 3) * (kBoxBytes / 16) + r * 8 + (c & 7)] = make_uint4(0, 0, 0, 0);
          }
          fence_proxy_async_smem();
          __syncwarp();
        }
      }
      tc_fence_after();
    };
    auto wait_k = [&](int j) {
      const int n = 2 * j;
      mbar_wait(&sm.full[slot_of(n)], phase_of(n));
      tc_fence_after();
    };

    mbar_wait(&sm.q_full, 0);
    wait_k(0);
    issue_qk(0, 0);
    issue_qk(1, 0);
    for (int j = 0; j < n_tiles; ++j) {
      const bool more = j + 1 < n_tiles;
      wait_v(j);
      issue_pv(0, j);
      if (more) {
        wait_k(j + 1);
        issue_qk(0, j + 1);
      }
      P2_TRACE(1, j);
      issue_pv(1, j);
      if (more) issue_qk(1, j + 1);
      P2_TRACE(3, j);
    }
  } else if (warp < 8) {
    // ====================== softmax / correction / epilogue ======================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    const int t = warp >> 2;        // which head of the pair
    const int quad = warp & 3;      // TMEM lane quadrant this warp may touch
    const int row = quad * 32 + lane;
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    const bool row_valid = (q0 + row) < La;
    const uint32_t s_tmem = tmem + t * kBN + lane_base;
    const uint32_t o_tmem = tmem + 256 + t * kHD + lane_base;
    // a sink: its score (log2 units, like every score here) and its term
    float m_ref = p.sink > 0.f ? (p.sink_logits ? p.sink_logits[hq0 + t] * 1.4426950408889634f : 0.f) : -INFINITY;
    float l = p.sink;
    const int pi = p0 + row;                                   // this thread's query position
    const int lo_i = first_key(pi);
    const int lo_max = first_key(p_last);
    const float slope2 = p.slopes ? p.slopes[hq0 + t] * 1.4426950408889634f : 0.f;
    // what the table's last row adds to every score beyond it
    const float far_bias = DIST ? p.dist_bias[(int64_t)(p.dist_rows - 1) * p.HQ + hq0 + t] * 1.4426950408889634f : 0.f;

    for (int j = 0; j < n_tiles; ++j) {
      mbar_wait(&sm.s_full[t], j & 1);
      if (quad == 0) P2_TRACE(4 + 2 * t, j);
      tc_fence_after();
#ifdef CVLLM_PROBE_NO_SOFTMAX  // timing probe only (wrong results): the issuer / TMA side alone — 6.4 ms at 32K
      tc_fence_before();
      mbar_arrive(&sm.p_half[t]);
      mbar_arrive(&sm.p_full[t]);
      if (quad == 0) P2_TRACE(5 + 2 * t, j);
      continue;
#endif
      float s[kBN];
#pragma unroll
      for (int c = 0; c < kBN / 32; ++c) {
        uint32_t tmp[32];
        tmem_ld32(s_tmem + c * 32, tmp);
#pragma unroll
        for (int i = 0; i < 32; ++i) s[c * 32 + i] = __uint_as_float(tmp[i]);
      }
      tc_wait_ld();

      // ---- logits in log2 units with the distance bias: s_c * scale + slope2 * (pj - pi), pj = base + c ----
      const int base = tile_base(j);
      {
        const float2 sc2 = make_float2(p.scale_log2, p.scale_log2), sl2 = make_float2(slope2, slope2);
        bool table = false;
        float off = slope2 * (float)(base - pi);
        if constexpr (DIST) {
          table = p0 - base - (kBN - 1) < p.dist_rows - 1;   // some row of the tile has a distance inside the table
          off += far_bias;
        }
        if (DIST && table) {
          const float* tb = sm.table[t] + kTabFront + (pi - base);
#pragma unroll
          for (int c = 0; c < kBN; c += 2) {
            const float2 v = __ffma2_rn(make_float2(s[c], s[c + 1]), sc2, make_float2(tb[-c], tb[-c - 1]));
            s[c] = v.x;
            s[c + 1] = v.y;
          }
        } else {
          const float2 off2 = make_float2(off, off);
#pragma unroll
          for (int c = 0; c < kBN; c += 2) {
            const float2 bias = __ffma2_rn(make_float2((float)c, (float)(c + 1)), sl2, off2);
            const float2 v = __ffma2_rn(make_float2(s[c], s[c + 1]), sc2, bias);
            s[c] = v.x;
            s[c + 1] = v.y;
          }
        }
      }
      // ---- masks (boundary tiles only): keys after the query, keys before the row's chunk or window ----
      if (base + kBN - 1 > p0 || base < lo_max) {
        const int c_hi = pi - base, c_lo = lo_i - base;   // visible columns: c_lo <= c <= c_hi, and kept ones
        const int c_keep = p.keep - base;
#pragma unroll
        for (int c = 0; c < kBN; ++c)
          if (c > c_hi || (c < c_lo && c >= c_keep)) s[c] = -INFINITY;
      }

      auto row_max = [&]() -> float {
        float mx0 = s[0], mx1 = s[1], mx2 = s[2], mx3 = s[3];
#pragma unroll
        for (int c = 4; c < kBN; c += 4) {
          mx0 = fmaxf(mx0, s[c]);
          mx1 = fmaxf(mx1, s[c + 1]);
          mx2 = fmaxf(mx2, s[c + 2]);
          mx3 = fmaxf(mx3, s[c + 3]);
        }
        // a row that sees no key of this tile (it lies before the row's chunk or window) keeps a finite reference; the
        // lowest there is, since any higher one would make lower scores weigh nothing among themselves
        return fmaxf(fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3)), -3.402823466e38f);
      };
      // O *= alpha, l *= alpha, m_ref <- m_to.  O holds PV(0..j-1); PV(j-1) may still be in flight.
      auto rescale_to = [&](float m_to) {
        const float alpha = ex2(m_ref - m_to);  // m_ref == -inf on the first tile -> 0
        m_ref = m_to;
        l *= alpha;
        if (j > 0) {
          mbar_wait(&sm.o_done[t], (j - 1) & 1);
          tc_fence_after();
#pragma unroll
          for (int c = 0; c < kHD / 32; ++c) {
            uint32_t o[32];
            tmem_ld32(o_tmem + c * 32, o);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            tmem_st32(o_tmem + c * 32, o);
          }
        }
      };
      // P = exp2(S*scale - m_ref) packed to 16 bit over the S columns; returns the row sum of this tile.
      // Packed fp32 pairs: one fp32x2 FMA scales and shifts two logits, one fp32x2 add sums two probabilities (A/B on B200,
      // 7.62-7.68 ms vs 7.95-8.05 ms scalar at 32K).
      auto write_p = [&]() -> float {
        const float neg_m = (m_ref == -INFINITY) ? 0.f : -m_ref;
        const float2 sc2 = make_float2(1.f, 1.f), nm2 = make_float2(neg_m, neg_m);   // the logits are scaled already
        float2 l2a = make_float2(0.f, 0.f), l2b = make_float2(0.f, 0.f);
#pragma unroll
        for (int c = 0; c < kBN / 32; ++c) {
          uint32_t pk[16], lo[EXACT ? 16 : 1];
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const float2 t0 = __ffma2_rn(make_float2(s[c * 32 + 2 * i], s[c * 32 + 2 * i + 1]), sc2, nm2);
            const float2 t1 = __ffma2_rn(make_float2(s[c * 32 + 2 * i + 2], s[c * 32 + 2 * i + 3]), sc2, nm2);
#ifdef CVLLM_PROBE_NO_EXP  // timing probe only (wrong results): the loop without its MUFU work — 7.6 ms, unchanged
            const float2 e0 = t0, e1 = t1;
#else
            // kPoly = e: e of every 8 logit pairs (two loop trips, four pairs each... slots b0 b2 b1 b3 a1 a3 a0 a2)
            const int slot = (i >> 1) & 3;
            const bool p1 = (kPoly >= 1 && slot == 0) || (kPoly >= 2 && slot == 2) || (kPoly >= 3 && slot == 1) ||
                            (kPoly >= 4 && slot == 3);
            const bool p0 = (kPoly >= 5 && slot == 1) || (kPoly >= 6 && slot == 3) || (kPoly >= 7 && slot == 0) ||
                            (kPoly >= 8 && slot == 2);
            const float2 e0 = p0 ? ex2_poly2_b(t0) : make_float2(ex2(t0.x), ex2(t0.y));
            const float2 e1 = p1 ? ex2_poly2_b(t1) : make_float2(ex2(t1.x), ex2(t1.y));
#endif
            l2a = __fadd2_rn(l2a, e0);
            l2b = __fadd2_rn(l2b, e1);
            pk[i] = pack2<BF16>(e0.x, e0.y);
            pk[i + 1] = pack2<BF16>(e1.x, e1.y);
            if constexpr (EXACT) {
              lo[i] = rounded_off(e0, pk[i]);
              lo[i + 1] = rounded_off(e1, pk[i + 1]);
            }
          }
          tmem_st16(s_tmem + c * 16, pk);
          if constexpr (EXACT) tmem_st16(s_tmem + kBN / 2 + c * 16, lo);
#if CVLLM_PREFILL_P_SPLIT > 0
          if (c == kPSplitB - 1) {  // the first part of P (and any O rescale before it) is in TMEM
            tc_wait_st();
            tc_fence_before();
            mbar_arrive(&sm.p_half[t]);
          }
#endif
        }
        return (l2a.x + l2b.x) + (l2a.y + l2b.y);
      };

      // The row maximum of the tile is known before the first exponential.  Taking it off the critical path
      // (exponentials against the previous tiles' reference, rescale deferred by one tile) was measured on B200
      // and changed nothing: 7.70-7.91 ms vs 7.60-7.80 ms at 32K — the chain of maxima already hides under the
      // TMEM load latency.
      {
        const float m_new = fmaxf(m_ref, row_max());
        const bool need = (j == 0) || (m_new > m_ref + p.rescale_threshold);
        if (__any_sync(0xffffffffu, need)) rescale_to(m_new);
        l += write_p();
      }
      tc_wait_st();
      tc_fence_before();
      mbar_arrive(&sm.p_full[t]);
      if (quad == 0) P2_TRACE(5 + 2 * t, j);
    }

    // ---- epilogue: O / l -> out ----
    mbar_wait(&sm.o_final[t], 0);
    tc_fence_after();
    const float inv = l > 0.f ? 1.f / l : 0.f;
    char* orow = reinterpret_cast<char*>(p.out) +
                 ((int64_t)(q_beg + q0 + row) * p.o_stride_n + (int64_t)(hq0 + t) * kHD) * 2;
#pragma unroll
    for (int c = 0; c < kHD / 32; ++c) {
      uint32_t o[32];
      tmem_ld32(o_tmem + c * 32, o);
      tc_wait_ld();
      if (row_valid) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          uint4 w;
          w.x = pack2<BF16>(__uint_as_float(o[8 * i + 0]) * inv, __uint_as_float(o[8 * i + 1]) * inv);
          w.y = pack2<BF16>(__uint_as_float(o[8 * i + 2]) * inv, __uint_as_float(o[8 * i + 3]) * inv);
          w.z = pack2<BF16>(__uint_as_float(o[8 * i + 4]) * inv, __uint_as_float(o[8 * i + 5]) * inv);
          w.w = pack2<BF16>(__uint_as_float(o[8 * i + 6]) * inv, __uint_as_float(o[8 * i + 7]) * inv);
          *reinterpret_cast<uint4*>(orow + c * 64 + i * 16) = w;
        }
      }
    }
  }

  else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));  // warps 10, 11
  }

  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, 512);
}

}  // namespace cvllm

using namespace cvllm;

// What the kernel serves, beside bfloat16 storage, an even number of query heads per KV head and contiguous page tables.
bool cvllm_prefill_bias_serves(int D, int Dv, int page_size, int dist_rows) {
  return D == Dv && (D == 128 || D == 64) &&
         (page_size % 128 == 0 || page_size == 64 || page_size == 32 || page_size == 16) && dist_rows <= pb::kMaxDistRows;
}

namespace {

template <int HD, bool DIST, bool EXACT>
int launch_bias(const CUtensorMap& tm_q, const CUtensorMap& tm_kc, const CUtensorMap& tm_vc, const PrefillBiasParams& p,
                int max_seqlen_q, cudaStream_t st) {
  const size_t smem = sizeof(PrefillBiasSmem<HD, DIST>) + 1024;
  static_assert(sizeof(PrefillBiasSmem<HD, DIST>) + 1024 <= 227 * 1024, "shared memory");
  const dim3 grid((max_seqlen_q + pb::kBM - 1) / pb::kBM, p.HQ / 2, p.B);
  static std::atomic<uint64_t> attr{0};
  CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)prefill_attn_bias_kernel<HD, DIST, EXACT>, (int)smem, attr));
  CVLLM_CHECK_CUDA(launch_behind(prefill_attn_bias_kernel<HD, DIST, EXACT>, grid, dim3(pb::kThreads), smem, st, tm_q, tm_kc, tm_vc, p));
  CVLLM_CHECK_LAUNCH();
  return CVLLM_OK;
}

}  // namespace

// Launch.  Called by cvllm_bias_attn_varlen (bias_attn.cu) for the shapes named at the top; returns a CVLLM_* code.
int cvllm_launch_prefill_bias(const void* q, const void* k_cache, const void* v_cache, int64_t cache_rows, void* out,
                              const int32_t* seq_start, const float* slopes, const int32_t* page_table,
                              const int32_t* batch_mapping, const int32_t* cu_seqlens_q, int B, int N, int HQ, int HKV, int HD,
                              int PS, int NLP, int max_seqlen_q, float scale, int chunk, int window, int keep, int sink,
                              const float* sink_logits, const float* dist_bias, int dist_rows, int64_t o_stride,
                              cudaStream_t st) {
  using namespace pb;
  CVLLM_CHECK_ALIGN(aligned16(q) && aligned16(out) && aligned16(k_cache) && aligned16(v_cache));
  CUtensorMap tm_q, tm_kc, tm_vc;
  {
    const uint32_t box3[3] = {64, 1, (uint32_t)kBM};
    const uint64_t dq[3] = {(uint64_t)HD, (uint64_t)HQ, (uint64_t)N};
    const uint64_t sq[2] = {(uint64_t)HD * 2, (uint64_t)HQ * HD * 2};
    int rc = make_tmap_16b(&tm_q, q, 3, dq, sq, box3, true);
    if (rc) return rc;
    const uint32_t box2[2] = {64, (uint32_t)(PS < kBN ? PS : kBN)};
    const uint64_t dc[2] = {(uint64_t)HD, (uint64_t)cache_rows};
    const uint64_t sc[1] = {(uint64_t)HD * 2};
    rc = make_tmap_16b(&tm_kc, k_cache, 2, dc, sc, box2, true);
    if (rc) return rc;
    rc = make_tmap_16b(&tm_vc, v_cache, 2, dc, sc, box2, true);
    if (rc) return rc;
  }
  PrefillBiasParams p;
  p.out = out; p.seq_start = seq_start; p.slopes = slopes; p.page_table = page_table;
  p.batch_mapping = batch_mapping; p.cu_seqlens_q = cu_seqlens_q;
  p.B = B; p.HQ = HQ; p.HKV = HKV; p.G = HQ / HKV; p.PS = PS; p.NLP = NLP;
  p.o_stride_n = o_stride;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.rescale_threshold = 8.0f;
  {
    const float t = test_options().prefill_threshold.load(std::memory_order_relaxed);
    if (t >= 0.f) p.rescale_threshold = t;
  }
  const bool exact = HD == 64 || dist_bias || PS % kBN;   // see the top
  p.chunk = chunk;
  p.window = window;
  p.keep = keep;
  p.sink = sink ? 1.f : 0.f;
  p.sink_logits = sink ? sink_logits : nullptr;
  p.dist_bias = dist_bias;
  p.dist_rows = dist_rows;
  p.by_tile = order_by_tile(dim3((max_seqlen_q + kBM - 1) / kBM, HQ / 2, B), N, kBM);
  if (HD == 64)
    return dist_bias ? launch_bias<64, true, true>(tm_q, tm_kc, tm_vc, p, max_seqlen_q, st)
                     : launch_bias<64, false, true>(tm_q, tm_kc, tm_vc, p, max_seqlen_q, st);
  if (dist_bias) return launch_bias<128, true, true>(tm_q, tm_kc, tm_vc, p, max_seqlen_q, st);
  return exact ? launch_bias<128, false, true>(tm_q, tm_kc, tm_vc, p, max_seqlen_q, st)
               : launch_bias<128, false, false>(tm_q, tm_kc, tm_vc, p, max_seqlen_q, st);
}

#ifdef CVLLM_PREFILL_TRACE
// profiling build only: copies the 8 x 256 clock64 stamps of the last launch's CTA (0,0,0) to host memory
extern "C" int cvllm_debug_prefill_bias_trace_read(void* host_out) {
  CVLLM_CHECK_CUDA(cudaDeviceSynchronize());
  CVLLM_CHECK_CUDA(cudaMemcpyFromSymbol(host_out, cvllm::g_pb_trace, sizeof(long long) * 8 * 256));
  return CVLLM_OK;
}
#endif
