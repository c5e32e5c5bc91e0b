// SnapKV observation-window scorer on tcgen05 (reference: compression/snapkv.py:39-276,332-448; K12 + K13).
//
// Rows = the last w query tokens x the G query heads of one kv head (w * G <= 256: R = 1 or 2 row tiles of 128), columns =
// 128-key tiles of the sequence's non-window keys.  A unit is a key tile against a row tile, R to a key tile, in turn
// through the four TMEM buffers.
// Two launches over the same (key split, kv head, sequence) grid, one CTA per split:
//   pass 1  S = Qwin . K_tile^T (lane = row, column = key): running (max, sum) of every row over the split's
//           keys -> stats[part][row]
//   pass 2  S^T = K_tile . Qwin^T (lane = key, column = row): column sums of exp2(s - m_row) / l_row with the
//           FINAL row statistics (all parts combined), causal kpool-tap mean inside pool_segment-key segments,
//           window keys <- +inf                                                            -> out[key, hk]
// Roles per CTA as in score_chunk_umma.cu: warp 8 TMA producer (Q window once: a 3-D box {64 d, G heads, w tokens}
// lands in shared memory already in row order (token, g); K tiles through a 4-slot ring), warp 9 UMMA issuer (four
// 128-column TMEM buffers), warps 0-7 two warpgroups.  Pass 1: the warpgroups take alternate tiles (with half the columns of every
// tile each they loaded TMEM at the same time and took exponentials at the same time), a thread keeps its row's 128
// logits in registers, and each writes its own partial statistics (parts = 2 x splits).  Pass 2: the warpgroups take
// alternate tiles; with the operands swapped a thread owns one KEY, so the sum over the rows stays in its registers, with the
// rows' statistics read from shared memory as broadcasts.  With lane = row it took 62 shuffles a thread, two barriers of
// all eight warps a tile and nothing to overlap them with.  40960 keys, 32 / 8 heads, both passes and the call: 88 -> 50 us
// with the splits below, 131072 keys 288 -> 130 us; error against 64 bits (rms, relative) 9.3e-8 -> 5.2e-8.
// What bounds the passes: pass 1 the read of K (84 MB of 40960 keys: 13 us), pass 2 the exponentials (128 x 128 a tile at 16
// per clock: 1024 clocks), both the start: a CTA holds the SM (TMEM, 200 KB of shared memory), so the grid runs in waves of 148
// CTAs and a start (barriers, TMEM, the first tile's latency, in pass 2 the statistics) costs as much as four tiles: see
// snap_split_tiles() for how many CTAs a call is cut into.  Alternate tiles in pass 1, a unit's row of TMEM in one load, all
// parts' statistics in flight together, and pass 2 launched while pass 1 ends: 50.0 -> 46.9 us, short prompts 18.2 -> 14.8.
// Two row tiles (16 / 2 heads, 32 tokens): 153 us on mma.sync, which served them, 26.6 here, and half the error.
// Two key tiles at a time in pass 2, to read the statistics once for both, took 33.8 us for 29.4: with nine pairs a CTA one
// warpgroup has a fifth more to do, and shared memory was not the bound.
#include <algorithm>

#include "common.cuh"
#include "tma.cuh"

namespace cvllm {

namespace sn {
constexpr int kTile = 128, kHD = 128;
constexpr int kTileBytes = kTile * kHD * 2;  // 32 KB
constexpr int kBoxBytes = kTileBytes / 2;
constexpr int kSlots = 4;
constexpr int kThreads = 384;
constexpr int kRegsSoftmax = 224, kRegsOther = 56;
constexpr int kMaxTilesManyCtas = 8;  // key tiles per CTA where (sequence, head) pairs alone fill the chip
}  // namespace sn

struct SnapUmmaParams {
  const int32_t* cu_q;
  const int32_t* cu_k;
  float* stats;  // [B, HKV, parts, 128, 2] partial (m, l) per row; parts = 2 * n_splits
  float* out;    // [Nk, HKV]
  int HKV, G, w, n_splits, split, kpool, pool_segment;  // split: keys per CTA, a multiple of 128
  float scale_log2;
};

struct SnapUmmaSmem {
  unsigned char q[2 * sn::kTileBytes];   // two halves of 64 numbers, each of 128 R rows
  unsigned char ring[sn::kSlots][sn::kTileBytes];
  float2 row_stat[2 * sn::kTile];  // pass 2: (-m, 1 / l) of every row; R = 1, second half: (m, l) of the other warpgroup
  float raw[2][2][sn::kTile];      // pass 2: [warpgroup][its tile's parity] column sums before the mean over taps
  uint64_t q_full;
  uint64_t full[sn::kSlots], empty[sn::kSlots];
  uint64_t s_full[4], s_empty[4];
  uint32_t tmem_base;
};

__device__ __forceinline__ void snap_bar_256() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ void snap_bar_wg(int wg) { asm volatile("bar.sync %0, 128;" ::"r"(2 + wg) : "memory"); }

template <bool BF16, bool PASS2, int R>
__global__ void __launch_bounds__(sn::kThreads, 1)
snap_umma_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const SnapUmmaParams p) {
  using namespace sn;
  extern __shared__ unsigned char smem_raw[];
  SnapUmmaSmem& sm = *reinterpret_cast<SnapUmmaSmem*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  // pass 2 is launched when the last CTAs of pass 1 are: its CTAs take over the SMs one by one, and set up, load and make
  // their first S while pass 1 ends elsewhere
  if constexpr (!PASS2) pdl_trigger();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sp = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
  const int kb = p.cu_k[b], len = p.cu_k[b + 1] - kb, q_end = p.cu_q[b + 1];
  const int rows = p.w * p.G;
  const int n_scored = len - p.w;  // keys [0, L - w) are scored, the window keys get +inf
  const int k_lo = sp * p.split;
  const int k_hi = min(n_scored, k_lo + p.split);  // scored keys of this split
  const int n_tiles = k_hi > k_lo ? (k_hi - k_lo + kTile - 1) / kTile : 0;
  const int parts = 2 * p.n_splits;
  float* st_base = p.stats + ((int64_t)b * p.HKV + hk) * parts * kTile * 2;

  if (n_tiles == 0) {  // uniform over the CTA; covers splits beyond the sequence (k_lo >= len) too
    // no scored key here: pass 1 publishes empty statistics; pass 2 writes +inf for window keys (0 when the whole
    // sequence is no longer than the window: the reference leaves those rows uninitialised, snapkv.py:94-95,204-205)
    if (!PASS2) {
      for (int i = threadIdx.x; i < 2 * kTile; i += kThreads) {
        float* st = st_base + ((int64_t)(2 * sp + i / kTile) * kTile + (i % kTile)) * 2;
        st[0] = -INFINITY;
        st[1] = 0.f;
      }
    } else {
      const float v = n_scored > 0 ? INFINITY : 0.f;
      for (int k = k_lo + threadIdx.x; k < min(len, k_lo + p.split); k += kThreads)
        p.out[(int64_t)(kb + k) * p.HKV + hk] = v;
      pdl_wait();   // nothing after this launch may begin before pass 1 is through
    }
    return;
  }

  if (threadIdx.x == 0) {
    mbar_init(&sm.q_full, 1);
    for (int i = 0; i < kSlots; ++i) { mbar_init(&sm.full[i], 1); mbar_init(&sm.empty[i], 1); }
    for (int i = 0; i < 4; ++i) { mbar_init(&sm.s_full[i], 1); mbar_init(&sm.s_empty[i], 128); }
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(&sm.tmem_base, 512);
    tmem_relinquish();
  }
  // rows >= w * G of the Q tile are never loaded: zero them (their logits are then 0, not NaN from stale smem)
  for (int i = threadIdx.x; i < (R * kTile - rows) * 16; i += kThreads) {
    const int r = rows + i / 16, c = i % 16;
    *reinterpret_cast<uint4*>(sm.q + (c >> 3) * R * kBoxBytes + r * 128 + (c & 7) * 16) = make_uint4(0, 0, 0, 0);
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp == 8) {
    // =========================== TMA producer ===========================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
    if (lane == 0) {
      mbar_expect_tx(&sm.q_full, 2 * rows * 128);
      tma_load_3d(sm.q, &tm_q, &sm.q_full, 0, hk * p.G, q_end - p.w);
      tma_load_3d(sm.q + R * kBoxBytes, &tm_q, &sm.q_full, 64, hk * p.G, q_end - p.w);
      for (int t = 0; t < n_tiles; ++t) {
        const int slot = t % kSlots;
        mbar_wait(&sm.empty[slot], ((t / kSlots) & 1) ^ 1);
        mbar_expect_tx(&sm.full[slot], kTileBytes);
        tma_load_3d(sm.ring[slot], &tm_k, &sm.full[slot], 0, hk, kb + k_lo + t * kTile);
        tma_load_3d(sm.ring[slot] + kBoxBytes, &tm_k, &sm.full[slot], 64, hk, kb + k_lo + t * kTile);
      }
    }
  } else if (warp == 9) {
    // ============================ UMMA issuer ============================
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));
    constexpr uint32_t idesc = umma_idesc(BF16, kTile, kTile, false, false);
    const uint32_t tmem_u = __shfl_sync(0xffffffffu, tmem, 0);  // provably warp-uniform for the compiler
    mbar_wait(&sm.q_full, 0);
    for (int t = 0; t < n_tiles; ++t) {
      const int slot = t % kSlots;
      mbar_wait(&sm.full[slot], (t / kSlots) & 1);
#pragma unroll
      for (int x = 0; x < R; ++x) {
        const int unit = t * R + x, buf = unit & 3;
        mbar_wait(&sm.s_empty[buf], ((unit >> 2) & 1) ^ 1);
        tc_fence_after();
        if (lane == 0) {
          const uint64_t q_desc = umma_smem_desc(smem_u32(sm.q) + x * kBoxBytes, 16, 1024);
          const uint64_t k_desc = umma_smem_desc(smem_u32(sm.ring[slot]), 16, 1024);
#pragma unroll
          for (int kk = 0; kk < kHD / 16; ++kk) {
            const uint64_t qd = umma_desc_add(q_desc, (kk >> 2) * R * kBoxBytes + (kk & 3) * 32);
            const uint64_t kd = umma_desc_add(k_desc, (kk >> 2) * kBoxBytes + (kk & 3) * 32);
            umma_ss(tmem_u + buf * kTile, PASS2 ? kd : qd, PASS2 ? qd : kd, idesc, kk > 0 ? 1u : 0u);
          }
          umma_commit(&sm.s_full[buf]);
          if (x == R - 1) umma_commit(&sm.empty[slot]);
        }
        __syncwarp();
      }
    }
  } else if (warp < 8) {
    // ====================== softmax statistics / column sums ======================
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsSoftmax));
    const int wg = warp >> 2, quad = warp & 3;
    const int row = quad * 32 + lane;  // TMEM lane: the query row (pass 1) or the key of the tile (pass 2)
    const int st = threadIdx.x;        // 0..255
    const uint32_t lane_base = (uint32_t)(quad * 32) << 16;
    if constexpr (!PASS2) {
      // the running statistics of the row over this warpgroup's units: every second tile, or with R = 2 its row tile's all
      float m_run = -INFINITY, l_run = 0.f;
      for (int unit = wg; unit < n_tiles * R; unit += 2) {
        const int buf = unit & 3;
        const int nk = min(kTile, k_hi - (k_lo + unit / R * kTile));  // scored keys in this tile
        mbar_wait(&sm.s_full[buf], (unit >> 2) & 1);
        tc_fence_after();
        float2 sv[kTile / 2];
#pragma unroll
        for (int c = 0; c < kTile / 32; ++c) {
          uint32_t r[32];
          tmem_ld32(tmem + buf * kTile + lane_base + 32 * c, r);
#pragma unroll
          for (int i = 0; i < 16; ++i) sv[16 * c + i] = make_float2(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
        }
        tc_wait_ld();
        tc_fence_before();
        mbar_arrive(&sm.s_empty[buf]);
        const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
#pragma unroll
        for (int i = 0; i < kTile / 2; ++i) sv[i] = __fmul2_rn(sv[i], sc2);
        if (nk < kTile) {
#pragma unroll
          for (int i = 0; i < kTile / 2; ++i) {
            if (2 * i >= nk) sv[i].x = -INFINITY;
            if (2 * i + 1 >= nk) sv[i].y = -INFINITY;
          }
        }
        float m0 = sv[0].x, m1 = sv[0].y, m2 = sv[1].x, m3 = sv[1].y;
#pragma unroll
        for (int i = 2; i < kTile / 2; i += 2) {
          m0 = fmaxf(m0, sv[i].x); m1 = fmaxf(m1, sv[i].y); m2 = fmaxf(m2, sv[i + 1].x); m3 = fmaxf(m3, sv[i + 1].y);
        }
        // The reference point is rounded up to a whole number: every later change of it, here and where the parts
        // meet, is then a power of two and adds no error (ex2's is one-sided and would add up along the chain).
        const float m_new = fmaxf(m_run, ceilf(fmaxf(fmaxf(m0, m1), fmaxf(m2, m3))));
        if (m_new > -INFINITY) {  // else: every key is masked so far
          const float2 nm2 = make_float2(-m_new, -m_new);
          float2 a[4];
#pragma unroll
          for (int i = 0; i < kTile / 2; ++i) {
            const float2 x = __fadd2_rn(sv[i], nm2), e = make_float2(ex2(x.x), ex2(x.y));
            a[i % 4] = i < 4 ? e : __fadd2_rn(a[i % 4], e);
          }
          const float2 u = __fadd2_rn(__fadd2_rn(a[0], a[1]), __fadd2_rn(a[2], a[3]));
          l_run = l_run * ex2(m_run - m_new) + (u.x + u.y);  // ex2(-inf) = 0 on the first live tile
          m_run = m_new;
        }
      }
      float* stp = st_base + ((int64_t)(2 * sp + wg) * kTile + row) * 2;
      stp[0] = m_run;
      stp[1] = l_run;
    } else {
      // the rows' final statistics: a thread combines one row's parts of one warpgroup (part & 1 == wg), then with R = 1 the
      // first 128 threads the two warpgroups'
      {
        pdl_wait();
        const float2* parts_of = reinterpret_cast<const float2*>(st_base) + (int64_t)wg * kTile + row;
        float M = -INFINITY, L = 0.f;
        constexpr int kAhead = 20;   // parts in flight together (one sequence of 8 KV heads has 18)
        for (int s0 = 0; s0 < p.n_splits; s0 += kAhead) {
          float2 ml[kAhead];
          float m = M;
#pragma unroll
          for (int s = 0; s < kAhead; ++s)
            ml[s] = s0 + s < p.n_splits ? parts_of[(int64_t)(s0 + s) * 2 * kTile] : make_float2(-INFINITY, 0.f);
#pragma unroll
          for (int s = 0; s < kAhead; ++s) m = fmaxf(m, ml[s].x);
          if (m > -INFINITY) {
            L *= ex2(M - m);          // whole references: a power of two
#pragma unroll
            for (int s = 0; s < kAhead; ++s) L += ml[s].y * ex2(ml[s].x - m);
            M = m;
          }
        }
        auto put = [&](int r, float m, float l) {
          sm.row_stat[r] = make_float2(m > -INFINITY ? -m : 0.f, (r < rows && l > 0.f) ? 1.f / l : 0.f);
        };
        if constexpr (R == 2) {
          put(wg * kTile + row, M, L);
        } else {
          if (wg == 1) sm.row_stat[kTile + row] = make_float2(M, L);
          snap_bar_256();
          if (wg == 0) {
            const float2 o = sm.row_stat[kTile + row];
            const float Mt = fmaxf(M, o.x);
            float Lt = 0.f;
            if (M > -INFINITY) Lt += L * ex2(M - Mt);
            if (o.x > -INFINITY) Lt += o.y * ex2(o.x - Mt);
            put(row, Mt, Lt);
          }
        }
        snap_bar_256();
      }
      const int blocks = (rows + 31) >> 5;  // 32-row column blocks that hold rows
      for (int t = wg; t < n_tiles; t += 2) {
        const int nk = min(kTile, k_hi - (k_lo + t * kTile));  // scored keys in this tile
        float total = 0.f;  // of at most four blocks a row tile, each a tree over eight chains of four: short chains of roundings
#pragma unroll
        for (int x = 0; x < R; ++x) {
          const int unit = t * R + x, buf = unit & 3;
          mbar_wait(&sm.s_full[buf], (unit >> 2) & 1);
          tc_fence_after();
          uint32_t r[4][32];   // the whole row: one wait a unit for TMEM, not four
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32(tmem + buf * kTile + lane_base + 32 * c, r[c]);
          tc_wait_ld();
          tc_fence_before();
          mbar_arrive(&sm.s_empty[buf]);
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (4 * x + c < blocks) {
              const float4* rs = reinterpret_cast<const float4*>(sm.row_stat + kTile * x + 32 * c);
              float a[8];
#pragma unroll
              for (int i = 0; i < 32; i += 2) {
                const float4 u = rs[i / 2];  // (-m, 1 / l) of two rows
                const float e0 = ex2(fmaf(__uint_as_float(r[c][i]), p.scale_log2, u.x));
                const float e1 = ex2(fmaf(__uint_as_float(r[c][i + 1]), p.scale_log2, u.z));
                a[i % 8] = i < 8 ? e0 * u.y : fmaf(e0, u.y, a[i % 8]);
                a[i % 8 + 1] = i < 8 ? e1 * u.w : fmaf(e1, u.w, a[i % 8 + 1]);
              }
              total += ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
            }
          }
        }
        // causal kpool-tap mean inside pool_segment-key segments (snapkv.py:253-262); window keys <- +inf.  The
        // buffer of this parity is written again two tiles on, behind the next tile's barrier, which every
        // reader of this one passes first
        float* raw = sm.raw[wg][(t >> 1) & 1];
        raw[row] = total;
        snap_bar_wg(wg);
        const int kabs = k_lo + t * kTile + row;
        if (kabs < len) {
          float v = INFINITY;
          if (row < nk) {
            const int lo = max(row - (p.kpool - 1), (row / p.pool_segment) * p.pool_segment);
            float s = 0.f;
            for (int u = lo; u <= row; ++u) s += raw[u];
            v = s / (float)(row + 1 - lo);
          }
          p.out[(int64_t)(kb + kabs) * p.HKV + hk] = v;
        }
      }
      // window keys of this split that lie beyond its last scored tile
      for (int k = k_lo + n_tiles * kTile + st; k < min(len, k_lo + p.split); k += 256)
        p.out[(int64_t)(kb + k) * p.HKV + hk] = INFINITY;
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsOther));  // warps 10, 11
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, 512);
}

}  // namespace cvllm

using namespace cvllm;

// Key tiles per CTA.  A CTA holds its SM, and its start costs about four tiles.  Few (sequence, head) pairs are cut into as
// many splits as make the waves of CTAs, each of a start and a split, shortest; the splits beyond a shorter sequence's
// end (the caller's bound may be all the keys of a batch) also take their turn on an SM, about 0.02 tiles of the whole
// launch each.  From 74 pairs on the pairs themselves fill the chip and a CTA takes 8 tiles, which keeps sequences of
// unequal length balanced.
// In a graph, 32 / 8 heads, us, fixed splits of 8 tiles / at least four splits a sequence in up to three waves / this:
// 1220 + 1987 + 1640 + 1076 keys 30.7 / 34.8 / 26.6, six of 864 to 1550 34.8 / 41.0 / 32.8, four of 8000
// 73.7 / 71.7 / 57.3, 500 + 20000 + 3000 + 9000 73.8 / 71.7 / 61.4; one sequence (the same as the second): 1000 30.7 / 16.4, 4096 30.7 / 20.5, 40960 96.2 / 55.3.
static int snap_split_tiles(int B, int HKV, int Nk, int max_seqlen_k) {
  const int sms = sm_count();
  if ((int64_t)B * HKV > sms / 2) return sn::kMaxTilesManyCtas;
  const int64_t longest = std::max(1, (max_seqlen_k + sn::kTile - 1) / sn::kTile);
  int64_t best = longest, best_cost = INT64_MAX;
  for (int64_t splits = 1; splits <= std::min<int64_t>(longest, sms / HKV); ++splits) {
    const int64_t tiles = (longest + splits - 1) / splits, padded = B * ((longest + tiles - 1) / tiles);
    const int64_t live = std::min(padded, Nk / (tiles * sn::kTile) + B);   // at most a partial split per sequence
    const int64_t waves = (live * HKV + sms - 1) / sms;
    const int64_t cost = waves * (4 + tiles) * sms + 3 * (padded - live) * HKV;
    if (cost < best_cost) best_cost = cost, best = tiles;
  }
  return (int)best;
}

// Tests: key tiles per CTA of such a call.
extern "C" int cvllm_selftest_snap_split(int B, int HKV, int Nk, int max_seqlen_k) {
  return B > 0 && HKV > 0 ? snap_split_tiles(B, HKV, Nk, max_seqlen_k) : 0;
}

size_t cvllm_snap_umma_workspace_bytes(int B, int max_seqlen_k, int HKV) {
  const size_t tiles = (size_t)(max_seqlen_k + sn::kTile - 1) / sn::kTile;
  const int sms = sm_count();
  // the most that snap_split_tiles() can make of it, whatever the total of the keys
  const size_t n_splits = (int64_t)B * HKV > sms / 2 ? (tiles + sn::kMaxTilesManyCtas - 1) / sn::kMaxTilesManyCtas
                                                          : std::min(tiles, (size_t)(sms / HKV));
  return (size_t)B * HKV * 2 * (n_splits ? n_splits : 1) * sn::kTile * 2 * sizeof(float);
}

int cvllm_launch_snap_umma(const void* q, const void* k, int64_t q_stride_n, int64_t k_stride_n,
                           const int32_t* cu_q, const int32_t* cu_k, int w, int B, int Nq, int Nk, int HQ, int HKV,
                           int max_seqlen_k, float scale_log2, int kpool, int pool_segment, float* out, float* stats,
                           bool bf16, cudaStream_t st) {
  const int G = HQ / HKV;
  CUtensorMap tm_q, tm_k;
  const uint32_t boxq[3] = {64, (uint32_t)G, (uint32_t)w};
  const uint64_t dq[3] = {(uint64_t)sn::kHD, (uint64_t)HQ, (uint64_t)Nq};   // (their packing may be another than the keys')
  const uint64_t sq[2] = {(uint64_t)sn::kHD * 2, (uint64_t)q_stride_n * 2};
  int rc = make_tmap_16b(&tm_q, q, 3, dq, sq, boxq, bf16);
  if (rc) return rc;
  const uint32_t boxk[3] = {64, 1, (uint32_t)sn::kTile};
  const uint64_t dk[3] = {(uint64_t)sn::kHD, (uint64_t)HKV, (uint64_t)Nk};
  const uint64_t sk[2] = {(uint64_t)sn::kHD * 2, (uint64_t)k_stride_n * 2};
  rc = make_tmap_16b(&tm_k, k, 3, dk, sk, boxk, bf16);
  if (rc) return rc;
  SnapUmmaParams p;
  p.cu_q = cu_q; p.cu_k = cu_k; p.stats = stats; p.out = out; p.HKV = HKV; p.G = G; p.w = w;
  p.split = snap_split_tiles(B, HKV, Nk, max_seqlen_k) * sn::kTile;
  p.n_splits = (max_seqlen_k + p.split - 1) / p.split;
  p.kpool = kpool; p.pool_segment = pool_segment; p.scale_log2 = scale_log2;
  const dim3 grid(p.n_splits, HKV, B);
  const int smem = (int)sizeof(SnapUmmaSmem) + 1024;
  using Kernel = void (*)(CUtensorMap, CUtensorMap, SnapUmmaParams);
  static std::atomic<uint64_t> attr[4][2] = {};
  auto both = [&](Kernel pass1, Kernel pass2, std::atomic<uint64_t>(&done)[2]) -> int {
    CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)pass1, smem, done[0]));
    CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)pass2, smem, done[1]));
    pass1<<<grid, sn::kThreads, smem, st>>>(tm_q, tm_k, p);
    CVLLM_CHECK_CUDA(launch_behind(pass2, grid, dim3(sn::kThreads), smem, st, tm_q, tm_k, p));
    return CVLLM_OK;
  };
  if (w * G <= sn::kTile)
    rc = bf16 ? both(snap_umma_kernel<true, false, 1>, snap_umma_kernel<true, true, 1>, attr[0])
              : both(snap_umma_kernel<false, false, 1>, snap_umma_kernel<false, true, 1>, attr[1]);
  else
    rc = bf16 ? both(snap_umma_kernel<true, false, 2>, snap_umma_kernel<true, true, 2>, attr[2])
              : both(snap_umma_kernel<false, false, 2>, snap_umma_kernel<false, true, 2>, attr[3]);
  if (rc) return rc;
  CVLLM_CHECK_LAUNCHES(2);
  return CVLLM_OK;
}
