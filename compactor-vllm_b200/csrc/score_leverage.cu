// Compactor pre-RoPE approximate leverage scores.
//
// Reference: compression/compactor.py:113-221 (torch: batched GEMM K.PHI,
// python loops over chunks, cuSOLVER gesvda on the 48x48 Grams, second GEMM,
// Triton z-score :224-269).  Here: ONE CTA per (chunk, kv head) does the whole
// chain in shared memory, then one small launch z-scores each chunk.
//
//   X   = round16(K_h . PHI)                mma.sync, K rows straight from global
//   Xc  = round16(X - round16(mean_t X))    per chunk
//   G   = fp32(round16(Xc^T Xc)) + reg*I    mma.sync on the transposed sketch
//   G   = V diag(lam) V^T                   Householder + divide and conquer, fp64, one CTA per matrix
//   u   = round16(Xc . round16(V |lam|^-1/2));  score = round16(sum_j round16(u_j^2))
//
// The reference keeps X, Xc, G, V S^-1/2, U and the row sums in K's 16-bit
// dtype; rounding G entrywise perturbs it by far more than the
// 5e-3 regulariser (it can even go indefinite: the SVD then yields |lam|), so
// those rounding points are part of the reference's scores and are reproduced
// here — an exact fp32 x^T G^-1 x only overlaps ~80 % with the reference's
// kept set (tests/test_oracle_golden.py).  Work is ~170 KFLOP/token: latency
// and launch count, not throughput, is what the fusion removes.
#include <stdlib.h>

#include "common.cuh"
#include "leverage_eig.cuh"
#include "mma.cuh"

namespace cvllm {

constexpr int kLevThreads = 256;
constexpr int kSk = 48;            // sketch columns
constexpr int kTokTile = 512;      // tokens per smem tile: the engine's chunk (512) is resident, one sketch pass
constexpr int kXtStride = kTokTile + 8;  // 16-bit elements per sketch row (pad: bank spread)

struct LevParams {
  const void* k;
  int64_t k_stride_n, k_stride_h;  // elements
  const int32_t* chunk_offsets;
  const void* phi;  // [128, 48] 16-bit
  const void* sketch;  // optional [N, HKV, 48] 16-bit = round16(K.PHI) from rope.cu; null: derive it from k
  float* raw;       // [N, HKV] fp32 (values already rounded to 16-bit)
  float* gram;      // [n_chunks*HKV][48][48] fp32
  float* sv;        // [n_chunks*HKV][48][48] fp32 (values rounded to 16-bit)
  uint16_t* xc;     // centred sketch, 16-bit: chunk ch / head h at (c_beg*HKV + h*c_len)*48, [48][c_len] sketch-major
  int HKV;
  float reg;
};

template <bool BF16>
__device__ __forceinline__ float round16(float x) {
  if constexpr (BF16) return __bfloat162float(__float2bfloat16_rn(x));
  else return __half2float(__float2half_rn(x));
}
template <bool BF16>
__device__ __forceinline__ uint16_t to16(float x) {
  if constexpr (BF16) return __bfloat16_as_ushort(__float2bfloat16_rn(x));
  else return __half_as_ushort(__float2half_rn(x));
}
template <bool BF16>
__device__ __forceinline__ float from16(uint16_t x) {
  if constexpr (BF16) return __uint_as_float((uint32_t)x << 16);
  else return __half2float(__ushort_as_half(x));
}

// 48 rows of 520 and 136 16-bit numbers: rows a multiple of 16 bytes apart and 4 banks on, so that eight rows' 16-byte pieces
// (ldmatrix, stmatrix) lie in separate banks
struct GramSmem {
  uint16_t phiT[kSk][128 + 8];        // PHI^T: sketch-major, d contiguous
  uint16_t xt[kSk][kXtStride];        // X^T tile: sketch-major, token contiguous
  uint16_t stage[kLevThreads / 32][16][128 + 8];   // 16 key rows per warp
  float g[kSk][kSk + 1];              // Gram accumulator (upper triangle)
  float colsum[kSk];
  float mean[kSk];
};
struct ScoreSmem {
  uint16_t xt[kSk][kXtStride];
  float sv[kSk][kSk];                 // round16(V |lam|^-1/2)
};

__device__ __forceinline__ uint32_t lev_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
// 16 bytes, or as many zeros
__device__ __forceinline__ void lev_copy16(void* dst, const void* src, bool real) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(lev_addr(dst)), "l"(src), "r"(real ? 16 : 0) : "memory");
}
__device__ __forceinline__ void lev_copies_done() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const void* row) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(lev_addr(row))
               : "memory");
}
// the right operand of two neighbouring column tiles (rows col, col + 1, .. of `m`, 16 numbers from k0 on): b[0..1] and b[2..3]
template <int PITCH>
__device__ __forceinline__ void load_pair(uint32_t (&b)[4], const uint16_t (*m)[PITCH], int col, int k0, int lane) {
  ldmatrix4(b, &m[col + (lane >> 4) * 8 + (lane & 7)][k0 + ((lane >> 3) & 1) * 8]);
}
// the left operand: rows row .. row + 15, 16 numbers from k0 on
template <int PITCH>
__device__ __forceinline__ void load_left(uint32_t (&a)[4], const uint16_t (*m)[PITCH], int row, int k0, int lane) {
  ldmatrix4(a, &m[row + ((lane >> 3) & 1) * 8 + (lane & 7)][k0 + (lane >> 4) * 8]);
}

// X^T tile for tokens [t0, t0+nt): xt[c][t] = round16(sum_d K[t][d] * PHI[d][c]) (optionally centred).  A warp's 16 key rows come
// by asynchronous copies while it multiplies the 16 before them; the product's fragments are stored transposed.  Loads of
// four bytes a lane, four stores of two bytes for every eight columns and the right operand's 96 loads a tile took two
// thirds of the L1's cycles (the kernel 33 us for 256 chunks, 22 now).
template <bool BF16>
__device__ __forceinline__ void sketch_tile(GramSmem& sm, const LevParams& p, int h, int tok0, int nt,
                                            bool centre) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, j = lane & 3;
  const char* kb = reinterpret_cast<const char*>(p.k);
  const int n_mt = (nt + 15) / 16;
  if (p.sketch) {
    // precomputed sketch rows (96 B per (token, head)): transpose into xt, zero the m-tile padding
    const uint16_t* xs = reinterpret_cast<const uint16_t*>(p.sketch);
    const int nt16 = n_mt * 16;
    for (int i = threadIdx.x; i < nt16 * (kSk / 8); i += kLevThreads) {
      const int cchunk = i / nt16, t = i - cchunk * nt16;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (t < nt) v = *reinterpret_cast<const uint4*>(xs + ((int64_t)(tok0 + t) * p.HKV + h) * kSk + cchunk * 8);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        uint16_t bits = (uint16_t)(w[e >> 1] >> ((e & 1) * 16));
        if (centre && t < nt)
          bits = to16<BF16>(round16<BF16>(from16<BF16>(bits) - sm.mean[cchunk * 8 + e]));
        sm.xt[cchunk * 8 + e][t] = bits;
      }
    }
    return;
  }
  uint16_t(*stage)[128 + 8] = sm.stage[warp];
  auto fetch = [&](int mt) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int row = 2 * i + (lane >> 4), piece = lane & 15, t = mt * 16 + row;
      lev_copy16(&stage[row][piece * 8], kb + ((int64_t)(tok0 + min(t, nt - 1)) * p.k_stride_n + (int64_t)h * p.k_stride_h) * 2 + piece * 16,
                 t < nt);
    }
  };
  if (warp < n_mt) fetch(warp);
  for (int mt = warp; mt < n_mt; mt += kLevThreads / 32) {
    uint32_t a[8][4];
    lev_copies_done();
    __syncwarp();
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) load_left(a[ks], stage, 0, 16 * ks, lane);
    __syncwarp();
    if (mt + kLevThreads / 32 < n_mt) fetch(mt + kLevThreads / 32);
    const int t_lo = mt * 16 + r, t_hi = t_lo + 8;
#pragma unroll
    for (int nn = 0; nn < kSk / 16; ++nn) {
      float acc[2][4] = {};
      // natural-k chain (mma.cuh): the bits of the reference's cuBLAS GEMM at compactor.py:158
#pragma unroll
      for (int ks = 0; ks < 8; ++ks) {
        uint32_t b[4];
        load_pair(b, sm.phiT, 16 * nn, 16 * ks, lane);
        mma16816<BF16>(acc[0], a[ks][0], a[ks][1], a[ks][2], a[ks][3], b[0], b[1]);
        mma16816<BF16>(acc[1], a[ks][0], a[ks][1], a[ks][2], a[ks][3], b[2], b[3]);
      }
      // acc[u]: rows t_lo / t_hi, sketch cols 16 nn + 8 u + 2 j, + 1
      uint32_t m[4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float x[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          x[e] = round16<BF16>(acc[u][e]);
          if (centre) x[e] = round16<BF16>(x[e] - sm.mean[16 * nn + 8 * u + 2 * j + (e & 1)]);
        }
        m[2 * u] = t_lo < nt ? pack2<BF16>(x[0], x[1]) : 0u;
        m[2 * u + 1] = t_hi < nt ? pack2<BF16>(x[2], x[3]) : 0u;
      }
      asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(
                       lev_addr(&sm.xt[16 * nn + (lane >> 4) * 8 + (lane & 7)][mt * 16 + ((lane >> 3) & 1) * 8])),
                   "r"(m[0]), "r"(m[1]), "r"(m[2]), "r"(m[3])
                   : "memory");
    }
  }
}

__device__ __forceinline__ void load_phi(GramSmem& sm, const LevParams& p) {
  if (reinterpret_cast<uintptr_t>(p.phi) & 15) {
    const uint16_t* phi = reinterpret_cast<const uint16_t*>(p.phi);
    for (int i = threadIdx.x; i < 128 * kSk; i += kLevThreads) sm.phiT[i % kSk][i / kSk] = phi[i];
    return;
  }
  const uint4* phi = reinterpret_cast<const uint4*>(p.phi);   // 6 pieces of eight columns a row
  for (int i = threadIdx.x; i < 128 * (kSk / 8); i += kLevThreads) {
    const int d = i / (kSk / 8), c = i % (kSk / 8) * 8;
    const uint4 v = phi[i];
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 8; ++e) sm.phiT[c + e][d] = (uint16_t)(w[e >> 1] >> ((e & 1) * 16));
  }
}

// ---- kernel 1: grid (n_chunks, HKV): column means + Gram of the centred sketch ----
// out: gram[(ch*HKV+h)][48][48] = fp32(round16(Xc^T Xc)) + reg*I
template <bool BF16>
__global__ void __launch_bounds__(kLevThreads, 2) leverage_gram_kernel(const LevParams p) {
  extern __shared__ __align__(16) unsigned char lev_smem_raw[];
  GramSmem& sm = *reinterpret_cast<GramSmem*>(lev_smem_raw);
  const int ch = blockIdx.x, h = blockIdx.y;
  const int c_beg = p.chunk_offsets[ch], c_len = p.chunk_offsets[ch + 1] - c_beg;
  if (c_len <= 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (!p.sketch) load_phi(sm, p);
  if (tid < kSk) sm.colsum[tid] = 0.f;
  for (int i = tid; i < kSk * (kSk + 1); i += kLevThreads) (&sm.g[0][0])[i] = 0.f;
  __syncthreads();

  // ---- pass A: column means of X over the chunk ----
  for (int t0 = 0; t0 < c_len; t0 += kTokTile) {
    const int nt = min(kTokTile, c_len - t0);
    sketch_tile<BF16>(sm, p, h, c_beg + t0, nt, false);
    __syncthreads();
    // 48 columns x 256 threads: warp w sums columns w, w+8, ...
    for (int c = warp; c < kSk; c += kLevThreads / 32) {
      float s = 0.f;
      for (int t = lane; t < nt; t += 32) s += from16<BF16>(sm.xt[c][t]);
      s = warp_sum(s);
      if (lane == 0) sm.colsum[c] += s;
    }
    __syncthreads();
  }
  if (tid < kSk) sm.mean[tid] = round16<BF16>(sm.colsum[tid] / (float)c_len);
  __syncthreads();

  // ---- pass B: Gram of the centred sketch, G[i][j] = sum_t xc[t][i] xc[t][j] ----
  for (int t0 = 0; t0 < c_len; t0 += kTokTile) {
    const int nt = min(kTokTile, c_len - t0);
    // Centre (one tile: the uncentred sketch is still resident; several tiles: re-derived centred), zero the
    // padded token columns (partial k16 steps must contribute nothing) and hand the centred sketch to the score
    // kernel — one vectorised pass, a warp per sketch row, 8 tokens per lane.  (A flat `i / nt` element loop
    // here was 65 % of the kernel's instructions, by ncu.)
    const bool resident = c_len <= kTokTile;
    if (!resident) {
      sketch_tile<BF16>(sm, p, h, c_beg + t0, nt, true);
      __syncthreads();
    }
    const int nt16 = (nt + 15) & ~15;
    {
      uint16_t* xc = p.xc + ((int64_t)c_beg * p.HKV + (int64_t)h * c_len) * kSk;
      const bool vec_ok = (c_len & 7) == 0;
      for (int c = warp; c < kSk; c += kLevThreads / 32) {
        const float mu = resident ? sm.mean[c] : 0.f;
        for (int t8 = lane * 8; t8 < nt16; t8 += 256) {
          uint4 v = *reinterpret_cast<const uint4*>(&sm.xt[c][t8]);
          uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            float lo = from16<BF16>((uint16_t)(w4[e] & 0xffffu)), hi = from16<BF16>((uint16_t)(w4[e] >> 16));
            if (resident) { lo = round16<BF16>(lo - mu); hi = round16<BF16>(hi - mu); }
            const uint32_t blo = (t8 + 2 * e < nt) ? to16<BF16>(lo) : 0u;
            const uint32_t bhi = (t8 + 2 * e + 1 < nt) ? to16<BF16>(hi) : 0u;
            w4[e] = blo | (bhi << 16);
          }
          v = make_uint4(w4[0], w4[1], w4[2], w4[3]);
          *reinterpret_cast<uint4*>(&sm.xt[c][t8]) = v;
          uint16_t* dst = xc + (int64_t)c * c_len + t0 + t8;
          if (vec_ok && t8 + 8 <= nt) {
            *reinterpret_cast<uint4*>(dst) = v;
          } else {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (t8 + e < nt) dst[e] = (uint16_t)(w4[e >> 1] >> ((e & 1) * 16));
          }
        }
      }
    }
    __syncthreads();
    // the tiles that hold the upper triangle: 16 sketch rows from `rows` on, columns 16 pair .. 16 pair + 15, for six warps
    if (warp < 6) {
      const int rows = warp < 3 ? 0 : warp < 5 ? 16 : 32, pair = warp < 3 ? warp : warp < 5 ? warp - 2 : 2;
      // the accumulator is CARRIED across token tiles (not summed per tile and added): one sequential
      // k16 chain over the whole chunk, the order a non-split-K library GEMM accumulates in — the Gram is
      // rounded to 16 bit next, and on low-rank keys one flipped ulp there moves a chunk's scores by O(1)
      const int gi = rows + (lane >> 2), gj = 16 * pair + 2 * (lane & 3);
      float acc[2][4];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[u][e] = sm.g[gi + 8 * (e >> 1)][gj + 8 * u + (e & 1)];
#pragma unroll 4
      for (int k0 = 0; k0 < nt16; k0 += 16) {
        uint32_t a[4], b[4];
        load_left(a, sm.xt, rows, k0, lane);
        load_pair(b, sm.xt, 16 * pair, k0, lane);
        mma16816<BF16>(acc[0], a[0], a[1], a[2], a[3], b[0], b[1]);
        mma16816<BF16>(acc[1], a[0], a[1], a[2], a[3], b[2], b[3]);
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) sm.g[gi + 8 * (e >> 1)][gj + 8 * u + (e & 1)] = acc[u][e];
    }
    __syncthreads();
  }
  // round the Gram to the 16-bit dtype (compactor.py:166,171,173), add the regulariser.
  // Symmetrise from the upper triangle so rounding cannot make G asymmetric.
  float* gout = p.gram + (int64_t)(ch * p.HKV + h) * kSk * kSk;
  for (int i = tid; i < kSk * kSk; i += kLevThreads) {
    const int a = i / kSk, b = i - a * kSk;
    gout[i] = round16<BF16>(a <= b ? sm.g[a][b] : sm.g[b][a]) + ((a == b) ? p.reg : 0.f);
  }
}

// ---- kernel 2: symmetric eigendecomposition, leverage_eig.cuh ----

// ---- kernel 3: grid (n_chunks, HKV): score_t = round16(sum_j round16(round16(xc_t . sv_j)^2)) ----
template <bool BF16>
__global__ void __launch_bounds__(kLevThreads, 2) leverage_score_kernel(const LevParams p) {
  extern __shared__ __align__(16) unsigned char lev_smem_raw[];
  ScoreSmem& sm = *reinterpret_cast<ScoreSmem*>(lev_smem_raw);
  pdl_wait();
  const int ch = blockIdx.x, h = blockIdx.y;
  const int c_beg = p.chunk_offsets[ch], c_len = p.chunk_offsets[ch + 1] - c_beg;
  if (c_len <= 0) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, r = lane >> 2, j = lane & 3;
  const bool vec_ok = (c_len & 7) == 0;
  const uint16_t* xc = p.xc + ((int64_t)c_beg * p.HKV + (int64_t)h * c_len) * kSk;
  // the centred sketch's tile from token t0 on; whole pieces in flight beside what follows
  auto fetch = [&](int t0) {
    const int nt = min(kTokTile, c_len - t0);
    for (int c = warp; c < kSk; c += kLevThreads / 32) {
      const uint16_t* src = xc + (int64_t)c * c_len + t0;
      for (int t8 = lane * 8; t8 < nt; t8 += 256) {
        if (vec_ok) {
          lev_copy16(&sm.xt[c][t8], src + t8, true);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) sm.xt[c][t8 + e] = (t8 + e < nt) ? src[t8 + e] : (uint16_t)0;
        }
      }
    }
  };
  fetch(0);
  {
    const float4* svin = reinterpret_cast<const float4*>(p.sv + (int64_t)(ch * p.HKV + h) * kSk * kSk);
    for (int i = tid; i < kSk * kSk / 4; i += kLevThreads) reinterpret_cast<float4*>(&sm.sv[0][0])[i] = svin[i];
  }
  __syncthreads();
  // B fragments of U = Xc . SV (k = sketch column c, n = eigen-column): SV's entries are 16-bit values held in fp32
  uint32_t bfr[3][6][2];
#pragma unroll
  for (int ks = 0; ks < 3; ++ks)
#pragma unroll
    for (int nn = 0; nn < 6; ++nn) {
      bfr[ks][nn][0] = pack2<BF16>(sm.sv[16 * ks + 2 * j][nn * 8 + r], sm.sv[16 * ks + 2 * j + 1][nn * 8 + r]);
      bfr[ks][nn][1] = pack2<BF16>(sm.sv[16 * ks + 8 + 2 * j][nn * 8 + r], sm.sv[16 * ks + 9 + 2 * j][nn * 8 + r]);
    }
  for (int t0 = 0; t0 < c_len; t0 += kTokTile) {
    const int nt = min(kTokTile, c_len - t0);
    if (t0 > 0) fetch(t0);
    lev_copies_done();
    __syncthreads();
    // U[16 tokens x 48] per m-tile on mma.sync (the scalar form was 48 x 48 FFMA per token); the A operand is read
    // straight out of the sketch-major tile with ldmatrix.trans
    const int n_mt = (nt + 15) / 16;
    for (int mt = warp; mt < n_mt; mt += kLevThreads / 32) {
      float acc[6][4];
#pragma unroll
      for (int nn = 0; nn < 6; ++nn) acc[nn][0] = acc[nn][1] = acc[nn][2] = acc[nn][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < 3; ++ks) {
        const int mid = lane >> 3;  // 8x8 matrix this lane addresses: (k half, token half)
        const uint16_t* rowp = &sm.xt[16 * ks + (mid >> 1) * 8 + (lane & 7)][mt * 16 + (mid & 1) * 8];
        uint32_t a0, a1, a2, a3;
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(a0), "=r"(a1), "=r"(a2), "=r"(a3)
                     : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(rowp))));
#pragma unroll
        for (int nn = 0; nn < 6; ++nn) mma16816<BF16>(acc[nn], a0, a1, a2, a3, bfr[ks][nn][0], bfr[ks][nn][1]);
      }
      // score = round16(sum_j round16(round16(u_j)^2)) (compactor.py:209-210), rows r and r + 8 of the m-tile
      float s_lo = 0.f, s_hi = 0.f;
#pragma unroll
      for (int nn = 0; nn < 6; ++nn) {
        const float u0 = round16<BF16>(acc[nn][0]), u1 = round16<BF16>(acc[nn][1]);
        const float u2 = round16<BF16>(acc[nn][2]), u3 = round16<BF16>(acc[nn][3]);
        s_lo += round16<BF16>(u0 * u0) + round16<BF16>(u1 * u1);
        s_hi += round16<BF16>(u2 * u2) + round16<BF16>(u3 * u3);
      }
      s_lo += __shfl_xor_sync(0xffffffffu, s_lo, 1);
      s_lo += __shfl_xor_sync(0xffffffffu, s_lo, 2);
      s_hi += __shfl_xor_sync(0xffffffffu, s_hi, 1);
      s_hi += __shfl_xor_sync(0xffffffffu, s_hi, 2);
      if (j == 0) {
        const int t_lo = mt * 16 + r, t_hi = t_lo + 8;
        if (t_lo < nt) p.raw[(int64_t)(c_beg + t0 + t_lo) * p.HKV + h] = fmaxf(round16<BF16>(s_lo), 0.f);
        if (t_hi < nt) p.raw[(int64_t)(c_beg + t0 + t_hi) * p.HKV + h] = fmaxf(round16<BF16>(s_hi), 0.f);
      }
    }
    __syncthreads();
  }
}

// grid (n_chunks): z-score a chunk over all heads (compactor.py:224-269) and cast to the output dtype
template <bool BF16>
__global__ void __launch_bounds__(256) leverage_finalize_kernel(const float* raw,
                                                                const int32_t* __restrict__ chunk_offsets,
                                                                void* __restrict__ out, int HKV, int normalize) {
  pdl_wait();
  const int ch = blockIdx.x;
  const int beg = chunk_offsets[ch], len = chunk_offsets[ch + 1] - beg;
  if (len <= 0) return;
  const int total = len * HKV;
  const float* src = raw + (int64_t)beg * HKV;
  uint16_t* dst = reinterpret_cast<uint16_t*>(out) + (int64_t)beg * HKV;
  __shared__ float s_red[2][8];
  __shared__ float s_stat[2];
  float mean = 0.f, invstd = 1.f;
  if (normalize) {
    float a1 = 0.f, a2 = 0.f;
    for (int i = threadIdx.x; i < total; i += 256) {
      const float v = src[i];
      a1 += v;
      a2 += v * v;
    }
    a1 = warp_sum(a1);
    a2 = warp_sum(a2);
    if ((threadIdx.x & 31) == 0) { s_red[0][threadIdx.x >> 5] = a1; s_red[1][threadIdx.x >> 5] = a2; }
    __syncthreads();
    if (threadIdx.x == 0) {
      float t1 = 0.f, t2 = 0.f;
      for (int w = 0; w < 8; ++w) { t1 += s_red[0][w]; t2 += s_red[1][w]; }
      const float cnt = (float)total;
      const float m = t1 / cnt;
      const float var = fmaxf(t2 / cnt - m * m, 0.f);
      s_stat[0] = m;
      s_stat[1] = 1.0f / sqrtf(var);
    }
    __syncthreads();
    mean = s_stat[0];
    invstd = s_stat[1];
  }
  for (int i = threadIdx.x; i < total; i += 256) {
    float v = src[i];
    if (normalize) v = (v - mean) * invstd;
    dst[i] = to16<BF16>(v);
  }
}

}  // namespace cvllm

using namespace cvllm;

template <bool BF16>
static cudaError_t ensure_eig_smem() {
  static std::atomic<uint64_t> done{0};
  return ensure_max_dyn_smem((const void*)leverage_eig_kernel<BF16>, (int)sizeof(EigSmem), done);
}

static size_t lev_align(size_t x) { return (x + 255) & ~(size_t)255; }

extern "C" size_t cvllm_leverage_scores_workspace_bytes(int N, int HKV, int sketch, int n_chunks) {
  (void)sketch;
  if (N <= 0 || HKV <= 0) return 256;
  const size_t mats = (size_t)(n_chunks > 0 ? n_chunks : 0) * HKV;
  return lev_align((size_t)N * HKV * sizeof(float)) + 2 * lev_align(mats * kSk * kSk * sizeof(float)) +
         lev_align((size_t)N * HKV * kSk * sizeof(uint16_t));
}

static int leverage_launch(const void* k_pre, int64_t k_stride_n, int64_t k_stride_h, const void* sketch_rows,
                           const int32_t* chunk_offsets, int n_chunks, int max_chunk,
                           const void* phi, void* out_scores, int N, int HKV, int D, int sketch,
                           float regularizer, int normalize, int dtype, void* workspace,
                           size_t workspace_bytes, cvllm_stream_t stream) {
  CVLLM_CHECK_ARG(N >= 0 && HKV > 0 && n_chunks >= 0 && max_chunk >= 0);
  if (N == 0 || n_chunks == 0) return CVLLM_OK;
  CVLLM_CHECK_ARG((sketch_rows || (k_pre && phi)) && chunk_offsets && out_scores && workspace);
  CVLLM_CHECK_ARG(dtype == CVLLM_F16 || dtype == CVLLM_BF16);
  CVLLM_CHECK_SUPPORTED(D == 128 && sketch == kSk);
  CVLLM_CHECK_ALIGN(aligned16(k_pre) && aligned16(sketch_rows) && k_stride_n % 8 == 0 && k_stride_h % 8 == 0);
  CVLLM_CHECK_ARG(workspace_bytes >= cvllm_leverage_scores_workspace_bytes(N, HKV, sketch, n_chunks));
  auto st = static_cast<cudaStream_t>(stream);
  const size_t mats = (size_t)n_chunks * HKV;
  char* wsb = reinterpret_cast<char*>(workspace);
  LevParams p;
  p.k = k_pre; p.k_stride_n = k_stride_n; p.k_stride_h = k_stride_h; p.chunk_offsets = chunk_offsets;
  p.phi = phi; p.sketch = sketch_rows; p.HKV = HKV; p.reg = regularizer;
  p.raw = reinterpret_cast<float*>(wsb);
  wsb += lev_align((size_t)N * HKV * sizeof(float));
  p.gram = reinterpret_cast<float*>(wsb);
  wsb += lev_align(mats * kSk * kSk * sizeof(float));
  p.sv = reinterpret_cast<float*>(wsb);
  wsb += lev_align(mats * kSk * kSk * sizeof(float));
  p.xc = reinterpret_cast<uint16_t*>(wsb);
  static std::atomic<uint64_t> attr_g[2] = {{0}, {0}}, attr_s[2] = {{0}, {0}};
  // the last two are scheduled beside the end of the kernel in front; the eigensolver is not: its CTAs would come two to the SMs
  // whose Gram is done first, where one each is faster (256 chunks 147 -> 149 us a call)
  const dim3 grid(n_chunks, HKV);
  if (dtype == CVLLM_BF16) {
    CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)leverage_gram_kernel<true>, (int)sizeof(GramSmem), attr_g[1]));
    CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)leverage_score_kernel<true>, (int)sizeof(ScoreSmem), attr_s[1]));
    CVLLM_CHECK_CUDA(ensure_eig_smem<true>());
    leverage_gram_kernel<true><<<grid, kLevThreads, sizeof(GramSmem), st>>>(p);
    leverage_eig_kernel<true><<<(unsigned)mats, kEigThreads, sizeof(EigSmem), st>>>(p.gram, p.sv, chunk_offsets, HKV, (int)mats, nullptr, nullptr, nullptr);
    CVLLM_CHECK_CUDA(launch_behind(leverage_score_kernel<true>, grid, dim3(kLevThreads), sizeof(ScoreSmem), st, p));
    CVLLM_CHECK_CUDA(launch_behind(leverage_finalize_kernel<true>, dim3(n_chunks), dim3(256), 0, st, p.raw, chunk_offsets, out_scores,
                                   HKV, normalize));
  } else {
    CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)leverage_gram_kernel<false>, (int)sizeof(GramSmem), attr_g[0]));
    CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)leverage_score_kernel<false>, (int)sizeof(ScoreSmem), attr_s[0]));
    CVLLM_CHECK_CUDA(ensure_eig_smem<false>());
    leverage_gram_kernel<false><<<grid, kLevThreads, sizeof(GramSmem), st>>>(p);
    leverage_eig_kernel<false><<<(unsigned)mats, kEigThreads, sizeof(EigSmem), st>>>(p.gram, p.sv, chunk_offsets, HKV, (int)mats, nullptr, nullptr, nullptr);
    CVLLM_CHECK_CUDA(launch_behind(leverage_score_kernel<false>, grid, dim3(kLevThreads), sizeof(ScoreSmem), st, p));
    CVLLM_CHECK_CUDA(launch_behind(leverage_finalize_kernel<false>, dim3(n_chunks), dim3(256), 0, st, p.raw, chunk_offsets, out_scores,
                                   HKV, normalize));
  }
  CVLLM_CHECK_LAUNCHES(4);
  return CVLLM_OK;
}

extern "C" int cvllm_leverage_scores(const void* k_pre, int64_t k_stride_n, int64_t k_stride_h,
                                     const int32_t* chunk_offsets, int n_chunks, int max_chunk,
                                     const void* phi, void* out_scores, int N, int HKV, int D, int sketch,
                                     float regularizer, int normalize, int dtype, void* workspace,
                                     size_t workspace_bytes, cvllm_stream_t stream) {
  if (N > 0 && n_chunks > 0) CVLLM_CHECK_ARG(k_pre != nullptr);
  return leverage_launch(k_pre, k_stride_n, k_stride_h, nullptr, chunk_offsets, n_chunks, max_chunk, phi,
                         out_scores, N, HKV, D, sketch, regularizer, normalize, dtype, workspace,
                         workspace_bytes, stream);
}

extern "C" int cvllm_leverage_scores_from_sketch(const void* sketch_rows, const int32_t* chunk_offsets,
                                                 int n_chunks, int max_chunk, const void* phi,
                                                 void* out_scores, int N, int HKV, int sketch,
                                                 float regularizer, int normalize, int dtype,
                                                 void* workspace, size_t workspace_bytes,
                                                 cvllm_stream_t stream) {
  if (N > 0 && n_chunks > 0) CVLLM_CHECK_ARG(sketch_rows != nullptr);
  return leverage_launch(nullptr, 0, 0, sketch_rows, chunk_offsets, n_chunks, max_chunk, phi, out_scores, N,
                         HKV, 128, sketch, regularizer, normalize, dtype, workspace, workspace_bytes, stream);
}

// Test entry (tests/test_gpu_scores.py): the eigensolver alone.  gram: fp32 [mats, 48, 48] symmetric;
// lam_out: fp64 [mats, 48]; vec_out: fp64 [mats, 48, 48] (columns = eigenvectors, arbitrary order);
// sv_out: fp32 [mats, 48, 48] = round16(V |lam|^-1/2), the product output.
extern "C" int cvllm_selftest_eig(const float* gram, double* lam_out, double* vec_out, float* sv_out, int mats,
                                  int dtype, long long* clk_out, cvllm_stream_t stream) {
  CVLLM_CHECK_ARG(gram && lam_out && vec_out && sv_out && mats > 0);
  CVLLM_CHECK_ARG(dtype == CVLLM_F16 || dtype == CVLLM_BF16);
  auto st = static_cast<cudaStream_t>(stream);
  CVLLM_CHECK_CUDA(dtype == CVLLM_BF16 ? ensure_eig_smem<true>() : ensure_eig_smem<false>());
  if (dtype == CVLLM_BF16)
    leverage_eig_kernel<true><<<mats, kEigThreads, sizeof(EigSmem), st>>>(gram, sv_out, nullptr, 1, mats, lam_out, vec_out, clk_out);
  else
    leverage_eig_kernel<false><<<mats, kEigThreads, sizeof(EigSmem), st>>>(gram, sv_out, nullptr, 1, mats, lam_out, vec_out, clk_out);
  CVLLM_CHECK_LAUNCH();
  return CVLLM_OK;
}
