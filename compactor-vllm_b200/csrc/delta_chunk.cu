// Gated delta rule over portions of prompts, in chunks of 64 tokens on tcgen05 / TMEM (the recurrence, its gates and norm:
// recurrent.cu, whose kernels keep short portions, single tokens and other sizes).
//
// With S [D, Dv] a head's state before a chunk, its tokens counted 0 .. 63, q and k the unit vectors, w_ts = g_(s+1) .. g_t
// and G_t = g_0 .. g_t (products, never quotients), token t writes k_t u_t^T with
//   u_t = beta_t (v_t - G_t S^T k_t) - sum_(s < t) beta_t w_ts (k_t . k_s) u_s
// - a triangular system that the value columns share.  With T its inverse (times diag(beta)), P = (w_ts (q_t . k_s)) for
// s <= t, C = K^T diag(w_63) T, and R = V - diag(G) K S,
//   S <- G_63 S + C R;   O = diag(G) Q S + (P T) R
// C and P T depend on the inputs alone: delta_rows_kernel and delta_coef_kernel make them for all chunks at once.
// delta_chunk_kernel walks a sequence's chunks with two products in sequence, [K; Q] S and C R, and P T R beside them.
//
// 32 bits on a 16-bit tensor pipe: every operand is the sum of three bfloat16 numbers (24 bits of fraction; the rest is below
// 2^-26 of the value), every product takes the six pairs of parts down to 2^-18, and pairs of one magnitude share an
// accumulator: with the three parts of the right operand side by side in N, the left operand's first part meets all three
// parts, its second part the first two (32 accumulator columns further on) and its third part the first.  Three products
// of 96, 64 and 32 columns read the left operand three times instead of six, and the three sums are added smallest first.  The
// tensor pipe truncates its sums, which with keys that share a direction is a bias: the largest sum of [K; Q] S has four
// accumulators of a quarter of the channels each (one accumulator: twice the state's error behind a last chunk of few tokens),
// and the coefficients are 64-bit (delta_coef_kernel).
//
// A chunk's images (operands as they lie in shared memory, 128-byte swizzle) are written once by the first kernels and copied
// by untiled bulk copies.
//
// A cluster of Dv / 32 CTAs serves one (head, sequence); each keeps 32 value columns of S in registers (a thread per key
// channel and 16 columns), rewritten as three parts into shared memory after every chunk.  Unit norms need all columns
// of a head: the CTAs exchange their sums of squares through distributed shared memory.
//
// What is not finite stays behind its token: an element of R that is infinite or NaN would meet zeros of P T in earlier
// tokens' rows, so it enters the products as 0 and its column becomes NaN from that token on.
//
// Measured (one portion of 4096 tokens, 32 / 16 heads of 128 x 128, which takes the kernel of blocks of four 927 us): rows 58 us (their
// bytes take 32; 45 with products in 32 bits), coefficients 126 us (barriers between short phases, 3.4 of the 11 cycles between two
// instructions of a warp, two CTAs an SM; 120 in 32 bits), chunks 214 us.  What bounds the last: a chain per chunk of two
// products (32 + 64, 64 and 32 columns of 128, 12 of 96, 64 and 32) and two turns through registers of some 1000 cycles each, on 128
// SMs; and shared memory, whose operand reads and copies take about two thirds of a chunk's cycles at 128 bytes each.  Tried: three
// products in sequence without C (248 us where this form then took 226); the columns in two groups that alternate (339: twice the
// operand reads); K S alone at 64 rows with Q S behind it (277); the gates' factors on two warps beside the issuing one (269);
// copies paced to arrive between the products (the same).
//
// Every wait has a limit.  A wait that runs out sets the CTA's abort flag; all roles then leave their loops, copies and
// products in flight are waited for (with a limit), the CTA's state and its columns of the launch's rows become NaN and a counter
// that the host can read (cvllm_delta_chunk_aborts) goes up, once per CTA.  In the coefficients' kernel it voids the chunk: its
// decays, and with them the outputs from there on and the state, become NaN.
#include <algorithm>
#include <utility>

#include "mma.cuh"
#include "recur_common.cuh"
#include "tma.cuh"

namespace cvllm {

__device__ int g_delta_chunk_aborts;

namespace {

constexpr int kChunk = 64;                       // tokens
constexpr int kCols = 32;                        // value columns of a CTA
constexpr int kPanel = 128 * 128;                // 128 rows of 64 16-bit numbers
constexpr int kParts = 3;
constexpr uint32_t kSpins = 1u << 20;            // tries of a wait, each up to kSleep ns: about two seconds
constexpr uint32_t kSpinsHeld = 1u << 9;         // in tests whose waits run out: about a millisecond
constexpr uint32_t kSleep = 2000;

struct DeltaChunkArgs {
  const float* qkv;            // [tokens, 2 G D + H Dv] (q | k | v) after the convolution
  int64_t qkv_stride, proj_stride, gate_stride, out_stride;
  const void *proj, *gate;
  int b_off, a_off, gate_off;
  const float *A_log, *dt_bias, *norm_w;
  int norm_head_stride;
  float eps;
  float* state;
  void* out;
  int H, G, Dv, reserved_slot;
  StepGeom g;
  // a launch takes a window of `slots` chunks, whose images lie at places from 0 on.  per_seq == 0: the chunks of all sequences in
  // a row, chunk c of sequence b at cu_q[b] / 64 + b + c, from `window` on.  per_seq > 0: the chunks from `window` on of every
  // sequence, per_seq places each.
  int B, window, slots, per_seq;
  unsigned char* kq;           // [slots, G, parts, D / 64, panel]: rows 0 .. 63 k, 64 .. 127 q
  unsigned char* cp;           // [slots, H, parts, D + 64 rows of 128 bytes]: rows 0 .. D - 1 C, then P T
  double* dots;                // [slots, G, 2, 10, 16, 16]: lower blocks of K K^T and Q K^T
  float* gw;                   // [slots, H, 64]: G_t
  float *carry_in, *carry_out; // [H, Dv, D]: the state of the sequence that the window before (this one) ends in, or every sequence's
  uint32_t spins;              // limit of a wait, in tries of up to kSleep ns
  int hold;                    // tests: copies of chunk hold - 1 never begin for CTA 0 (coefficients: of chunk -hold - 1 for head 0)
};
// the chunk at place blockIdx.x of the window: false where a sequence's last chunk is not followed by the next sequence's first
__device__ __forceinline__ bool chunk_of_block(const DeltaChunkArgs& a, int& b, int& c, int& t0, int& n) {
  const int at = a.window + blockIdx.x;
  b = 0;
  if (a.per_seq > 0) {
    b = blockIdx.x / a.per_seq;
  } else if (a.B > 1) {
    int before = 0;      // sequences that begin here or before
    for (int i0 = 0; i0 < a.B && before == i0; i0 += blockDim.x) {
      const int i = i0 + threadIdx.x;
      before += __syncthreads_count(i < a.B && a.g.cu_q[i] / kChunk + i <= at);
    }
    if (before == 0) return false;
    b = before - 1;
  }
  int n_new, start;
  portion(a.g, b, t0, n_new, start);
  c = a.per_seq > 0 ? at - b * a.per_seq : at - (t0 / kChunk + b);
  n = min(kChunk, n_new - c * kChunk);
  return c >= 0 && n > 0;
}

// x = hi + mid + lo, each a bfloat16; two numbers a word
__device__ __forceinline__ void split3(float2 x, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const float2 minus = make_float2(-1.f, -1.f);
  hi = pack2<true>(x.x, x.y);
  x = __ffma2_rn(unpack2<true>(hi), minus, x);
  mid = pack2<true>(x.x, x.y);
  x = __ffma2_rn(unpack2<true>(mid), minus, x);
  lo = pack2<true>(x.x, x.y);
}
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  split3(make_float2(x, y), hi, mid, lo);
}

__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
// A number of a unit row (|x| <= 1) as x0 + 2^-12 x1 + 2^-24 x2, each a float16: x0 a multiple of 2^-11, so that a sum of such
// products (multiples of 2^-22, at most 1 for two unit rows) is exact in fp32; x1 and x2 what is left, 11 bits each.
__device__ __forceinline__ void slice3(float2 x, uint32_t& x0, uint32_t& x1, uint32_t& x2) {
  const float2 near0 = make_float2((x.x + 6144.f) - 6144.f, (x.y + 6144.f) - 6144.f);   // 6144: last place 2^-11
  x0 = pack2<false>(near0.x, near0.y);
  x = make_float2((x.x - near0.x) * 4096.f, (x.y - near0.y) * 4096.f);
  x1 = pack2<false>(x.x, x.y);
  const float2 h = unpack2<false>(x1);
  x2 = pack2<false>((x.x - h.x) * 4096.f, (x.y - h.y) * 4096.f);
}
// acc of two 8-column tiles (i: which) += A . B on three parts each; the largest pair apart from the others
__device__ __forceinline__ void mma_parts(float (&big)[4], float (&rest)[4], const uint32_t (&fa)[3][4], const uint32_t (&fb)[3][4],
                                          int i) {
  auto mul = [&](float (&acc)[4], int ea, int eb) {
    mma16816<true>(acc, fa[ea][0], fa[ea][1], fa[ea][2], fa[ea][3], fb[eb][2 * i], fb[eb][2 * i + 1]);
  };
  mul(rest, 0, 2);
  mul(rest, 1, 1);
  mul(rest, 2, 0);
  mul(big, 0, 0);
  mul(rest, 0, 1);
  mul(rest, 1, 0);
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, int bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
// A try sleeps until the phase ends (kSleep at most): a dozen warps that poll shared memory instead slow the products' operand
// reads down.
__device__ __forceinline__ bool dc_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\t"
               "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity), "r"(kSleep) : "memory");
  return ok != 0;
}

// byte offset of (row, 16-byte piece) in a panel
__device__ __forceinline__ int panel_at(int row, int piece) { return row * 128 + ((piece ^ (row & 7)) << 4); }

// ---------------------------------------------------------------------------------------------------------
// Unit rows and their products.  grid (chunks, G), 256 threads: k and q rows to unit length and into parts, the image out
// by a bulk copy; K K^T and Q K^T (lower blocks of 16) on mma.sync, from float16 slices that take the image's place.  The largest
// sum is exact and the others are 2^-12 and 2^-24 of it, so a product is good to 2^-32: 63 of them enter every u_t, and keys that
// share a direction (products near 1) make the sum as large as the values.
// ---------------------------------------------------------------------------------------------------------
constexpr int kPrepThreads = 256;
constexpr int kUnits = 20;    // lower blocks of 16 x 16 of two matrices
__device__ __forceinline__ void unit_of(int u, int& m, int& mt, int& nt) {
  m = u / 10;
  const int i = u % 10;
  mt = i < 1 ? 0 : i < 3 ? 1 : i < 6 ? 2 : 3;
  nt = i - mt * (mt + 1) / 2;
}

template <int D>
__global__ void __launch_bounds__(kPrepThreads, 2) delta_rows_kernel(const DeltaChunkArgs a) {
  pdl_wait();      // each of the three kernels may be scheduled beside the one in front
  pdl_trigger();
  extern __shared__ unsigned char smem_raw[];
  const int grp = blockIdx.y;
  int b, c, t0, n;
  if (!chunk_of_block(a, b, c, t0, n)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, slot = blockIdx.x;
  unsigned char* img = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  constexpr int kPartBytes = (D / 64) * kPanel;

  // ---- unit rows in parts: a thread has four numbers of 2 x 8 (heads of 64: 2 x 4) rows ----
  {
    constexpr int LR = D / 4, RW = 32 / LR, kPasses = kChunk / (8 * RW), kRows = 2 * kPasses;
    const int sub = lane / LR, l = lane % LR, d = l * 4;
    const float* base = a.qkv + (int64_t)(t0 + c * kChunk) * a.qkv_stride + grp * D + d;
    const int off0 = (d >> 6) * kPanel + (d & 7) * 2, piece = (d & 63) >> 3;
    float4 x[kRows];           // q rows, then k rows
    float ss[kRows];
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      const int t = (i % kPasses) * (8 * RW) + warp * RW + sub;
      x[i] = t < n ? *reinterpret_cast<const float4*>(base + (int64_t)t * a.qkv_stride + (i / kPasses) * a.G * D)
                   : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < kRows; ++i)
      ss[i] = fmaf(x[i].w, x[i].w, fmaf(x[i].z, x[i].z, fmaf(x[i].y, x[i].y, x[i].x * x[i].x)));
    // sums over a row's lanes, all rows together: every exchange halves the sums that a lane is left with
    int mine = 0;
#pragma unroll
    for (int o = 1, left = kRows; o < LR; o <<= 1) {
      if (left > 1) {
        const bool up = (l & o) != 0;
        left >>= 1;
#pragma unroll
        for (int i = 0; i < kRows / 2; ++i)
          if (i < left) {
            const float send = up ? ss[i] : ss[i + left], keep = up ? ss[i + left] : ss[i];
            ss[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
        if (up) mine += left;
      } else {
        ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], o);
      }
    }
    const float inv_mine = (mine < kPasses ? rsqrtf((float)D) : 1.0f) / sqrtf(ss[0] + 1e-6f);
#pragma unroll
    for (int i = 0; i < kRows; ++i) {
      // the lane that row i's sum ended up in: bit k of its number is set where the k-th exchange kept the upper half
      int from = 0;
#pragma unroll
      for (int o = 1, left = kRows, at = i; left > 1; o <<= 1) {
        left >>= 1;
        if (at >= left) from |= o, at -= left;
      }
      const float inv = __shfl_sync(0xffffffffu, inv_mine, from, LR);
      x[i] = make_float4(x[i].x * inv, x[i].y * inv, x[i].z * inv, x[i].w * inv);
    }
    auto put = [&](auto&& cut) {
#pragma unroll
      for (int i = 0; i < kRows; ++i) {
        uint32_t p[kParts][2];
        cut(make_float2(x[i].x, x[i].y), p[0][0], p[1][0], p[2][0]);
        cut(make_float2(x[i].z, x[i].w), p[0][1], p[1][1], p[2][1]);
        const int t = (i % kPasses) * (8 * RW) + warp * RW + sub, row = i < kPasses ? kChunk + t : t;
#pragma unroll
        for (int e = 0; e < kParts; ++e)
          *reinterpret_cast<uint2*>(img + e * kPartBytes + off0 + panel_at(row, piece)) = make_uint2(p[e][0], p[e][1]);
      }
    };
    put([](float2 v, uint32_t& e0, uint32_t& e1, uint32_t& e2) { split3(v, e0, e1, e2); });
    fence_proxy_async_smem();
    __syncthreads();
    if (tid == 0) {
      unsigned char* dst = a.kq + ((int64_t)slot * a.G + grp) * (kParts * kPartBytes);
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(img)),
                   "r"(kParts * kPartBytes)
                   : "memory");
      bulk_commit();
      bulk_wait_read<0>();
    }
    __syncthreads();
    put([](float2 v, uint32_t& e0, uint32_t& e1, uint32_t& e2) { slice3(v, e0, e1, e2); });
  }
  __syncthreads();

  // ---- K K^T and Q K^T: 20 lower blocks over eight warps ----
  constexpr int kRounds = (kUnits + 7) / 8;
#pragma unroll 1
  for (int r = 0; r < kRounds; ++r) {
    float acc[3][2][4] = {};     // sums of 1, 2^-12, 2^-24
    const int u = warp + 8 * r;
    if (u < kUnits) {
      int m, mt, nt;
      unit_of(u, m, mt, nt);
      const int row_a = m * kChunk + mt * 16 + (lane & 15), row_b = nt * 16 + (lane & 7) + ((lane >> 4) << 3);
      const uint32_t base = smem_u32(img);
#pragma unroll 2
      for (int ks = 0; ks < D / 16; ++ks) {
        const int pa = ks * 2 + (lane >> 4), pb = ks * 2 + ((lane >> 3) & 1);
        uint32_t fa[kParts][4], fb[kParts][4];
#pragma unroll
        for (int e = 0; e < kParts; ++e) {
          ldmatrix4(fa[e], base + e * kPartBytes + (pa >> 3) * kPanel + panel_at(row_a, pa & 7));
          ldmatrix4(fb[e], base + e * kPartBytes + (pb >> 3) * kPanel + panel_at(row_b, pb & 7));
        }
#pragma unroll
        for (int ea = 0; ea < kParts; ++ea)
#pragma unroll
          for (int eb = 0; eb + ea < kParts; ++eb)
#pragma unroll
            for (int i = 0; i < 2; ++i)
              mma16816<false>(acc[ea + eb][i], fa[ea][0], fa[ea][1], fa[ea][2], fa[ea][3], fb[eb][2 * i], fb[eb][2 * i + 1]);
      }
      double* dst = a.dots + (((int64_t)slot * a.G + grp) * kUnits + u) * 256;
      auto sum = [&](int i, int e) { return (double)acc[0][i][e] + 0x1p-12 * ((double)acc[1][i][e] + 0x1p-12 * (double)acc[2][i][e]); };
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          *reinterpret_cast<double2*>(dst + ((lane >> 2) + 8 * e) * 16 + i * 8 + (lane & 3) * 2) =
              make_double2(sum(i, 2 * e), sum(i, 2 * e + 1));
    }
  }
  if (tid == 0) bulk_wait<0>();
}

// ---------------------------------------------------------------------------------------------------------
// Coefficients of the chunks.  grid (chunks, H), 256 threads: decays; A (beta_t w_ts k_t . k_s, t > s); the inverse X of
// I + A in blocks of 16 tokens - diagonal blocks by forward substitution, a column per thread, then halves of 32 and of 64 from
// X_21 = -X_22 (A_21 X_11); C = K^T diag(w_63) X diag(beta) from three parts on mma.sync; P and P X diag(beta).
//
// A, X, P and P X are 64-bit (the products on mma.sync in f64, 64 multiply-adds per cycle and SM, as many as without it): with keys
// that share a direction their sums cancel, and what 32 bits lose there is two to three times what the kernel of blocks of four
// loses in all.  Rounded once, into the parts of C and P T.
//
// A token whose decay, beta or key is not finite makes itself and all that follow NaN, and no more: its rows of A are left out
// (a product would carry them to earlier tokens as 0 * NaN), its rows of P T and all of C become NaN.  A query's own row needs
// no care.
// ---------------------------------------------------------------------------------------------------------
constexpr int kPitchD = 20;              // numbers per row of a block of 16 x 16: fragment loads without bank conflicts
constexpr int kBlk = 16 * kPitchD;
template <int D>
struct CoefSmem {
  static constexpr int kRow = kChunk * 128;                  // one part's panel of K rows
  static constexpr int k = 0;                                // [parts][D / 64][64 rows], then C's image
  static constexpr int a = kParts * (D / 64) * kRow;         // A, then the parts of diag(w) T, then P, then P T's image
  static constexpr int x = a + 10 * kBlk * 8;
  static constexpr int total = x + 10 * kBlk * 8;
};
static_assert(kParts * kChunk * 128 <= 10 * kBlk * 8, "the parts fit in A's place");

// lower block (i, j)
__device__ __forceinline__ int blk_at(int i, int j) { return (i * (i + 1) / 2 + j) * kBlk; }

// acc (16 x 8) += left (16 x 16) . right (16 rows, 8 columns from `right` on)
__device__ __forceinline__ void block_mul(double (&acc)[4], const double* left, const double* right, int lane) {
  const double* pa = left + (lane >> 2) * kPitchD + (lane & 3);
  const double* pb = right + (lane & 3) * kPitchD + (lane >> 2);
  double fa[8], fb[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    fa[2 * k] = pa[4 * k];
    fa[2 * k + 1] = pa[8 * kPitchD + 4 * k];
    fb[k] = pb[4 * k * kPitchD];
  }
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7,%8,%9,%10,%11}, {%12,%13,%14,%15}, "
      "{%0,%1,%2,%3};"
      : "+d"(acc[0]), "+d"(acc[1]), "+d"(acc[2]), "+d"(acc[3])
      : "d"(fa[0]), "d"(fa[1]), "d"(fa[2]), "d"(fa[3]), "d"(fa[4]), "d"(fa[5]), "d"(fa[6]), "d"(fa[7]), "d"(fb[0]), "d"(fb[1]),
        "d"(fb[2]), "d"(fb[3]));
}
__device__ __forceinline__ void block_put(double* m, const double (&v)[4], double sign, int lane) {
  double* p = m + (lane >> 2) * kPitchD + (lane & 3) * 2;
  *reinterpret_cast<double2*>(p) = make_double2(sign * v[0], sign * v[1]);
  *reinterpret_cast<double2*>(p + 8 * kPitchD) = make_double2(sign * v[2], sign * v[3]);
}
// the three parts of two 64-bit numbers
__device__ __forceinline__ void split3(double x, double y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack2<true>((float)x, (float)y);
  const float2 h = unpack2<true>(hi);
  const float2 r = make_float2((float)(x - (double)h.x), (float)(y - (double)h.y));
  mid = pack2<true>(r.x, r.y);
  const float2 m = unpack2<true>(mid);
  lo = pack2<true>(r.x - m.x, r.y - m.y);
}

template <typename T, int D>
__global__ void __launch_bounds__(kPrepThreads, 2) delta_coef_kernel(const DeltaChunkArgs a) {
  pdl_wait();
  pdl_trigger();
  using L = CoefSmem<D>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ float2 s_tok[kChunk];                    // decays and betas
  __shared__ uint64_t s_bar;
  __shared__ double s_pre[kChunk], s_suf[kChunk];     // products of the decays of a token's block up to it, and behind it
  __shared__ int s_bad;                               // first token that is not finite
  const int h = blockIdx.y, grp = h / (a.H / a.G);
  int b, c, t0, n;
  if (!chunk_of_block(a, b, c, t0, n)) return;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, slot = blockIdx.x;
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  double *A = reinterpret_cast<double*>(sm + L::a), *X = reinterpret_cast<double*>(sm + L::x);
  const double* dots = a.dots + ((int64_t)slot * a.G + grp) * kUnits * 256;

  if (tid == 0) {       // k's rows, used by the product at the end
    mbar_init(&s_bar, 1);
    mbar_fence_init();
    const unsigned char* kq = a.kq + ((int64_t)slot * a.G + grp) * (kParts * (D / 64) * kPanel);
    mbar_expect_tx(&s_bar, kParts * (D / 64) * L::kRow);
    if (h > 0 || a.hold >= 0 || c != -a.hold - 1)
      for (int i = 0; i < kParts * (D / 64); ++i) bulk_load(sm + L::k + i * L::kRow, kq + i * kPanel, L::kRow, &s_bar);
    s_bad = kChunk;
  }
  // of the dots: threads 0 .. 63 a column of a diagonal block, the others eight numbers of the blocks below
  const int dblk = tid >> 4, dcol = tid & 15;
  auto diag_at = [&](int m) { return dots + (m * 10 + dblk * (dblk + 1) / 2 + dblk) * 256 + dcol; };
  auto below = [&](int i, int& bi, int& bj, int& t, int& s) {   // number i of this thread
    const int e = (i * 192 + tid - kChunk), q = e >> 8;         // blocks (1,0) (2,0) (2,1) (3,0) (3,1) (3,2)
    bi = q < 1 ? 1 : q < 3 ? 2 : 3;
    bj = q - (bi * (bi - 1)) / 2;
    t = (e >> 4) & 15;
    s = e & 15;
  };
  double dot[16];
  auto load_dots = [&](int m) {
    if (tid < kChunk) {
#pragma unroll
      for (int t = 0; t < 16; ++t) dot[t] = t >= dcol ? diag_at(m)[t * 16] : 0.0;
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        int bi, bj, t, s;
        below(i, bi, bj, t, s);
        dot[i] = dots[(m * 10 + bi * (bi + 1) / 2 + bj) * 256 + t * 16 + s];
      }
    }
  };
  load_dots(0);
  __syncthreads();      // s_bad
  if (tid < kChunk) {
    float2 tok = make_float2(1.f, 0.f);     // missing tokens: decay 1, beta 0
    if (tid < n) {
      const T* pr = static_cast<const T*>(a.proj) + (int64_t)(t0 + c * kChunk + tid) * a.proj_stride;
      tok = make_float2(exp_1ulp(-expf(a.A_log[h]) * softplus_f(to_f<T>(pr[a.a_off + h]) + a.dt_bias[h])),
                        sigmoid_f(to_f<T>(pr[a.b_off + h])));
    }
    s_tok[tid] = tok;
    double own = 0.0;                       // the key's product with itself
#pragma unroll
    for (int t = 0; t < 16; ++t)
      if (t == dcol) own = dot[t];
    if (!(fabsf(tok.x) + fabsf(tok.y) + fabsf((float)own) < 1e30f)) atomicMin(&s_bad, tid);
    double up = tok.x, down = tok.x;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
      const double lo = __shfl_up_sync(0xffffffffu, up, o, 16), hi = __shfl_down_sync(0xffffffffu, down, o, 16);
      if (dcol >= o) up *= lo;
      if (dcol + o < 16) down *= hi;
    }
    const double behind = __shfl_down_sync(0xffffffffu, down, 1, 16);
    s_pre[tid] = up;
    s_suf[tid] = dcol < 15 ? behind : 1.0;
  }
  __syncthreads();
  const int bad = s_bad;
  auto whole = [&](int i) { return s_pre[i * 16 + 15]; };   // a block's decays
  // w of the blocks below: behind s, the blocks between, up to t
  auto below_w = [&](int bi, int bj, int t, int s) {
    double w = s_suf[bj * 16 + s] * s_pre[bi * 16 + t];
    for (int i = bj + 1; i < bi; ++i) w *= whole(i);
    return w;
  };
  if (tid < kChunk) {   // G_t, and the diagonal blocks of A and X
    double g = s_pre[tid];
    for (int i = 0; i < dblk; ++i) g *= whole(i);
    a.gw[((int64_t)slot * a.H + h) * kChunk + tid] = (float)g;
    double* d = A + blk_at(dblk, dblk);
    double w = 1.0;
#pragma unroll
    for (int t = 1; t < 16; ++t)
      if (t > dcol) {
        w *= (double)s_tok[dblk * 16 + t].x;
        d[t * kPitchD + dcol] = dblk * 16 + t < bad ? (double)s_tok[dblk * 16 + t].y * w * dot[t] : 0.0;
      }
    __syncwarp();
    double x[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      double acc0 = t == dcol ? 1.0 : 0.0, acc1 = 0.0;
#pragma unroll
      for (int s = 0; s < t; ++s) {
        const double r = d[t * kPitchD + s];
        if (s & 1) acc1 = fma(-r, x[s], acc1);
        else acc0 = fma(-r, x[s], acc0);
      }
      x[t] = acc0 + acc1;
      X[blk_at(dblk, dblk) + t * kPitchD + dcol] = t < dcol ? 0.0 : x[t];
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      int bi, bj, t, s;
      below(i, bi, bj, t, s);
      A[blk_at(bi, bj) + t * kPitchD + s] =
          bi * 16 + t < bad ? (double)s_tok[bi * 16 + t].y * below_w(bi, bj, t, s) * dot[i] : 0.0;
    }
  }
  __syncthreads();

  // ---- X below the diagonal: eight columns a warp; sums on the way lie in A's diagonal blocks ----
  const int half = (warp & 1) * 8, pair = warp >> 1;
  auto S_at = [&](int i) { return A + blk_at(i, i) + half; };
  if (pair < 2) {          // blocks (1, 0) and (3, 2)
    const int i = 2 * pair + 1, j = 2 * pair;
    double acc[4] = {}, res[4] = {};
    block_mul(acc, A + blk_at(i, j), X + blk_at(j, j) + half, lane);
    block_put(S_at(j), acc, -1.0, lane);
    __syncwarp();
    block_mul(res, X + blk_at(i, i), S_at(j), lane);
    block_put(X + blk_at(i, j) + half, res, 1.0, lane);
  }
  __syncthreads();
  if (pair < 2) {          // blocks (2, j) and (3, j)
    const int j = pair;
    double s2[4] = {}, s3[4] = {}, x2[4] = {}, x3[4] = {};
    for (int k = j; k < 2; ++k) {
      block_mul(s2, A + blk_at(2, k), X + blk_at(k, j) + half, lane);
      block_mul(s3, A + blk_at(3, k), X + blk_at(k, j) + half, lane);
    }
    block_put(S_at(2 * j), s2, -1.0, lane);
    block_put(S_at(2 * j + 1), s3, -1.0, lane);
    __syncwarp();
    block_mul(x2, X + blk_at(2, 2), S_at(2 * j), lane);
    block_mul(x3, X + blk_at(3, 2), S_at(2 * j), lane);
    block_mul(x3, X + blk_at(3, 3), S_at(2 * j + 1), lane);
    block_put(X + blk_at(2, j) + half, x2, 1.0, lane);
    block_put(X + blk_at(3, j) + half, x3, 1.0, lane);
  }
  __syncthreads();

  // ---- diag(w) X diag(beta) in parts: the lower blocks' rows in pieces of eight (the others are not read) ----
  for (int i = tid; i < 320; i += kPrepThreads) {
    const int q = i >> 5, bi = q < 1 ? 0 : q < 3 ? 1 : q < 6 ? 2 : 3, bj = q - bi * (bi + 1) / 2, t = (i >> 1) & 15, s0 = (i & 1) * 8;
    double w = s_suf[bi * 16 + t];
    for (int k = bi + 1; k < 4; ++k) w *= whole(k);
    const double2* x = reinterpret_cast<const double2*>(X + blk_at(bi, bj) + t * kPitchD + s0);
    uint32_t p[kParts][4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const double2 v = x[e];
      const int s = bj * 16 + s0 + 2 * e;
      split3(v.x * (w * (double)s_tok[s].y), v.y * (w * (double)s_tok[s + 1].y), p[0][e], p[1][e], p[2][e]);
    }
#pragma unroll
    for (int e = 0; e < kParts; ++e)
      *reinterpret_cast<uint4*>(sm + L::a + e * L::kRow + panel_at(bi * 16 + t, bj * 2 + (i & 1))) =
          make_uint4(p[e][0], p[e][1], p[e][2], p[e][3]);
  }
  load_dots(1);
  {
    uint32_t spins = 0;
    bool ok = dc_try(&s_bar, 0);
    while (!ok && spins < a.spins) {
      ++spins;
      ok = dc_try(&s_bar, 0);
    }
    if (!__syncthreads_and(ok)) {    // the chunk is void
      if (tid < kChunk) a.gw[((int64_t)slot * a.H + h) * kChunk + tid] = __int_as_float(0x7fc00000);
      if (tid == 0) {
        atomicAdd(&g_delta_chunk_aborts, 1);
        for (spins = 0; !dc_try(&s_bar, 0) && spins < a.spins; ++spins) {}   // the loads land before the CTA ends
      }
      return;
    }
  }

  // ---- C: 16 channels a warp, all 64 columns; column block nb has rows of token blocks kb >= nb.  The largest pair's sums
  // leave the tensor pipe, which truncates, after each 16 tokens ----
  float big[4][2][4] = {}, rest[4][2][4] = {};
  if (warp < D / 16) {
    const uint32_t kb_at = smem_u32(sm + L::k), tb_at = smem_u32(sm + L::a);
    const int piece_a = 2 * warp + ((lane >> 3) & 1), row_a = (lane & 7) + ((lane >> 4) << 3), row_b = (lane & 7) + (((lane >> 3) & 1) << 3);
#pragma unroll
    for (int kb = 0; kb < 4; ++kb) {
      uint32_t fa[kParts][4];
#pragma unroll
      for (int e = 0; e < kParts; ++e)
        ldmatrix4_trans(fa[e], kb_at + (e * (D / 64) + (piece_a >> 3)) * L::kRow + panel_at(kb * 16 + row_a, piece_a & 7));
#pragma unroll
      for (int nb = 0; nb <= kb; ++nb) {
        uint32_t fb[kParts][4];
#pragma unroll
        for (int e = 0; e < kParts; ++e) ldmatrix4_trans(fb[e], tb_at + e * L::kRow + panel_at(kb * 16 + row_b, nb * 2 + (lane >> 4)));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          float part[4] = {};
          mma_parts(part, rest[nb][i], fa, fb, i);
#pragma unroll
          for (int e = 0; e < 4; ++e) big[nb][i][e] += part[e];
        }
      }
    }
  }
  __syncthreads();   // K and the parts are read: C's image and P take their places
  if (warp < D / 16) {
    const float nan = __int_as_float(0x7fc00000);
#pragma unroll
    for (int nb = 0; nb < 4; ++nb)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          uint32_t p[kParts];
          const float u = big[nb][i][2 * e] + rest[nb][i][2 * e], v = big[nb][i][2 * e + 1] + rest[nb][i][2 * e + 1];
          split3(bad < kChunk ? nan : u, bad < kChunk ? nan : v, p[0], p[1], p[2]);
          const int at = panel_at(warp * 16 + (lane >> 2) + 8 * e, nb * 2 + i) + (lane & 3) * 4;
#pragma unroll
          for (int q = 0; q < kParts; ++q) *reinterpret_cast<uint32_t*>(sm + L::k + q * D * 128 + at) = p[q];
        }
  }
  if (tid < kChunk) {
    double* d = A + blk_at(dblk, dblk);
    double w = 1.0;
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      if (t > dcol) w *= (double)s_tok[dblk * 16 + t].x;
      d[t * kPitchD + dcol] = t >= dcol ? w * dot[t] : 0.0;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      int bi, bj, t, s;
      below(i, bi, bj, t, s);
      A[blk_at(bi, bj) + t * kPitchD + s] = below_w(bi, bj, t, s) * dot[i];
    }
  }
  __syncthreads();

  // ---- P X: the ten lower blocks, five block products a pair of warps, eight columns a warp ----
  const uint32_t blocks = pair == 0 ? 0x0030u : pair == 1 ? 0x3220u : pair == 2 ? 0x1031u : 0x33221121u;   // a byte each: row, column
  double acc[4][4] = {};
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (q < 2 || pair == 3) {
      const int i = (blocks >> (8 * q + 4)) & 15, j = (blocks >> (8 * q)) & 15;
#pragma unroll 1
      for (int k = j; k <= i; ++k) block_mul(acc[q], A + blk_at(i, k), X + blk_at(k, j) + half, lane);
    }
  __syncthreads();   // P is read: the image takes its place
  auto put_pt = [&](int i, int j, const double (&v)[4]) {
    const int s = j * 16 + half + (lane & 3) * 2;
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int t = i * 16 + (lane >> 2) + 8 * e;
      double u0 = s <= t ? v[2 * e] * (double)s_tok[s].y : 0.0, u1 = s < t ? v[2 * e + 1] * (double)s_tok[s + 1].y : 0.0;
      if (t >= bad) u0 = s <= t ? nan : 0.0, u1 = s < t ? nan : 0.0;
      uint32_t p[kParts];
      split3(u0, u1, p[0], p[1], p[2]);
#pragma unroll
      for (int q = 0; q < kParts; ++q)
        *reinterpret_cast<uint32_t*>(sm + L::a + q * L::kRow + panel_at(t, s >> 3) + (s & 7) * 2) = p[q];
    }
  };
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (q < 2 || pair == 3) put_pt((blocks >> (8 * q + 4)) & 15, (blocks >> (8 * q)) & 15, acc[q]);
  {
    const double zero[4] = {};
    for (int q = pair; q < 6; q += 4) {
      const int i = q < 3 ? 0 : q < 5 ? 1 : 2, j = q < 3 ? q + 1 : q < 5 ? q - 1 : 3;
      put_pt(i, j, zero);
    }
  }
  fence_proxy_async_smem();
  __syncthreads();
  if (tid == 0) {
    unsigned char* dst = a.cp + ((int64_t)slot * a.H + h) * (kParts * (D + kChunk) * 128);
    for (int e = 0; e < kParts; ++e) {
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst + e * (D + kChunk) * 128),
                   "r"(smem_u32(sm + L::k + e * D * 128)), "r"(D * 128)
                   : "memory");
      asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst + e * (D + kChunk) * 128 + D * 128),
                   "r"(smem_u32(sm + L::a + e * L::kRow)), "r"(L::kRow)
                   : "memory");
    }
    bulk_commit();
    bulk_wait<0>();
  }
}

// ---------------------------------------------------------------------------------------------------------
// The chunks of one (head, sequence).  grid (H * Dv / 32, B), clusters of Dv / 32; 512 threads: warps 0 - 7 turn products
// into operands (TMEM lane = row: token or key channel; warps 4 - 7 the second 16 columns), warp 8 issues the products,
// warp 9 the copies; warps 10, 11, 14 and 15 read the lanes of Q S and P T R and make the outputs (12 and 13 only fill the
// place that gives those warps their quarter of TMEM).
// ---------------------------------------------------------------------------------------------------------
template <int D>
struct ChunkSmem {
  static constexpr int kqPart = (D / 64) * kPanel;          // [K; Q], one part
  static constexpr int cpPart = (D + kChunk) * 128;         // [C; P T], one part
  static constexpr int kq = 0;
  static constexpr int cp = kParts * kqPart;
  static constexpr int s = cp + kParts * cpPart;            // [parts][D rows][64 bytes]
  static constexpr int sPart = D * kCols * 2;
  static constexpr int r = s + kParts * sPart;              // [parts][64 rows][64 bytes]
  static constexpr int rPart = kChunk * kCols * 2;
  static constexpr int total = r + kParts * rPart;
};

struct ChunkBars {
  uint64_t kq_full[kParts], cp_full;
  uint64_t y_done, s_done, o_done;       // the products [K; Q] S, C R and P T R
  uint64_t s_full, r_full;               // their right operands
  uint64_t o_free;                       // P T R is read
  uint64_t norm[2], drain;
  float part[2][16][kChunk];             // sums of squares: [CTA * 2 + column half][token]
  float norm_w[kCols];
  int bad[2][kCols], any_bad[2];         // first token of the chunk whose R is not finite, per column
  uint32_t tmem_base, spins;
  volatile uint32_t abort;
};

__device__ __forceinline__ bool dc_wait(uint64_t* bar, uint32_t parity, ChunkBars& b) {
  uint32_t spins = 0;
  while (!dc_try(bar, parity)) {
    if (b.abort) return false;
    if (++spins > b.spins) {
      b.abort = 1;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool dc_wait_warp(uint64_t* bar, uint32_t parity, ChunkBars& b) {
  return __all_sync(0xffffffffu, dc_wait(bar, parity, b));
}
// right operands: N runs along the rows of memory (64 bytes of 32 columns a part), 64-byte swizzle
__device__ __forceinline__ uint64_t cols_desc(uint32_t addr, int part_bytes) {
  return (umma_smem_desc(addr, part_bytes, 512) & ~((uint64_t)7 << 61)) | ((uint64_t)4 << 61);
}
// 16 columns (`half` of the 32) of row `row` -> the three parts of a right operand
__device__ __forceinline__ void put_parts(unsigned char* base, int part_bytes, int row, int half, const float2 (&v)[8]) {
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    uint32_t p[kParts][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) split3(v[4 * q + i], p[0][i], p[1][i], p[2][i]);
    const int at = row * 64 + (((half * 2 + q) ^ ((row >> 1) & 3)) << 4);
#pragma unroll
    for (int e = 0; e < kParts; ++e)
      *reinterpret_cast<uint4*>(base + e * part_bytes + at) = make_uint4(p[e][0], p[e][1], p[e][2], p[e][3]);
  }
}
// the three sums of a product, smallest first
__device__ __forceinline__ void take_product(uint32_t addr, float2 (&v)[8]) {
  uint32_t x[3][16];
#pragma unroll
  for (int e = 0; e < 3; ++e) tmem_ld16(addr + e * kCols, x[e]);
  tc_wait_ld();
  auto pair = [&](int e, int j) { return make_float2(__uint_as_float(x[e][2 * j]), __uint_as_float(x[e][2 * j + 1])); };
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = __fadd2_rn(pair(0, j), __fadd2_rn(pair(1, j), pair(2, j)));
}

// [K; Q] S: the largest sum lies in four accumulators, a quarter of the key channels each, behind them the two others
constexpr int kFirst = 4;
__device__ __forceinline__ void take_first(uint32_t addr, float2 (&v)[8]) {
  auto pair = [](const uint32_t (&x)[16], int j) { return make_float2(__uint_as_float(x[2 * j]), __uint_as_float(x[2 * j + 1])); };
  uint32_t x[2][16];
  tmem_ld16(addr, x[0]);
  tmem_ld16(addr + kCols, x[1]);
  tc_wait_ld();
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = __fadd2_rn(pair(x[0], j), pair(x[1], j));
  tmem_ld16(addr + 2 * kCols, x[0]);
  tmem_ld16(addr + 3 * kCols, x[1]);
  tc_wait_ld();
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = __fadd2_rn(v[j], __fadd2_rn(pair(x[0], j), pair(x[1], j)));
  tmem_ld16(addr + 4 * kCols, x[0]);
  tmem_ld16(addr + 5 * kCols, x[1]);
  tc_wait_ld();
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = __fadd2_rn(v[j], __fadd2_rn(pair(x[0], j), pair(x[1], j)));
}

template <typename T, int D>
__global__ void __launch_bounds__(512, 1) delta_chunk_kernel(const DeltaChunkArgs a) {
  pdl_wait();
  using L = ChunkSmem<D>;
  extern __shared__ unsigned char smem_raw[];
  __shared__ ChunkBars bars;
  const int VT = a.Dv / kCols, h = blockIdx.x / VT, vt = blockIdx.x % VT, b = blockIdx.y;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int t0, n_all, start;
  portion(a.g, b, t0, n_all, start);
  const int base = a.per_seq > 0 ? 0 : t0 / kChunk + b, first = max(0, a.window - base);
  const int chunks = min(cdiv(max(n_all, 0), kChunk), a.window + (a.per_seq > 0 ? a.per_seq : a.slots) - base) - first;
  if (chunks <= 0) return;                 // the same for every CTA of the cluster
  const int seq_slot = a.g.slots[b], grp = h / (a.H / a.G);
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));

  if (tid == 0) {
    for (int e = 0; e < kParts; ++e) mbar_init(&bars.kq_full[e], 1);
    mbar_init(&bars.cp_full, 1);
    mbar_init(&bars.y_done, 1);
    mbar_init(&bars.s_done, 1);
    mbar_init(&bars.o_done, 1);
    mbar_init(&bars.s_full, 384);          // eight warps of the state, four of the outputs (Q S is read)
    mbar_init(&bars.r_full, 128);
    mbar_init(&bars.o_free, 128);
    mbar_init(&bars.norm[0], VT > 1 ? 1 : 2 * kChunk);
    mbar_init(&bars.norm[1], VT > 1 ? 1 : 2 * kChunk);
    mbar_init(&bars.drain, 1);
    bars.any_bad[0] = bars.any_bad[1] = 0;
    bars.abort = 0;
    bars.spins = a.spins;
    mbar_fence_init();
  }
  if (tid < kCols) {
    bars.norm_w[tid] = a.norm_w[h * a.norm_head_stride + vt * kCols + tid];
    bars.bad[0][tid] = bars.bad[1][tid] = kChunk;
  }
  if (warp == 8) {
    tmem_alloc(&bars.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (VT > 1) cluster_sync_all();          // barriers exist before a neighbour writes to them
  const uint32_t tmem = bars.tmem_base;
  constexpr uint32_t kY = 0, kS = 256, kO = 384;   // TMEM columns of the products
  const int first_slot = base + first - a.window + b * a.per_seq;
  bool ok = true;

  if (warp == 9) {
    // ------------------------------ copies ------------------------------
    if (lane == 0) {
      const unsigned char* kq = a.kq + ((int64_t)first_slot * a.G + grp) * (kParts * L::kqPart);
      const unsigned char* cp = a.cp + ((int64_t)first_slot * a.H + h) * (kParts * L::cpPart);
      const int64_t kq_step = (int64_t)a.G * kParts * L::kqPart, cp_step = (int64_t)a.H * kParts * L::cpPart;
      int begun = 0, begun_cp = 0;
      for (int c = 0; c < chunks; ++c) {
        // the images' places are free behind the last chunk's first product and its last one
        if (c > 0) ok = dc_wait(&bars.y_done, (c - 1) & 1, bars);
        if (!ok) break;
        for (int e = 0; e < kParts; ++e) {
          mbar_expect_tx(&bars.kq_full[e], L::kqPart);
          if (blockIdx.x > 0 || first + c != a.hold - 1)
            bulk_load(sm + L::kq + e * L::kqPart, kq + c * kq_step + e * L::kqPart, L::kqPart, &bars.kq_full[e]);
        }
        ++begun;
        if (c > 0) ok = dc_wait(&bars.o_done, (c - 1) & 1, bars);
        if (!ok) break;
        mbar_expect_tx(&bars.cp_full, kParts * L::cpPart);
        bulk_load(sm + L::cp, cp + c * cp_step, kParts * L::cpPart, &bars.cp_full);
        ++begun_cp;
      }
      {                  // copies in flight land before the CTA ends, also those that nobody waits for any more
        auto land = [&](uint64_t* bar, int n) {
          for (uint32_t spins = 0; n > 0 && !dc_try(bar, (n - 1) & 1) && spins < a.spins; ++spins) {}
        };
        for (int e = 0; e < kParts; ++e) land(&bars.kq_full[e], begun);
        land(&bars.cp_full, begun_cp);
      }
    }
  } else if (warp == 8) {
    // ----------------------------- products -----------------------------
    const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
    const uint64_t kq_d = umma_smem_desc(smem_u32(sm + L::kq), 16, 1024);
    const uint64_t cp_d = umma_smem_desc(smem_u32(sm + L::cp), 16, 1024);
    const uint64_t s_d = cols_desc(smem_u32(sm + L::s), L::sPart);
    const uint64_t r_d = cols_desc(smem_u32(sm + L::r), L::rPart);
    // the left operand's part e meets the first 3 - e parts of the right one
    auto product = [&](uint32_t d, int e, int ks, uint64_t left, uint64_t right) {
      umma_ss_warp(tm + d + e * kCols, left, right, umma_idesc(true, 128, kCols * (kParts - e), false, true),
                   (e > 0 || ks > 0) ? 1u : 0u);
    };
    // 128 rows of [C; P T] from row `row` on, times R
    auto product_r = [&](uint32_t d, int row) {
#pragma unroll
      for (int e = 0; e < kParts; ++e)
#pragma unroll
        for (int ks = 0; ks < kChunk / 16; ++ks)
          product(d, e, ks, umma_desc_add(cp_d, e * L::cpPart + row * 128 + ks * 32), umma_desc_add(r_d, ks * 1024));
    };
    for (int c = 0; c < chunks && ok; ++c) {
      const uint32_t ph = c & 1;
      ok = dc_wait_warp(&bars.s_full, ph, bars);
#pragma unroll
      for (int e = 0; e < kParts; ++e) {
        ok = ok && dc_wait_warp(&bars.kq_full[e], ph, bars);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          constexpr int kStep = D / 16 / kFirst;      // products per accumulator of the largest sum
          const uint64_t left = umma_desc_add(kq_d, e * L::kqPart + (ks >> 2) * kPanel + (ks & 3) * 32), right = umma_desc_add(s_d, ks * 1024);
          if (e == 0)
            umma_ss_warp(tm + kY + (ks / kStep) * kCols, left, right, umma_idesc(true, 128, kCols, false, true), ks % kStep > 0);
          umma_ss_warp(tm + kY + (kFirst + (e == 2)) * kCols, left, e == 0 ? umma_desc_add(right, L::sPart) : right,
                       umma_idesc(true, 128, e == 2 ? kCols : 2 * kCols, false, true), e > 0 || ks > 0);
        }
      }
      if (!ok) break;
      umma_commit_warp(&bars.y_done);
      ok = dc_wait_warp(&bars.cp_full, ph, bars) && dc_wait_warp(&bars.r_full, ph, bars) &&
           (c == 0 || dc_wait_warp(&bars.o_free, ph ^ 1, bars));
      if (!ok) break;
      tc_fence_after();
      product_r(kS, 0);                    // heads of 64: C and P T at once
      umma_commit_warp(&bars.s_done);
      if (D == 128) product_r(kO, 64);     // lanes 64 .. 127: P T (the others: C's second half again, not read)
      umma_commit_warp(&bars.o_done);
    }
    if (!ok) {           // products in flight end before TMEM is given back
      umma_commit_warp(&bars.drain);
      for (uint32_t spins = 0; !dc_try(&bars.drain, 0) && spins < a.spins; ++spins) {}
    }
    __syncwarp();
  } else if (warp < 8) {
    // -------------------- products to operands, state --------------------
    const int q4 = warp & 3, half = warp >> 2, row = q4 * 32 + lane;   // TMEM lane
    const bool early = q4 < 2;             // rows 0 .. 63, the chunk's tokens: R
    const int col0 = vt * kCols + half * 16;
    const uint32_t my = tmem + ((uint32_t)(q4 * 32) << 16) + half * 16;
    const bool keyed = row < D;            // a key channel's thread
    float* st = a.state + (((int64_t)seq_slot * a.H + h) * a.Dv + col0) * D + row;
    const int64_t carried = (((int64_t)(a.per_seq > 0 ? b : 0) * a.H + h) * a.Dv + col0) * D + row;
    const float* gw = a.gw + ((int64_t)first_slot * a.H + h) * kChunk;
    float2 S[8];
    {
      const float* from = first > 0 ? a.carry_in + carried : st;
      const bool zero = !keyed || (first == 0 && start <= 0);
#pragma unroll
      for (int j = 0; j < 8; ++j)
        S[j] = zero ? make_float2(0.f, 0.f) : make_float2(from[(int64_t)(2 * j) * D], from[(int64_t)(2 * j + 1) * D]);
    }
    if (keyed) put_parts(sm + L::s, L::sPart, row, half, S);
    fence_proxy_async_smem();
    mbar_arrive(&bars.s_full);

    for (int c = 0; c < chunks; ++c) {
      const uint32_t ph = c & 1;
      const float g_all = gw[kChunk - 1];
      // ---- K S -> R = V - G K S ----
      if (early) {
        const int tok = (first + c) * kChunk + row;       // within the portion
        const float g_t = -gw[row];
        float4 v[4];
        {
          const float4* p = reinterpret_cast<const float4*>(a.qkv + (int64_t)(t0 + tok) * a.qkv_stride + 2 * a.G * D + h * a.Dv + col0);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] = tok < n_all ? p[j] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        ok = dc_wait_warp(&bars.y_done, ph, bars);
        if (!ok) break;
        tc_fence_after();
        float2 o[8], not_finite = make_float2(0.f, 0.f);
        take_first(my + kY, o);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          o[j] = __ffma2_rn(make_float2(g_t, g_t), o[j], j & 1 ? make_float2(v[j / 2].z, v[j / 2].w) : make_float2(v[j / 2].x, v[j / 2].y));
          not_finite = __ffma2_rn(o[j], make_float2(0.f, 0.f), not_finite);
        }
        if (!(not_finite.x + not_finite.y == 0.f)) {
          auto check = [&](float& x, int j) {
            if (!(fabsf(x) <= 3.3e38f)) {
              atomicMin(&bars.bad[ph][half * 16 + j], row);
              x = 0.f;
            }
          };
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            check(o[j].x, 2 * j);
            check(o[j].y, 2 * j + 1);
          }
          bars.any_bad[ph] = 1;
        }
        put_parts(sm + L::r, L::rPart, row, half, o);
        fence_proxy_async_smem();
        tc_fence_before();
        mbar_arrive(&bars.r_full);
      }
      // ---- the state behind the chunk ----
      ok = dc_wait_warp(&bars.s_done, ph, bars);
      if (!ok) break;
      tc_fence_after();
      if (warp == 0) {                     // the last chunk's, whose readers are through (s_full, o_free)
        bars.bad[ph ^ 1][lane] = kChunk;
        if (lane == 0) bars.any_bad[ph ^ 1] = 0;
      }
      float2 x[8];
      take_product(my + kS, x);
      if (*const_cast<volatile int*>(&bars.any_bad[ph])) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (bars.bad[ph][half * 16 + 2 * j] < kChunk) x[j].x = __int_as_float(0x7fc00000);
          if (bars.bad[ph][half * 16 + 2 * j + 1] < kChunk) x[j].y = __int_as_float(0x7fc00000);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) S[j] = __ffma2_rn(make_float2(g_all, g_all), S[j], x[j]);
      if (keyed) put_parts(sm + L::s, L::sPart, row, half, S);
      fence_proxy_async_smem();
      tc_fence_before();
      mbar_arrive(&bars.s_full);
      gw += (int64_t)a.H * kChunk;
    }
    if (keyed) {
      const bool ends = (first + chunks) * kChunk >= n_all;
      float* to = ends ? (seq_slot != a.reserved_slot ? st : nullptr) : a.carry_out + carried;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (to) {
          to[(int64_t)(2 * j) * D] = S[j].x;
          to[(int64_t)(2 * j + 1) * D] = S[j].y;
        }
    }
  } else if ((warp & 3) >= 2) {
    // ------------------------------ outputs ------------------------------
    const int q4 = warp & 3, half = (warp >> 2) - 2, t = (q4 - 2) * 32 + lane;   // TMEM lanes 64 .. 127: tokens
    const int col0 = vt * kCols + half * 16;
    const uint32_t my = tmem + ((uint32_t)(q4 * 32) << 16) + half * 16;
    const float* gw = a.gw + ((int64_t)first_slot * a.H + h) * kChunk + t;
    T* out = static_cast<T*>(a.out) + (int64_t)(t0 + first * kChunk + t) * a.out_stride + h * a.Dv + col0;
    const T* gate = static_cast<const T*>(a.gate) + (int64_t)(t0 + first * kChunk + t) * a.gate_stride + a.gate_off + h * a.Dv + col0;
    constexpr int kPieces = sizeof(T);     // 16 numbers in 16-byte pieces
    uint4 z[kPieces];
    int left = n_all - first * kChunk - t;   // tokens of the portion from this thread's on
    auto load_gate = [&]() {
#pragma unroll
      for (int j = 0; j < kPieces; ++j) z[j] = left > 0 ? *reinterpret_cast<const uint4*>(gate + j * (16 / sizeof(T))) : make_uint4(0, 0, 0, 0);
    };
    float g_t = *gw;
    load_gate();
    mbar_arrive(&bars.s_full);
    for (int c = 0; c < chunks; ++c) {
      const uint32_t ph = c & 1;
      float2 o[8], x[8];
      ok = dc_wait_warp(&bars.y_done, ph, bars);
      if (!ok) break;
      tc_fence_after();
      take_first(my + kY, o);
      tc_fence_before();
      mbar_arrive(&bars.s_full);           // Q S may be overwritten
      ok = dc_wait_warp(&bars.o_done, ph, bars);
      if (!ok) break;
      tc_fence_after();
      take_product(my + (D == 128 ? kO : kS), x);
      tc_fence_before();
      if (*const_cast<volatile int*>(&bars.any_bad[ph])) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          if (t >= bars.bad[ph][half * 16 + 2 * j]) x[j].x = __int_as_float(0x7fc00000);
          if (t >= bars.bad[ph][half * 16 + 2 * j + 1]) x[j].y = __int_as_float(0x7fc00000);
        }
      }
      mbar_arrive(&bars.o_free);
      float2 sq = make_float2(0.f, 0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o[j] = __ffma2_rn(make_float2(g_t, g_t), o[j], x[j]);
        sq = __ffma2_rn(o[j], o[j], sq);
      }
      float ss = sq.x + sq.y;
      float* mine = &bars.part[ph][vt * 2 + half][t];
      if (VT > 1) {
        if (t == 0 && half == 0) mbar_expect_tx(&bars.norm[ph], VT * 2 * kChunk * sizeof(float));
        for (int r = 0; r < VT; ++r)
          asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(mapa_u32(mine, r)),
                       "r"(__float_as_uint(ss)), "r"(mapa_u32(&bars.norm[ph], r))
                       : "memory");
      } else {       // a launch without clusters: st.async is an illegal instruction there
        *mine = ss;
        mbar_arrive(&bars.norm[ph]);
      }
      // ---- weight and gate, and the next chunk's ----
      auto gated = [&](float v, int j, float gz) { return v * bars.norm_w[half * 16 + j] * silu_fast(gz); };
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float2 gz;
        if constexpr (sizeof(T) == 2) {
          const uint32_t w[4] = {z[j / 4].x, z[j / 4].y, z[j / 4].z, z[j / 4].w};
          gz = unpack2<true>(w[j & 3]);
        } else {
          gz = j & 1 ? make_float2(__uint_as_float(z[j / 2].z), __uint_as_float(z[j / 2].w))
                     : make_float2(__uint_as_float(z[j / 2].x), __uint_as_float(z[j / 2].y));
        }
        o[j] = make_float2(gated(o[j].x, 2 * j, gz.x), gated(o[j].y, 2 * j + 1, gz.y));
      }
      const bool real = left > 0;
      if (c + 1 < chunks) {
        left -= kChunk;
        gw += (int64_t)a.H * kChunk;
        gate += (int64_t)kChunk * a.gate_stride;
        g_t = *gw;
        load_gate();
      }
      // ---- unit norm over the columns of all CTAs ----
      ok = dc_wait_warp(&bars.norm[ph], (c >> 1) & 1, bars);
      if (!ok) break;
      ss = 0.f;
      for (int r = 0; r < 2 * VT; ++r) ss += bars.part[ph][r][t];
      const float inv = 1.0f / sqrtf(ss / (float)a.Dv + a.eps);
      if (real) {
#pragma unroll
        for (int j = 0; j < 8; ++j) o[j] = __fmul2_rn(o[j], make_float2(inv, inv));
        if constexpr (sizeof(T) == 2) {
#pragma unroll
          for (int j = 0; j < 2; ++j)
            *reinterpret_cast<uint4*>(out + 8 * j) =
                make_uint4(pack2<true>(o[4 * j].x, o[4 * j].y), pack2<true>(o[4 * j + 1].x, o[4 * j + 1].y),
                           pack2<true>(o[4 * j + 2].x, o[4 * j + 2].y), pack2<true>(o[4 * j + 3].x, o[4 * j + 3].y));
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<float4*>(out + 4 * j) = make_float4(o[2 * j].x, o[2 * j].y, o[2 * j + 1].x, o[2 * j + 1].y);
        }
      }
      out += (int64_t)kChunk * a.out_stride;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (bars.abort) {                        // whichever role gave up
    const float nan = __int_as_float(0x7fc00000);
    const int64_t cols = (int64_t)h * a.Dv + vt * kCols;
    const bool ends = (first + chunks) * kChunk >= n_all;
    float* to = ends ? (seq_slot != a.reserved_slot ? a.state + (int64_t)seq_slot * a.H * a.Dv * D : nullptr)
                     : a.carry_out + (int64_t)(a.per_seq > 0 ? b : 0) * a.H * a.Dv * D;
    if (to)
      for (int i = tid; i < kCols * D; i += 512) to[cols * D + i] = nan;
    const int rows = min(n_all - first * kChunk, chunks * kChunk);
    T* out = static_cast<T*>(a.out) + (int64_t)(t0 + first * kChunk) * a.out_stride + cols;
    for (int i = tid; i < rows * kCols; i += 512) out[(int64_t)(i / kCols) * a.out_stride + i % kCols] = from_f<T>(nan);
    if (tid == 0) atomicAdd(&g_delta_chunk_aborts, 1);
  }
  if (VT > 1) {
    cluster_sync_all();                    // nobody leaves while its sums may still be written:
    if (bars.abort) __nanosleep(20000);    // here a neighbour's last ones may be under way, for nobody waited for them
  }
  if (warp == 8) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

struct ChunkPlan {
  int windows, slots, per_seq;
  size_t cp, dots, gw, carry, other_carry, bytes;
};

// Images take 98 KB per chunk and key head and 74 KB per chunk and head (heads of 128), products 41 KB per key head: 0.3 GB per 4096
// tokens of 16 / 32 heads.  Above `kMost` the chunks are taken in windows of equal length: the row of all chunks is cut, so that a
// window is full however the tokens are spread (8000 tokens beside 15 times 500, 32 / 16 heads: 2.83 -> 1.64 ms against a range of
// every sequence's chunks; 6000 beside 31 single tokens: 3.38 -> 0.93 ms), and ends in at most one sequence, whose state is
// carried to the next.  Where a window of the row would hold too few sequences for the SMs and the sequences are about equally long,
// a window takes a range of every sequence's chunks instead (8 times 4096 tokens, 8 heads of 128 x 64: 1.10 -> 0.74 ms).
constexpr size_t kMost = (size_t)320 << 20;

ChunkPlan chunk_plan(int64_t tokens, int B, int max_new, int H, int G, int D, int Dv) {
  ChunkPlan p{};
  const size_t kq = (size_t)G * kParts * (D / 64) * kPanel, cp = (size_t)H * kParts * (D + kChunk) * 128;
  const size_t dots = (size_t)G * kUnits * 256 * sizeof(double), gw = (size_t)H * kChunk * sizeof(float);
  const size_t state = (size_t)H * Dv * D * sizeof(float);
  const int64_t all = tokens / kChunk + B;      // cu_q[b] / 64 + b + c is below this
  const int64_t most = std::max<int64_t>(1, (int64_t)(kMost / (kq + cp + dots + gw)));
  const int chunks = cdiv(max_new, kChunk);
  p.windows = (int)((all + most - 1) / most);
  p.slots = (int)((all + p.windows - 1) / p.windows);
  if (p.windows > 1 && B <= most && B * state <= kMost / 4 && 4 * tokens >= 3 * (int64_t)B * max_new &&
      (p.slots / chunks + 1) * (int64_t)H * (Dv / kCols) < sm_count()) {
    p.per_seq = (int)std::min<int64_t>(most / B, chunks);
    p.windows = cdiv(chunks, p.per_seq);
    p.per_seq = cdiv(chunks, p.windows);
    p.slots = p.per_seq * B;
  }
  p.cp = p.slots * kq;
  p.dots = p.cp + p.slots * cp;
  p.gw = p.dots + p.slots * dots;
  p.carry = p.gw + p.slots * gw;
  p.other_carry = p.carry + (p.per_seq > 0 ? 0 : state);       // of its own: one sequence's is read while another's is written
  p.bytes = p.windows == 1 ? p.carry : p.per_seq > 0 ? p.carry + B * state : p.other_carry + state;
  return p;
}

template <typename T, int D>
int launch_chunks(DeltaChunkArgs a, const ChunkPlan& p, int B, cudaStream_t st) {
  static std::atomic<uint64_t> attr_r{0}, attr_k{0}, attr_c{0};
  constexpr size_t smem_r = (size_t)kParts * (D / 64) * kPanel + 1024, smem_k = CoefSmem<D>::total + 1024,
                   smem_c = ChunkSmem<D>::total + 1024;
  CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)delta_rows_kernel<D>, (int)smem_r, attr_r));
  CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)delta_coef_kernel<T, D>, (int)smem_k, attr_k));
  CVLLM_CHECK_CUDA(ensure_max_dyn_smem((const void*)delta_chunk_kernel<T, D>, (int)smem_c, attr_c));
  const int VT = a.Dv / kCols;
  for (int w = 0; w < p.windows; ++w) {
    a.window = w * (p.per_seq > 0 ? p.per_seq : p.slots);
    if (w > 0) std::swap(a.carry_in, a.carry_out);
    // Each beside the end of the one in front, for heads of 64.  With heads of 128 the next kernel's CTAs then come two to the SMs that are
    // free first, where one each is faster: 300 + 200 tokens, 16 / 8 heads, 68.4 us for 63.3 one behind the other, 400 + 100 73.5 for
    // 68.5, 400 with 32 / 16 93.3 for 89.9, 2000 183.2 for 180.6; heads of 64: 600 tokens 66.6 for 67.7, 2000 150.0 for 151.9.
    constexpr bool kBehind = D == 64;
    if constexpr (kBehind) {
      CVLLM_CHECK_CUDA(launch_behind(delta_rows_kernel<D>, dim3(p.slots, a.G), dim3(kPrepThreads), smem_r, st, a));
      CVLLM_CHECK_CUDA(launch_behind(delta_coef_kernel<T, D>, dim3(p.slots, a.H), dim3(kPrepThreads), smem_k, st, a));
    } else {
      delta_rows_kernel<D><<<dim3(p.slots, a.G), kPrepThreads, smem_r, st>>>(a);
      delta_coef_kernel<T, D><<<dim3(p.slots, a.H), kPrepThreads, smem_k, st>>>(a);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.H * VT, B);
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = smem_c;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = kBehind;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = VT;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = VT > 1 ? 2 : 1;
    CVLLM_CHECK_CUDA(cudaLaunchKernelEx(&cfg, delta_chunk_kernel<T, D>, a));
  }
  CVLLM_CHECK_LAUNCHES(3 * p.windows);
  return CVLLM_OK;
}

}  // namespace
}  // namespace cvllm

using namespace cvllm;

// From where the chunks are faster than the blocks of four (cvllm_delta_rule).  The three launches take 35 to 45 us for 64 tokens, the
// blocks of four 0.23 us a token (heads of 128) or 0.16 (64) while they are few; with `pairs` (head, sequence) pairs at work at once
// both grow.  Coefficients cost the same whatever Dv, and the blocks of four pass value sizes of 32 and 64 at twice the rate per column.
// Blocks' time / chunks' in us, at the lines (32 or 16 heads, lengths x sequences):
//   128 x 128: 192 x 1: 54 / 46; 128 x 1: 39 / 43; 128 x 4, 16 heads (64 pairs): 56 / 62; 128 x 4, 32 heads (128): 108 / 83
//   64 x 256: 256 x 1, 32 heads: 70 / 74; 384 x 1: 99 / 90; 64 x 128: 128 x 16, 16 heads (256): 137 / 141; 192 x 16: 210 / 187
//   128 x 64: 256 x 2, 16 heads: 53 / 56; 512 x 2, 32 heads: 125 / 92; 512 x 16, 8 heads (128): 177 / 203
//   128 x 32: 512 x 2, 16 heads: 90 / 67; 1024 x 4, 16 heads (64): 178 / 191; 64 x 32: 1024 x 8, 16 heads: 168 / 239
// Every sequence fills whole chunks: 96 tokens a sequence on average at least (7 single tokens and 762: 293 / 179).
// Of 2886 measured batches (D 64 and 128, Dv 32 to 256, 4 to 64 heads, 1 to 32 equal or ragged sequences) none is slower by the rule.
static bool chunks_are_faster(int64_t tokens, int B, int max_new, int H, int D, int Dv) {
  if (max_new < 2 * kChunk || tokens < 96 * (int64_t)B) return false;
  const int64_t work = H * tokens;             // pairs * max_new
  auto pairs_above = [&](int64_t n) { return work > n * max_new; };
  if (Dv >= 3 * kCols) {
    if (D == 128) return max_new >= 192 || pairs_above(64);
    return max_new >= (pairs_above(32) ? 256 : 384) || pairs_above(256);
  }
  return max_new >= (pairs_above(16) ? 512 : 256) && !pairs_above(sm_count() / (Dv == 2 * kCols ? 2 : 3));
}

extern "C" size_t cvllm_delta_rule_chunks_workspace_bytes(int64_t tokens, int B, int max_new, int H, int G, int D, int Dv) {
  if (tokens <= 0 || B <= 0 || max_new <= 0 || H <= 0 || G <= 0) return 0;
  const int forced = test_options().gla_layout.load();   // tests and measurements: > 0 the other kernel, < 0 chunks
  if (forced > 0 || (forced == 0 && !chunks_are_faster(tokens, B, max_new, H, D, Dv))) return 0;
  if ((D != 64 && D != 128) || Dv <= 0 || Dv % kCols != 0 || Dv > 8 * kCols || H % G != 0) return 0;
  const size_t bytes = chunk_plan(tokens, B, max_new, H, G, D, Dv).bytes;
  return bytes <= 2 * kMost ? bytes : 0;   // one chunk of very many heads
}

extern "C" int cvllm_delta_rule_chunks(const float* qkv, int64_t qkv_stride, const void* proj, int64_t proj_stride, int b_off,
                                       int a_off, const float* A_log, const float* dt_bias, float* state, const void* gate,
                                       int64_t gate_stride, int gate_off, const float* norm_w, int norm_head_stride, float eps,
                                       const int32_t* cu_seqlens_q, const int32_t* seq_start, const int32_t* batch_mapping,
                                       int64_t tokens, int B, int max_new, void* out, int64_t out_stride, int H, int G, int D,
                                       int Dv, int reserved_slot, int dtype, void* workspace, size_t workspace_bytes,
                                       cvllm_stream_t stream) {
  drop_stale_error();
  CVLLM_CHECK_ARG(tokens >= 0 && B >= 0 && max_new >= 0 && H > 0 && G > 0 && H % G == 0 && D > 0 && Dv > 0);
  if (B == 0 || max_new == 0 || tokens == 0) return CVLLM_OK;
  CVLLM_CHECK_ARG(qkv && proj && A_log && dt_bias && state && gate && norm_w && cu_seqlens_q && seq_start && batch_mapping &&
                  out && workspace && (dtype == CVLLM_BF16 || dtype == CVLLM_F32));
  CVLLM_CHECK_SUPPORTED((D == 64 || D == 128) && Dv % kCols == 0 && Dv <= 8 * kCols && H <= 65535 && B <= 65535 &&
                        tokens / kChunk + B < (1 << 24));
  const int64_t E = dtype == CVLLM_BF16 ? 8 : 4;
  CVLLM_CHECK_ALIGN(aligned16(qkv) && qkv_stride % 4 == 0 && aligned16(out) && out_stride % E == 0 && aligned16(gate) &&
                    gate_stride % E == 0 && gate_off % E == 0 && aligned16(workspace));
  const ChunkPlan p = chunk_plan(tokens, B, max_new, H, G, D, Dv);
  if (workspace_bytes < p.bytes) {
    set_last_error("workspace too small for cvllm_delta_rule_chunks");
    return CVLLM_E_WORKSPACE;
  }
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  DeltaChunkArgs a{qkv, qkv_stride, proj_stride, gate_stride, out_stride, proj, gate, b_off, a_off, gate_off, A_log, dt_bias, norm_w,
                   norm_head_stride, eps, state, out, H, G, Dv, reserved_slot, {cu_seqlens_q, seq_start, nullptr, batch_mapping},
                   B, 0, p.slots, p.per_seq, ws, ws + p.cp,
                   reinterpret_cast<double*>(ws + p.dots), reinterpret_cast<float*>(ws + p.gw),
                   reinterpret_cast<float*>(ws + p.carry), reinterpret_cast<float*>(ws + p.other_carry), kSpins, test_options().delta_chunk_hold.load()};
  if (a.hold != 0) a.spins = kSpinsHeld;
  auto st = static_cast<cudaStream_t>(stream);
  if (dtype == CVLLM_BF16)
    return D == 128 ? launch_chunks<__nv_bfloat16, 128>(a, p, B, st) : launch_chunks<__nv_bfloat16, 64>(a, p, B, st);
  return D == 128 ? launch_chunks<float, 128>(a, p, B, st) : launch_chunks<float, 64>(a, p, B, st);
}

extern "C" int cvllm_delta_chunk_aborts(int* count) {
  CVLLM_CHECK_ARG(count);
  CVLLM_CHECK_CUDA(cudaMemcpyFromSymbol(count, g_delta_chunk_aborts, sizeof(int)));
  return CVLLM_OK;
}
