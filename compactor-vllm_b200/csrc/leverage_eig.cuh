// Symmetric eigendecomposition of 48 x 48 matrices in fp64, one CTA of 192 threads per matrix (score_leverage.cu, whose scores
// need round16(V |lam|^-1/2)).
//
// Why fp64: |lam| ranges over 1e-2 .. 1e5, and an absolute error of eps32 * |lam|_max ~ 1e-2 destroys the small eigenpairs that
// dominate x^T |G|^-1 x (profiles/leverage_selfdistance_before.json: fp32 solvers agree with the exact scores to 60-85 %).
//
// What bounds it: one matrix is a chain of dependent fp64 operations (9 cycles each) and exchanges between threads, so the
// steps are laid out for few links, not for few operations:
//   1. Householder reduction, T = Q^T G Q, the matrix in registers of three warps (thread 4 c + p: rows of residue p mod 4
//      of columns c and c + 24, twelve numbers each).  Two barriers a step: the row's norm and the product with it need the same exchange, as
//      A u = A x - g A e differs from A x by a column.
//   2. Divide and conquer on T (Cuppen): leaves of three by Jacobi, then four rounds of merges 3 -> 6 -> 12 -> 24 -> 48, all merges
//      of a round at once.  A merge's eigenvalues are the roots of 1 + sum w_i / (d_i - x), one per four threads, each found on its own
//      from the nearer pole (the step with that pole's weight fixed of Li, "Solving secular equations stably and efficiently", 1994,
//      inside a bracket);
//      the vectors come from the z that has these roots exactly (Gu and Eisenstat 1994), which makes them orthogonal however
//      close the roots are.  No deflation, hence no data-dependent sizes and no serial scan: equal poles are set kSep apart and
//      z has a floor (both perturb G by less than 2^-42 of its norm).
//   3. V = Q W on mma.sync in f64, W in its fragments, eight reflectors at a time (I - Y T Y^T; T and the leaves at the same time).
// Two columns a thread in step 1 halve what is read from shared memory (a register pair of 32 lanes takes two cycles whether or
// not lanes share an address): 45 -> 36 thousand cycles.  The merges want more warps, whose chains fill one another's gaps.
// Measured: 41.6 us for one matrix (76 thousand cycles: reduction 37, leaves 4, merges 20 + 10, V 4), 54 us for 256, 105 us for 512;
// implicit QL, a chain of some 1800 rotations of 86 cycles, took 192, 250 and 250 us.  Three CTAs an SM instead of two would leave 96
// registers a thread, which the reduction overflows (50, 62 and 122 us).
#pragma once
#include "common.cuh"

namespace cvllm {

constexpr int kEigN = 48, kEigHalf = 24;
constexpr int kEigThreads = 4 * kEigN, kEigReduceThreads = 4 * kEigHalf;
constexpr int kEigPitchW = kEigHalf + 2, kEigPitchU = kEigN + 4, kEigPitchR = kEigN + 2;   // fragment loads without bank conflicts
constexpr int kEigPart = 25;                    // numbers per residue of an exchanged vector: twelve, then zeros for reads past them
constexpr double kEigSep = 0x1p-52, kEigZFloor = 0x1p-52, kEigRhoFloor = 0x1p-60;   // T is scaled below 1
constexpr int kEigRootSteps = 40;

struct EigSmem {
  double w[kEigN][kEigPitchW];                  // vectors of T so far: columns c and c + 24 (blocks of 24 rows) side by side
  double u[kEigN][kEigPitchU];                  // vectors of the merge, in the end those of T
  double refl[kEigN][kEigPitchR];               // u of every Householder step, zero up to its own row
  double tm[kEigN / 8][8][8];                   // -T of eight reflectors
  double rh[kEigN];                             // 2 / |u|^2
  double d[kEigN], e[kEigN + 1];                // T; e[i] couples i - 1 and i
  double ds[kEigN], zs[kEigN], pole[kEigN];     // a merge's poles in ascending order (before and after the separation), its z
  double near[kEigN], tau[kEigN];               // root = near + tau
  double zh[kEigN];
  double x[4 * kEigPart], ax[4 * kEigPart];
  int orig[kEigN];
};

// x > 0, normal: 1 / sqrt(x) = y (1 - e)^(-1/2) with e = 1 - x y^2, the binomial series cut behind e^2 (a seed of 2^-22)
__device__ __forceinline__ double rsqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
// x != 0, normal: 1 / x = y / (1 - e) with e = 1 - x y, the geometric series y (1 + e + e^2) cut behind e^2 (a seed of 2^-23: 2^-69 left)
__device__ __forceinline__ double rcp64(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// sum over the four threads of a column: the same bits in each
__device__ __forceinline__ double quad_sum(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}
__device__ __forceinline__ long long order_key(double v) {   // integers in the numbers' order (total: NaN too)
  const long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
// 8 x 8 += 8 x 4 . 4 x 8: a is (lane / 4, lane % 4), b (lane % 4, lane / 4), c (lane / 4, 2 (lane % 4) + 0, 1)
__device__ __forceinline__ void mma884(double (&c)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

__device__ __forceinline__ void eig_bar(int id, int count) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory"); }

// Householder steps [from, to) of Q^T G Q = T.  a[e]: this thread's rows of column q + 24 e (only e = 1 where C0 is 1: the other is
// reduced): a[e][j] is row 4 (j + from / 4) + p on entry, in steps where at most 4 NB such rows are left (the others are zero).
// Straight code: a branch here waits for what it orders.
template <int NB, int C0>
__device__ __forceinline__ void eig_steps(EigSmem& s, double (&a)[2][12], int q, int p, int from, int to) {
  constexpr int L = 4 * NB;
  const int own[2] = {(q & 3) * kEigPart + (q >> 2), (q & 3) * kEigPart + (q >> 2) + kEigHalf / 4};
#pragma unroll 1
  for (int i = from; i < to; ++i) {
    const int i1 = i + 1;
    const bool wrap = (i1 & 3) == 0;            // row i + 1 is the first of the next four
    const bool next = p == (i1 & 3);            // this thread holds it
#pragma unroll
    for (int e = C0; e < 2; ++e) {
      const int c = q + kEigHalf * e;
      if (p == (i & 3)) s.x[own[e]] = c > i ? a[e][0] : 0.0;
      if (p == (i & 3) && c == i) s.d[i] = a[e][0];
    }
    eig_bar(1, kEigReduceThreads);
    const int at = p * kEigPart + (i >> 2);
    const double f = s.x[(i1 & 3) * kEigPart + (i1 >> 2)];
    double uc[2], x[L], px[2][2] = {}, ss[2] = {};
#pragma unroll
    for (int j = 0; j < L; ++j) x[j] = s.x[at + j];
#pragma unroll
    for (int e = C0; e < 2; ++e) uc[e] = s.x[own[e]];
#pragma unroll
    for (int j = 0; j < L; ++j) {
      ss[j & 1] = fma(x[j], x[j], ss[j & 1]);
#pragma unroll
      for (int e = C0; e < 2; ++e) px[e][j & 1] = fma(a[e][j], x[j], px[e][j & 1]);
    }
    const double h = quad_sum(ss[0] + ss[1]);
#pragma unroll
    for (int e = C0; e < 2; ++e) px[e][0] = quad_sum(px[e][0] + px[e][1]);
    const bool act = h > 1e-280;                // else the row is reduced already: H_i = I.  The same in all threads.
    const double g = act ? -copysign(h * rsqrt64(h), f) : 0.0, u1 = f - g;
#pragma unroll
    for (int e = C0; e < 2; ++e) {
      const double v = fma(-g, wrap ? a[e][1] : a[e][0], px[e][0]);   // A u
      if (next) s.ax[own[e]] = q + kEigHalf * e > i ? v : 0.0;
    }
    eig_bar(1, kEigReduceThreads);
    double ax[L], axc[2];
#pragma unroll
    for (int j = 0; j < L; ++j) ax[j] = s.ax[at + j];
#pragma unroll
    for (int e = C0; e < 2; ++e) axc[e] = s.ax[own[e]];
    const double rh = act ? rcp64(fma(-f, g, h)) : 0.0;        // 2 / |u|^2
    if (next) {
      if (wrap) x[1] = u1;
      else x[0] = u1;
    }
    if (C0 == 1) s.refl[i][q] = 0.0;
#pragma unroll
    for (int e = C0; e < 2; ++e) {
      if (q + kEigHalf * e == i1) uc[e] = u1;
      s.refl[i][q + kEigHalf * e] = uc[e];      // by the column's four threads, the same number
    }
    s.e[i1] = g;
    s.rh[i] = rh;
    double k[2] = {};
#pragma unroll
    for (int j = 0; j < L; ++j) k[j & 1] = fma(x[j], ax[j], k[j & 1]);
    // A <- A - u q^T - q u^T with q = rh A u - k u, k = rh^2 u^T A u / 2: column c loses u (rh (A u)_c - 2 k u_c) + (A u) rh u_c
    const double rk = rh * quad_sum(k[0] + k[1]);
#pragma unroll
    for (int e = C0; e < 2; ++e) {
      const double m1 = -rh * uc[e], m0 = fma(rk, m1, rh * axc[e]);
#pragma unroll
      for (int j = 0; j < L; ++j) a[e][j] = fma(-m0, x[j], fma(m1, ax[j], a[e][j]));
      if (wrap) {
#pragma unroll
        for (int j = 0; j < 11; ++j) a[e][j] = a[e][j + 1];
        a[e][11] = 0.0;
      }
    }
  }
}
// T and the reflectors from G's columns q and q + 24, rows p, p + 4, ..., in a
__device__ __forceinline__ void eig_tridiagonal(EigSmem& s, double (&a)[2][12], int q, int p) {
  eig_steps<3, 0>(s, a, q, p, 0, 16);
  eig_steps<2, 0>(s, a, q, p, 16, 24);
  eig_steps<2, 1>(s, a, q, p, 24, 32);
  eig_steps<1, 1>(s, a, q, p, 32, kEigN - 2);
  // rows 46 and 47: residues 2 and 3 of the last four
  if (q == kEigHalf - 2 && p == 2) s.d[kEigN - 2] = a[1][0];
  if (q == kEigHalf - 1 && p == 3) s.d[kEigN - 1] = a[1][0];
  if (q == kEigHalf - 2 && p == 3) s.e[kEigN - 1] = a[1][0];
}

// one rotation of a 3 x 3 matrix: zeroes pq; r is the third index
__device__ __forceinline__ void jacobi3(double& app, double& aqq, double& apq, double& arp, double& arq, double (&v)[9], int cp, int cq) {
  const double dl = aqq - app, t2 = fma(dl, dl, 4.0 * apq * apq);
  const bool act = t2 > 1e-290;
  const double r = rsqrt64(act ? t2 : 1.0);
  const double cc = act ? fma(0.5 * fabs(dl), r, 0.5) : 1.0;
  const double ic = rsqrt64(cc), c = cc * ic;
  const double sn = act ? copysign(1.0, dl) * apq * r * ic : 0.0;
  const double t = sn * ic * apq;               // tan * apq = sn / c * apq, 1 / c = ic
  app -= t;
  aqq += t;
  apq = 0.0;
  const double rp = arp, rq = arq;
  arp = fma(c, rp, -sn * rq);
  arq = fma(sn, rp, c * rq);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double vp = v[3 * k + cp], vq = v[3 * k + cq];
    v[3 * k + cp] = fma(c, vp, -sn * vq);
    v[3 * k + cq] = fma(sn, vp, c * vq);
  }
}

// A round of merges of N / 2 + N / 2: threads 4 c + p serve column c.  s.w and s.d become the new vectors and eigenvalues; N = 48: the
// vectors stay in `v` (N = 24: scratch), row tiles of eight: v[t][i] is row 8 t + 2 (lane % 4) + i of column 8 warp + lane / 4.
template <int N>
__device__ __forceinline__ void eig_merge(EigSmem& s, double (&v)[6][2], int c, int p) {
  constexpr int M = (N + 3) / 4, H = N / 2;
  constexpr bool kEven = N % 4 == 0;
  const int j = c % N, b0 = c - j, cw = c % kEigHalf;
  // number m of this thread among the block's: p + 4 m (past its end: the first one, to be left out)
  auto at = [&](int m) { return b0 + (kEven || p + 4 * m < N ? p + 4 * m : 0); };
  auto in = [&](int m) { return kEven || p + 4 * m < N; };
  const double beta = s.e[b0 + H], rho = fmax(fabs(beta), kEigRhoFloor);
  // ---- poles in ascending order ----
  {
    const double dc = s.d[c];
    const long long key = order_key(dc);
    int rank = 0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const long long o = order_key(s.d[at(m)]);
      rank += in(m) && (o < key || (o == key && p + 4 * m < j));
    }
    rank += __shfl_xor_sync(0xffffffffu, rank, 1);
    rank += __shfl_xor_sync(0xffffffffu, rank, 2);
    double z = s.w[b0 + H - (j < H ? 1 : 0)][cw];
    if (j >= H && beta < 0.0) z = -z;
    z = fabs(z) < kEigZFloor ? copysign(kEigZFloor, z) : z;
    if (p == 0) {
      s.ds[b0 + rank] = dc;
      s.zs[b0 + rank] = z;
      s.orig[b0 + rank] = c;
    }
  }
  __syncthreads();
  // ---- at least kEigSep apart ----
  {
    double top = -8.0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const double x = fma(-(double)(p + 4 * m), kEigSep, s.ds[at(m)]);
      top = p + 4 * m <= j ? fmax(top, x) : top;
    }
    top = fmax(top, __shfl_xor_sync(0xffffffffu, top, 1));
    top = fmax(top, __shfl_xor_sync(0xffffffffu, top, 2));
    if (p == 0) s.pole[c] = fma((double)j, kEigSep, top);
  }
  __syncthreads();
  // ---- root j: between poles j and j + 1, the last one behind pole N - 1 ----
  double near, tau;
  {
    const bool last = j == N - 1;
    const int p1 = last ? N - 2 : j;            // the two poles that a step keeps: p1 and p1 + 1
    auto root_of = [&](double a, double b, double c2) {         // of c2 t^2 - a t + b, the one in the interval
      const double disc = fmax(fma(a, a, -4.0 * b * c2), 1e-300), sq = disc * rsqrt64(disc);
      const double big = a + (a > 0.0 ? sq : -sq);
      const bool other = (a > 0.0) != last;
      return (other ? 2.0 * b : big) * rcp64(other ? big : 2.0 * c2);
    };
    double dk[M], w[M], tot = 0.0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const double z = s.zs[at(m)], d = s.pole[at(m)];
      dk[m] = in(m) ? d : 4.0;                  // a pole without weight
      w[m] = in(m) ? rho * z * z : 0.0;
      tot += w[m];
    }
    tot = quad_sum(tot);
    const double dj = s.pole[c], d1 = s.pole[b0 + p1], d2 = s.pole[b0 + p1 + 1];
    const double z1 = s.zs[b0 + p1], z2 = s.zs[b0 + p1 + 1], w1 = rho * z1 * z1, w2 = rho * z2 * z2;
    const double gap = last ? tot : d2 - dj;
    double rest = 0.0, two = 0.0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const double t = w[m] * rcp64((dk[m] - dj) - 0.5 * gap);
      const bool kept = p + 4 * m == p1 || p + 4 * m == p1 + 1;
      two += kept ? t : 0.0;
      rest += kept ? 0.0 : t;
    }
    rest = 1.0 + quad_sum(rest);
    const bool right = !(rest + quad_sum(two) >= 0.0);          // in the right half
    near = (last || !right) ? dj : d2;
    double lo = right ? (last ? 0.5 : -0.5) * gap : 0.0, hi = right ? (last ? gap : 0.0) : 0.5 * gap;
    const double e1 = d1 - near, e2 = d2 - near;                // one of the two is zero
    const bool first = near == d1;
    const double wn = first ? w1 * (e1 - e2) : w2 * (e2 - e1);
    tau = root_of(fma(rest, e1 + e2, w1 + w2), fma(w1, e2, w2 * e1), rest);
    if (!(tau > lo && tau < hi)) tau = 0.5 * (lo + hi);
#pragma unroll
    for (int m = 0; m < M; ++m) dk[m] -= near;
    bool done = false;
#pragma unroll 1
    for (int it = 0; it < kEigRootSteps; ++it) {
      double f = 0.0, mag = 0.0, df = 0.0;
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const double r = rcp64(dk[m] - tau);
        f = fma(w[m], r, f);
        mag = fma(w[m], fabs(r), mag);
        df = fma(w[m], r * r, df);
      }
      f = 1.0 + quad_sum(f);
      mag = 1.0 + quad_sum(mag);
      df = quad_sum(df);
      const bool zero = done || !(fabs(f) > 0x1p-50 * mag);
      lo = f < 0.0 && !zero ? tau : lo;
      hi = f < 0.0 || zero ? hi : tau;
      const double q1 = e1 - tau, q2 = e2 - tau, q12 = q1 * q2, qn = first ? q1 : q2, rn = rcp64(qn);
      const double c2 = f - fma(first ? q2 : q1, df, wn * rn * rn);
      double t = tau + root_of(fma(q1 + q2, f, -q12 * df), q12 * f, c2);
      const bool inside = t > lo && t < hi;
      t = inside ? t : 0.5 * (lo + hi);
      // a step of 2^-30 leaves an error of the order of its square
      done = zero || (inside ? !(fabs(t - tau) > 0x1p-30 * fabs(t)) : t == tau);
      tau = zero ? tau : t;
      if (__all_sync(0xffffffffu, done)) break;
    }
    if (p == 0) {
      s.near[c] = near;
      s.tau[c] = tau;
    }
  }
  __syncthreads();
  // ---- the z whose roots these are: z_i^2 = (x_last - d_i) prod_j (x_j - d_i) / (d_j or j + 1 - d_i), each factor in [0, 1] ----
  {
    const double di = s.pole[c];
    double pr[2] = {1.0, 1.0};
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int i = p + 4 * m;
      const double num = (s.near[at(m)] - di) + s.tau[at(m)];
      const double den = s.pole[i < N - 1 ? at(m) + (i < j ? 0 : 1) : at(m)] - di;
      const double x = num * rcp64(i < N - 1 ? den : 1.0);
      pr[m & 1] *= in(m) ? x : 1.0;
    }
    double z2 = pr[0] * pr[1];
    z2 *= __shfl_xor_sync(0xffffffffu, z2, 1);
    z2 *= __shfl_xor_sync(0xffffffffu, z2, 2);
    z2 = fmax(fabs(z2), 1e-300);
    if (p == 0) {
      s.zh[c] = copysign(z2 * rsqrt64(z2), s.zs[c]);
      s.d[c] = near + tau;
    }
  }
  __syncthreads();
  {
    double x[M], ss = 0.0;
#pragma unroll
    for (int m = 0; m < M; ++m) {
      x[m] = s.zh[at(m)] * rcp64((s.pole[at(m)] - near) - tau);
      if (!in(m)) x[m] = 0.0;
      ss = fma(x[m], x[m], ss);
    }
    const double inv = rsqrt64(quad_sum(ss));
#pragma unroll
    for (int m = 0; m < M; ++m)
      if (in(m)) s.u[s.orig[at(m)]][c] = x[m] * inv;
  }
  __syncthreads();
  // ---- W U: the halves' rows of W meet their rows of U ----
  if constexpr (N >= 24) {
    const int col = (threadIdx.x >> 5) * 8, r8 = (threadIdx.x & 31) >> 2, k4 = threadIdx.x & 3, blk = col / N * N;
#pragma unroll
    for (int t = 0; t < N / 8; ++t) v[t][0] = v[t][1] = 0.0;
#pragma unroll
    for (int k = 0; k < N; k += 4) {
      const double a = s.u[blk + k + k4][col + r8];
#pragma unroll
      for (int t = 0; t < N / 8; ++t) {
        const bool low = 8 * t < H, high = 8 * t + 8 > H;       // the halves that rows 8 t .. 8 t + 7 lie in
        if (k < H ? low : high) {
          double b = s.w[blk + 8 * t + r8][k % kEigHalf + k4];
          if (low && high) b = (8 * t + r8 < H) == (k < H) ? b : 0.0;
          mma884(v[t], a, b);
        }
      }
    }
    if constexpr (N < kEigN) {
      __syncthreads();
#pragma unroll
      for (int t = 0; t < N / 8; ++t)
#pragma unroll
        for (int i = 0; i < 2; ++i) s.w[blk + 8 * t + 2 * k4 + i][col % kEigHalf + r8] = v[t][i];
      __syncthreads();
    }
  } else {
    double acc[M] = {};
#pragma unroll
    for (int m = 0; m < M; ++m) {
      const int off = at(m) - b0 < H ? 0 : H;
#pragma unroll
      for (int k = 0; k < H; ++k) acc[m] = fma(s.w[at(m)][b0 % kEigHalf + off + k], s.u[b0 + off + k][c], acc[m]);
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < M; ++m)
      if (in(m)) s.w[at(m)][cw] = acc[m];
    __syncthreads();
  }
}

// gram: [mats][48][48] fp32, symmetric.  sv_out[mat][48][48] = round16(V |lam|^-1/2); the order of the columns is arbitrary (the
// score sums over all of them).  A matrix with an entry that is not finite gives NaN.
template <bool BF16>
__global__ void __launch_bounds__(kEigThreads, 2) leverage_eig_kernel(const float* __restrict__ gram, float* __restrict__ sv_out,
                                                                      const int32_t* __restrict__ chunk_offsets, int HKV, int mats,
                                                                      double* __restrict__ dbg_lam, double* __restrict__ dbg_vec,
                                                                      long long* __restrict__ dbg_clk) {
  extern __shared__ __align__(16) unsigned char eig_smem_raw[];
  EigSmem& s = *reinterpret_cast<EigSmem*>(eig_smem_raw);
  constexpr int n = kEigN;
  const int tid = threadIdx.x, lane = tid & 31, c = tid >> 2, p = tid & 3;
  const int mat = blockIdx.x;
  if (mat >= mats) return;
  if (chunk_offsets) {
    const int ch = mat / HKV;
    if (chunk_offsets[ch + 1] - chunk_offsets[ch] <= 0) return;
  }
  auto stamp = [&](int i) {
    if (dbg_clk && tid == 0) dbg_clk[mat * 6 + i] = clock64();
  };
  for (int i = tid; i < 4 * kEigPart; i += kEigThreads) s.x[i] = s.ax[i] = 0.0;
  if (tid == 0) s.e[0] = s.e[n] = 0.0;
  if (tid < 2) s.rh[n - 2 + tid] = 0.0;
  if (tid < 2 * kEigPitchR) s.refl[n - 2][tid] = 0.0;           // the last block's missing two
  __syncthreads();
  stamp(0);
  if (tid < kEigReduceThreads) {
    const float* gin = gram + (int64_t)mat * n * n;
    double a[2][12];
#pragma unroll
    for (int e = 0; e < 2; ++e)
#pragma unroll
      for (int m = 0; m < 12; ++m) a[e][m] = (double)gin[(4 * m + p) * n + c + kEigHalf * e];
    eig_tridiagonal(s, a, c, p);
  }
  __syncthreads();
  stamp(1);

  // ---- T scaled below 1 by a power of two; the leaves' ends without their couplings ----
  double back;
  {
    double top = fmax(fabs(s.d[lane]), fabs(s.e[lane]));
    if (lane + 32 < n) top = fmax(top, fmax(fabs(s.d[lane + 32]), fabs(s.e[lane + 32])));
    // fmax drops NaN: a sum keeps it
    double bad = s.d[lane] + s.e[lane] + (lane + 32 < n ? s.d[lane + 32] + s.e[lane + 32] : 0.0);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
      bad += __shfl_xor_sync(0xffffffffu, bad, o);
    }
    if (!(fabs(bad) < 1e300)) {                 // the same in all threads
      const float nan = __int_as_float(0x7fffffff);
      for (int i = tid; i < n * n; i += kEigThreads) {
        sv_out[(int64_t)mat * n * n + i] = nan;
        if (dbg_vec) dbg_vec[(int64_t)mat * n * n + i] = nan;
      }
      if (dbg_lam && tid < n) dbg_lam[(int64_t)mat * n + tid] = nan;
      return;
    }
    const int ex = top > 1e-280 ? ilogb(top) + 3 : 0;
    const double sc = scalbn(1.0, -ex);
    back = top > 1e-280 ? scalbn(1.0, ex) : 0.0;
    double dn = 0.0, en = 0.0;
    if (tid < n) {
      const bool first = tid % 3 == 0 && tid > 0, end = tid % 3 == 2 && tid < n - 1;
      dn = (s.d[tid] - (first ? fabs(s.e[tid]) : 0.0) - (end ? fabs(s.e[tid + 1]) : 0.0)) * sc;
      en = s.e[tid] * sc;
    }
    __syncthreads();
    if (tid < n) {
      s.d[tid] = dn;
      s.e[tid] = en;
    }
    __syncthreads();
  }
  if (tid < 32) {
    const int b = 3 * (tid & 15);
    double a0 = s.d[b], a1 = s.d[b + 1], a2 = s.d[b + 2], o01 = s.e[b + 1], o12 = s.e[b + 2], o02 = 0.0;
    double v[9] = {1.0, 0.0, 0.0, 0.0, 1.0, 0.0, 0.0, 0.0, 1.0};
#pragma unroll 1
    for (int sweep = 0; sweep < 10; ++sweep) {
      if (__all_sync(0xffffffffu, !(fabs(o01) + fabs(o02) + fabs(o12) > 0x1p-58))) break;
      jacobi3(a0, a1, o01, o02, o12, v, 0, 1);
      jacobi3(a0, a2, o02, o01, o12, v, 0, 2);
      jacobi3(a1, a2, o12, o01, o02, v, 1, 2);
    }
    if (tid < 16) {
      s.d[b] = a0;
      s.d[b + 1] = a1;
      s.d[b + 2] = a2;
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k) s.w[b + r][b % kEigHalf + k] = v[3 * r + k];
    }
  } else {
    // T of H_i0 ... H_i0+7 = I - Y T Y^T: T_rr = rh_r, T_rj = -rh_j sum_(r <= i < j) T_ri (u_i . u_j)
    double* dots = &s.u[0][0];                  // [block][i][j]
    const int t = tid - 32, blk = t / 28, at = t % 28;
    int j = 1;
    while ((j + 1) * j / 2 <= at) ++j;
    const int i = at - j * (j - 1) / 2;
    if (8 * blk + j < n - 2) {
      const double *ui = s.refl[8 * blk + i], *uj = s.refl[8 * blk + j];
      double d0 = 0.0, d1 = 0.0;
      for (int k = 8 * blk; k < n; k += 2) {
        d0 = fma(ui[k], uj[k], d0);
        d1 = fma(ui[k + 1], uj[k + 1], d1);
      }
      dots[blk * 64 + i * 8 + j] = d0 + d1;
    }
    eig_bar(1, kEigThreads - 32);
    if (t < n) {
      const int b8 = t / 8, r = t % 8;
      double tr[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        double sum = 0.0;
#pragma unroll
        for (int l = 0; l < k; ++l) sum = fma(tr[l], dots[b8 * 64 + l * 8 + k], sum);
        const double rh = s.rh[8 * b8 + k];
        tr[k] = k < r || 8 * b8 + k >= n - 2 ? 0.0 : k == r ? rh : -rh * sum;
        s.tm[b8][r][k] = -tr[k];
      }
    }
  }
  __syncthreads();
  stamp(2);
  double v[6][2];
  eig_merge<6>(s, v, c, p);
  eig_merge<12>(s, v, c, p);
  eig_merge<24>(s, v, c, p);
  stamp(3);
  eig_merge<48>(s, v, c, p);
  stamp(4);

  // ---- V = H_0 H_1 ... W, transposed: V^T = W^T - (W^T Y) T^T Y^T; a result's fragment is the next product's left one where the
  // right one takes its rows in the order 0 2 4 6, 1 3 5 7 ----
  const int r8 = lane >> 2, k4 = lane & 3;
#pragma unroll
  for (int b = n / 8 - 1; b >= 0; --b) {
    double d0[2] = {}, d1[2] = {}, c0[2] = {}, c1[2] = {};
#pragma unroll
    for (int t = b; t < 6; ++t) {               // reflector i is zero up to row i
      const double2 y = *reinterpret_cast<const double2*>(&s.refl[8 * b + r8][8 * t + 2 * k4]);
      mma884(d0, v[t][0], y.x);
      mma884(d1, v[t][1], y.y);
    }
    const double2 m = *reinterpret_cast<const double2*>(&s.tm[b][r8][2 * k4]);
    mma884(c0, d0[0] + d1[0], m.x);
    mma884(c1, d0[1] + d1[1], m.y);
#pragma unroll
    for (int t = b; t < 6; ++t) {
      mma884(v[t], c0[0] + c1[0], s.refl[8 * b + 2 * k4][8 * t + r8]);
      mma884(v[t], c0[1] + c1[1], s.refl[8 * b + 2 * k4 + 1][8 * t + r8]);
    }
  }
  pdl_trigger();   // late: kernels that wait on an SM keep others from it
  float* out = sv_out + (int64_t)mat * n * n;
  const int col = 8 * (tid >> 5) + r8;
  const double lam = s.d[col] * back, rs = rsqrt(fabs(lam));
#pragma unroll
  for (int t = 0; t < 6; ++t)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int at = (8 * t + 2 * k4 + i) * n + col;
      const float x = (float)(v[t][i] * rs);
      out[at] = BF16 ? __bfloat162float(__float2bfloat16_rn(x)) : __half2float(__float2half_rn(x));
      if (dbg_vec) dbg_vec[(int64_t)mat * n * n + at] = v[t][i];
    }
  if (dbg_lam && k4 == 0) dbg_lam[(int64_t)mat * n + col] = lam;
  stamp(5);
}

}  // namespace cvllm
