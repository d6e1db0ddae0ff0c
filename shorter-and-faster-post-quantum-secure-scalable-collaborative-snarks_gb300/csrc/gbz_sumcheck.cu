// Sumcheck round kernels, the eq (beta) table and the WHIR beta update.
//
// Round message (coSumcheck_MPI.cpp:199, Whir.cpp:215-221,
// delegate_protocol.cpp:16-21): over pairs j of two vectors,
//   H(x) = sum_j (a1 x + b1)(a2 x + b2),  a = v[2j+1] - v[2j], b = v[2j],
// so H = (sum a1 a2, sum a1 b2 + b1 a2, sum b1 b2).  With
// D = v1[2j+1] v2[2j+1] the middle term is D - A - C, three products per
// pair instead of four (exact arithmetic, same value).
// Fold (coSumcheck_MPI.cpp:215-218, Whir.cpp:223-231):
//   v[j] = r (v[2j+1] - v[2j]) + v[2j].
// The fold of round i and the message of round i+1 are one pass: each
// thread reads four consecutive entries of both vectors, writes the two
// folded entries of each and accumulates the next message from them.
#include <algorithm>

#include "gbz_internal.cuh"

namespace gbz {

namespace {

constexpr int kScThreads = 256;

__device__ __forceinline__ fe shfl_down_fe(fe v, int d) {
  fe r;
  r.re = __shfl_down_sync(0xffffffffu, v.re, d);
  r.im = __shfl_down_sync(0xffffffffu, v.im, d);
  return r;
}

// Block-wide sum of three field elements; result valid in thread 0.
__device__ void block_sum3(fe &x, fe &y, fe &z) {
  __shared__ fe red[3][kScThreads / 32];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    x = fadd(x, shfl_down_fe(x, d));
    y = fadd(y, shfl_down_fe(y, d));
    z = fadd(z, shfl_down_fe(z, d));
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { red[0][w] = x; red[1][w] = y; red[2][w] = z; }
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    x = lane < nw ? red[0][lane] : fe_zero();
    y = lane < nw ? red[1][lane] : fe_zero();
    z = lane < nw ? red[2][lane] : fe_zero();
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      x = fadd(x, shfl_down_fe(x, d));
      y = fadd(y, shfl_down_fe(y, d));
      z = fadd(z, shfl_down_fe(z, d));
    }
  }
}

__device__ __forceinline__ void acc_pair(fe a0, fe a1, fe b0, fe b1, facc &A, facc &C, facc &D) {
  facc_mul(A, fsub_lazy(a1, a0), fsub(b1, b0));
  facc_mul(C, a0, b0);
  facc_mul(D, a1, b1);
}

// partial[3*blk + {0,1,2}] = (sum A, sum C, sum D) of the block.
__global__ void __launch_bounds__(kScThreads)
sc_reduce_kernel(const fe *__restrict__ a, const fe *__restrict__ b, uint64_t pairs, fe *partial) {
  pdl_wait();
  facc sA = facc_zero(), sC = facc_zero(), sD = facc_zero();
  const uint64_t stride = (uint64_t)gridDim.x * kScThreads;
  for (uint64_t j = (uint64_t)blockIdx.x * kScThreads + threadIdx.x; j < pairs; j += stride) {
    fe a0 = a[2 * j], a1 = a[2 * j + 1], b0 = b[2 * j], b1 = b[2 * j + 1];
    acc_pair(a0, a1, b0, b1, sA, sC, sD);
  }
  fe A = facc_value(sA), C = facc_value(sC), D = facc_value(sD);
  block_sum3(A, C, D);
  if (threadIdx.x == 0) {
    partial[3 * blockIdx.x] = A;
    partial[3 * blockIdx.x + 1] = C;
    partial[3 * blockIdx.x + 2] = D;
  }
}

// Fold (a, b) of length m by *chal into (a2, b2) of length m/2; when
// reduce, accumulate the message of the folded pair sequence.
__global__ void __launch_bounds__(kScThreads)
sc_fold_kernel(const fe *__restrict__ a, const fe *__restrict__ b, uint64_t m, const fe *chal,
               fe *__restrict__ a2, fe *__restrict__ b2, int reduce, fe *partial) {
  pdl_wait();
  const fe r = *chal;
  facc sA = facc_zero(), sC = facc_zero(), sD = facc_zero();
  const uint64_t stride = (uint64_t)gridDim.x * kScThreads;
  const uint64_t quads = m / 4;
  for (uint64_t t = (uint64_t)blockIdx.x * kScThreads + threadIdx.x; t < quads; t += stride) {
    fe x0 = a[4 * t], x1 = a[4 * t + 1], x2 = a[4 * t + 2], x3 = a[4 * t + 3];
    fe y0 = b[4 * t], y1 = b[4 * t + 1], y2 = b[4 * t + 2], y3 = b[4 * t + 3];
    const fe fa0 = ffold(x0, x1, r), fa1 = ffold(x2, x3, r), fb0 = ffold(y0, y1, r), fb1 = ffold(y2, y3, r);
    a2[2 * t] = fa0; a2[2 * t + 1] = fa1;
    b2[2 * t] = fb0; b2[2 * t + 1] = fb1;
    if (reduce) acc_pair(fa0, fa1, fb0, fb1, sA, sC, sD);
  }
  if (m == 2 && blockIdx.x == 0 && threadIdx.x == 0) {  // fold to a single entry
    a2[0] = fadd(fmul(r, fsub(a[1], a[0])), a[0]);
    b2[0] = fadd(fmul(r, fsub(b[1], b[0])), b[0]);
  }
  if (!reduce) return;
  fe A = facc_value(sA), C = facc_value(sC), D = facc_value(sD);
  block_sum3(A, C, D);
  if (threadIdx.x == 0) {
    partial[3 * blockIdx.x] = A;
    partial[3 * blockIdx.x + 1] = C;
    partial[3 * blockIdx.x + 2] = D;
  }
}

// Two WHIR sumcheck rounds in one pass (Whir.cpp:215-231 twice): the
// challenges r0, r1 are drawn before the round messages exist (F::_random),
// so a thread takes four consecutive entries of both vectors, adds the two
// pairs to the first round's message, folds them by r0, adds the folded pair
// to the second round's message and folds it by r1 into (a4, b4) of length
// m/4.  One read of (a, b) instead of three passes.
__global__ void __launch_bounds__(kScThreads, 2)
sc_fold2_kernel(const fe *__restrict__ a, const fe *__restrict__ b, uint64_t m, const fe *chal0, const fe *chal1,
                fe *__restrict__ a4, fe *__restrict__ b4, fe *partial0, fe *partial1, BStr bs) {
  pdl_wait();
  const uint32_t pb = blockIdx.y;
  a = badv(a, bs.s[0], pb);
  b = badv(b, bs.s[1], pb);
  chal0 = badv(chal0, bs.s[2], pb);
  chal1 = badv(chal1, bs.s[3], pb);
  a4 = badv(a4, bs.s[4], pb);
  b4 = badv(b4, bs.s[5], pb);
  partial0 = badv(partial0, bs.s[6], pb);
  partial1 = badv(partial1, bs.s[7], pb);
  const fe r0 = *chal0, r1 = *chal1;
  facc sA0 = facc_zero(), sC0 = facc_zero(), sD0 = facc_zero();
  facc sA1 = facc_zero(), sC1 = facc_zero(), sD1 = facc_zero();
  const uint64_t stride = (uint64_t)gridDim.x * kScThreads;
  const uint64_t quads = m / 4;
  for (uint64_t t = (uint64_t)blockIdx.x * kScThreads + threadIdx.x; t < quads; t += stride) {
    const fe x0 = a[4 * t], x1 = a[4 * t + 1], x2 = a[4 * t + 2], x3 = a[4 * t + 3];
    const fe y0 = b[4 * t], y1 = b[4 * t + 1], y2 = b[4 * t + 2], y3 = b[4 * t + 3];
    acc_pair(x0, x1, y0, y1, sA0, sC0, sD0);
    acc_pair(x2, x3, y2, y3, sA0, sC0, sD0);
    const fe fa0 = ffold(x0, x1, r0), fa1 = ffold(x2, x3, r0), fb0 = ffold(y0, y1, r0), fb1 = ffold(y2, y3, r0);
    acc_pair(fa0, fa1, fb0, fb1, sA1, sC1, sD1);
    a4[t] = ffold(fa0, fa1, r1);
    b4[t] = ffold(fb0, fb1, r1);
  }
  fe A0 = facc_value(sA0), C0 = facc_value(sC0), D0 = facc_value(sD0);
  fe A1 = facc_value(sA1), C1 = facc_value(sC1), D1 = facc_value(sD1);
  block_sum3(A0, C0, D0);
  if (threadIdx.x == 0) {
    partial0[3 * blockIdx.x] = A0;
    partial0[3 * blockIdx.x + 1] = C0;
    partial0[3 * blockIdx.x + 2] = D0;
  }
  __syncthreads();  // block_sum3's shared scratch is reused
  block_sum3(A1, C1, D1);
  if (threadIdx.x == 0) {
    partial1[3 * blockIdx.x] = A1;
    partial1[3 * blockIdx.x + 1] = C1;
    partial1[3 * blockIdx.x + 2] = D1;
  }
}

// The same two rounds for the first WHIR iteration, whose b is the eq
// vector of the sumcheck challenges c (precompute_beta, utils.cpp:198-243):
// b[4t + 2 x1 + x0] = eq1(c0, x0) eq1(c1, x1) E2[t] with E2 the eq table of
// c2.. (m/4 entries), so b is never read.  Per pair the messages need only
// S0 = sum a0 g and S1 = sum a1 g (g the pair's factor without eq1(c0, .)):
// A = (e1 - e0)(S1 - S0), C = e0 S0, D = e1 S1 (e_x = eq1(c0, x)), and after
// the fold by r0 the pair's b is lambda0 eq1(c1, x1) E2[t], lambda0 =
// eq1(c0, r0); b4 = lambda0 lambda1 E2 (lambda1 = eq1(c1, r1)).
__global__ void __launch_bounds__(kScThreads, 2)
sc_fold2_eq_kernel(const fe *__restrict__ a, const fe *__restrict__ E2, uint64_t m, const fe *c, const fe *chal0,
                   const fe *chal1, fe *__restrict__ a4, fe *__restrict__ b4, fe *partial0, fe *partial1, BStr bs) {
  pdl_wait();
  const uint32_t pb = blockIdx.y;
  a = badv(a, bs.s[0], pb);
  E2 = badv(E2, bs.s[1], pb);
  c = badv(c, bs.s[2], pb);
  chal0 = badv(chal0, bs.s[3], pb);
  chal1 = badv(chal1, bs.s[4], pb);
  a4 = badv(a4, bs.s[5], pb);
  b4 = badv(b4, bs.s[6], pb);
  partial0 = badv(partial0, bs.s[7], pb);
  partial1 = badv(partial1, bs.s[8], pb);
  const fe r0 = *chal0, r1 = *chal1, c0 = c[0], c1 = c[1];
  const fe e0 = fsub(fe_one(), c0), f0 = fsub(fe_one(), c1);
  const fe lam0 = fadd(fmul(r0, fsub(c0, e0)), e0), lam1 = fadd(fmul(r1, fsub(c1, f0)), f0);
  const fe lam = fmul(lam0, lam1);
  facc sS0 = facc_zero(), sS1 = facc_zero(), sT0 = facc_zero(), sT1 = facc_zero();
  const uint64_t stride = (uint64_t)gridDim.x * kScThreads;
  const uint64_t quads = m / 4;
  for (uint64_t t = (uint64_t)blockIdx.x * kScThreads + threadIdx.x; t < quads; t += stride) {
    const fe x0 = a[4 * t], x1 = a[4 * t + 1], x2 = a[4 * t + 2], x3 = a[4 * t + 3];
    const fe E = E2[t];
    const fe g0 = fmul_fold(f0, E), g1 = fmul_fold(c1, E);
    fe fa0, fa1;
    if (!(x0.im | x1.im | x2.im | x3.im)) {
      // base-field entries (the witness of the configurations): products
      // with a base-field factor need two of the four partial products
      facc_mul_base(sS0, g0, x0.re);
      facc_mul_base(sS0, g1, x2.re);
      facc_mul_base(sS1, g0, x1.re);
      facc_mul_base(sS1, g1, x3.re);
      fa0 = ffold_base(x0.re, x1.re, r0);
      fa1 = ffold_base(x2.re, x3.re, r0);
    } else {
      facc_mul(sS0, g0, x0);
      facc_mul(sS0, g1, x2);
      facc_mul(sS1, g0, x1);
      facc_mul(sS1, g1, x3);
      fa0 = ffold(x0, x1, r0);
      fa1 = ffold(x2, x3, r0);
    }
    facc_mul(sT0, fa0, E);
    facc_mul(sT1, fa1, E);
    a4[t] = ffold(fa0, fa1, r1);
    b4[t] = fmul(lam, E);
  }
  fe S0 = facc_value(sS0), S1 = facc_value(sS1), T0 = facc_value(sT0), T1 = facc_value(sT1);
  fe Z = fe_zero();
  block_sum3(S0, S1, Z);
  if (threadIdx.x == 0) {
    partial0[3 * blockIdx.x] = fmul(fsub(c0, e0), fsub(S1, S0));
    partial0[3 * blockIdx.x + 1] = fmul(e0, S0);
    partial0[3 * blockIdx.x + 2] = fmul(c0, S1);
  }
  __syncthreads();  // block_sum3's shared scratch is reused
  Z = fe_zero();
  block_sum3(T0, T1, Z);
  if (threadIdx.x == 0) {
    partial1[3 * blockIdx.x] = fmul(lam0, fmul(fsub(c1, f0), fsub(T1, T0)));
    partial1[3 * blockIdx.x + 1] = fmul(lam0, fmul(f0, T0));
    partial1[3 * blockIdx.x + 2] = fmul(lam0, fmul(c1, T1));
  }
}

// Sumcheck of sum_x w(x) eq(z, x) without folding the eq vector, two rounds
// a pass.  After i rounds the folded eq vector is
// epre * eq1(z_i, x_0) * E_i[x'], E_i the eq table of z_{i+1..}
// (eq1(z, x) = z x + (1 - z)(1 - x)), so the round polynomial is
// epre * eq1(z_i, X) * S(X), S(X) linear with S(0) = sum w[2j] E_i[j] and
// S(1) = sum w[2j+1] E_i[j] (the same polynomial as the pairwise products of
// the reference's loop).  E_i[2j + x] = eq1(z_{i+1}, x) E_{i+1}[j], so with
//   T_k = sum_j w[4j + k] E_{i+1}[j], k < 4,
// round i has S(X) = (1 - z_{i+1}) T_X + z_{i+1} T_{2+X}, and round i + 1,
// after the challenge c, S(X) = T_{2X} + c (T_{2X+1} - T_{2X}): one pass over
// w and one launch between hash chains for both (a pass a round took twice
// the reads and multiplies, and 11 us a round where launches are short).
// E_{i+3}[t] = sum of the four entries of E_{i+1} from 4t on.
// partial[4 blk + k] = T_k.  A thread's entries all have the same index mod 4.
__device__ void block_sum_classes(const facc &acc, fe *partial) {
  __shared__ fe red[kScThreads / 32][4];
  fe x = facc_value(acc);
#pragma unroll
  for (int d = 4; d < 32; d <<= 1)
    x = fadd(x, fe_make(__shfl_xor_sync(0xffffffffu, x.re, d), __shfl_xor_sync(0xffffffffu, x.im, d)));
  if ((threadIdx.x & 31) < 4) red[threadIdx.x >> 5][threadIdx.x & 3] = x;
  __syncthreads();
  if (threadIdx.x >= 4) return;
  x = red[0][threadIdx.x];
#pragma unroll
  for (int w = 1; w < kScThreads / 32; w++) x = fadd(x, red[w][threadIdx.x]);
  partial[4 * blockIdx.x + threadIdx.x] = x;
}

__global__ void __launch_bounds__(kScThreads)
sc_eq_reduce_kernel(const fe *__restrict__ a, const fe *__restrict__ E, uint64_t m, fe *partial, BStr bs) {
  pdl_wait();
  a = badv(a, bs.s[0], blockIdx.y);
  E = badv(E, bs.s[1], blockIdx.y);
  partial = badv(partial, bs.s[2], blockIdx.y);
  facc acc = facc_zero();
  const uint64_t stride = (uint64_t)gridDim.x * kScThreads;
#pragma unroll 4
  for (uint64_t x = (uint64_t)blockIdx.x * kScThreads + threadIdx.x; x < m; x += stride) {
    const fe e = E[x >> 2], w = a[x];
    if (!w.im) facc_mul_base(acc, e, w.re);  // a base-field entry: two partial products
    else facc_mul(acc, w, e);
  }
  block_sum_classes(acc, partial);
}

// Fold a (m entries, a multiple of 128) by chal[0] and chal[1] into a4 and E
// (m / 4 entries) into E4, which the tail reads after the last pass too; with
// reduce also the T sums of a4 with E4.
__global__ void __launch_bounds__(kScThreads)
sc_eq_fold_kernel(const fe *__restrict__ a, uint64_t m, const fe *chal, fe *__restrict__ a4,
                  const fe *__restrict__ E, fe *__restrict__ E4, int reduce, fe *partial, BStr bs) {
  pdl_wait();
  a = badv(a, bs.s[0], blockIdx.y);
  chal = badv(chal, bs.s[1], blockIdx.y);
  a4 = badv(a4, bs.s[2], blockIdx.y);
  E = badv(E, bs.s[3], blockIdx.y);
  E4 = badv(E4, bs.s[4], blockIdx.y);
  partial = badv(partial, bs.s[5], blockIdx.y);
  const fe c0 = chal[0], c1 = chal[1];
  facc acc = facc_zero();
  const uint64_t stride = (uint64_t)gridDim.x * kScThreads;
  for (uint64_t j = (uint64_t)blockIdx.x * kScThreads + threadIdx.x; j < m / 4; j += stride) {
    const fe x0 = a[4 * j], x1 = a[4 * j + 1], x2 = a[4 * j + 2], x3 = a[4 * j + 3];
    fe e = E[j];
    fe f0, f1;
    if (!(x0.im | x1.im | x2.im | x3.im)) {  // base-field entries (the first fold of the witness)
      f0 = ffold_base(x0.re, x1.re, c0);
      f1 = ffold_base(x2.re, x3.re, c0);
    } else {
      f0 = ffold(x0, x1, c0);
      f1 = ffold(x2, x3, c0);
    }
    f0 = ffold(f0, f1, c1);
    a4[j] = f0;
#pragma unroll
    for (int d = 1; d < 4; d <<= 1)
      e = fadd(e, fe_make(__shfl_xor_sync(0xffffffffu, e.re, d), __shfl_xor_sync(0xffffffffu, e.im, d)));
    if ((j & 3) == 0) E4[j >> 2] = e;
    if (reduce) facc_mul(acc, f0, e);
  }
  if (reduce) block_sum_classes(acc, partial);
}

// out = (a, b, c) of the round message from (A, C, D) partials.
__global__ void __launch_bounds__(kScThreads) sc_sum_kernel(const fe *partial, int blocks, fe *out) {
  pdl_wait();
  fe A = fe_zero(), C = fe_zero(), D = fe_zero();
  for (int i = threadIdx.x; i < blocks; i += kScThreads) {
    A = fadd(A, partial[3 * i]);
    C = fadd(C, partial[3 * i + 1]);
    D = fadd(D, partial[3 * i + 2]);
  }
  block_sum3(A, C, D);
  if (threadIdx.x == 0) {
    out[0] = A;
    out[1] = fsub(fsub(D, A), C);
    out[2] = C;
  }
}

// precompute_beta, one CTA per block of 2^11 consecutive entries: thread 0
// forms the product over the index bits from 11 up, then the CTA doubles the
// table in shared memory from bit 10 down to bit 0 (T[2j+1] = T[j] r_i,
// T[2j] = T[j] - T[j] r_i, one product per entry) and writes the block with
// coalesced 16-byte stores.
constexpr int kBetaBlockLog = 11;
__global__ void __launch_bounds__(256) beta_block_kernel(const fe *r, int nr, fe *B, BStr bs) {
  pdl_wait();
  __shared__ fe T[1 << kBetaBlockLog];
  __shared__ fe rs[64];
  r = badv(r, bs.s[0], blockIdx.y);
  B = badv(B, bs.s[1], blockIdx.y);
  const int low = nr < kBetaBlockLog ? nr : kBetaBlockLog;
  if ((int)threadIdx.x < nr) rs[threadIdx.x] = r[threadIdx.x];
  __syncthreads();
  if (threadIdx.x == 0) {
    fe pre = fe_one();
    const uint64_t hi = (uint64_t)blockIdx.x;
    for (int i = low; i < nr; i++) pre = fmul(pre, ((hi >> (i - low)) & 1) ? rs[i] : fsub(fe_one(), rs[i]));
    T[0] = pre;
  }
  __syncthreads();
  for (int i = low - 1; i >= 0; i--) {
    const int len = 1 << (low - 1 - i);  // entries before this level (at most 2^10)
    const fe ri = rs[i];
    fe v[4];
    int cnt = 0;
    for (int j = threadIdx.x; j < len; j += blockDim.x) v[cnt++] = T[j];
    __syncthreads();
    cnt = 0;
    for (int j = threadIdx.x; j < len; j += blockDim.x) {
      const fe t = v[cnt++];
      const fe x = fmul(t, ri);
      T[2 * j + 1] = x;
      T[2 * j] = fsub(t, x);
    }
    __syncthreads();
  }
  fe *o = B + ((uint64_t)blockIdx.x << low);
  for (int j = threadIdx.x; j < (1 << low); j += blockDim.x) o[j] = T[j];
}

// Tables of 2^15 entries or more: a CTA writes 16 blocks of 2^11 entries.
// The table is the tensor product of the eq table LO over the 11 low
// variables (built once per CTA by doubling in shared memory) and the
// products over the high variables of each block (16 threads, one block
// each), so every output entry costs one product and the serial part of a
// CTA is amortised over 2^15 entries.
constexpr int kBetaChunksLog = 4;  // at most 16 blocks of 2^11 entries per CTA
__global__ void __launch_bounds__(256) beta_tensor_kernel(const fe *r, int nr, int chunks_log, fe *B, BStr bs) {
  pdl_wait();
  __shared__ fe T[1 << kBetaBlockLog];
  __shared__ fe hi_pre[1 << kBetaChunksLog];
  __shared__ fe rs[64];
  r = badv(r, bs.s[0], blockIdx.y);
  B = badv(B, bs.s[1], blockIdx.y);
  if ((int)threadIdx.x < nr) rs[threadIdx.x] = r[threadIdx.x];
  __syncthreads();
  if (threadIdx.x < (1u << chunks_log)) {
    const uint64_t c = ((uint64_t)blockIdx.x << chunks_log) + threadIdx.x;  // block of 2^11 entries
    fe pre = fe_one();
    for (int i = kBetaBlockLog; i < nr; i++)
      pre = fmul(pre, ((c >> (i - kBetaBlockLog)) & 1) ? rs[i] : fsub(fe_one(), rs[i]));
    hi_pre[threadIdx.x] = pre;
  }
  if (threadIdx.x == 32) T[0] = fe_one();
  __syncthreads();
  for (int i = kBetaBlockLog - 1; i >= 0; i--) {
    const int len = 1 << (kBetaBlockLog - 1 - i);
    const fe ri = rs[i];
    fe v[4];
    int cnt = 0;
    for (int j = threadIdx.x; j < len; j += blockDim.x) v[cnt++] = T[j];
    __syncthreads();
    cnt = 0;
    for (int j = threadIdx.x; j < len; j += blockDim.x) {
      const fe t = v[cnt++];
      const fe x = fmul(t, ri);
      T[2 * j + 1] = x;
      T[2 * j] = fsub(t, x);
    }
    __syncthreads();
  }
  fe lo[(1 << kBetaBlockLog) / 256];
#pragma unroll
  for (int k = 0; k < (1 << kBetaBlockLog) / 256; k++) lo[k] = T[threadIdx.x + 256 * k];
  fe *o = B + ((uint64_t)blockIdx.x << (kBetaBlockLog + chunks_log));
  for (int c = 0; c < (1 << chunks_log); c++) {
    const fe h = hi_pre[c];
#pragma unroll
    for (int k = 0; k < (1 << kBetaBlockLog) / 256; k++)
      o[((uint64_t)c << kBetaBlockLog) + threadIdx.x + 256 * k] = fmul(h, lo[k]);
  }
}

// update_betas: b[j] += sum_i c_i * w_i^j.  A CTA owns 32 PER consecutive
// entries: lane L of every warp owns the PER entries starting at cta0 + PER L,
// and warp g takes the queries i = g (mod 8), so the l * 32 PER multiply-adds
// of a CTA are spread over all its threads; the eight warps' partial sums are
// added in shared memory.  A thread starts each of its queries' geometric runs
// from s_i * pw_i[L] (s_i = c_i w_i^{cta0}, pw_i[L] = w_i^{PER L}) and steps
// it by w_i.
constexpr int kUbThreads = 256;
constexpr int kUbWarps = kUbThreads / 32;

// pw[i*32 + L] = w_i^(L * per)
__global__ void __launch_bounds__(32) ub_table_kernel(const fe *w, int per, fe *pw) {
  pdl_wait();
  const int i = blockIdx.x, t = threadIdx.x;
  pw[i * 32 + t] = fpow(w[i], (uint64_t)t * per);
}

template <int PER>
__global__ void __launch_bounds__(kUbThreads)
ub_kernel(fe *b, uint64_t nb, const fe *w, const fe *c, int l, const fe *pw, uint64_t b_stride, uint64_t u_stride) {
  pdl_wait();
  constexpr int SPAN = 32 * PER;
  __shared__ fe s_start[kMaxQueries], s_w[kMaxQueries];
  __shared__ fe part[kUbWarps][SPAN];
  b = badv(b, b_stride, blockIdx.y);
  w = badv(w, u_stride, blockIdx.y);
  c = badv(c, u_stride, blockIdx.y);
  pw = badv(pw, u_stride, blockIdx.y);
  const uint64_t cta0 = (uint64_t)blockIdx.x * SPAN;
  for (int i = threadIdx.x; i < l; i += kUbThreads) {
    const fe wi = w[i];
    s_w[i] = wi;
    s_start[i] = fmul(c[i], fpow(wi, cta0));
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  fe acc[PER];  // sums of folded words, folded again after each
#pragma unroll
  for (int k = 0; k < PER; k++) acc[k] = fe_zero();
#pragma unroll(PER == 1 ? 4 : 1)
  for (int i = warp; i < l; i += kUbWarps) {
    const fe wi = s_w[i];
    fe d = fmul_fold(s_start[i], pw[i * 32 + lane]);
#pragma unroll
    for (int k = 0; k < PER; k++) {
      acc[k] = fe_make(fold64(acc[k].re + d.re), fold64(acc[k].im + d.im));
      if (k + 1 < PER) d = fmul_fold(d, wi);
    }
  }
#pragma unroll
  for (int k = 0; k < PER; k++) part[warp][lane * PER + k] = fe_make(canon64(acc[k].re), canon64(acc[k].im));
  __syncthreads();
  // thread t finishes entry cta0 + t
  const uint64_t j = cta0 + threadIdx.x;
  if (threadIdx.x >= SPAN || j >= nb) return;
  fe sum = part[0][threadIdx.x];
#pragma unroll
  for (int g = 1; g < kUbWarps; g++) sum = fadd(sum, part[g][threadIdx.x]);
  b[j] = fadd(b[j], sum);
}

}  // namespace

int sc_blocks(uint64_t pairs) {
  uint64_t want = (pairs + kScThreads - 1) / kScThreads;
  const uint64_t cap = 152 * 8;  // 8 CTAs per SM on 152 SMs, grid-stride beyond that
  if (want > cap) want = cap;
  return want ? (int)want : 1;
}

void sc_step_launch(const fe *a, const fe *b, uint64_t m, const fe *chal, fe *a2, fe *b2, bool reduce,
                    fe *partial, int blocks, cudaStream_t s) {
  if (!chal) {
    launch_kernel(sc_reduce_kernel, blocks, kScThreads, 0, s, a, b, m / 2, partial);
  } else {
    launch_kernel(sc_fold_kernel, blocks, kScThreads, 0, s, a, b, m, chal, a2, b2, reduce ? 1 : 0, partial);
  }
  GBZ_CUDA(cudaGetLastError());
}

void sc_fold2_launch(const fe *a, const fe *b, uint64_t m, const fe *chal0, const fe *chal1, fe *a4, fe *b4,
                     fe *partial0, fe *partial1, int blocks, cudaStream_t s, int batch, const BStr &bs) {
  if (m < 4) throw ArgError("two-round fold needs at least 4 entries");
  launch_kernel(sc_fold2_kernel, dim3(blocks, batch), kScThreads, 0, s, a, b, m, chal0, chal1, a4, b4, partial0,
                partial1, bs);
  GBZ_CUDA(cudaGetLastError());
}

void sc_fold2_eq_launch(const fe *a, const fe *E2, uint64_t m, const fe *c, const fe *chal0, const fe *chal1, fe *a4,
                        fe *b4, fe *partial0, fe *partial1, int blocks, cudaStream_t s, int batch, const BStr &bs) {
  if (m < 4) throw ArgError("two-round fold needs at least 4 entries");
  launch_kernel(sc_fold2_eq_kernel, dim3(blocks, batch), kScThreads, 0, s, a, E2, m, c, chal0, chal1, a4, b4,
                partial0, partial1, bs);
  GBZ_CUDA(cudaGetLastError());
}

void sc_eq_reduce_launch(const fe *a, const fe *E, uint64_t m, fe *partial, int blocks, cudaStream_t s, int batch,
                         const BStr &bs) {
  launch_kernel(sc_eq_reduce_kernel, dim3(blocks, batch), kScThreads, 0, s, a, E, m, partial, bs);
  GBZ_CUDA(cudaGetLastError());
}

void sc_eq_fold_launch(const fe *a, const fe *E, uint64_t m, const fe *chal, fe *a4, fe *E4, bool reduce, fe *partial,
                       int blocks, cudaStream_t s, int batch, const BStr &bs) {
  if (m < 128 || m % 128) throw ArgError("two-round fold of w needs a multiple of 128 entries");
  launch_kernel(sc_eq_fold_kernel, dim3(blocks, batch), kScThreads, 0, s, a, m, chal, a4, E, E4, reduce ? 1 : 0,
                partial, bs);
  GBZ_CUDA(cudaGetLastError());
}

void sc_sum_launch(const fe *partial, int blocks, fe *out3, cudaStream_t s) {
  launch_kernel(sc_sum_kernel, 1, kScThreads, 0, s, partial, blocks, out3);
  GBZ_CUDA(cudaGetLastError());
}

void beta_launch(const fe *r, int nr, fe *B, cudaStream_t s, int batch, uint64_t r_stride, uint64_t B_stride) {
  if (nr < 0 || nr > 60) throw ArgError("beta table: bad number of variables");
  BStr bs;
  bs.s[0] = r_stride;
  bs.s[1] = B_stride;
  if (nr >= kBetaBlockLog + 4) {
    // enough CTAs to cover the SMs (at least 2^9), up to 16 blocks each
    const int chunks_log = std::max(0, std::min(kBetaChunksLog, nr - kBetaBlockLog - 9));
    launch_kernel(beta_tensor_kernel, dim3((unsigned)(1ull << (nr - kBetaBlockLog - chunks_log)), batch), 256, 0, s,
                  r, nr, chunks_log, B, bs);
    GBZ_CUDA(cudaGetLastError());
    return;
  }
  const int low = nr < kBetaBlockLog ? nr : kBetaBlockLog;
  launch_kernel(beta_block_kernel, dim3((unsigned)(1ull << (nr - low)), batch), 256, 0, s, r, nr, B, bs);
  GBZ_CUDA(cudaGetLastError());
}

int update_betas_per(uint64_t nb, int batch) {
  const uint64_t entries = nb * (uint64_t)batch;
  return entries >= (1ull << 15) ? 8 : entries >= (1ull << 13) ? 2 : 1;
}

void update_betas_powers_launch(fe *b, uint64_t nb, const fe *w, const fe *c, int l, const fe *pw, cudaStream_t s,
                                int batch, uint64_t b_stride, uint64_t u_stride) {
  if (l <= 0) return;
  if (l > kMaxQueries) throw ArgError("update_betas: too many queries");
  const int per = update_betas_per(nb, batch), span = 32 * per;
  const dim3 grid((unsigned)((nb + span - 1) / span), batch);
  if (!grid.x) return;
  if (per == 8) launch_kernel(ub_kernel<8>, grid, kUbThreads, 0, s, b, nb, w, c, l, pw, b_stride, u_stride);
  else if (per == 2) launch_kernel(ub_kernel<2>, grid, kUbThreads, 0, s, b, nb, w, c, l, pw, b_stride, u_stride);
  else launch_kernel(ub_kernel<1>, grid, kUbThreads, 0, s, b, nb, w, c, l, pw, b_stride, u_stride);
  GBZ_CUDA(cudaGetLastError());
}

void update_betas_launch(fe *b, uint64_t nb, const ProofState *st, int l, fe *pw_scratch, cudaStream_t s) {
  if (l <= 0) return;
  if (l > kMaxQueries) throw ArgError("update_betas: too many queries");
  launch_kernel(ub_table_kernel, l, 32, 0, s, st->omega_q, update_betas_per(nb, 1), pw_scratch);
  GBZ_CUDA(cudaGetLastError());
  update_betas_powers_launch(b, nb, st->omega_q, st->comb, l, pw_scratch, s, 1, 0, 0);
}

}  // namespace gbz
