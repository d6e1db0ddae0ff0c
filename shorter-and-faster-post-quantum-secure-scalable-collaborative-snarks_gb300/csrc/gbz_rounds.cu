// Round forms of the multilinear sumcheck provers and the device-resident
// distributed sumcheck (gbz_rounds.cuh).
//
// Every form sums, over the pairs (v[2j], v[2j+1]) of its vectors, a product
// of the lines l(x) = (v[2j+1] - v[2j]) x + v[2j] (linear_poly,
// polynomial.h:46-59), coefficients highest degree first:
//   quadratic (v1, v2)            sum l1 l2                    coSumcheck_MPI.cpp:199
//   cubic (v1, v2, v3)            sum l1 l2 l3                 Distributed_Sumcheck.cpp:1144-1151
//   batch (v1..v4, r1, r2; b)     sum l1 l2 + l3 l4 + b lr1 lr2 coSumcheck_MPI.cpp:156-176
//   zero-check (v1, v2, v3, beta, r1, r2; b)
//                                 sum (l1 l2 + b lr1 lr2 - x l3) lbeta   coSumcheck_MPI.cpp:12-32
//   quadruple (v1..v4)            sum l1 l2 l3 l4              delegate_protocol.cpp:66-76
// and folds every vector by the round challenge r: v[j] = v[2j] + r (v[2j+1]
// - v[2j]) (coSumcheck_MPI.cpp:34-44, 178-187).  The fold of round i and the
// message of round i + 1 are one pass (four entries of every vector per
// thread).  All arithmetic is exact, so the summation order does not change
// a single bit of the result.
#include "gbz_rounds.cuh"

#include <type_traits>

namespace gbz {

namespace {

constexpr int kThreads = 256;

template <int FORM> struct Form;
template <> struct Form<SC_QUADRATIC> { static constexpr int NV = 2, NC = 3; };
template <> struct Form<SC_CUBIC> { static constexpr int NV = 3, NC = 4; };
template <> struct Form<SC_BATCH> { static constexpr int NV = 6, NC = 3; };
template <> struct Form<SC_ZEROCHECK> { static constexpr int NV = 6, NC = 4; };
template <> struct Form<SC_QUADRUPLE> { static constexpr int NV = 4, NC = 5; };

struct Line {
  fe a, b, h;  // a x + b, h = a + b (the value at 1)
};
__device__ __forceinline__ Line line(fe lo, fe hi) { return Line{fsub(hi, lo), lo, hi}; }

// x / 2 in F_p: (x + p x_0) / 2 of each word.
__device__ __forceinline__ uint64_t halfp(uint64_t x) { return (x & 1) ? (x + P) >> 1 : x >> 1; }
__device__ __forceinline__ fe fhalf(fe x) { return fe_make(halfp(x.re), halfp(x.im)); }

// The cubic form accumulates, per thread, the sums of its products at 0, 1,
// -1 and the leading coefficient (7 products a pair instead of 9); this
// turns them into the coefficients (x^3, x^2, x, 1) before the sums are
// combined across threads.  The map is linear and exact, so the messages
// are the coefficient sums the reference forms pair by pair.
template <int FORM>
__device__ __forceinline__ void acc_to_coeffs(fe *acc) {
  if (FORM == SC_QUADRATIC) acc[1] = fsub(fsub(acc[1], acc[0]), acc[2]);  // q(1) = q2 + q1 + q0
  if (FORM == SC_CUBIC) {
    const fe e_inf = acc[0], e1 = acc[1], em = acc[2], e0 = acc[3];
    acc[1] = fsub(fhalf(fadd(e1, em)), e0);     // c(1) + c(-1) = 2 (c2 + c0)
    acc[2] = fsub(fhalf(fsub(e1, em)), e_inf);  // c(1) - c(-1) = 2 (c3 + c1)
  }
}

// (a1 x + b1)(a2 x + b2) with three products
__device__ __forceinline__ void lmul(const Line &x, const Line &y, fe q[3]) {
  q[0] = fmul(x.a, y.a);
  q[2] = fmul(x.b, y.b);
  q[1] = fsub(fsub(fmul(fadd(x.a, x.b), fadd(y.a, y.b)), q[0]), q[2]);
}
// (q0 x^2 + q1 x + q2)(a x + b)
__device__ __forceinline__ void qlmul(const fe q[3], const Line &l, fe c[4]) {
  c[0] = fmul(q[0], l.a);
  c[1] = fadd(fmul(q[0], l.b), fmul(q[1], l.a));
  c[2] = fadd(fmul(q[1], l.b), fmul(q[2], l.a));
  c[3] = fmul(q[2], l.b);
}

// The sums of a thread: 96-bit accumulators for the forms of plain products
// (quadratic, cubic, quadruple), reduced once per thread; canonical sums for
// the two weighted forms, whose coefficients are combined before they are
// added.
template <int FORM> struct Sums {
  static constexpr bool kLazy = FORM == SC_QUADRATIC || FORM == SC_CUBIC || FORM == SC_QUADRUPLE;
  typedef typename std::conditional<kLazy, facc, fe>::type type;
};
__device__ __forceinline__ void sum_zero(facc &s) { s = facc_zero(); }
__device__ __forceinline__ void sum_zero(fe &s) { s = fe_zero(); }
__device__ __forceinline__ fe sum_value(const facc &s) { return facc_value(s); }
__device__ __forceinline__ fe sum_value(const fe &s) { return s; }

// What each accumulator of a form holds: quadratic the leading coefficient,
// the values at 1 and 0; cubic the leading coefficient, the values at 1, -1
// and 0; the others the coefficients.  acc_to_coeffs turns a thread's sums
// into coefficients.
template <int FORM>
__device__ __forceinline__ void accumulate(const Line *l, fe b, typename Sums<FORM>::type *acc) {
  fe q[3], c[4];
  if constexpr (FORM == SC_QUADRATIC) {
    facc_mul(acc[0], l[0].a, l[1].a);
    facc_mul(acc[1], l[0].h, l[1].h);
    facc_mul(acc[2], l[0].b, l[1].b);
  } else if constexpr (FORM == SC_CUBIC) {
    // the first two lines' product at the leading coefficient, 1 and 0 gives
    // its value at -1: 2 (q_inf + q_0) - q_1, with 2p to stay positive
    const fe qi = fmul_fold(l[0].a, l[1].a), q1 = fmul_fold(l[0].h, l[1].h), q0 = fmul_fold(l[0].b, l[1].b);
    const fe qm = fe_make(fold64(2 * (qi.re + q0.re) + (2 * P - q1.re)), fold64(2 * (qi.im + q0.im) + (2 * P - q1.im)));
    facc_mul(acc[0], qi, l[2].a);
    facc_mul(acc[1], q1, l[2].h);
    facc_mul(acc[2], qm, fsub(l[2].b, l[2].a));
    facc_mul(acc[3], q0, l[2].b);
  } else if constexpr (FORM == SC_QUADRUPLE) {
    // ((l1 l2) l3) l4 as the reference multiplies them (polynomial.cpp:91-101)
    lmul(l[0], l[1], q);
    qlmul(q, l[2], c);
    facc_mul(acc[0], c[0], l[3].a);
    facc_mul(acc[1], c[1], l[3].a);
    facc_mul(acc[1], c[0], l[3].b);
    facc_mul(acc[2], c[2], l[3].a);
    facc_mul(acc[2], c[1], l[3].b);
    facc_mul(acc[3], c[3], l[3].a);
    facc_mul(acc[3], c[2], l[3].b);
    facc_mul(acc[4], c[3], l[3].b);
  } else if constexpr (FORM == SC_BATCH) {
    fe q2[3], qr[3];
    lmul(l[0], l[1], q);
    lmul(l[2], l[3], q2);
    lmul(l[4], l[5], qr);
    for (int k = 0; k < 3; k++) acc[k] = fadd(acc[k], fadd(fadd(q[k], q2[k]), fmul(b, qr[k])));
  } else {
    fe qr[3];
    lmul(l[0], l[1], q);
    lmul(l[4], l[5], qr);
    q[0] = fadd(q[0], fmul(b, qr[0]));
    q[1] = fsub(fadd(q[1], fmul(b, qr[1])), l[2].a);
    q[2] = fsub(fadd(q[2], fmul(b, qr[2])), l[2].b);
    qlmul(q, l[3], c);
    for (int k = 0; k < 4; k++) acc[k] = fadd(acc[k], c[k]);
  }
}

__device__ __forceinline__ fe shfl_down_fe(fe v, int d) {
  fe r;
  r.re = __shfl_down_sync(0xffffffffu, v.re, d);
  r.im = __shfl_down_sync(0xffffffffu, v.im, d);
  return r;
}

// Block sum of NC field elements; valid in thread 0.
template <int NC>
__device__ void block_sum(fe *x) {
  __shared__ fe red[kMaxFormCoeffs][kThreads / 32];
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
#pragma unroll
    for (int k = 0; k < NC; k++) x[k] = fadd(x[k], shfl_down_fe(x[k], d));
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0)
    for (int k = 0; k < NC; k++) red[k][w] = x[k];
  __syncthreads();
  if (w == 0) {
    const int nw = blockDim.x >> 5;
    for (int k = 0; k < NC; k++) x[k] = lane < nw ? red[k][lane] : fe_zero();
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
#pragma unroll
      for (int k = 0; k < NC; k++) x[k] = fadd(x[k], shfl_down_fe(x[k], d));
  }
}

// MODE 0: message over the pairs of in (pairs = m / 2).
// MODE 1: fold in (length 4 * pairs) by *r into out and message of the folded vectors.
// MODE 2: fold only (pairs = outputs).
// scale (optional): vector 2 of pair entry e is multiplied by scale[e >> scale_log]
// as it is read (the parties' weights of the cubic form).
template <int FORM, int MODE>
__global__ void __launch_bounds__(kThreads) form_step_kernel(RoundArgs a) {
  pdl_wait();
  constexpr int NV = Form<FORM>::NV, NC = Form<FORM>::NC;
  typename Sums<FORM>::type sums[NC];
#pragma unroll
  for (int k = 0; k < NC; k++) sum_zero(sums[k]);
  const fe r = MODE ? *a.r : fe_zero();
  const fe b = a.b ? *a.b : fe_zero();
  const uint64_t stride = (uint64_t)gridDim.x * kThreads;
  for (uint64_t g = (uint64_t)blockIdx.x * kThreads + threadIdx.x; g < a.pairs; g += stride) {
    Line l[NV];
    if (MODE == 0) {
#pragma unroll
      for (int k = 0; k < NV; k++) {
        fe lo = a.in[k][2 * g], hi = a.in[k][2 * g + 1];
        if (k == 2 && a.scale) {  // a pair may straddle two parties when M = 1
          lo = fmul(lo, a.scale[(2 * g) >> a.scale_log]);
          hi = fmul(hi, a.scale[(2 * g + 1) >> a.scale_log]);
        }
        l[k] = line(lo, hi);
      }
      accumulate<FORM>(l, b, sums);
    } else if (MODE == 1) {
      // every vector's four entries are loaded before any output is stored
      // (the stores could alias later loads, so the compiler would not
      // hoist them): one memory round trip per step instead of one per vector
      fe xs[NV][4];
#pragma unroll
      for (int k = 0; k < NV; k++) {
        const fe *p = a.in[k] + 4 * g;
#pragma unroll
        for (int q = 0; q < 4; q++) xs[k][q] = p[q];
      }
#pragma unroll
      for (int k = 0; k < NV; k++) {
        fe x0 = xs[k][0], x1 = xs[k][1], x2 = xs[k][2], x3 = xs[k][3];
        if (k == 2 && a.scale) {
          x0 = fmul(x0, a.scale[(4 * g) >> a.scale_log]);
          x1 = fmul(x1, a.scale[(4 * g + 1) >> a.scale_log]);
          x2 = fmul(x2, a.scale[(4 * g + 2) >> a.scale_log]);
          x3 = fmul(x3, a.scale[(4 * g + 3) >> a.scale_log]);
        }
        const fe f0 = ffold(x0, x1, r), f1 = ffold(x2, x3, r);
        a.out[k][2 * g] = f0;
        a.out[k][2 * g + 1] = f1;
        l[k] = line(f0, f1);
      }
      accumulate<FORM>(l, b, sums);
    } else {
#pragma unroll
      for (int k = 0; k < NV; k++) {
        fe x0 = a.in[k][2 * g], x1 = a.in[k][2 * g + 1];
        if (k == 2 && a.scale) {
          x0 = fmul(x0, a.scale[(2 * g) >> a.scale_log]);
          x1 = fmul(x1, a.scale[(2 * g + 1) >> a.scale_log]);
        }
        a.out[k][g] = ffold(x0, x1, r);
      }
    }
  }
  if (MODE == 2) return;
  fe acc[NC];
#pragma unroll
  for (int k = 0; k < NC; k++) acc[k] = sum_value(sums[k]);
  acc_to_coeffs<FORM>(acc);
  block_sum<NC>(acc);
  if (threadIdx.x == 0)
#pragma unroll
    for (int k = 0; k < NC; k++) a.partial[(uint64_t)blockIdx.x * NC + k] = acc[k];
}

// Copies the first entry of every vector (with the weight scale of vector
// 2) to fin: the final values when no round is left.
__global__ void form_first_kernel(RoundArgs a, int nv, fe *fin) {
  pdl_wait();
  const int k = threadIdx.x;
  if (k >= nv) return;
  fe x = a.in[k][0];
  if (k == 2 && a.scale) x = fmul(x, a.scale[0]);
  fin[k] = x;
}

__device__ fe eval_poly(const fe *c, int nc, fe x) {
  fe acc = c[0];
  for (int k = 1; k < nc; k++) acc = fadd(fmul(acc, x), c[k]);
  return acc;
}

// Thread-0 part of a round: checks H(0) + H(1) against the running claim y,
// stores H, draws the challenge (Fiat-Shamir hash chain fs over the
// coefficients, or the leader's glibc challenge drawn ahead of time by
// prng_draw_kernel when drawn is set) and updates the claim.  The state is
// passed by reference so that the one-CTA tail keeps it in registers.
__device__ fe finish_round(const fe *H, int nc, fe &fs, fe &y, uint32_t &error, int round, const fe *drawn,
                           fe *polys, fe *chal) {
  // H(0) + H(1) = 2 c_last + sum of the other coefficients
  fe s = H[nc - 1];
  for (int k = 0; k < nc; k++) s = fadd(s, H[k]);
  if (!fe_eq(s, y)) error |= 1u;
  for (int k = 0; k < nc; k++) polys[(uint64_t)round * nc + k] = H[k];
  fe ch;
  if (drawn) {
    ch = *drawn;
  } else {
    for (int k = 0; k < nc; k++) fs = hash_F(fs, H[k]);
    ch = fs;
  }
  chal[round] = ch;
  y = eval_poly(H, nc, ch);
  return ch;
}

__device__ __forceinline__ fe shfl_xor_fe(fe x, int d) {
  return fe_make(__shfl_xor_sync(0xffffffffu, x.re, d), __shfl_xor_sync(0xffffffffu, x.im, d));
}

// Sum of coefficient k of `blocks` partials over a warp's lanes.
__device__ __forceinline__ fe warp_partial_sum(const fe *partial, int blocks, int nc, int k, int first, int step) {
  fe x = fe_zero();
#pragma unroll 4
  for (int i = first; i < blocks; i += step) x = fadd(x, partial[(uint64_t)i * nc + k]);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) x = fadd(x, shfl_xor_fe(x, d));
  return x;
}

// Sums the partials into the round polynomial H (nc coefficients, two warps
// each) and finishes the round.
__global__ void __launch_bounds__(256)
form_finalize_kernel(const fe *partial, int blocks, int nc, RoundState *st, int round, const fe *drawn, fe *polys,
                     fe *chal) {
  pdl_wait();
  __shared__ fe red[4][2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k = warp >> 1;
  fe fs = st->fs, y = st->y;
  uint32_t error = st->error;
  if (k < nc) {
    const fe x = warp_partial_sum(partial, blocks, nc, k, lane + 32 * (warp & 1), 64);
    if (lane == 0) red[k][warp & 1] = x;
  }
  __syncthreads();
  if (threadIdx.x) return;
  fe H[4];
#pragma unroll
  for (int q = 0; q < 4; q++)
    if (q < nc) H[q] = fadd(red[q][0], red[q][1]);
  finish_round(H, nc, fs, y, error, round, drawn, polys, chal);
  st->fs = fs;
  st->y = y;
  st->error = error;
}

// The leader's rounds take the fourth of every four F::_random() draws
// (Distributed_Sumcheck.cpp), 160 outputs of the generator; the glibc stream
// depends on nothing the rounds compute, so a warp draws its n challenges
// while the first, largest rounds run, and the stream's final state goes back
// to st->prng.  Of a challenge's outputs the last 40 are its digits.  (One
// thread took 22 us a challenge.)
__global__ void __launch_bounds__(32) prng_draw_kernel(RoundState *st, int n, fe *out) {
  pdl_wait();
  constexpr int kDraws = 160, kFull = kDraws / 31, kRest = kDraws % 31;
  __shared__ int32_t d[kDraws + 31];
  const int lane = threadIdx.x, f0 = st->prng.f;
  uint32_t x = prng_warp_load(st->prng, lane);
#pragma unroll 1
  for (int j = 0; j < n; j++) {
#pragma unroll 1
    for (int b = 0; b < kFull; b++) {
      x = prng_warp_next(x, lane);
      if (lane < 31) d[31 * b + lane] = (int32_t)(x >> 1);
    }
    const uint32_t y = prng_warp_next(x, lane);
    if (lane < kRest) d[31 * kFull + lane] = (int32_t)(y >> 1);
    x = prng_warp_shift(x, y, kRest, lane);
    __syncwarp();
    uint64_t v = 0;
    if (lane < 2) v = prng_number_from(d + kDraws - 40 + 20 * lane) % P;
    const uint64_t im = __shfl_sync(0xffffffffu, v, 1);
    if (lane == 0) out[j] = fe_make(v, im);
    __syncwarp();
  }
  __syncwarp();
  prng_warp_store(st->prng, x, f0, (uint64_t)kDraws * n, lane);
}

constexpr int kTailThreads = 512, kTailWarps = kTailThreads / 32;

// One round of a one-CTA tail: folds the form's vectors (cur entries) by r
// into out and leaves the message's sums, a warp each, in red[k][warp].
// Returns the number of warps that had work.
template <int FORM>
__device__ __forceinline__ int tail_round(const fe *const *in, fe *const *out, uint64_t cur, fe r,
                                          fe (*red)[kTailWarps]) {
  constexpr int NV = Form<FORM>::NV, NC = Form<FORM>::NC;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int pairs = (int)(cur / 4), active = min(kTailWarps, (pairs + 31) / 32);
  if (wid < active) {
    typename Sums<FORM>::type sums[NC];
#pragma unroll
    for (int k = 0; k < NC; k++) sum_zero(sums[k]);
    for (int g = threadIdx.x; g < pairs; g += kTailThreads) {
      Line l[NV];
#pragma unroll
      for (int k = 0; k < NV; k++) {
        const fe *p = in[k] + 4 * g;
        const fe f0 = ffold(p[0], p[1], r), f1 = ffold(p[2], p[3], r);
        out[k][2 * g] = f0;
        out[k][2 * g + 1] = f1;
        l[k] = line(f0, f1);
      }
      accumulate<FORM>(l, fe_zero(), sums);
    }
    fe acc[NC];
#pragma unroll
    for (int k = 0; k < NC; k++) acc[k] = sum_value(sums[k]);
    acc_to_coeffs<FORM>(acc);
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
#pragma unroll
      for (int k = 0; k < NC; k++) acc[k] = fadd(acc[k], shfl_down_fe(acc[k], d));
    if (lane == 0)
#pragma unroll
      for (int k = 0; k < NC; k++) red[k][wid] = acc[k];
  }
  return active;
}

// Shared memory of a tail entered with `cur` entries: the vectors' folds,
// cur/2 entries and cur/4 in turn.
template <int FORM>
constexpr size_t tail_shared(uint64_t cur) {
  return sizeof(fe) * Form<FORM>::NV * (cur / 2 + cur / 4);
}
template <int FORM>
__device__ __forceinline__ void tail_buffers(fe *sm, uint64_t cur, fe *(*buf)[Form<FORM>::NV]) {
  constexpr int NV = Form<FORM>::NV;
  for (int k = 0; k < NV; k++) {
    buf[0][k] = sm + k * (cur / 2);
    buf[1][k] = sm + NV * (cur / 2) + k * (cur / 4);
  }
}

struct TailArgs {
  const fe *in[3];  // entries entering round i0, before its fold
  uint64_t cur;     // entries of every vector entering round i0
  int i0, total, fs_rounds;
  RoundState *st;
  const fe *drawn;  // glibc challenges of rounds fs_rounds.. (or null)
  fe *polys, *chal, *fin;
};

// Rounds i0..total-1 of the party sumcheck and the final fold in one CTA,
// once the vectors are small: every round is the fused fold + message of
// form_step_kernel<FORM, 1> in shared memory, a reduction and finish_round.
// A round costs its four hashes (2.2 us) and about as much again, where a
// launch of a step and one of the finish take 9; from 2^13 entries on the
// folds of one SM take longer than that.  (From 2^14 entries and through L2
// the last 14 rounds took 116 us; these last 12 take 51.)
template <int FORM>
__global__ void __launch_bounds__(kTailThreads) form_tail_kernel(TailArgs t) {
  pdl_wait();
  constexpr int NV = Form<FORM>::NV, NC = Form<FORM>::NC;
  extern __shared__ fe tail_sm[];
  __shared__ fe red[NC][kTailWarps];
  __shared__ fe sh_r;
  const fe *in[NV];
  fe *buf[2][NV];
  tail_buffers<FORM>(tail_sm, t.cur, buf);
#pragma unroll
  for (int k = 0; k < NV; k++) in[k] = t.in[k];
  fe r = t.chal[t.i0 - 1];
  fe fs = fe_zero(), y = fe_zero();  // the running state, in thread 0's registers
  uint32_t error = 0;
  if (threadIdx.x == 0) {
    fs = t.st->fs;
    y = t.st->y;
    error = t.st->error;
  }
  uint64_t cur = t.cur;
  int pp = 0;
#pragma unroll 1
  for (int i = t.i0; i < t.total; i++) {
    const int active = tail_round<FORM>(in, buf[pp], cur, r, red);
    __syncthreads();
    if (threadIdx.x < 32) {
      // lane 8 k + w takes warps w and w + 8 of coefficient k
      const int k = threadIdx.x >> 3, w = threadIdx.x & 7;
      fe x = fe_zero();
      if (k < NC && w < active) x = red[k][w];
      if (k < NC && w + 8 < active) x = fadd(x, red[k][w + 8]);
#pragma unroll
      for (int d = 4; d > 0; d >>= 1) x = fadd(x, shfl_xor_fe(x, d));
      fe H[4];
#pragma unroll
      for (int q = 0; q < 4; q++)
        H[q] = fe_make(__shfl_sync(0xffffffffu, x.re, 8 * q), __shfl_sync(0xffffffffu, x.im, 8 * q));
      if (threadIdx.x == 0)
        sh_r = finish_round(H, NC, fs, y, error, i,
                            i >= t.fs_rounds && t.drawn ? t.drawn + (i - t.fs_rounds) : nullptr, t.polys, t.chal);
    }
    __syncthreads();
    r = sh_r;
#pragma unroll
    for (int k = 0; k < NV; k++) in[k] = buf[pp][k];
    pp ^= 1;
    cur /= 2;
  }
  if (threadIdx.x == 0) {
    t.st->fs = fs;
    t.st->y = y;
    t.st->error = error;
  }
  // final fold of the last length-2 vectors: the leader's v[0] values
#pragma unroll
  for (int k = 0; k < NV; k++)
    if ((int)threadIdx.x == k) t.fin[k] = fadd(in[k][0], fmul(r, fsub(in[k][1], in[k][0])));
}

// Rounds i0..rounds-1 of a sumcheck whose challenges were drawn ahead
// (the leader's glibc sumchecks of delegate_protocol.cpp) and its final
// fold, in one CTA, and the messages of all its rounds.  No fold waits for a
// message, so they are finished together at the end, a warp a round: the sum
// of its partials, H(0) + H(1) against the claim that the round before leaves
// (flag `bit` when it differs, none when bit is 0), H and the challenge.  A
// round takes a fold and a barrier (finished one by one, and through L2 from
// 2^14 entries on, the quadruple form took 111 us and the cubic 105, now 46 and 31).
template <int FORM>
__global__ void __launch_bounds__(kTailThreads) form_tail_drawn_kernel(DrawnTailArgs t) {
  pdl_wait();
  constexpr int NV = Form<FORM>::NV, NC = Form<FORM>::NC;
  extern __shared__ fe tail_sm[];
  __shared__ fe red[kDrawnTailLog][NC][kTailWarps];
  __shared__ fe claim[kMaxLogN + 2];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  auto challenge = [&](int i) { return t.draw[t.first + (uint64_t)t.stride * i]; };
  const fe *in[NV];
  fe *buf[2][NV];
  uint64_t cur = t.n >> (t.i0 - 1);
  tail_buffers<FORM>(tail_sm, cur, buf);
#pragma unroll
  for (int k = 0; k < NV; k++) in[k] = t.in[k];
  int pp = 0;
#pragma unroll 1
  for (int i = t.i0; i < t.rounds; i++) {
    tail_round<FORM>(in, buf[pp], cur, challenge(i - 1), red[i - t.i0]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NV; k++) in[k] = buf[pp][k];
    pp ^= 1;
    cur /= 2;
  }
  // the final fold of the length-2 vectors: their v[0]
  if ((int)threadIdx.x < NV) {
    const fe *p = in[threadIdx.x];
    const fe v = fadd(p[0], fmul(challenge(t.rounds - 1), fsub(p[1], p[0])));
    t.fin[threadIdx.x] = v;
    put_fe(t.tr, t.off_fin + 16ull * threadIdx.x, v);
  }
  if (threadIdx.x == 0) claim[0] = *t.y;
  // a warp a round; claim[i + 1] is what round i leaves
  fe at01[(kMaxLogN + 2 + kTailWarps - 1) / kTailWarps];
  int q = 0;
#pragma unroll
  for (int base = 0; base < kMaxLogN + 2; base += kTailWarps, q++) {
    const int i = base + wid;
    if (i >= t.rounds) continue;
    fe H[NC];
    if (i < t.i0) {
#pragma unroll
      for (int k = 0; k < NC; k++) H[k] = warp_partial_sum(t.partial[i], t.blocks[i], NC, k, lane, 32);
    } else {
      const int active = min(kTailWarps, (int)(((t.n >> (i + 1)) + 31) / 32));
#pragma unroll
      for (int k = 0; k < NC; k++) {
        fe x = lane < active ? red[i - t.i0][k][lane] : fe_zero();
#pragma unroll
        for (int d = kTailWarps / 2; d > 0; d >>= 1) x = fadd(x, shfl_xor_fe(x, d));
        H[k] = x;
      }
    }
    if (lane == 0) {
      const fe c = challenge(i);
      fe e = H[NC - 1];
#pragma unroll
      for (int k = 0; k < NC; k++) {
        e = fadd(e, H[k]);
        put_fe(t.tr, t.off_polys + 16ull * ((uint64_t)i * NC + k), H[k]);
      }
      at01[q] = e;
      t.ch[i] = c;
      claim[i + 1] = eval_poly(H, NC, c);
    }
  }
  __syncthreads();
  q = 0;
#pragma unroll
  for (int base = 0; base < kMaxLogN + 2; base += kTailWarps, q++) {
    const int i = base + wid;
    if (i < t.rounds && lane == 0 && t.bit && !fe_eq(at01[q], claim[i])) atomicOr(t.flags, t.bit);
  }
  if (threadIdx.x == 0) *t.y = claim[t.rounds];
}

__global__ void form_sum_kernel(const fe *partial, int blocks, int nc, fe *out) {
  pdl_wait();
  __shared__ fe red[kMaxFormCoeffs][kThreads];
  fe acc[kMaxFormCoeffs];
  for (int k = 0; k < kMaxFormCoeffs; k++) acc[k] = fe_zero();
  for (int i = threadIdx.x; i < blocks; i += kThreads)
    for (int k = 0; k < nc; k++) acc[k] = fadd(acc[k], partial[(uint64_t)i * nc + k]);
  for (int k = 0; k < kMaxFormCoeffs; k++) red[k][threadIdx.x] = acc[k];
  __syncthreads();
  for (int w = kThreads / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w)
      for (int k = 0; k < kMaxFormCoeffs; k++) red[k][threadIdx.x] = fadd(red[k][threadIdx.x], red[k][threadIdx.x + w]);
    __syncthreads();
  }
  if (threadIdx.x < (unsigned)nc) out[threadIdx.x] = red[threadIdx.x][0];
}

template <int FORM, int MODE>
void launch_step(const RoundArgs &a, int blocks, cudaStream_t s) {
  launch_kernel(form_step_kernel<FORM, MODE>, blocks, kThreads, 0, s, a);
  GBZ_CUDA(cudaGetLastError());
}

template <int FORM>
void launch_form(const RoundArgs &a, int mode, int blocks, cudaStream_t s) {
  if (mode == 0) launch_step<FORM, 0>(a, blocks, s);
  else if (mode == 1) launch_step<FORM, 1>(a, blocks, s);
  else launch_step<FORM, 2>(a, blocks, s);
}

}  // namespace

int form_vectors(int form) {
  switch (form) {
    case SC_QUADRATIC: return 2;
    case SC_CUBIC: return 3;
    case SC_BATCH: return 6;
    case SC_ZEROCHECK: return 6;
    case SC_QUADRUPLE: return 4;
    default: return 0;
  }
}
int form_coeffs(int form) {
  switch (form) {
    case SC_QUADRATIC: return 3;
    case SC_CUBIC: return 4;
    case SC_BATCH: return 3;
    case SC_ZEROCHECK: return 4;
    case SC_QUADRUPLE: return 5;
    default: return 0;
  }
}

int round_blocks(uint64_t pairs) {
  uint64_t want = (pairs + kThreads - 1) / kThreads;
  const uint64_t cap = 152 * 8;
  if (want > cap) want = cap;
  return want ? (int)want : 1;
}

void form_step_launch(int form, const RoundArgs &a, int mode, int blocks, cudaStream_t s) {
  switch (form) {
    case SC_QUADRATIC: launch_form<SC_QUADRATIC>(a, mode, blocks, s); break;
    case SC_CUBIC: launch_form<SC_CUBIC>(a, mode, blocks, s); break;
    case SC_BATCH: launch_form<SC_BATCH>(a, mode, blocks, s); break;
    case SC_ZEROCHECK: launch_form<SC_ZEROCHECK>(a, mode, blocks, s); break;
    case SC_QUADRUPLE: launch_form<SC_QUADRUPLE>(a, mode, blocks, s); break;
    default: throw ArgError("sumcheck: unknown round form");
  }
}

namespace {
template <int FORM>
void launch_tail_drawn(const DrawnTailArgs &a, cudaStream_t s) {
  const size_t sh = tail_shared<FORM>(a.n >> (a.i0 - 1));
  GBZ_CUDA(cudaFuncSetAttribute(form_tail_drawn_kernel<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tail_shared<FORM>(1ull << kDrawnTailLog)));
  launch_kernel(form_tail_drawn_kernel<FORM>, 1, kTailThreads, sh, s, a);
}
template <int FORM>
void launch_tail(const TailArgs &a, cudaStream_t s) {
  GBZ_CUDA(cudaFuncSetAttribute(form_tail_kernel<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tail_shared<FORM>(kTailEntries)));
  launch_kernel(form_tail_kernel<FORM>, 1, kTailThreads, tail_shared<FORM>(a.cur), s, a);
}
}  // namespace

void form_tail_drawn_launch(int form, const DrawnTailArgs &a, cudaStream_t s) {
  if (a.rounds > kMaxLogN || (a.n >> (a.i0 - 1)) > (1ull << kDrawnTailLog))
    throw ArgError("sumcheck tail: too many rounds or entries");
  switch (form) {
    case SC_QUADRATIC: launch_tail_drawn<SC_QUADRATIC>(a, s); break;
    case SC_CUBIC: launch_tail_drawn<SC_CUBIC>(a, s); break;
    case SC_QUADRUPLE: launch_tail_drawn<SC_QUADRUPLE>(a, s); break;
    default: throw ArgError("sumcheck tail: quadratic, cubic or quadruple form");
  }
  GBZ_CUDA(cudaGetLastError());
}

void form_sum_launch(const fe *partial, int blocks, int nc, fe *out, cudaStream_t s) {
  launch_kernel(form_sum_kernel, 1, kThreads, 0, s, partial, blocks, nc, out);
  GBZ_CUDA(cudaGetLastError());
}

void form_finalize_launch(const fe *partial, int blocks, int nc, RoundState *st, int round, const fe *drawn, fe *polys,
                          fe *chal, cudaStream_t s) {
  launch_kernel(form_finalize_kernel, 1, kThreads, 0, s, partial, blocks, nc, st, round, drawn, polys, chal);
  GBZ_CUDA(cudaGetLastError());
}

void form_first_launch(const RoundArgs &a, int nv, fe *fin, cudaStream_t s) {
  launch_kernel(form_first_kernel, 1, 32, 0, s, a, nv, fin);
  GBZ_CUDA(cudaGetLastError());
}

int party_sumcheck_rounds(uint64_t M, int N, int offset, int *fs_rounds) {
  const int lm = ilog2(M);
  int rounds = lm - offset, off = offset;
  if (rounds <= 0) {
    rounds = 0;
    off = lm;
  }
  if (fs_rounds) *fs_rounds = rounds;
  return rounds + ilog2((uint64_t)N << off);
}

void party_sumcheck_enqueue(int form, const fe *const *v, uint64_t M, int N, const fe *w, int offset, RoundState *st,
                            fe *const *scratch, fe *partial, fe *polys, fe *chal, fe *fin, fe *drawn,
                            const SideStream &side, cudaStream_t s) {
  // The N parties' vectors are held party-major, so pair g of the
  // concatenation is pair g mod (cur/2) of party g / (cur/2) while every
  // party still has two entries or more: the parties' round polynomials
  // summed (with the weights w folded into v3 for the cubic form, which is
  // what aggregate_poly computes) are the round polynomial of the
  // concatenation, and the leader's gathered vectors are the concatenation
  // itself.  So the N-party prover is one sumcheck over N * M entries whose
  // first rounds draw Fiat-Shamir challenges and whose last log2(N * 2^offset)
  // rounds draw the leader's glibc challenges.
  const int nv = form_vectors(form), nc = form_coeffs(form);
  int fs_rounds = 0;
  const int total = party_sumcheck_rounds(M, N, offset, &fs_rounds);
  uint64_t cur = M * (uint64_t)N;
  RoundArgs a{};
  a.b = nullptr;
  a.partial = partial;
  a.scale = form == SC_CUBIC ? w : nullptr;
  a.scale_log = ilog2(M);
  for (int k = 0; k < nv; k++) a.in[k] = v[k];
  if (total == 0) {
    form_first_launch(a, nv, fin, s);
    return;
  }
  // the leader's glibc challenges, drawn on the side stream while the first
  // rounds run; the stream joins before the first round that takes one
  const bool glibc = total > fs_rounds;
  if (glibc) {
    cudaStream_t ds = side.stream ? side.stream : s;
    if (side.stream) {
      GBZ_CUDA(cudaEventRecord(side.fork, s));
      GBZ_CUDA(cudaStreamWaitEvent(side.stream, side.fork, 0));
    }
    launch_kernel(prng_draw_kernel, 1, 32, 0, ds, st, total - fs_rounds, drawn);
    GBZ_CUDA(cudaGetLastError());
    if (side.stream) GBZ_CUDA(cudaEventRecord(side.join, side.stream));
  }
  bool joined = !glibc || !side.stream;
  auto join = [&](int upto) {  // before a launch that finishes rounds up to upto
    if (!joined && upto >= fs_rounds) {
      GBZ_CUDA(cudaStreamWaitEvent(s, side.join, 0));
      joined = true;
    }
  };
  int pp = 0;
  for (int i = 0; i < total; i++) {
    int blocks;
    if (i == 0) {
      a.pairs = cur / 2;
      blocks = round_blocks(a.pairs);
      form_step_launch(form, a, 0, blocks, s);
    } else {
      if (i >= 2 && cur <= kTailEntries) {
        // the remaining rounds and the final fold in one CTA
        TailArgs t{};
        for (int k = 0; k < nv; k++) t.in[k] = a.in[k];
        t.cur = cur;
        t.i0 = i;
        t.total = total;
        t.fs_rounds = fs_rounds;
        t.st = st;
        t.drawn = glibc ? drawn : nullptr;
        t.polys = polys;
        t.chal = chal;
        t.fin = fin;
        join(total - 1);
        if (form == SC_QUADRATIC) launch_tail<SC_QUADRATIC>(t, s);
        else launch_tail<SC_CUBIC>(t, s);
        GBZ_CUDA(cudaGetLastError());
        return;
      }
      // fold by the previous challenge into scratch[pp], message of the result
      a.pairs = cur / 4;
      a.r = chal + (i - 1);
      for (int k = 0; k < nv; k++) a.out[k] = scratch[pp * 6 + k];
      blocks = round_blocks(a.pairs);
      form_step_launch(form, a, 1, blocks, s);
      for (int k = 0; k < nv; k++) a.in[k] = a.out[k];
      a.scale = nullptr;
      pp ^= 1;
      cur /= 2;
    }
    join(i);
    form_finalize_launch(partial, blocks, nc, st, i, i >= fs_rounds ? drawn + (i - fs_rounds) : nullptr, polys, chal,
                         s);
  }
  // final fold of the last length-2 vectors: the leader's v[0] values
  a.pairs = 1;
  a.r = chal + (total - 1);
  for (int k = 0; k < nv; k++) a.out[k] = fin + k;
  form_step_launch(form, a, 2, 1, s);
}

}  // namespace gbz
