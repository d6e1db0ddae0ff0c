// F_{p^2} arithmetic, p = 2^61 - 1, i^2 = -1, for device and host code.
//
// Replaces virgo::fieldElement (fieldElement.hpp:20-108, fieldElement.cpp).
// Layout: {uint64 re, uint64 im}, 16 bytes, `real` first, exactly the bytes
// the reference memcpy's into Merkle leaves and Fiat-Shamir blocks.
//
// All operations take canonical inputs (each word in [0, p)) and return
// canonical outputs.  For canonical inputs the reference's operators also
// return canonical values equal to the exact field result, so any exact
// evaluation order gives identical bytes; the multiply below uses fewer
// conditional steps than the reference's literal sequence
// (fieldElement.cpp:49-78) but the same value.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define GBZ_HD __host__ __device__ __forceinline__
#else
#define GBZ_HD inline
#endif

namespace gbz {

constexpr uint64_t P = 0x1FFFFFFFFFFFFFFFull;  // 2^61 - 1 (fieldElement.cpp:7)

struct alignas(16) fe {
  uint64_t re, im;
};

GBZ_HD fe fe_make(uint64_t re, uint64_t im) { fe r; r.re = re; r.im = im; return r; }
GBZ_HD fe fe_zero() { return fe_make(0, 0); }
GBZ_HD fe fe_one() { return fe_make(1, 0); }
GBZ_HD bool fe_eq(fe a, fe b) { return a.re == b.re && a.im == b.im; }

// Full 64x64 -> 128 product.
GBZ_HD void mul64wide(uint64_t x, uint64_t y, uint64_t &lo, uint64_t &hi) {
#ifdef __CUDA_ARCH__
  lo = x * y;
  hi = __umul64hi(x, y);
#else
  unsigned __int128 t = (unsigned __int128)x * y;
  lo = (uint64_t)t;
  hi = (uint64_t)(t >> 64);
#endif
}

// x*y mod p without the final reduction: for x, y < 2^62 the value is
// congruent to x*y and below 2^63 + 2^61 (the reference's mymult,
// fieldElement.cpp:341-361, computes the same quantity).
GBZ_HD uint64_t mulp_lazy(uint64_t x, uint64_t y) {
  uint64_t lo, hi;
  mul64wide(x, y, lo, hi);
  return ((hi << 3) | (lo >> 61)) + (lo & P);
}

// Full reduction of any 64-bit value to [0, p).
GBZ_HD uint64_t redp(uint64_t t) {
  t = (t >> 61) + (t & P);  // <= p + 7
  return t >= P ? t - P : t;
}

GBZ_HD uint64_t addp(uint64_t a, uint64_t b) {
  uint64_t s = a + b;
  return s >= P ? s - P : s;
}
GBZ_HD uint64_t subp(uint64_t a, uint64_t b) {
  uint64_t s = a + (P - b);
  return s >= P ? s - P : s;
}

// operator+ (fieldElement.cpp:34-47)
GBZ_HD fe fadd(fe a, fe b) { return fe_make(addp(a.re, b.re), addp(a.im, b.im)); }
// operator- (fieldElement.cpp:80-96)
GBZ_HD fe fsub(fe a, fe b) { return fe_make(subp(a.re, b.re), subp(a.im, b.im)); }
GBZ_HD fe fneg(fe a) { return fsub(fe_zero(), a); }

// Reduction of a value below 2^125 to [0, p): 2^61 = 1 (mod p) folds the
// high part onto the low 61 bits twice, then one conditional subtraction.
GBZ_HD uint64_t red125(unsigned __int128 v) {
  const uint64_t lo = (uint64_t)v, hi = (uint64_t)(v >> 64);
  uint64_t t = ((hi << 3) | (lo >> 61)) + (lo & P);  // < 2^63 + 2^61
  t = (t >> 61) + (t & P);                            // <= p + 4
  return t >= P ? t - P : t;
}

#ifdef __CUDACC__
// The device multiply works on sums of two products, S = a b + c d, in
// 32-bit columns.  What bounds it on sm_103a: IMAD.WIDE occupies the FMA
// pipe for 4 cycles a warp and every other integer instruction one of the
// two pipes (FMA, ALU) for 2, so the eight wide products a component (64
// cycles an F_{p^2} multiply) are the floor and each instruction beside them
// counts.  The columns are chosen so that none of them needs a register
// move: the cross products share one 64-bit accumulator (they stay below
// 2^64 because the high words are short), the low ones chain their carry
// into the high ones.  48.6 instructions canonical and 42.6 folded, against
// 66.8 for the 128-bit form that the host uses below.  gbz_calibrate (four
// chains a thread on every SM): 445 G canonical multiplies/s, 345 before;
// folded ones are 7 % faster.
struct dot_cols {
  uint32_t x0, x1, x2, x3;  // S, least significant word first
};
// Requires a, c < 2^62 and b, d <= 2^61: S < 2^124.
// add: a constant added to S.
__device__ __forceinline__ dot_cols dot2_cols(uint64_t a, uint64_t b, uint64_t c, uint64_t d, uint32_t add = 0) {
  dot_cols s;
  asm("{\n\t"
      ".reg .u32 al, ah, bl, bh, cl, ch, dl, dh, ml, mh;\n\t"
      ".reg .u64 m;\n\t"
      "mov.b64 {al, ah}, %4;\n\t"
      "mov.b64 {bl, bh}, %5;\n\t"
      "mov.b64 {cl, ch}, %6;\n\t"
      "mov.b64 {dl, dh}, %7;\n\t"
      "mul.wide.u32 m, al, bh;\n\t"
      "mad.wide.u32 m, ah, bl, m;\n\t"
      "mad.wide.u32 m, cl, dh, m;\n\t"
      "mad.wide.u32 m, ch, dl, m;\n\t"
      "mov.b64 {ml, mh}, m;\n\t"
      "mad.lo.cc.u32 %0, al, bl, %8;\n\t"
      "madc.hi.u32 %1, al, bl, 0;\n\t"
      "mad.lo.cc.u32 %0, cl, dl, %0;\n\t"
      "madc.hi.cc.u32 %1, cl, dl, %1;\n\t"
      "madc.lo.cc.u32 %2, ah, bh, 0;\n\t"
      "madc.hi.u32 %3, ah, bh, 0;\n\t"
      "mad.lo.cc.u32 %2, ch, dh, %2;\n\t"
      "madc.hi.u32 %3, ch, dh, %3;\n\t"
      "add.cc.u32 %1, %1, ml;\n\t"
      "addc.cc.u32 %2, %2, mh;\n\t"
      "addc.u32 %3, %3, 0;\n\t"
      "}"
      : "=&r"(s.x0), "=&r"(s.x1), "=&r"(s.x2), "=&r"(s.x3)
      : "l"(a), "l"(b), "l"(c), "l"(d), "r"(add));
  return s;
}
// A single product a b, a < 2^62, b < 2^62.
__device__ __forceinline__ dot_cols dot1_cols(uint64_t a, uint64_t b) {
  dot_cols s;
  asm("{\n\t"
      ".reg .u32 al, ah, bl, bh, ml, mh;\n\t"
      ".reg .u64 m;\n\t"
      "mov.b64 {al, ah}, %4;\n\t"
      "mov.b64 {bl, bh}, %5;\n\t"
      "mul.wide.u32 m, al, bh;\n\t"
      "mad.wide.u32 m, ah, bl, m;\n\t"
      "mov.b64 {ml, mh}, m;\n\t"
      "mul.lo.u32 %0, al, bl;\n\t"
      "mul.hi.u32 %1, al, bl;\n\t"
      "mul.lo.u32 %2, ah, bh;\n\t"
      "mul.hi.u32 %3, ah, bh;\n\t"
      "add.cc.u32 %1, %1, ml;\n\t"
      "addc.cc.u32 %2, %2, mh;\n\t"
      "addc.u32 %3, %3, 0;\n\t"
      "}"
      : "=&r"(s.x0), "=&r"(s.x1), "=&r"(s.x2), "=&r"(s.x3)
      : "l"(a), "l"(b));
  return s;
}
__device__ __forceinline__ uint64_t words64(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }
// S < 2^124 to t = S (mod p), t < 2^63 + 2^61, in two words.
__device__ __forceinline__ void dot_wrap(const dot_cols &s, uint32_t &tl, uint32_t &th) {
  const uint32_t ul = __funnelshift_l(s.x1, s.x2, 3), uh = __funnelshift_l(s.x2, s.x3, 3);
  asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, %5;"
      : "=r"(tl), "=r"(th)
      : "r"(ul), "r"(s.x0), "r"(uh), "r"(s.x1 & 0x1fffffffu));
}
// S (mod p) in [0, p + 4].
__device__ __forceinline__ uint64_t dot_fold(const dot_cols &s) {
  uint32_t tl, th, ol, oh;
  dot_wrap(s, tl, th);
  asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, 0;"
      : "=r"(ol), "=r"(oh)
      : "r"(tl), "r"(th >> 29), "r"(th & 0x1fffffffu));
  return words64(ol, oh);
}
// t mod p in [0, p) for t < 2^64 - 16, in two words: the quotient is
// floor((t + floor(t / 2^61) + 1) / 2^61).
__device__ __forceinline__ uint64_t canon_words(uint32_t tl, uint32_t th) {
  uint32_t qh, ol, oh;
  asm("{\n\t"
      ".reg .u32 t;\n\t"
      "add.cc.u32 t, %1, %2;\n\t"
      "addc.u32 %0, %3, 0;\n\t"
      "}"
      : "=r"(qh)
      : "r"(tl), "r"((th >> 29) + 1), "r"(th));
  asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, 0;" : "=r"(ol), "=r"(oh) : "r"(tl), "r"(qh >> 29), "r"(th));
  return words64(ol, oh & 0x1fffffffu);
}
__device__ __forceinline__ uint64_t canon64(uint64_t t) { return canon_words((uint32_t)t, (uint32_t)(t >> 32)); }
// S mod p in [0, p).
__device__ __forceinline__ uint64_t dot_canon(const dot_cols &s) {
  uint32_t tl, th;
  dot_wrap(s, tl, th);
  return canon_words(tl, th);
}
__device__ __forceinline__ uint64_t dot_wrap64(const dot_cols &s) {
  uint32_t tl, th;
  dot_wrap(s, tl, th);
  return words64(tl, th);
}
// Products with lazy words.  a's words may be up to 2p (a difference below),
// b's at most p.
__device__ __forceinline__ dot_cols mul_re(fe a, fe b) { return dot2_cols(a.re, b.re, a.im, b.im ^ P); }  // p - b.im
__device__ __forceinline__ dot_cols mul_im(fe a, fe b) { return dot2_cols(a.re, b.im, a.im, b.re); }
// Each component folded to [0, p + 4].
__device__ __forceinline__ fe fmul_fold(fe a, fe b) { return fe_make(dot_fold(mul_re(a, b)), dot_fold(mul_im(a, b))); }
// a - b + p, words in [0, 2p], for words in [0, p].
__device__ __forceinline__ fe fsub_lazy(fe a, fe b) { return fe_make(a.re + (b.re ^ P), a.im + (b.im ^ P)); }
__device__ __forceinline__ fe fadd_lazy(fe a, fe b) { return fe_make(a.re + b.re, a.im + b.im); }
// x0 + r (x1 - x0), canonical: x0 joins the wrapped sum.
__device__ __forceinline__ fe ffold(fe x0, fe x1, fe r) {
  const fe d = fsub_lazy(x1, x0);
  return fe_make(canon64(dot_wrap64(mul_re(d, r)) + x0.re), canon64(dot_wrap64(mul_im(d, r)) + x0.im));
}
// The same for base-field x0, x1 (imaginary words zero).
__device__ __forceinline__ fe ffold_base(uint64_t x0, uint64_t x1, fe r) {
  const uint64_t d = x1 + (x0 ^ P);
  return fe_make(canon64(dot_wrap64(dot1_cols(d, r.re)) + x0), dot_canon(dot1_cols(d, r.im)));
}

// A sum of products, each component 96 bits wide: a product is added after
// the first wrap (below 2^63 + 2^61), so a term costs 34 instructions beside
// its wide products instead of the 45 of a canonical product and a canonical
// addition, and the reduction comes once at the end.  Up to 2^32 terms.
struct facc {
  uint32_t re[3], im[3];
};
__device__ __forceinline__ facc facc_zero() { return facc{{0, 0, 0}, {0, 0, 0}}; }
__device__ __forceinline__ void acc96(uint32_t *w, const dot_cols &s) {
  uint32_t tl, th;
  dot_wrap(s, tl, th);
  asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, 0;"
      : "+r"(w[0]), "+r"(w[1]), "+r"(w[2])
      : "r"(tl), "r"(th));
}
__device__ __forceinline__ void facc_mul(facc &s, fe a, fe b) {
  acc96(s.re, mul_re(a, b));
  acc96(s.im, mul_im(a, b));
}
__device__ __forceinline__ void facc_mul_base(facc &s, fe a, uint64_t c) {
  acc96(s.re, dot1_cols(a.re, c));
  acc96(s.im, dot1_cols(a.im, c));
}
__device__ __forceinline__ uint64_t canon96(const uint32_t *w) {
  const uint64_t lo = words64(w[0], w[1]);  // 2^64 = 8 (mod p)
  return canon64((lo & P) + (lo >> 61) + 8ull * w[2]);
}
__device__ __forceinline__ fe facc_value(const facc &s) { return fe_make(canon96(s.re), canon96(s.im)); }

// The same sum in four registers instead of six (kernels with many of them):
// each component folded after every term, ten instructions instead of three.
struct facc64 {
  uint64_t re, im;
};
__device__ __forceinline__ uint64_t fold64(uint64_t t) { return (t & P) + (t >> 61); }
__device__ __forceinline__ void facc_mul(facc64 &s, fe a, fe b) {
  s.re = fold64(s.re + dot_fold(mul_re(a, b)));
  s.im = fold64(s.im + dot_fold(mul_im(a, b)));
}
__device__ __forceinline__ fe facc_value(const facc64 &s) { return fe_make(canon64(s.re), canon64(s.im)); }
#endif

// operator* (fieldElement.cpp:49-78).  Both forms combine the four 122-bit
// products exactly (re = ac - bd plus a multiple of p, im = ad + bc) and
// reduce each component once; the reference's Karatsuba form with lazy
// reductions gives the same canonical value.  a's words may be up to 2^62.
GBZ_HD fe fmul(fe a, fe b) {
#ifdef __CUDA_ARCH__
  const uint64_t nb = b.im ^ P;  // p - b.im
  return fe_make(dot_canon(dot2_cols(a.re, b.re, a.im, nb)), dot_canon(dot2_cols(a.re, b.im, a.im, b.re)));
#else
  typedef unsigned __int128 u128;
  const u128 ac = (u128)a.re * b.re, bd = (u128)a.im * b.im;
  const u128 ad = (u128)a.re * b.im, bc = (u128)a.im * b.re;
  const u128 bias = (u128)P * P * 2;  // a multiple of p above any bd
  return fe_make(red125(ac + (bias - bd)), red125(ad + bc));
#endif
}

GBZ_HD fe fsqr(fe a) { return fmul(a, a); }

// Multiply by a base-field value (img == 0): two products.
GBZ_HD fe fmul_base(fe a, uint64_t c) {
#ifdef __CUDA_ARCH__
  return fe_make(dot_canon(dot1_cols(a.re, c)), dot_canon(dot1_cols(a.im, c)));
#else
  return fe_make(redp(mulp_lazy(a.re, c)), redp(mulp_lazy(a.im, c)));
#endif
}

// fastPow (fieldElement.cpp:323-335) for exponents below 2^64.
GBZ_HD fe fpow(fe x, uint64_t e) {
  fe r = fe_one();
  while (e) {
    if (e & 1) r = fmul(r, x);
    x = fmul(x, x);
    e >>= 1;
  }
  return r;
}

// inv (fieldElement.cpp:207-210), 0 for 0: 1 / x = conj(x) / (re^2 + im^2), the
// norm (zero for x = 0 only, p = 3 mod 4) inverted as N^(p - 2), p - 2 =
// 2^61 - 3: N^(2^k - 1) up to k = 59, then N^(4 (2^59 - 1) + 1).  70 products
// in the base field where x^(p^2 - 2) took 300 in the extension (2 us instead
// of 20 on one thread).
GBZ_HD uint64_t mulp_red(uint64_t a, uint64_t b) { return redp(mulp_lazy(a, b)); }
GBZ_HD fe finv(fe x) {
  const uint64_t n = addp(mulp_red(x.re, x.re), mulp_red(x.im, x.im));
  uint64_t r = n;  // n^(2^k - 1)
  int k = 1;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
  for (int bit = 4; bit >= 0; bit--) {  // 59 = 111011 in binary
    uint64_t t = r;
    for (int q = 0; q < k; q++) t = mulp_red(t, t);
    r = mulp_red(t, r);
    k *= 2;
    if ((59 >> bit) & 1) {
      r = mulp_red(mulp_red(r, r), n);
      k++;
    }
  }
  r = mulp_red(r, r);
  r = mulp_red(mulp_red(r, r), n);
  return fe_make(mulp_red(x.re, r), mulp_red(x.im ? P - x.im : 0, r));
}

// getRootOfUnity (utils.cpp:706-717): generator of order 2^61 squared
// (62 - log_order) times.
GBZ_HD fe root_of_unity(int log_order) {
  fe r = fe_make(2147483648ull, 1033321771269002680ull);
  for (int i = 0; i < 62 - log_order; i++) r = fmul(r, r);
  return r;
}

// quadratic_poly::eval (polynomial.cpp:111-113): ((a x) + b) x + c
GBZ_HD fe quad_eval(fe a, fe b, fe c, fe x) { return fadd(fmul(fadd(fmul(a, x), b), x), c); }

}  // namespace gbz
