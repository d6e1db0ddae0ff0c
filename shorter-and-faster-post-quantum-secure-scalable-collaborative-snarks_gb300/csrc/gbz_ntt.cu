// Number-theoretic transform over F_{p^2} for power-of-two lengths.
//
// Replaces fft (utils.cpp:904-964), _fft/__fft (:966-1110) and pfft
// (:1583-1673).  All of them compute out[k] = sum_j in[j] w^{jk} with
// w = getRootOfUnity(logn) (its inverse, plus a 2^-logn scale, for the
// inverse transform); pfft is a 16-thread four-step split of the same
// forward transform.  Exact field arithmetic makes the result independent
// of the factorisation, so the GPU uses its own:
//
//  * lengths up to 2^13: one shared-memory pass;
//  * longer lengths: two or three passes (schedule()).  With L = S C, a pass
//    over columns computes, for each column l < C, the length-S DFT of
//    x[l + C j] (zero beyond n_valid: the Reed-Solomon padding is never
//    read), times omega_L^{l k}, stored at l + C k; what remains are S rows
//    of length C, transformed by the next passes.  The last pass stores in
//    natural order (no bit reversal pass).
//
// Inside a pass every CTA holds B sub-transforms of length S in shared
// memory and runs self-sorting (Stockham) stages on them, radix 8 after one
// radix-2 or radix-4 stage when log2 S is not a multiple of 3.  The first
// stage runs on the values as they are loaded from global memory and the
// last one stores from registers; between stages the values cross shared
// memory, with a barrier among the threads of one sub-transform only.
// Groups of B >= 2 neighbouring columns make the strided pass read whole
// 32-byte sectors.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "gbz_internal.cuh"

namespace gbz {

namespace {

constexpr int kSubLog = 13;          // largest sub-transform held in shared memory
constexpr int kTwLoBits = 12;        // outer twiddle table split
constexpr int kMaxThreads = 1024;
constexpr int kCtaElems = 1 << kSubLog;  // most elements staged per CTA
constexpr int kSmallLog = 10;        // longest sub-transform of the small kernel
constexpr int kCosetLog = 10;        // longest transform taken in cosets
constexpr int kPerThread = 8;            // elements per thread (CTA = max(32, E/8) threads)

// Two-pass shape of a length set by ntt_set_shape (the autotuner): k1 = log2
// of the contiguous second pass and the sub-transforms staged per CTA in each
// pass.  Lengths without one (k1 = -1) take the passes of schedule().
NttShape g_shape[kMaxLogN + 1];

struct PassArgs {
  const fe *in;
  fe *out;
  uint64_t n_valid;
  // Sub-transform g = h 2^logG + l reads its entry j at l in_gstride + h
  // in_hstride + j in_jstride and writes its output k at l out_gstride + h
  // out_hstride + k out_kstride; l is the column of the outer twiddle.
  uint64_t in_gstride, in_hstride, in_jstride, out_gstride, out_hstride, out_kstride;
  int logG;
  const fe *stages;  // twiddles of the direction: of the stages, or the small kernel's (set at launch)
  // The outer twiddle of output k is omega_L^{l k 2^tw_shift}.
  const fe *tw_lo;   // omega_L^t, t < 2^12 (nullptr: no outer twiddle)
  const fe *tw_hi;   // omega_L^{2^12 t}
  const fe *tw_full; // the twiddle at l out_gstride + k out_kstride + h tw_hstride (optional)
  uint64_t tw_hstride;
  int tw_shift;
  fe scale;
  int logS, logB, has_scale, inverse;
  // Sparse rows (second pass of a sparse transform, the first pass folded
  // in): the input is sum_i sp_c[i] e_{q_i}, q_i = sp_q[i] >> sp_shift;
  // entries of one column (q mod the row length) are chained by sp_next
  // from the one flagged in sp_lead; sp_lo / sp_hi give omega_L^e and
  // sp_mask = L - 1.
  const int32_t *sp_q;
  const fe *sp_c;
  int sp_l, sp_shift;
  const int16_t *sp_next;
  const uint8_t *sp_lead;
  const fe *sp_lo, *sp_hi;
  uint64_t sp_mask;
  // Accumulating output: out[addr] += v for addr < acc_n, other outputs dropped.
  uint64_t acc_n;
  int acc;
  // Every entry is present: n_valid and j_valid need no test (set at launch).
  int dense;
  // Coset form of a padded transform (the small kernel): entry j of
  // sub-transform l is multiplied by omega_L^{l j} (in_lo, in_hi as tw_lo,
  // tw_hi) when it is loaded.
  const fe *in_lo, *in_hi;
  // Entries j >= j_valid of every sub-transform are zero (per-transform
  // padding of batched transforms; S when unused).
  uint32_t j_valid;
  // Independent transforms side by side: grid row y works on in + y row_in
  // and out + y row_out (0 for one transform).
  uint64_t row_in, row_out;
  // Packed real input: input entry j is (in[2j].re, in[2j+1].re) (two
  // base-field values as one extension element); a non-zero imaginary word
  // among them sets *nonreal.
  int pack_real;
  uint32_t *nonreal;
  // Scattered output: output i of the row, with the fields (m, r, j) of
  // sc_n, sc_n and sc_lo bits from the top, goes to r sc_stride + m 2^sc_lo + j.
  int sc_lo, sc_n;
  uint64_t sc_stride;
  // When set, the pass does nothing unless *run_if is non-zero.
  const uint32_t *run_if;
};

// ---- lazy arithmetic inside one butterfly --------------------------------
// Words are residues held mod 2^64: additions and subtractions are plain
// 64-bit instructions, and the window of every word is argued once, here, so
// that a result is read as the integer it stands for when it is folded.
// Fold any 64-bit value to [0, p + 7] (p itself stands for zero).
__device__ __forceinline__ uint64_t fold(uint64_t x) { return (x & P) + (x >> 61); }
__device__ __forceinline__ uint64_t canon(uint64_t x) {  // [0, p + 7] -> [0, p)
  return x >= P ? x - P : x;
}
// A staged value (folded to [0, p + 7] by the last stage, or canonical) made
// canonical for the output.
__device__ __forceinline__ fe canon_fe(fe x) { return fe_make(canon(x.re), canon(x.im)); }
__device__ __forceinline__ fe lz_add(fe a, fe b) { return fe_make(a.re + b.re, a.im + b.im); }
__device__ __forceinline__ fe lz_sub(fe a, fe b) { return fe_make(a.re - b.re, a.im - b.im); }
__device__ __forceinline__ fe lz_fold(fe a) { return fe_make(fold(a.re), fold(a.im)); }
// a + w4 b (PLUS) or a - w4 b: getRootOfUnity(2) = -i, inverse i.
template <bool INV, bool PLUS>
__device__ __forceinline__ fe lz_w4_add(fe a, fe b) {
  return INV == PLUS ? fe_make(a.re - b.im, a.im + b.re) : fe_make(a.re + b.im, a.im - b.re);
}
// z 2^30 (mod p) for a signed z, |z| < 2^63: z = h 2^31 + l gives
// h 2^61 + l 2^30 = h + l 2^30, in [-2^32, p + 2^32].
__device__ __forceinline__ uint64_t mul2e30(uint64_t z) { return ((z << 30) & P) + (uint64_t)((int64_t)z >> 31); }

// x w + (1 + i) for a staged x (words <= p + 7) and a table twiddle w, each
// word in [1, p + 1].  The constant keeps the fold away from zero, which
// makes the window p wide instead of p + 1: with S + 1 <= (p + 7)(2p - 64) + 1
// (tw_margin) the wrapped sum stays below 3 2^61 - 50, so its quotient 2
// leaves at most p - 50 and quotients 0, 1 at most p and p + 1.
__device__ __forceinline__ fe tw_mul(fe x, fe w) {
  const uint64_t nb = w.im ^ P;
  return fe_make(dot_fold(dot2_cols(x.re, w.re, x.im, nb, 1)), dot_fold(dot2_cols(x.re, w.im, x.im, w.re, 1)));
}
// In-register DFTs with natural-order output: V[k] = sum_q v[q] w_R^{qk},
// words folded to [0, p + 7].
// dft2 and dft4 only run as a first stage, on words in [0, p + 7]: a sum of
// four of them and a difference biased by 2p or 4p stay within 64 bits.
template <bool INV>
__device__ __forceinline__ void dft2(fe *v) {
  const fe a = v[0], b = v[1], c = fe_make(a.re + 2 * P, a.im + 2 * P);
  v[0] = lz_fold(lz_add(a, b));
  v[1] = lz_fold(lz_sub(c, b));
}
template <bool INV>
__device__ __forceinline__ void dft4(fe *v) {
  const fe z = fe_make(v[0].re + 4 * P, v[0].im + 4 * P);
  const fe c0 = lz_add(v[0], v[2]), c1 = lz_add(v[1], v[3]);
  const fe c0b = lz_add(z, v[2]), d0 = lz_sub(z, v[2]), d1 = lz_sub(v[1], v[3]);
  v[0] = lz_fold(lz_add(c0, c1));
  v[2] = lz_fold(lz_sub(c0b, c1));
  v[1] = lz_fold(lz_w4_add<INV, true>(d0, d1));
  v[3] = lz_fold(lz_w4_add<INV, false>(d0, d1));
}
// Radix 8.  v[0] in [0, p + 7]; v[1..7] hold x + (1 + i) in [1, p + 1]
// (OFF, the outputs of tw_mul) or x in [0, p + 7] with x <= p - 1 except for
// v[0] (first stage, canonical).  Every output is v[0] plus signed inputs:
// v[0] carries the bias 4p (and the constant, which then cancels everywhere
// but in V[0], where both are taken out again), so
//   V[0] = sum of eight                                  in [0, 8p + 7],
//   V[2], V[4], V[6] + 4p: four inputs with either sign  in [0, 8p + 7],
//   odd V + 4p: b0 and w4 b2 in +-p, c1 and d1 of the rotated pair in
//     +-(p + 2^33) once the sum of two of them is shifted by p,
//     so within +-(3p + 2^34)                            in [0, 8p],
// and 8p + 7 = 2^64 - 1: no word wraps, and one fold each ends the stage.
// Against the previous form (biased subtractions of two instructions more
// and canonical products) a radix-8 stage issues 62 instead of 106
// arithmetic instructions an element.
template <bool INV, bool OFF>
__device__ __forceinline__ void dft8(fe *v) {
  constexpr uint64_t B = 4 * P + (OFF ? 1 : 0);  // bias of v[0]
  constexpr uint64_t Z = 4 * P + (OFF ? 8 : 0);  // what V[0] holds of biases and constants
  v[0] = fe_make(v[0].re + B, v[0].im + B);
  fe a[4], b[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    a[q] = lz_add(v[q], v[q + 4]);
    b[q] = lz_sub(v[q], v[q + 4]);
  }
  {
    const fe c0 = lz_add(a[0], a[2]), c1 = lz_add(a[1], a[3]);
    const fe d0 = lz_sub(a[0], a[2]), d1 = lz_sub(a[1], a[3]);
    v[0] = lz_fold(fe_make(c0.re + c1.re - Z, c0.im + c1.im - Z));
    v[4] = lz_fold(lz_sub(c0, c1));
    v[2] = lz_fold(lz_w4_add<INV, true>(d0, d1));
    v[6] = lz_fold(lz_w4_add<INV, false>(d0, d1));
  }
  // w8 = 2^30 (1 - i) and w8^3 = 2^30 (-1 - i), inverse conjugates: with
  // s = re + im, d = im - re
  //   forward: w8 b1 = (m(s1), m(d1)),   w8^3 b3 = (m(d3), -m(s3))
  //   inverse: w8 b1 = (m(-d1), m(s1)),  w8^3 b3 = (-m(s3), m(-d3))
  const uint64_t m1s = mul2e30(b[1].re + b[1].im), m3s = mul2e30(b[3].re + b[3].im);
  const uint64_t m1d = mul2e30(INV ? b[1].re - b[1].im : b[1].im - b[1].re);
  const uint64_t m3d = mul2e30(INV ? b[3].re - b[3].im : b[3].im - b[3].re);
  const fe c0 = lz_w4_add<INV, true>(b[0], b[2]), d0 = lz_w4_add<INV, false>(b[0], b[2]);
  fe c1, d1;
  if (INV) {
    c1 = fe_make(m1d - m3s, m1s + m3d - P);
    d1 = fe_make(m1d + m3s - P, m1s - m3d);
  } else {
    c1 = fe_make(m1s + m3d - P, m1d - m3s);
    d1 = fe_make(m1s - m3d, m1d + m3s - P);
  }
  v[1] = lz_fold(lz_add(c0, c1));
  v[5] = lz_fold(lz_sub(c0, c1));
  v[3] = lz_fold(lz_w4_add<INV, true>(d0, d1));
  v[7] = lz_fold(lz_w4_add<INV, false>(d0, d1));
}

// ---- one pass ------------------------------------------------------------
// The stages of a length-2^LOGS sub-transform: a first one of radix 2, 4 or
// 8 (whatever makes the rest a multiple of three levels), then radix 8.
__host__ __device__ constexpr int first_log(int logs) { return logs <= 3 ? logs : (logs % 3 == 0 ? 3 : logs % 3); }
// Stage twiddles: the products of a stage depend on Ns alone (omega_{8 Ns}^{r
// k}, k < Ns, r = 1..7), so one table in global memory serves every length:
// Ns = 2, 4, ..., 2^10 one after the other, each [r - 1][k].  Lanes of a warp
// read neighbouring k, whole lines out of L1 (57 KB for the last stage of
// S = 2^12, beside 128 KB of staged data).  As a half table of omega_S in
// shared memory, loaded by every CTA, the strided reads cost up to eight
// wavefronts for one (a pass's loads took three times their ideal wavefronts;
// of the 12 million that a pass of 2^9 over 2^24 elements takes now, one is
// a conflict) and r = 5..7 a conditional negation.
__host__ __device__ constexpr uint32_t stage_table_offset(int logns) { return 7u * ((1u << logns) - 2); }

// Entry j of sub-transform b in shared memory.  The exclusive or with j / 8
// keeps contiguous and stride-8 runs of 16-byte elements free of bank
// conflicts, the one with xb the runs that take the same j of neighbouring
// sub-transforms.
template <int LOGS>
__device__ __forceinline__ uint32_t slot(uint32_t b, uint32_t xb, uint32_t j) {
  return (b << LOGS) + (j ^ ((j >> 3) & 7u) ^ xb);
}
// The slot of entry j + (r << LR) from the slot s0 of entry j, where j has
// zeros at those bits: the exclusive or is linear.
template <int LR>
__device__ __forceinline__ uint32_t slot_step(uint32_t s0, uint32_t r) {
  const uint32_t x = r << LR;
  return LR >= 6 ? s0 + x : s0 ^ (x ^ ((x >> 3) & 7u));
}
// Spreads neighbouring sub-transforms over the banks so that eight lanes with
// 2 or 4 of them and 4 or 2 consecutive butterflies of radix 2, 4 or 8 meet
// no bank twice (the shifts lie outside the spans of the lanes' own offsets).
__device__ __forceinline__ uint32_t bank_shift(uint32_t b, int logB) {
  if (logB >= 3) return b & 7u;
  return logB == 2 ? (b & 1 ? 3u : 0u) ^ (b & 2 ? 5u : 0u) : (b & 1 ? 7u : 0u);
}

// Waits for the threads that share a sub-transform: a warp, or a named
// barrier of the S/8 threads where a CTA holds several sub-transforms, so
// that one group's memory phase overlaps another's arithmetic.
template <int LOGS>
__device__ __forceinline__ void group_sync() {
  constexpr uint32_t G = LOGS >= 3 ? 1u << (LOGS - 3) : 1u;
  if (G <= 32) {
    __syncwarp();
  } else if (blockDim.x <= G || blockDim.x / G > 15) {
    __syncthreads();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + threadIdx.x / G), "r"(G) : "memory");
  }
}

// Twiddle products of one butterfly of a stage with Ns = 2^LOGNS.
template <int LOGNS>
__device__ __forceinline__ void twiddle_inputs(fe *v, const fe *stages, uint32_t j) {
  const uint4 *t = reinterpret_cast<const uint4 *>(stages + stage_table_offset(LOGNS) + (j & ((1u << LOGNS) - 1)));
#pragma unroll
  for (int r = 1; r < 8; r++) {
    const uint4 w = __ldg(t + ((r - 1) << LOGNS));
    v[r] = tw_mul(v[r], fe_make(words64(w.x, w.y), words64(w.z, w.w)));
  }
}

// The stages between the first and the last, in place in shared memory:
//   v[r] = x[j + r S/8] omega_{8 Ns}^{r (j mod Ns)}, DFT_8(v),
//   x'[(j / Ns) 8 Ns + (j mod Ns) + r Ns] = v[r].
template <bool INV, int LOGS, int LOGNS>
__device__ __forceinline__ void middle_stages(fe *sm, const fe *stages, int logB, uint32_t nb, uint32_t u) {
  if constexpr (LOGNS + 3 < LOGS) {
    const uint32_t b = u >> (LOGS - 3), j = u & ((1u << (LOGS - 3)) - 1), xb = bank_shift(b, logB);
    fe v[8];
    if (u < nb) {
      const uint32_t s0 = slot<LOGS>(b, xb, j);
#pragma unroll
      for (int r = 0; r < 8; r++) v[r] = sm[slot_step<LOGS - 3>(s0, r)];
      twiddle_inputs<LOGNS>(v, stages, j);
      dft8<INV, true>(v);
    }
    group_sync<LOGS>();
    if (u < nb) {
      const uint32_t s0 = slot<LOGS>(b, xb, ((j >> LOGNS) << (LOGNS + 3)) + (j & ((1u << LOGNS) - 1)));
#pragma unroll
      for (int r = 0; r < 8; r++) sm[slot_step<LOGNS>(s0, r)] = v[r];
    }
    if constexpr (LOGNS + 6 < LOGS) group_sync<LOGS>();  // the caller waits before the last stage
    middle_stages<INV, LOGS, LOGNS + 3>(sm, stages, logB, nb, u);
  }
}

// A 16-byte copy from global to shared memory, waited for by copies_wait.
__device__ __forceinline__ void copy_async(fe *dst, const fe *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// Staged data is read once: it should not displace the twiddles in L1.
__device__ __forceinline__ fe load_once(const fe *p) {
  fe x;
  asm volatile("ld.global.L1::no_allocate.v2.u64 {%0, %1}, [%2];" : "=l"(x.re), "=l"(x.im) : "l"(p));
  return x;
}

// Writes one output group: values v[q] at positions k + q dk of column l,
// times the outer twiddle and the scale where the pass has them (SCATTER: at
// the places of a scattered output, hoff the block's offset in the row).
template <int N, bool SCATTER>
__device__ __forceinline__ void emit(const PassArgs &a, fe *out, uint64_t hoff, const fe *tw_full, uint64_t l,
                                     uint32_t k, uint32_t dk, const fe *v) {
  const uint64_t base = l * a.out_gstride + (uint64_t)k * a.out_kstride, step = (uint64_t)dk * a.out_kstride;
#pragma unroll
  for (int q = 0; q < N; q++) {
    fe x = v[q];
    const uint64_t addr = base + q * step;
    if (tw_full) {
      x = fmul(x, tw_full[addr]);
    } else if (a.tw_lo) {
      const uint64_t ex = l * (k + q * dk) << a.tw_shift;
      x = fmul(x, fmul(a.tw_lo[ex & ((1u << kTwLoBits) - 1)], a.tw_hi[ex >> kTwLoBits]));
    }
    if (a.has_scale) x = fmul(x, a.scale);
    else if (!a.tw_lo && !tw_full) x = canon_fe(x);
    if (SCATTER) {
      const uint64_t i = addr + hoff;
      out[((i >> a.sc_lo) & ((1u << a.sc_n) - 1)) * a.sc_stride + ((i >> (a.sc_lo + a.sc_n)) << a.sc_lo) +
          (i & ((1ull << a.sc_lo) - 1))] = x;
    } else if (!a.acc) out[addr] = x;
    else if (addr < a.acc_n) out[addr] = fadd(out[addr], x);
  }
}

// One pass: a CTA takes tiles of B = 2^logB sub-transforms of length S, E =
// S B elements, with E/8 threads.  The first stage runs on the values as
// they arrive from global memory, the last one ends in registers and stores
// them: a tile crosses shared memory once less than it has stages.  What
// bounds it: the integer pipes and the register file's read ports (a
// radix-8 stage alone takes 115 cycles an element on a full SM, 64 of them
// the FMA pipe's for the wide products); small CTAs (64 to 256 threads, 1024
// threads an SM at 64 registers) keep other tiles computing while one waits
// for memory or a barrier.  A pass of 2^8 over 2^24 elements takes 183 us,
// 0.8 of the sum of its stages alone.
// MODE: a plain pass, the first pass of a packed real transform, or the last
// pass of one with a scattered output.
enum { PASS_PLAIN, PASS_PACKED, PASS_SCATTER };
template <int LOGS, bool INV, int MODE>
__global__ void __launch_bounds__(kMaxThreads, 1) ntt_pass_kernel(const PassArgs a) {
  pdl_wait();
  if (a.run_if && *a.run_if == 0) return;  // uniform over the grid
  extern __shared__ fe smem[];
  constexpr bool PACK = MODE == PASS_PACKED, SCATTER = MODE == PASS_SCATTER;
  constexpr int LOGR = first_log(LOGS), R = 1 << LOGR, PER = kPerThread / R, LOGJ = LOGS - LOGR;
  constexpr uint32_t S = 1u << LOGS;
  const int logB = a.logB;
  const uint32_t total = S << logB;
  fe *sm = smem;
  const bool in_rows = a.in_jstride == 1, out_rows = a.out_kstride == 1 || logB == 0;
  const uint32_t tid = threadIdx.x;
  const uint64_t g0 = (uint64_t)blockIdx.x << logB;
  const uint64_t l0 = g0 & ((1ull << a.logG) - 1), h = g0 >> a.logG;
  const fe *in = a.in + blockIdx.y * a.row_in + h * a.in_hstride;
  const uint64_t hoff = h * a.out_hstride;
  fe *out = a.out + blockIdx.y * a.row_out + (SCATTER ? 0 : hoff);
  const fe *tw_full = a.tw_full ? a.tw_full + h * a.tw_hstride : nullptr;
  fe v[PER][R];
  // first stage: v[r] = x[j + r S/R]
  if (a.sp_l > 0) {
    // Sparse rows: row k2 of the intermediate holds, in column n1, the sum
    // over the entries q = n1 (mod row length) of c * omega_L^{q k2}: the
    // first pass's column transform of a few nonzeros times its outer
    // twiddle, formed directly, so the first pass and its intermediate
    // array are skipped.  One thread per (first entry of a column, row).
    for (uint32_t e = threadIdx.x; e < total; e += blockDim.x) sm[e] = fe_zero();
    __syncthreads();
    const uint32_t l = (uint32_t)a.sp_l;
    for (uint32_t t = threadIdx.x; t < (l << logB); t += blockDim.x) {
      const uint32_t i = t % l, b = t / l;
      if (!a.sp_lead[i]) continue;
      const uint64_t k2 = g0 + b;
      fe x = fe_zero();
      int u = (int)i;
      for (uint32_t it = 0; it < l && u >= 0; it++, u = a.sp_next[u]) {
        const uint64_t q = (uint64_t)((uint32_t)a.sp_q[u] >> a.sp_shift);
        const uint64_t ex = (q * k2) & a.sp_mask;
        x = fadd(x, fmul(a.sp_c[u], fmul(a.sp_lo[ex & ((1u << kTwLoBits) - 1)], a.sp_hi[ex >> kTwLoBits])));
      }
      sm[(b << LOGS) + (((uint32_t)a.sp_q[i] >> a.sp_shift) & (S - 1))] = x;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; i++) {
      const uint32_t u = tid + i * blockDim.x;
#pragma unroll
      for (int r = 0; r < R; r++) {
        const uint32_t e = (u >> LOGJ << LOGS) + (u & ((1u << LOGJ) - 1)) + ((uint32_t)r << LOGJ);
        v[i][r] = e < total ? sm[e] : fe_zero();
      }
    }
    __syncthreads();
  } else {
    uint64_t nonreal = 0;
#pragma unroll
    for (int i = 0; i < PER; i++) {  // all loads first: PER * R = 8 in flight
      const uint32_t u = tid + i * blockDim.x;
      const uint32_t b = in_rows ? u >> LOGJ : u & ((1u << logB) - 1);
      const uint32_t j = in_rows ? u & ((1u << LOGJ) - 1) : u >> logB;
      const uint64_t base = (l0 + b) * a.in_gstride + (uint64_t)j * a.in_jstride;
      const uint64_t step = a.in_jstride << LOGJ;
      if (u >= (total >> LOGR)) {
#pragma unroll
        for (int r = 0; r < R; r++) v[i][r] = fe_zero();
      } else if (a.dense) {
        const fe *p = in + (PACK ? 2 * base : base);
#pragma unroll
        for (int r = 0; r < R; r++) {
          if (!PACK) {
            v[i][r] = load_once(p + r * step);
          } else {
            const fe e0 = load_once(p + 2 * r * step), e1 = load_once(p + 2 * r * step + 1);
            nonreal |= e0.im | e1.im;
            v[i][r] = fe_make(e0.re, e1.re);
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; r++) {
          const uint64_t addr = base + r * step;
          const bool ok = addr < a.n_valid && j + ((uint32_t)r << LOGJ) < a.j_valid;
          if (!PACK) {
            v[i][r] = ok ? in[addr] : fe_zero();
          } else {
            const fe e0 = ok ? in[2 * addr] : fe_zero(), e1 = ok ? in[2 * addr + 1] : fe_zero();
            nonreal |= e0.im | e1.im;
            v[i][r] = fe_make(e0.re, e1.re);
          }
        }
      }
    }
    if (PACK && nonreal) atomicOr(a.nonreal, 1u);
  }
#pragma unroll
  for (int i = 0; i < PER; i++) {
    if (R == 8) dft8<INV, false>(v[i]);
    else if (R == 4) dft4<INV>(v[i]);
    else if (R == 2) dft2<INV>(v[i]);
  }
  const bool in_order = in_rows || a.sp_l > 0;
  if constexpr (LOGS <= 3) {  // the first stage is the last
    if constexpr (LOGS == 3 && MODE == PASS_PLAIN) {
      // A batch's outputs lie back to back: by way of shared memory neighbouring
      // threads store neighbouring elements instead of a line each (block sums of
      // 2^24 entries in pairs, extended fourfold: 2660 -> 2148 us).
      if (in_order && a.out_kstride == 1 && a.out_gstride == S && !a.acc && !a.tw_lo && !tw_full) {
        if (tid < (total >> 3)) {
#pragma unroll
          for (int r = 0; r < 8; r++) {
            const fe x = v[0][r];
            sm[(tid << 3) + (r ^ (tid & 7))] = a.has_scale ? fmul(x, a.scale) : canon_fe(x);
          }
        }
        __syncthreads();
        for (uint32_t e = tid; e < total; e += blockDim.x) out[l0 * S + e] = sm[(e & ~7u) + ((e ^ (e >> 3)) & 7)];
        return;
      }
    }
#pragma unroll
    for (int i = 0; i < PER; i++) {
      const uint32_t u = tid + i * blockDim.x;
      const uint32_t b = in_order ? u >> LOGJ : u & ((1u << logB) - 1);
      if (u < (total >> LOGR)) emit<R, SCATTER>(a, out, hoff, tw_full, l0 + b, 0, 1, v[i]);
    }
  } else {
#pragma unroll
    for (int i = 0; i < PER; i++) {  // x'[R j + r]
      const uint32_t u = tid + i * blockDim.x;
      const uint32_t b = in_order ? u >> LOGJ : u & ((1u << logB) - 1);
      const uint32_t j = in_order ? u & ((1u << LOGJ) - 1) : u >> logB;
      const uint32_t s0 = slot<LOGS>(b, bank_shift(b, logB), j << LOGR);
      if (u < (total >> LOGR)) {
#pragma unroll
        for (int r = 0; r < R; r++) sm[slot_step<0>(s0, r)] = v[i][r];
      }
    }
    __syncthreads();
    const uint32_t nb = total >> 3;
    middle_stages<INV, LOGS, LOGR>(sm, a.stages, logB, nb, tid);
    if (LOGR + 3 < LOGS) {
      if (out_rows) group_sync<LOGS>();
      else __syncthreads();
    }
    // last stage (Ns = S/8): outputs k = j + r S/8 leave from registers.
    // Columns stored side by side are taken by neighbouring threads.
    const uint32_t u = tid;
    const uint32_t b = out_rows ? u >> (LOGS - 3) : u & ((1u << logB) - 1);
    const uint32_t j = out_rows ? u & (S / 8 - 1) : u >> logB;
    const uint32_t s0 = slot<LOGS>(b, bank_shift(b, logB), j);
    fe w[8];
    if (u < nb) {
#pragma unroll
      for (int r = 0; r < 8; r++) w[r] = sm[slot_step<LOGS - 3>(s0, r)];
      const uint64_t base = (l0 + b) * a.out_gstride + (uint64_t)j * a.out_kstride;
      const uint64_t step = a.out_kstride * (S / 8);
      const bool staged_tw = !SCATTER && tw_full && !a.has_scale && !a.acc;
      twiddle_inputs<LOGS - 3>(w, a.stages, j);
      if (staged_tw) {
        // The outer twiddles arrive during the butterfly, in the slots that
        // this thread alone has read.  Those reads have returned: w[1..7]
        // went through the products, and the first address waits for w[0]
        // (below 2^62, so its top bit adds nothing).
        copy_async(sm + s0, tw_full + base + (w[0].re >> 63));
#pragma unroll
        for (int r = 1; r < 8; r++) copy_async(sm + slot_step<LOGS - 3>(s0, r), tw_full + base + r * step);
      }
      dft8<INV, true>(w);
      if (staged_tw) {
        copies_wait();
#pragma unroll
        for (int r = 0; r < 8; r++) out[base + r * step] = fmul(w[r], sm[slot_step<LOGS - 3>(s0, r)]);
      } else {
        emit<8, SCATTER>(a, out, hoff, tw_full, l0 + b, j, S / 8, w);
      }
    }
  }
}

// A launch of few short transforms is over before a pass kernel's 20 to 60 KB
// of unrolled butterflies have come in, each run through once: 8 to 12 us for
// transforms of 2^4 to 2^10.  Here a thread takes one radix-2 butterfly a
// level, in a loop of 2 KB that every length and both directions share, with
// the half table of omega_n in shared memory: half as much arithmetic again,
// which such a launch does not notice (2^6 to 2^10 by 4 cosets 10.4 -> 3.7 us,
// 2^8 to 2^15 by 128 13.3 -> 5.0, 2^10 to 2^16 by 64 14.8 -> 8.9; one
// transform of 2^11 gains nothing).
// stages: omega_{2^kSmallLog}^k of the direction, k < 2^(kSmallLog - 1).
__global__ void __launch_bounds__(1 << (kSmallLog - 1)) ntt_small_kernel(const PassArgs a) {
  pdl_wait();
  if (a.run_if && *a.run_if == 0) return;
  extern __shared__ fe smem[];
  const int logS = a.logS, logB = a.logB;
  const uint32_t half = 1u << (logS - 1), total = 2u << (logS - 1 + logB), tid = threadIdx.x;
  const uint32_t b = tid >> (logS - 1), j = tid & (half - 1);
  const uint64_t l = ((uint64_t)blockIdx.x << logB) + b;
  const fe *in = a.in + blockIdx.y * a.row_in;
  fe *out = a.out + blockIdx.y * a.row_out;
  fe *tw = smem, *buf[2] = {smem + half, smem + half + total};
  fe x[2];
#pragma unroll 1
  for (int r = 0; r < 2; r++) {
    const uint32_t jj = j + r * half;
    const uint64_t addr = l * a.in_gstride + (uint64_t)jj * a.in_jstride;
    const bool ok = addr < a.n_valid && jj < a.j_valid;
    fe v = fe_zero();
    if (a.pack_real) {
      if (ok) {
        const fe e0 = in[2 * addr], e1 = in[2 * addr + 1];
        if (e0.im | e1.im) atomicOr(a.nonreal, 1u);
        v = fe_make(e0.re, e1.re);
      }
    } else if (ok) {
      v = in[addr];
      if (a.in_lo) {
        const uint64_t ex = l * jj;
        fe w = a.in_lo[ex & ((1u << kTwLoBits) - 1)];
        if (ex >> kTwLoBits) w = fmul(w, a.in_hi[ex >> kTwLoBits]);
        v = fmul(v, w);
      }
    }
    if (r) x[1] = v;
    else x[0] = v;
  }
  for (uint32_t t = tid; t < half; t += blockDim.x) tw[t] = a.stages[t << (kSmallLog - logS)];
  fe y0 = fadd(x[0], x[1]), y1 = fsub(x[0], x[1]);
#pragma unroll 1
  for (int s = 1; s < logS; s++) {  // x'[(j / Ns) 2 Ns + j mod Ns (+ Ns)], Ns = 2^(s-1), then the next level
    fe *o = buf[s & 1] + (b << logS);
    const uint32_t low = j & ((1u << (s - 1)) - 1), at = ((j - low) << 1) + low;
    o[at] = y0;
    o[at + (1u << (s - 1))] = y1;
    __syncthreads();
    const fe u = o[j], t = fmul(o[j + half], tw[(j & ((1u << s) - 1)) << (logS - 1 - s)]);
    y0 = fadd(u, t);
    y1 = fsub(u, t);
  }
  if (a.has_scale) {
    y0 = fmul(y0, a.scale);
    y1 = fmul(y1, a.scale);
  }
  fe *o = out + l * a.out_gstride + j * a.out_kstride;
  *o = y0;
  o[half * a.out_kstride] = y1;
}

// ---- extension of evaluations to a larger subgroup --------------------------
// One transform of length S = 2^LOGS of a tile, from and to the registers of
// the threads that own it: thread (b, j) holds entries j + q S/8 of
// sub-transform b on both sides, the first stage's inputs and the last one's
// outputs alike.  Inputs canonical, outputs in [0, p + 7].
template <bool INV, int LOGS>
__device__ __forceinline__ void tile_transform(fe *w, fe *sm, const fe *stages, int logB, uint32_t nb, uint32_t u) {
  constexpr int LOGR = first_log(LOGS), R = 1 << LOGR, PER = 8 / R;
  const uint32_t b = u >> (LOGS - 3), j = u & ((1u << (LOGS - 3)) - 1), xb = bank_shift(b, logB);
#pragma unroll
  for (int i = 0; i < PER; i++) {  // butterfly j + i S/8
    fe x[R];
#pragma unroll
    for (int r = 0; r < R; r++) x[r] = w[i + PER * r];
    if constexpr (R == 8) dft8<INV, false>(x);
    else if constexpr (R == 4) dft4<INV>(x);
    else dft2<INV>(x);
    if constexpr (LOGS <= 3) {
#pragma unroll
      for (int r = 0; r < R; r++) w[r] = x[r];
    } else {
      const uint32_t s0 = slot<LOGS>(b, xb, (j + ((uint32_t)i << (LOGS - 3))) << LOGR);
#pragma unroll
      for (int r = 0; r < R; r++) sm[slot_step<0>(s0, r)] = x[r];
    }
  }
  if constexpr (LOGS > 3) {
    __syncthreads();
    middle_stages<INV, LOGS, LOGR>(sm, stages, logB, nb, u);
    if (LOGR + 3 < LOGS) __syncthreads();
    const uint32_t s0 = slot<LOGS>(b, xb, j);
#pragma unroll
    for (int r = 0; r < 8; r++) w[r] = sm[slot_step<LOGS - 3>(s0, r)];
    twiddle_inputs<LOGS - 3>(w, stages, j);
    dft8<INV, true>(w);
  }
}

// Blocks of S = 2^LOGS evaluations over the subgroup of order S, extended to
// the one of order S 2^EXT: its points w^(k 2^EXT) are the given ones, those of
// coset s are the transform of the coefficients times w^(s j).  One pass: the
// inverse transform ends in registers, where each forward one begins, and only
// the new evaluations are stored, coset s - 1 at out + (s - 1) total + the
// block's place.  (As an inverse and a forward transform of all points, 2^24
// entries in blocks of 128: 187 + 314 us, 805 and 805 MB; in this one 271 us, 537 MB.)
// factors: w^(s j) / S at (s - 1) S + j.
constexpr int kExtendThreads = 256, kExtendLog = 11;  // entries of a tile
template <int LOGS, int EXT>
__global__ void __launch_bounds__(kExtendThreads, EXT == 1 ? 4 : 3)
coset_extend_kernel(const fe *in, fe *out, uint64_t total, const fe *inv_stages, const fe *fwd_stages,
                    const fe *factors) {
  pdl_wait();
  __shared__ fe sm[1 << kExtendLog];
  constexpr uint32_t S = 1u << LOGS;
  constexpr int logB = kExtendLog - LOGS;
  const uint32_t u = threadIdx.x, j = u & (S / 8 - 1);
  const uint64_t at = ((uint64_t)blockIdx.x << kExtendLog) + ((u >> (LOGS - 3)) << LOGS) + j;
  fe c[8];
#pragma unroll
  for (int q = 0; q < 8; q++) c[q] = load_once(in + at + q * (S / 8));
  tile_transform<true, LOGS>(c, sm, inv_stages, logB, kExtendThreads, u);
#pragma unroll 1
  for (int s = 0; s + 1 < (1 << EXT); s++) {
    fe w[8];
#pragma unroll
    for (int q = 0; q < 8; q++) w[q] = fmul(c[q], factors[s * S + j + q * (S / 8)]);
    if (LOGS > 3) __syncthreads();  // the tile has been read
    tile_transform<false, LOGS>(w, sm, fwd_stages, logB, kExtendThreads, u);
#pragma unroll
    for (int q = 0; q < 8; q++) out[s * total + at + q * (S / 8)] = canon_fe(w[q]);
  }
}

__global__ void coset_extend_factors_kernel(fe *f, int logS, int ext, const fe *lo, fe scale) {
  pdl_wait();
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (((1u << ext) - 1) << logS)) return;
  f[t] = fmul(scale, lo[((t >> logS) + 1) * (t & ((1u << logS) - 1))]);  // below 2^12: one table
}

// Column chains of a sparse input: next[t] = the next entry with the same
// column ((q >> shift) & colmask), -1 at the end; lead[t] = 1 for the first
// entry of each column.  One thread per entry (l <= kMaxQueries).
__global__ void sparse_chain_kernel(const int32_t *q, int l, int shift, uint32_t colmask, int16_t *next,
                                    uint8_t *lead) {
  pdl_wait();
  __shared__ uint32_t col[kMaxQueries];
  const int t = threadIdx.x;
  if (t < l) col[t] = ((uint32_t)q[t] >> shift) & colmask;
  __syncthreads();
  if (t >= l) return;
  int nx = -1;
  uint8_t first = 1;
  for (int u = 0; u < l; u++) {
    if (col[u] != col[t]) continue;
    if (u < t) first = 0;
    else if (u > t && nx < 0) nx = u;
  }
  next[t] = (int16_t)nx;
  lead[t] = first;
}

typedef void (*PassKernel)(const PassArgs);
template <int LOGS>
PassKernel pass_kernel(bool inverse, int mode) {
  if (mode == PASS_PACKED) return ntt_pass_kernel<LOGS, false, PASS_PACKED>;
  if (mode == PASS_SCATTER) return ntt_pass_kernel<LOGS, false, PASS_SCATTER>;
  return inverse ? ntt_pass_kernel<LOGS, true, PASS_PLAIN> : ntt_pass_kernel<LOGS, false, PASS_PLAIN>;
}
PassKernel pass_kernel(int logS, bool inverse, int mode) {
  switch (logS) {
    case 0: return pass_kernel<0>(inverse, mode);
    case 1: return pass_kernel<1>(inverse, mode);
    case 2: return pass_kernel<2>(inverse, mode);
    case 3: return pass_kernel<3>(inverse, mode);
    case 4: return pass_kernel<4>(inverse, mode);
    case 5: return pass_kernel<5>(inverse, mode);
    case 6: return pass_kernel<6>(inverse, mode);
    case 7: return pass_kernel<7>(inverse, mode);
    case 8: return pass_kernel<8>(inverse, mode);
    case 9: return pass_kernel<9>(inverse, mode);
    case 10: return pass_kernel<10>(inverse, mode);
    case 11: return pass_kernel<11>(inverse, mode);
    case 12: return pass_kernel<12>(inverse, mode);
    default: return pass_kernel<13>(inverse, mode);
  }
}

// A device's tables that every length shares, per direction: the stage
// twiddles and the small kernel's half table.
struct DeviceTables {
  fe *stages[2] = {nullptr, nullptr}, *half[2] = {nullptr, nullptr};
};

void upload_table(fe **d, const std::vector<fe> &h) {
  GBZ_CUDA(device_malloc((void **)d, sizeof(fe) * h.size()));
  GBZ_CUDA(cudaMemcpy(*d, h.data(), sizeof(fe) * h.size(), cudaMemcpyHostToDevice));
}

DeviceTables device_tables_build() {
  DeviceTables t;
  try {
    std::vector<fe> h(stage_table_offset(kSubLog - 2)), half(1u << (kSmallLog - 1));
    for (int dir = 0; dir < 2; dir++) {
      for (int ns = 1; ns <= kSubLog - 3; ns++) {
        fe w = root_of_unity(ns + 3);
        if (dir) w = finv(w);
        fe wr = w;
        for (int r = 1; r < 8; r++, wr = fmul(wr, w)) {
          fe x = fe_one();
          for (uint32_t k = 0; k < (1u << ns); k++, x = fmul(x, wr)) h[stage_table_offset(ns) + ((r - 1) << ns) + k] = x;
        }
      }
      upload_table(&t.stages[dir], h);
      fe w = root_of_unity(kSmallLog), x = fe_one();
      if (dir) w = finv(w);
      for (size_t k = 0; k < half.size(); k++, x = fmul(x, w)) half[k] = x;
      upload_table(&t.half[dir], half);
    }
    // a copy from pageable memory may return before its last part has arrived
    GBZ_CUDA(cudaStreamSynchronize(cudaStreamLegacy));
    GBZ_CUDA(cudaFuncSetAttribute(ntt_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(sizeof(fe) * (5u << (kSmallLog - 1)))));
    for (int logS = 0; logS <= kSubLog; logS++)
      for (PassKernel k : {pass_kernel(logS, false, PASS_PLAIN), pass_kernel(logS, true, PASS_PLAIN),
                           pass_kernel(logS, false, PASS_PACKED), pass_kernel(logS, false, PASS_SCATTER)})
        GBZ_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(fe) * kCtaElems)));
  } catch (...) {
    for (int dir = 0; dir < 2; dir++) {
      cudaFree(t.stages[dir]);
      cudaFree(t.half[dir]);
    }
    throw;
  }
  return t;
}

// The current device's, built on first use and kept for the process.  A
// thread gets them when they are filled and the kernels' attributes are set;
// launches take the pointers from the NttTables of their own device.
DeviceTables device_tables() {
  static std::mutex mu;
  static std::map<int, DeviceTables> built;
  int dev = 0;
  GBZ_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  const auto it = built.find(dev);
  return it != built.end() ? it->second : built.emplace(dev, device_tables_build()).first->second;
}

// Launches of up to 2^kSmallTotal elements in sub-transforms of up to
// 2^kSmallLog take the small kernel, cosets up to 2^kCosetTotal (below).  The
// proofs and openings that were timed do not tell 2^13 from 2^17 for the
// first, nor 2^16 from 2^19 for the second.
constexpr int kSmallTotal = 16, kCosetTotal = 18;

bool small_launch(const PassArgs &a, uint64_t groups, int rows) {
  return a.in_lo || (a.logS >= 1 && a.logS <= kSmallLog && a.logG == 0 && !a.tw_lo && !a.tw_full && !a.sp_l &&
                     !a.acc && !a.sc_n &&
                     ((groups * (uint64_t)rows) << a.logS) <= (1ull << kSmallTotal));
}

// Launches with the tables of the transform's own device (t).
void launch_pass(const NttTables &t, PassArgs a, uint64_t groups, cudaStream_t s, int rows = 1) {
  if (rows < 1 || rows > 65535) throw ArgError("transform: 1..65535 rows per launch");
  if (small_launch(a, groups, rows)) {
    a.stages = a.inverse ? t.half_inv : t.half_fwd;
    // a warp of butterflies a CTA at least
    a.logB = std::min(std::max(0, 6 - a.logS), ilog2(groups & (~groups + 1)));
    const uint32_t threads = 1u << (a.logS - 1 + a.logB);
    launch_kernel(ntt_small_kernel, dim3((unsigned)(groups >> a.logB), (unsigned)rows), threads,
                  sizeof(fe) * 5 * threads, s, a);
    GBZ_CUDA(cudaGetLastError());
    return;
  }
  a.stages = a.inverse ? t.sub_inv : t.sub_fwd;
  const uint64_t tiles = groups >> a.logB;
  const uint32_t E = 1u << (a.logS + a.logB);
  const size_t smem = a.logS >= 3 || a.sp_l > 0 ? sizeof(fe) * E : 0;
  const unsigned threads = E / kPerThread > 32 ? E / kPerThread : 32;
  if (a.logG == 0) a.logG = 40;  // every g is a column of its own
  const uint64_t last = (groups - 1) * a.in_gstride + ((1ull << a.logS) - 1) * a.in_jstride;
  a.dense = a.j_valid >= (1u << a.logS) && (a.n_valid == ~0ull || last < a.n_valid);
  const int mode = a.pack_real ? PASS_PACKED : a.sc_n ? PASS_SCATTER : PASS_PLAIN;
  launch_kernel(pass_kernel(a.logS, a.inverse != 0, mode), dim3((unsigned)tiles, (unsigned)rows), threads, smem, s, a);
  GBZ_CUDA(cudaGetLastError());
}

}  // namespace

// Full outer-twiddle tables of the first pass, per (device, length, split,
// direction): T[n1 + N1 k2] = omega_L^{n1 k2}, so the pass multiplies once
// per element instead of forming the twiddle from the two-level table.
// The integer pipes bound the transform and HBM has room, so reading
// 16 B per element is the cheaper side of the trade.
std::mutex g_outer_mu;
std::map<std::tuple<int, int, int, int>, fe *> g_outer;
bool g_use_outer = true;  // gbz_ntt_full_twiddles

// T[n1 + N1 k] = w^(n1 k) for n1 < N1, k < N2: thread (n1, chunk) walks 64
// consecutive k from w^(n1 k0) by products with w^n1.
__global__ void outer_table_kernel(fe w, int logL, int k1, fe *T) {
  pdl_wait();
  const uint64_t N1 = 1ull << k1, N2 = 1ull << (logL - k1);
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t chunks = (N2 + 63) / 64;
  if (tid >= N1 * chunks) return;
  const uint64_t n1 = tid % N1, k0 = (tid / N1) * 64;
  const fe wn1 = fpow(w, n1);
  fe x = fpow(wn1, k0);
  for (uint64_t k = k0; k < k0 + 64 && k < N2; k++) {
    T[n1 + N1 * k] = x;
    x = fmul(x, wn1);
  }
}

// The schedules' tables have kScheduleTable added to the split.
constexpr int kScheduleTable = 64;

const fe *outer_table_get(int logn, int key_k1, bool inverse) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
  std::lock_guard<std::mutex> lk(g_outer_mu);
  auto it = g_outer.find(std::make_tuple(dev, logn, key_k1, inverse ? 1 : 0));
  return it == g_outer.end() ? nullptr : it->second;
}

void outer_table_build(int logn, int key_k1) {
  const int k1 = key_k1 & (kScheduleTable - 1);
  if (k1 < 1 || k1 >= logn) return;
  int dev = 0;
  GBZ_CUDA(cudaGetDevice(&dev));
  for (int dir = 0; dir < 2; dir++) {
    const auto key = std::make_tuple(dev, logn, key_k1, dir);
    {
      std::lock_guard<std::mutex> lk(g_outer_mu);
      if (g_outer.count(key)) continue;
    }
    const uint64_t L = 1ull << logn;
    fe *T = nullptr;
    if (device_malloc((void **)&T, sizeof(fe) * L) != cudaSuccess) {
      cudaGetLastError();  // no room: the pass keeps the two-level twiddles
      return;
    }
    fe w = root_of_unity(logn);
    if (dir) w = finv(w);
    const uint64_t threads = (1ull << k1) * (((L >> k1) + 63) / 64);
    launch_kernel(outer_table_kernel, (unsigned)((threads + 255) / 256), 256, 0, 0, w, logn, k1, T);
    GBZ_CUDA(cudaGetLastError());
    GBZ_CUDA(cudaDeviceSynchronize());
    std::lock_guard<std::mutex> lk(g_outer_mu);
    g_outer[key] = T;
  }
}

std::vector<int> outer_table_splits(int logn) {
  int dev = 0;
  GBZ_CUDA(cudaGetDevice(&dev));
  std::vector<int> out;
  std::lock_guard<std::mutex> lk(g_outer_mu);
  for (const auto &e : g_outer)
    if (std::get<0>(e.first) == dev && std::get<1>(e.first) == logn) out.push_back(std::get<2>(e.first));
  return out;
}

// After autotuning: the tables that it built for shapes it did not choose.
// Those that were there before stay, as captured proofs may read them.
void outer_table_keep_only(int logn, const std::vector<int> &splits) {
  int dev = 0;
  GBZ_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_outer_mu);
  for (auto it = g_outer.begin(); it != g_outer.end();) {
    if (std::get<0>(it->first) == dev && std::get<1>(it->first) == logn &&
        std::find(splits.begin(), splits.end(), std::get<2>(it->first)) == splits.end()) {
      GBZ_CUDA(cudaDeviceSynchronize());
      cudaFree(it->second);
      it = g_outer.erase(it);
    } else {
      ++it;
    }
  }
}

void ntt_use_full_twiddles(bool on) { g_use_outer = on; }

namespace {
// The passes of a transform whose shape nobody set: sub-transforms of 2^log[i]
// and 2^logB[i] of them a CTA, in order.
struct Schedule {
  int passes, log[3], logB[3];
};

// Cycles an element of a pass of length 2^log, as measured for its parts with
// every SM busy: a first stage of radix 2, 4 or 8, twiddled radix-8 stages,
// loads, stores and the outer product.  From 2^10 on the barriers of a
// sub-transform span several warps and cost more the longer it is (a pass of
// 2^8 reaches 0.8 of its arithmetic, one of 2^12 0.55).
double pass_cost(int log) {
  static const double first[4] = {0, 17, 23, 34};
  const double c = first[first_log(log)] + 115.0 * ((log - first_log(log)) / 3);
  return c * (log < 10 ? 1.0 : log == 10 ? 1.05 : log == 11 ? 1.1 : 1.35) + 125;
}

// Two or three passes by that cost: two up to 2^20 (2^20 as 9 + 11: 41 us,
// three passes 43), three above, where each further level would fall into
// passes of 2^11 and more (one transform, two passes of the old shapes ->
// three: 2^21 85 -> 74 us, 2^22 163 -> 142, 2^23 335 -> 280, 2^24 677 -> 541,
// 2^25 1594 -> 1121, 2^26 3908 -> 2223).  A pass of 2^6 goes last and the
// others in ascending order (2^22 as 8 + 8 + 6: 140 us, 6 + 8 + 8: 147).
// Equal costs: the longer shortest pass.  CTAs stage 2^11 elements (2^10 in
// three passes up to 2^22: 2^22 140 us, with 2^11 147), less where the rows
// of a launch are too short to give every SM one.
Schedule schedule(int logn, int rows = 1) {
  Schedule best{};
  double least = 1e30;
  for (int x = 5; x <= 12; x++)
    for (int y = x; y <= 12; y++) {
      if (x + y == logn && pass_cost(x) + pass_cost(y) <= least) {
        least = pass_cost(x) + pass_cost(y);
        best = Schedule{2, {x, y, 0}, {0, 0, 0}};
      }
      const int z = logn - x - y;
      if (z >= y && z <= 12 && pass_cost(x) + pass_cost(y) + pass_cost(z) <= least) {
        least = pass_cost(x) + pass_cost(y) + pass_cost(z);
        best = Schedule{3, {x, y, z}, {0, 0, 0}};
      }
    }
  int *l = best.log;
  if (l[0] == 6) std::rotate(l, l + 1, l + best.passes);
  if (best.passes == 3 && l[0] > l[1]) std::swap(l[0], l[1]);
  const int stage = std::min(best.passes == 3 && logn <= 22 ? 10 : 11, logn + ilog2((uint64_t)rows) - 8);
  int rest = logn;
  for (int i = 0; i < best.passes; i++) {
    rest -= l[i];
    const int cols = i + 1 < best.passes ? rest : l[0];  // neighbouring sub-transforms
    best.logB[i] = std::min(cols, std::max(stage - l[i], logn >= 18 ? 1 : 0));
  }
  return best;
}
}  // namespace

void ntt_tables_build(NttTables &t, int logn) {
  const DeviceTables dt = device_tables();
  t.logn = logn;
  t.sub_fwd = dt.stages[0];
  t.sub_inv = dt.stages[1];
  t.half_fwd = dt.half[0];
  t.half_inv = dt.half[1];
  t.inv_len = finv(fe_make(1ull << logn, 0));
  const uint64_t L = 1ull << logn;
  const int nlo = 1 << kTwLoBits;
  const uint64_t nhi = (L >> kTwLoBits) > 0 ? (L >> kTwLoBits) : 1;
  std::vector<fe> lo(nlo), hi(nhi);
  for (int dir = 0; dir < 2; dir++) {
    fe w = root_of_unity(logn);
    if (dir) w = finv(w);
    fe x = fe_one();
    for (int i = 0; i < nlo; i++) { lo[i] = x; x = fmul(x, w); }
    fe w12 = x;  // w^(2^12)
    x = fe_one();
    for (uint64_t i = 0; i < nhi; i++) { hi[i] = x; x = fmul(x, w12); }
    fe **plo = dir ? &t.lo_inv : &t.lo_fwd, **phi = dir ? &t.hi_inv : &t.hi_fwd;
    upload_table(plo, lo);
    upload_table(phi, hi);
  }
  GBZ_CUDA(cudaStreamSynchronize(cudaStreamLegacy));  // as for the device's tables
  if (logn > kSubLog) {
    if (g_shape[logn].k1 > 0) outer_table_build(logn, g_shape[logn].k1);
    const Schedule sc = schedule(logn);
    int rest = logn;
    for (int i = 0; i + 1 < sc.passes; i++) {
      outer_table_build(rest, (rest - sc.log[i]) + kScheduleTable);
      rest -= sc.log[i];
    }
  }
}

namespace {
// A transform of n <= 2^kCosetLog entries padded to L >= 8 n is L / n
// transforms of length n: X[k + (L/n) m] = DFT_n(x_j omega_L^{jk})[m], log n
// levels and a product instead of log L levels in one or two passes, and L / n
// or so CTAs where a whole transform in one CTA leaves the chip idle (2^4 to
// 2^13 28.3 us in one CTA, 3.5 in cosets; 2^8 to 2^15 15.6 us in two passes,
// 5.0).  Longer launches (above 2^kCosetTotal elements) keep the passes, which
// issue less.
bool coset_form(int logn, uint64_t n_valid, int rows) {
  return n_valid > 1 && n_valid <= (1u << kCosetLog) && logn >= 3 + ilog2(2 * n_valid - 1) &&
         ((uint64_t)rows << logn) <= (1ull << kCosetTotal);
}
}  // namespace

int ntt_launch_count(int logn, uint64_t n_valid, int rows) {
  if (coset_form(logn, n_valid, rows)) return 1;
  if (logn <= kSubLog) return 1;
  return g_shape[logn].k1 > 0 ? 2 : schedule(logn).passes;
}

namespace {
// The shape of a sparse transform (one second pass) whose length has none set.
NttShape sparse_shape(int logn) {
  NttShape sh;
  sh.k1 = (logn + 1) / 2;
  const int k2 = logn - sh.k1;
  // Strided pass: at least two neighbouring columns per CTA (whole 32-byte
  // sectors) and up to 2^13 staged elements, fewer when the transform is
  // small so that it still spreads over many CTAs.
  sh.logBA = std::min(sh.k1, std::max(k2 < kSubLog ? 1 : 0, std::min(kSubLog, logn - 8) - k2));
  sh.logBB = std::min(k2, std::max(0, std::min(kSubLog - 1, logn - 8) - sh.k1));
  return sh;
}
}  // namespace

bool ntt_shape_length(int logn) { return logn > kSubLog && logn <= kMaxNttLogN; }

bool ntt_shape_valid(int logn, const NttShape &sh) {
  if (!ntt_shape_length(logn)) return false;
  if (sh.k1 == -1) return true;
  const int k2 = logn - sh.k1;
  if (sh.k1 < 1 || sh.k1 > kSubLog || k2 < 1 || k2 > kSubLog) return false;
  if (sh.logBA < 0 || sh.logBA > sh.k1 || k2 + sh.logBA > kSubLog) return false;
  if (sh.logBB < 0 || sh.logBB > k2 || sh.k1 + sh.logBB > kSubLog) return false;
  return true;
}

NttShape ntt_get_shape(int logn) { return ntt_shape_length(logn) ? g_shape[logn] : NttShape{}; }

void ntt_set_shape(int logn, const NttShape &sh) {
  if (!ntt_shape_valid(logn, sh)) throw ArgError("ntt shape: invalid split or staging for this length");
  if (sh.k1 > 0) outer_table_build(logn, sh.k1);
  g_shape[logn] = sh.k1 > 0 ? sh : NttShape{};
}

std::vector<NttShape> ntt_shape_candidates(int logn) {
  std::vector<NttShape> out;
  for (int k1 = 1; k1 <= kSubLog; k1++) {
    const int k2 = logn - k1;
    if (k2 < 1 || k2 > kSubLog || std::abs(k1 - k2) > 2) continue;
    for (int a = 0; a <= std::min(k1, kSubLog - k2); a++)
      for (int b = 0; b <= std::min(k2, kSubLog - k1); b++) {
        NttShape sh{k1, a, b};
        if (a > 4 || b > 3) continue;
        if (ntt_shape_valid(logn, sh)) out.push_back(sh);
      }
  }
  return out;
}

void ntt_tables_free(NttTables &t) {
  cudaFree(t.lo_fwd);
  cudaFree(t.hi_fwd);
  cudaFree(t.lo_inv);
  cudaFree(t.hi_inv);
  t.lo_fwd = t.hi_fwd = t.lo_inv = t.hi_inv = nullptr;
  t.logn = -1;
}

namespace {

// Shared by the dense transform and the sparse/accumulating variant.
// Options of a transform: packed real input (the pass that reads `in`) and
// a device flag that gates every pass.
struct PassGate {
  int pack_real = 0;
  uint32_t *nonreal = nullptr;
  const uint32_t *run_if = nullptr;
  const fe *out_tab = nullptr;  // output k is multiplied by out_tab[k] (the inverse transform's scale included)
  int sc_lo = 0, sc_n = 0;      // scattered output (PassArgs)
  uint64_t sc_stride = 0;
};

void ntt_passes(const NttTables &t, const fe *in, uint64_t n_valid, fe *out, fe *tmp, bool inverse,
                  cudaStream_t s, int rows = 1, uint64_t row_in = 0, uint64_t row_out = 0,
                  const PassGate &gate = PassGate(), uint64_t out_elem_stride = 1) {
  const int logn = t.logn;
  const uint64_t L = 1ull << logn;
  if (logn > kMaxNttLogN) throw ArgError("transform longer than 2^26");
  if (gate.pack_real && (logn < 1 || rows != 1)) throw ArgError("packed real transform: one row, length >= 2");
  if (n_valid > L) n_valid = L;
  PassArgs a{};
  a.pack_real = gate.pack_real;
  a.nonreal = gate.nonreal;
  a.run_if = gate.run_if;
  a.row_in = row_in;
  a.row_out = row_out;
  a.scale = t.inv_len;
  a.inverse = inverse ? 1 : 0;
  a.j_valid = 1u << kSubLog;
  const int logv = n_valid ? ilog2(2 * n_valid - 1) : 0;  // 2^logv >= n_valid
  const fe *in_end = in + (uint64_t)(rows - 1) * row_in + n_valid;
  const fe *out_end = out + (uint64_t)(rows - 1) * row_out + ((L - 1) * out_elem_stride + 1);
  if (gate.out_tab && out_elem_stride != 1) throw ArgError("transform: output factors need unit stride");
  if (gate.sc_n && (inverse || out_elem_stride != 1 || gate.sc_lo + 2 * gate.sc_n != logn))
    throw ArgError("transform: scattered output");
  if (!gate.pack_real && !gate.out_tab && !gate.sc_n && coset_form(logn, n_valid, rows) &&
      (in_end <= out || out_end <= in)) {
    a.in = in;
    a.out = out;
    a.n_valid = n_valid;
    a.in_gstride = 0;
    a.in_jstride = 1;
    a.in_lo = inverse ? t.lo_inv : t.lo_fwd;
    a.in_hi = inverse ? t.hi_inv : t.hi_fwd;
    a.out_gstride = out_elem_stride;
    a.out_kstride = out_elem_stride << (logn - logv);
    a.logS = logv;
    a.has_scale = inverse;
    launch_pass(t, a, 1ull << (logn - logv), s, rows);
    return;
  }
  if (logn <= kSubLog) {
    a.in = in;
    a.out = out;
    a.n_valid = n_valid;
    a.in_gstride = L;
    a.in_jstride = 1;
    a.out_gstride = L;
    a.out_kstride = out_elem_stride;
    a.logS = logn;
    a.logB = 0;
    a.has_scale = inverse && !gate.out_tab;
    a.tw_lo = nullptr;
    a.tw_hi = nullptr;
    a.tw_full = gate.out_tab;
    a.sc_lo = gate.sc_lo;
    a.sc_n = gate.sc_n;
    a.sc_stride = gate.sc_stride;
    // Rows too short to fill a CTA of 2^11 elements share one, as neighbouring
    // sub-transforms, where that leaves enough CTAs for every SM; what is left
    // over of them goes row by row.  (The output factors and the scattered
    // output are addressed by row.)  A CTA for every row of 2^9, 65535 of them
    // from 2^5 entries, took 657 us, so 443.
    if (rows <= 65535 && !gate.out_tab && !gate.sc_n && !small_launch(a, 1, rows)) {
      int logB = std::max(0, 11 - logn);
      while (logB > 0 && (rows >> logB) < 608) logB--;
      const int full = rows >> logB << logB;
      if (logB > 0) {
        PassArgs b = a;
        b.in_gstride = row_in;
        b.out_gstride = row_out;
        b.row_in = b.row_out = 0;
        b.n_valid = ~0ull;
        b.j_valid = (uint32_t)n_valid;
        b.logB = logB;
        launch_pass(t, b, (uint64_t)full, s);
        if (full == rows) return;
        a.in += full * row_in;
        a.out += full * row_out;
        rows -= full;
      }
    }
    launch_pass(t, a, 1, s, rows);
    return;
  }
  Schedule sc;
  const bool set = g_shape[logn].k1 > 0;
  if (set) {
    const NttShape sh = g_shape[logn];
    sc = Schedule{2, {logn - sh.k1, sh.k1, 0}, {sh.logBA, sh.logBB, 0}};
  } else {
    sc = schedule(logn, rows);
  }
  // Pass i transforms the columns of what is left of the length, 2^rest: for
  // each of the 2^done blocks that earlier passes made, columns l < C = 2^rest
  // / S at stride C, times omega_{2^rest}^{l k}, in place.  The last pass
  // transforms contiguous rows; its outputs go to natural order.
  int done = 0, rest = logn;
  for (int i = 0; i + 1 < sc.passes; i++) {
    const int lc = rest - sc.log[i];
    const uint64_t C = 1ull << lc;
    PassArgs b = a;
    b.pack_real = i == 0 ? gate.pack_real : 0;  // only the first pass reads the input
    b.in = i == 0 ? in : tmp;
    b.row_in = i == 0 ? row_in : L;
    b.n_valid = i == 0 ? n_valid : ~0ull;
    b.out = tmp;
    b.row_out = L;  // the intermediate holds one full row per transform
    b.in_gstride = b.out_gstride = 1;
    b.in_hstride = b.out_hstride = 1ull << rest;
    b.in_jstride = b.out_kstride = C;
    b.logG = lc;
    b.logS = sc.log[i];
    b.logB = sc.logB[i];
    b.tw_lo = inverse ? t.lo_inv : t.lo_fwd;
    b.tw_hi = inverse ? t.hi_inv : t.hi_fwd;
    b.tw_shift = done;
    b.tw_full = g_use_outer ? outer_table_get(rest, lc + (set ? 0 : kScheduleTable), inverse) : nullptr;
    launch_pass(t, b, L >> sc.log[i], s, rows);
    done += sc.log[i];
    rest = lc;
  }
  // Row (k0, k1) of the last pass starts at k0 2^(logn - log0) + k1 2^rest and
  // its output k goes to k0 + 2^log0 k1 + 2^done k; neighbouring k0 are taken
  // together, so that a CTA's outputs lie side by side.
  PassArgs b = a;
  b.pack_real = 0;
  b.in = tmp;
  b.row_in = L;
  b.n_valid = ~0ull;
  b.out = out;
  b.row_out = row_out;
  b.logG = sc.log[0];
  b.in_gstride = 1ull << (logn - sc.log[0]);
  b.in_hstride = 1ull << rest;
  b.in_jstride = 1;
  b.out_gstride = out_elem_stride;
  b.out_hstride = out_elem_stride << sc.log[0];
  b.out_kstride = out_elem_stride << done;
  b.logS = rest;
  b.logB = sc.logB[sc.passes - 1];
  b.has_scale = inverse && !gate.out_tab;
  b.tw_full = gate.out_tab;
  b.tw_hstride = gate.out_tab ? b.out_hstride : 0;
  b.sc_lo = gate.sc_lo;
  b.sc_n = gate.sc_n;
  b.sc_stride = gate.sc_stride;
  launch_pass(t, b, L >> rest, s, rows);
}

}  // namespace

void ntt_launch(const NttTables &t, const fe *in, uint64_t n_valid, fe *out, fe *tmp, bool inverse,
                cudaStream_t s) {
  ntt_passes(t, in, n_valid, out, tmp, inverse, s);
}

namespace {
// x / 2 mod p for canonical x: 2 is invertible and x + p is even when x is odd.
__device__ __forceinline__ uint64_t half_p(uint64_t x) { return (x + ((x & 1) ? P : 0)) >> 1; }
__device__ __forceinline__ fe conj_fe(fe x) { return fe_make(x.re, x.im ? P - x.im : 0); }

// Real-input transform, last step.  Z = DFT_M(z), z_j = x_2j + i x_2j+1
// (M = N/2, omega_M = omega_N^2).  In F_{p^2} conjugation is the Frobenius
// x -> x^p and p = -1 mod N, so conj(omega_N) = omega_N^{-1}; for base-field
// x this gives E[k] = (Z[k] + conj Z[M-k]) / 2 = DFT_M(x_even)[k] and
// O[k] = (Z[k] - conj Z[M-k]) / 2i = DFT_M(x_odd)[k], then X[k] = E + w^k O,
// X[k+M] = E - w^k O (w = omega_N), and X[N-k] = conj X[k].  Thread t takes
// k = t and M - t (t = 0 and t = M/2 alone): 2 reads, 4 writes, 2 multiplies.
__global__ void real_unpack_kernel(const fe *__restrict__ Z, uint64_t M, const fe *lo, const fe *hi,
                                   fe *__restrict__ X) {
  pdl_wait();
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t > M / 2) return;
  const fe a = Z[t], b = Z[t == 0 ? 0 : M - t];
  const fe E = fe_make(half_p(addp(a.re, b.re)), half_p(subp(a.im, b.im)));
  const fe O = fe_make(half_p(addp(a.im, b.im)), half_p(subp(b.re, a.re)));
  const fe w = fmul(lo[t & ((1u << kTwLoBits) - 1)], hi[t >> kTwLoBits]);
  const fe wo = fmul(w, O);
  const fe xk = fadd(E, wo), xkm = fsub(E, wo);
  X[t] = xk;
  X[t + M] = xkm;
  if (t != 0 && t != M / 2) {
    X[M - t] = conj_fe(xkm);
    X[2 * M - t] = conj_fe(xk);
  }
}
}  // namespace

void ntt_launch_real(const NttTables &t_half, const NttTables &t_full, const fe *in, uint64_t n_valid, fe *out,
                     fe *tmp, uint32_t *nonreal, cudaStream_t s) {
  const int logn = t_full.logn;
  if (t_half.logn != logn - 1 || logn < 2) throw ArgError("real transform: tables of lengths N/2 and N, N >= 4");
  if (n_valid & 1) throw ArgError("real transform: even number of input entries");
  const uint64_t N = 1ull << logn, M = N / 2;
  fe *Z = tmp + M;  // tmp holds N entries: the half-length intermediate, then Z
  PassGate g;
  g.pack_real = 1;
  g.nonreal = nonreal;
  ntt_passes(t_half, in, n_valid / 2, Z, tmp, false, s, 1, 0, 0, g);
  const uint64_t threads = M / 2 + 1;
  launch_kernel(real_unpack_kernel, (unsigned)((threads + 255) / 256), 256, 0, s, Z, M, t_full.lo_fwd, t_full.hi_fwd,
                out);
  GBZ_CUDA(cudaGetLastError());
  // any imaginary word: the general transform replaces the result
  PassGate f;
  f.run_if = nonreal;
  ntt_passes(t_full, in, n_valid, out, tmp, false, s, 1, 0, 0, f);
}

int ntt_launch_real_count(int logn, uint64_t n_valid) {
  return ntt_launch_count(logn - 1) + 1 + ntt_launch_count(logn, n_valid);
}

void ntt_launch_rows(const NttTables &t, const fe *in, uint64_t n_valid, uint64_t in_stride, fe *out,
                     uint64_t out_stride, int rows, fe *tmp, bool inverse, cudaStream_t s, uint64_t out_elem_stride,
                     const fe *out_tab) {
  if (rows < 1) return;
  if (out_elem_stride < 1) throw ArgError("transform: output element stride >= 1");
  PassGate g;
  g.out_tab = out_tab;
  ntt_passes(t, in, n_valid, out, tmp, inverse, s, rows, in_stride, out_stride, g, out_elem_stride);
}

void ntt_launch_rows_scatter(const NttTables &t, const fe *in, uint64_t n_valid, uint64_t in_stride, fe *out,
                             uint64_t out_stride, int rows, fe *tmp, int log_parts, uint64_t part_stride,
                             cudaStream_t s) {
  if (rows < 1) return;
  PassGate g;
  g.sc_n = log_parts;
  g.sc_lo = t.logn - 2 * log_parts;
  g.sc_stride = part_stride;
  ntt_passes(t, in, n_valid, out, tmp, false, s, rows, in_stride, out_stride, g);
}

void ntt_batched(const NttTables &t, const fe *in, uint64_t in_stride, uint32_t j_valid, fe *out, uint64_t count,
                 bool inverse, cudaStream_t s) {
  const int logS = t.logn;
  if (logS > kSubLog) throw ArgError("batched transform longer than 2^13");
  if (!count) return;
  PassArgs a{};
  a.scale = t.inv_len;
  a.inverse = inverse ? 1 : 0;
  a.in = in;
  a.out = out;
  a.n_valid = ~0ull;
  a.j_valid = j_valid;
  a.in_gstride = in_stride;
  a.in_jstride = 1;
  a.out_gstride = 1ull << logS;
  a.out_kstride = 1;
  a.logS = logS;
  a.has_scale = inverse;
  // up to 2^12 staged elements per CTA, never more transforms than there are
  int logB = std::max(0, 12 - logS);
  while (logB > 0 && (1ull << logB) > count) logB--;
  a.logB = logB;
  const uint64_t B = 1ull << logB;
  const uint64_t full = count / B * B;
  if (full) launch_pass(t, a, full, s);
  if (full < count) {  // remaining transforms one per CTA
    PassArgs r = a;
    r.in = in + full * in_stride;
    r.out = out + (full << logS);
    r.logB = 0;
    launch_pass(t, r, count - full, s);
  }
}

bool coset_extend_fits(uint64_t total, int logS, int ext) {
  return logS >= 3 && logS <= 10 && (ext == 1 || ext == 2) && total && total % (1ull << kExtendLog) == 0;
}

void coset_extend_factors_launch(const NttTables &tS, const NttTables &tL, int ext, fe *f, cudaStream_t s) {
  const unsigned n = ((1u << ext) - 1) << tS.logn;
  launch_kernel(coset_extend_factors_kernel, (n + 255) / 256, 256, 0, s, f, tS.logn, ext, tL.lo_fwd, tS.inv_len);
  GBZ_CUDA(cudaGetLastError());
}

namespace {
template <int LOGS>
void extend_launch(const NttTables &t, const fe *in, uint64_t total, int ext, const fe *f, fe *out, cudaStream_t s) {
  auto k = ext == 1 ? coset_extend_kernel<LOGS, 1> : coset_extend_kernel<LOGS, 2>;
  launch_kernel(k, (unsigned)(total >> kExtendLog), kExtendThreads, 0, s, in, out, total, t.sub_inv, t.sub_fwd, f);
}
}  // namespace

void coset_extend_launch(const NttTables &tS, const fe *in, uint64_t total, int ext, const fe *factors, fe *out,
                         cudaStream_t s) {
  if (!coset_extend_fits(total, tS.logn, ext)) throw ArgError("extension: block or total length");
  switch (tS.logn) {
    case 3: extend_launch<3>(tS, in, total, ext, factors, out, s); break;
    case 4: extend_launch<4>(tS, in, total, ext, factors, out, s); break;
    case 5: extend_launch<5>(tS, in, total, ext, factors, out, s); break;
    case 6: extend_launch<6>(tS, in, total, ext, factors, out, s); break;
    case 7: extend_launch<7>(tS, in, total, ext, factors, out, s); break;
    case 8: extend_launch<8>(tS, in, total, ext, factors, out, s); break;
    case 9: extend_launch<9>(tS, in, total, ext, factors, out, s); break;
    default: extend_launch<10>(tS, in, total, ext, factors, out, s); break;
  }
  GBZ_CUDA(cudaGetLastError());
}

void ntt_batched_strided(const NttTables &t, const fe *in, uint64_t col_stride, uint32_t j_valid, fe *out,
                         uint64_t count, bool inverse, cudaStream_t s) {
  const int logS = t.logn;
  if (logS > kSubLog) throw ArgError("batched transform longer than 2^13");
  if (!count) return;
  PassArgs a{};
  a.scale = t.inv_len;
  a.inverse = inverse ? 1 : 0;
  a.in = in;
  a.out = out;
  a.n_valid = ~0ull;
  a.j_valid = j_valid;
  a.in_gstride = 1;            // transform g starts at in[g]
  a.in_jstride = col_stride;   // its entry j at in[g + j * col_stride]
  a.out_gstride = 1ull << logS;
  a.out_kstride = 1;
  a.logS = logS;
  a.has_scale = inverse;
  // neighbouring transforms share 32-byte sectors: stage at least two per CTA
  int logB = std::max(0, 12 - logS);
  while (logB > 0 && (1ull << logB) > count) logB--;
  a.logB = logB;
  const uint64_t B = 1ull << logB;
  const uint64_t full = count / B * B;
  if (full) launch_pass(t, a, full, s);
  if (full < count) {
    PassArgs r = a;
    r.in = in + full;
    r.out = out + (full << logS);
    r.logB = 0;
    launch_pass(t, r, count - full, s);
  }
}

void ntt_sparse_accumulate(const NttTables &t, const int32_t *q, const fe *c, int l, fe *acc, uint64_t nacc,
                           fe *tmp, cudaStream_t s, int q_shift) {
  if (t.logn <= kSubLog) throw ArgError("sparse transform needs a two-pass length");
  if (q_shift < 0 || q_shift > 8) throw ArgError("sparse transform: position shift out of range");
  if (l < 1 || l > kMaxQueries) throw ArgError("sparse transform: 1..256 entries");
  const int logn = t.logn;
  const uint64_t L = 1ull << logn;
  const NttShape sh = g_shape[logn].k1 > 0 ? g_shape[logn] : sparse_shape(logn);
  const int k1 = sh.k1, k2 = logn - k1;
  const uint64_t N1 = 1ull << k1, N2 = 1ull << k2;
  // column chains in the (otherwise unused) scratch
  int16_t *next = reinterpret_cast<int16_t *>(tmp);
  uint8_t *lead = reinterpret_cast<uint8_t *>(next + kMaxQueries);
  launch_kernel(sparse_chain_kernel, 1, kMaxQueries, 0, s, q, l, q_shift, (uint32_t)(N1 - 1), next, lead);
  GBZ_CUDA(cudaGetLastError());
  PassArgs b{};
  b.scale = t.inv_len;
  b.inverse = 0;
  b.j_valid = 1u << kSubLog;
  b.in = nullptr;
  b.out = acc;
  b.n_valid = L;
  b.in_gstride = N1;
  b.in_jstride = 1;
  b.out_gstride = 1;
  b.out_kstride = N2;
  b.logS = k1;
  b.logB = sh.logBB;
  b.has_scale = 0;
  b.acc = 1;
  b.acc_n = nacc;
  b.sp_q = q;
  b.sp_c = c;
  b.sp_l = l;
  b.sp_shift = q_shift;
  b.sp_next = next;
  b.sp_lead = lead;
  b.sp_lo = t.lo_fwd;
  b.sp_hi = t.hi_fwd;
  b.sp_mask = L - 1;
  launch_pass(t, b, N2, s);
}

}  // namespace gbz
