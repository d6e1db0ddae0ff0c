// The plain single-party prover on one GPU.
//
// One proof = the reference's call sequence
//   Whir_Commit_initial (Whir.cpp:158-190)          -> root
//   hash_to_field({0}) x log n (main.cpp:83-85)      -> evaluation point z
//   quadratic sumcheck of sum_x w(x) eq(z, x) with Fiat-Shamir challenges
//     (round body of _quadratic_cosumcheck, coSumcheck_MPI.cpp:195-219)
//   Whir_Open of the resulting claim, whir_k = 4 (Whir.cpp:388-467)
// and its transcript is the ordered record stream documented in
// include/gbz.h.  Everything, including the Fiat-Shamir chain and the glibc
// random() draws that the reference uses for WHIR challenges and queries,
// runs on the device: a proof is a fixed sequence of launches on one
// stream with no host synchronisation, so it can be replayed from a CUDA
// graph and overlapped with other proofs on other streams.
#include <math.h>

#include <cstring>
#include <memory>
#include <mutex>

#include "gbz_prover.cuh"

namespace gbz {

namespace {

// ------------------------------------------------------------ kernels


// The generator of a proof (a batch: one CTA per proof).
__global__ void __launch_bounds__(32) k_init(ProofState *st, uint32_t seed, int seed_in_state) {
  pdl_wait();
  st += blockIdx.x;
  prng_warp_seed(st->prng, seed_in_state ? st->seed_in : seed, threadIdx.x);
}
__global__ void k_init_open(ProofState *st, glibc_prng g, const fe *point, int logn, fe K) {
  pdl_wait();
  if (threadIdx.x == 0) {
    st->fs = fe_zero();
    st->prng = g;
    st->y = fe_zero();
    st->K = K;
    st->error = 0;
  }
  for (int i = threadIdx.x; i < logn; i += blockDim.x) st->chal[i] = point[i];
}

// z_i = hash_to_field({0}) for i < logn.
// The start of a proof's protocol state and its evaluation point.
__global__ void k_point(ProofState *st, int logn, uint8_t *tr, uint64_t off, uint64_t trs) {
  pdl_wait();
  st += blockIdx.x;
  tr += trs * blockIdx.x;
  if (threadIdx.x) return;
  st->y = fe_zero();
  st->K = fe_zero();
  st->error = 0;
  fe s = fe_zero();
#pragma unroll 1
  for (int i = 0; i < logn; i++) {
    s = hash_F(s, fe_zero());
    st->z[i] = s;
    put_fe(tr, off + 16 * i, s);
  }
  st->fs = s;
}

__device__ void sum_partials(const fe *partial, int blocks, fe out[3]) {
  __shared__ fe red[3][32];
  fe A = fe_zero(), C = fe_zero(), D = fe_zero();
  for (int i = threadIdx.x; i < blocks; i += blockDim.x) {
    A = fadd(A, partial[3 * i]);
    C = fadd(C, partial[3 * i + 1]);
    D = fadd(D, partial[3 * i + 2]);
  }
  for (int d = 16; d > 0; d >>= 1) {
    fe t;
    t.re = __shfl_down_sync(0xffffffffu, A.re, d); t.im = __shfl_down_sync(0xffffffffu, A.im, d); A = fadd(A, t);
    t.re = __shfl_down_sync(0xffffffffu, C.re, d); t.im = __shfl_down_sync(0xffffffffu, C.im, d); C = fadd(C, t);
    t.re = __shfl_down_sync(0xffffffffu, D.re, d); t.im = __shfl_down_sync(0xffffffffu, D.im, d); D = fadd(D, t);
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { red[0][w] = A; red[1][w] = C; red[2][w] = D; }
  __syncthreads();
  if (threadIdx.x == 0) {
    A = C = D = fe_zero();
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) {
      A = fadd(A, red[0][k]);
      C = fadd(C, red[1][k]);
      D = fadd(D, red[2][k]);
    }
    out[0] = A;
    out[1] = fsub(fsub(D, A), C);
    out[2] = C;
  }
}

// Batched plans: codewords of 2^kBatchRealLog entries or more are committed
// proof by proof with the real-input transform, shorter ones in one batched
// general transform.
constexpr int kBatchRealLog = 18;

// The Fiat-Shamir state of the sumcheck of sum w(x) eq(z, x): the hash chain,
// the running claim, prod_{k < i} eq1(z_k, chal_k) and the verdict.
struct ScChain {
  fe fs, y, ep;
  uint32_t bad;
};

// Round i of that sumcheck from S(0), S(1):
// H(X) = epre * eq1(z_i, X) * (S0 + X (S1 - S0)) (the reference's round
// message of the pairs of w and the folded eq vector); claim check (the first
// round records it); the challenge hash_to_field({H.a, H.b, H.c}); y = H(c);
// and epre *= eq1(z_i, c).  Payload of the message at off_poly, the challenge
// 56 bytes after it.
__device__ __forceinline__ fe sc_round_eq(ScChain &v, fe S0, fe S1, fe z, fe *chal, uint8_t *tr, int64_t off_claim,
                                          uint64_t off_poly) {
  const fe a1 = fsub(fadd(z, z), fe_one()), b1 = fsub(fe_one(), z), d = fsub(S1, S0);
  const fe A = fmul(v.ep, a1), B = fmul(v.ep, b1);
  const fe h0 = fmul(A, d), h1 = fadd(fmul(A, S0), fmul(B, d)), h2 = fmul(B, S0);
  const fe h01 = fadd(h2, fadd(fadd(h0, h1), h2));  // H(0) + H(1)
  if (off_claim >= 0) put_fe(tr, (uint64_t)off_claim, h01);
  else if (!fe_eq(h01, v.y)) v.bad = 1;
  put_fe(tr, off_poly, h0);
  put_fe(tr, off_poly + 16, h1);
  put_fe(tr, off_poly + 32, h2);
  fe s = v.fs;
#pragma unroll 1
  for (int k = 0; k < 3; k++) s = hash_F(s, k == 0 ? h0 : k == 1 ? h1 : h2);
  v.fs = s;
  *chal = s;
  put_fe(tr, off_poly + 56, s);
  v.y = fadd(fmul(fadd(fmul(h0, s), h1), s), h2);
  v.ep = fadd(fmul(A, s), B);
  return s;
}

__device__ __forceinline__ fe shfl_xor_fe(fe x, int d) {
  return fe_make(__shfl_xor_sync(0xffffffffu, x.re, d), __shfl_xor_sync(0xffffffffu, x.im, d));
}

// Rounds i and i + 1 from the T sums of a pass (gbz_sumcheck.cu): the sum of
// the partials, then thread 0 alone through both rounds' hash chains (3.4 us
// of the 5 a launch takes).
__global__ void __launch_bounds__(256)
k_sc_rounds_eq(const fe *partial, int blocks, ProofState *st, int round, uint8_t *tr, int64_t off_claim,
               uint64_t off_poly, uint64_t ps, uint64_t trs) {
  pdl_wait();
  __shared__ fe red[8][4];
  partial = badv(partial, ps, blockIdx.x);
  st += blockIdx.x;
  tr += trs * blockIdx.x;
  const fe z0 = st->z[round], z1 = st->z[round + 1];
  ScChain v{st->fs, st->y, round ? st->epre : fe_one(), 0};
  fe x = fe_zero();
  for (int i = threadIdx.x; i < 4 * blocks; i += 256) x = fadd(x, partial[i]);
  for (int d = 4; d < 32; d *= 2) x = fadd(x, shfl_xor_fe(x, d));
  if ((threadIdx.x & 31) < 4) red[threadIdx.x >> 5][threadIdx.x & 3] = x;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  x = red[threadIdx.x >> 2][threadIdx.x & 3];
  for (int d = 4; d < 32; d *= 2) x = fadd(x, shfl_xor_fe(x, d));
  if (threadIdx.x < 4) red[0][threadIdx.x] = x;
  __syncwarp();
  if (threadIdx.x) return;
  const fe T0 = red[0][0], T1 = red[0][1], T2 = red[0][2], T3 = red[0][3];
  const fe c = sc_round_eq(v, fadd(T0, fmul(z1, fsub(T2, T0))), fadd(T1, fmul(z1, fsub(T3, T1))), z0,
                           &st->chal[round], tr, off_claim, off_poly);
  (void)sc_round_eq(v, fadd(T0, fmul(c, fsub(T1, T0))), fadd(T2, fmul(c, fsub(T3, T2))), z1, &st->chal[round + 1],
                    tr, -1, off_poly + 80);
  st->fs = v.fs;
  st->y = v.y;
  st->epre = v.ep;
  if (v.bad) atomicOr(&st->error, 1u);
}

// The last rounds of the same sumcheck in one CTA, from w of m <= kScTailMax
// entries and its table E (m / 4) on, then the final fold and the SC_FINAL
// record.  The hash chain of a round is serial (1.7 us); everything else runs
// beside it: with the T sums of w_r in hand, thread 0 knows round r + 1's
// message as soon as it has challenge r, and while it hashes it the workers
// fold w by challenge r and form the next T sums.  (The fold, the sums and
// the reductions in turn with the hashes took 7 us a round, 63 us for 2^10.)
// The workers are the warps outside the first one's quarter of the SM, whose
// issue slots the compressions fill.  Round r's SC_POLY payload is at
// off_poly0 + 80 (r - round0), its SC_CHALLENGE 56 bytes after it.
constexpr int kScTailMax = 4096;
constexpr int kScTailThreads = 1024, kScTailWorkers = kScTailThreads / 4 * 3;
constexpr size_t kScTailShared = sizeof(fe) * (kScTailMax / 2 + kScTailMax / 4 + kScTailMax / 8 + kScTailMax / 16);
__global__ void __launch_bounds__(kScTailThreads)
k_sc_tail(ProofState *st, const fe *a, const fe *E, int m, int round0, int logn, uint8_t *tr, int64_t off_claim,
          uint64_t off_poly0, uint64_t off_final, BStr bs) {
  pdl_wait();
  extern __shared__ fe tail_sm[];
  __shared__ fe red[kScTailWorkers / 32][4], T[2][4], zs[64], chal[2];
  // a batch: one CTA per proof; bs = strides of (a, E, tr)
  st += blockIdx.x;
  a = badv(a, bs.s[0], blockIdx.x);
  E = badv(E, bs.s[1], blockIdx.x);
  tr = badv(tr, bs.s[2], blockIdx.x);
  fe *w[2] = {tail_sm, tail_sm + kScTailMax / 2};
  fe *e[2] = {tail_sm + kScTailMax / 2 + kScTailMax / 4, tail_sm + kScTailMax / 2 + kScTailMax / 4 + kScTailMax / 8};
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool worker = (warp & 3) != 0;
  const int wid = (warp >> 2) * 3 + (warp & 3) - 1;  // worker warp
  const int t = wid * 32 + lane;
  // T sums from the workers' accumulators (a thread's entries all have the
  // same index mod 4)
  auto sum_classes = [&](const facc &acc, fe *out) {
    fe x = facc_value(acc);
    for (int d = 4; d < 32; d *= 2) x = fadd(x, shfl_xor_fe(x, d));
    if (lane < 4) red[wid][lane] = x;
    asm volatile("bar.sync 1, %0;" ::"n"(kScTailWorkers) : "memory");
    if (wid) return;
    x = fe_zero();
    for (int k = lane >> 2; k < kScTailWorkers / 32; k += 8) x = fadd(x, red[k][lane & 3]);
    for (int d = 4; d < 32; d *= 2) x = fadd(x, shfl_xor_fe(x, d));
    if (lane < 4) out[lane] = x;
  };
  ScChain v{};
  if (threadIdx.x < logn) zs[threadIdx.x] = st->z[threadIdx.x];
  if (threadIdx.x == 0) v = ScChain{st->fs, st->y, round0 ? st->epre : fe_one(), 0};
  if (worker) {
    facc acc = facc_zero();
    for (int x = t; x < m; x += kScTailWorkers) facc_mul(acc, a[x], E[x >> 2]);
    sum_classes(acc, T[round0 & 1]);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const fe *q = T[round0 & 1], z1 = zs[round0 + 1];
    chal[round0 & 1] = sc_round_eq(v, fadd(q[0], fmul(z1, fsub(q[2], q[0]))), fadd(q[1], fmul(z1, fsub(q[3], q[1]))),
                                   zs[round0], &st->chal[round0], tr, off_claim, off_poly0);
  }
  __syncthreads();
  int pp = 0;
#pragma unroll 1
  for (int r = round0; r < logn; r++) {  // w_r of m entries, its E and T, challenge r
    const fe c = chal[r & 1];
    fe *wn = w[pp], *en = e[pp];
    if (!worker) {
      if (threadIdx.x == 0 && r + 1 < logn) {
        const fe *q = T[r & 1];
        chal[(r + 1) & 1] = sc_round_eq(v, fadd(q[0], fmul(c, fsub(q[1], q[0]))), fadd(q[2], fmul(c, fsub(q[3], q[2]))),
                                        zs[r + 1], &st->chal[r + 1], tr, -1,
                                        off_poly0 + 80ull * (uint64_t)(r + 1 - round0));
      }
    } else {
      facc acc = facc_zero();
      for (int x = t; x < m / 2; x += kScTailWorkers) {
        const fe f = ffold(a[2 * x], a[2 * x + 1], c);
        wn[x] = f;
        if (m >= 8) {
          const fe ee = fadd(E[2 * (x >> 2)], E[2 * (x >> 2) + 1]);
          if ((x & 3) == 0) en[x >> 2] = ee;
          facc_mul(acc, f, ee);
        }
      }
      if (m >= 8) sum_classes(acc, T[(r + 1) & 1]);
    }
    a = wn;
    E = en;
    m /= 2;
    pp ^= 1;
    __syncthreads();
  }
  if (threadIdx.x == 0) {  // the folded w and the eq prefix
    put_fe(tr, off_final, a[0]);
    put_fe(tr, off_final + 16, v.ep);
    st->K = a[0];
    st->fs = v.fs;
    if (v.bad) atomicOr(&st->error, 1u);
  }
}

// omega^e from a two-level power table (lo[e & 4095] * hi[e >> 12]).
__device__ __forceinline__ fe pow_table(const fe *lo, const fe *hi, uint64_t e) {
  return fmul(lo[e & 4095u], hi[e >> 12]);
}

struct UbSlots;

constexpr int kOpenThreads = 128;

// One iteration of the opening on the query stream.
struct QueryArgs {
  ProofState *st;
  uint64_t cws, ps, trs;  // per-proof strides of cw, the partials and tr in a batch (grid.y = proof)
  const fe *cw;           // the codeword it opens
  uint64_t L;             // its length
  int l;                  // number of queries
  const fe *partial0, *partial1;  // the two round messages' partials
  int blocks;
  uint8_t *tr;
  uint64_t off_poly[kWhirLogK], off_chal[kWhirLogK];
  uint64_t off_root, off_q, off_rep, off_ans, off_path, off_comb, off_K;
  const UbSlots *u;       // c_i at slot base + i
  uint64_t us;
  int base;
  // omega_L^{-e} table, and the iteration's constants of
  // get_RS_multifold_segment_tensor for a segment of 4 (coPCS_utils.cpp:333-383)
  const fe *inv_lo, *inv_hi;
  fe step0;    // (omega_L^{-1})^(L/4): advance of inv_omegas at level 0
  fe len_inv;  // 4^{-1}
};



// The WHIR randomness of a proof, drawn up front.  Every F::_random() and
// rand() of the opening comes from the glibc generator seeded once, and no
// draw depends on the data, so the draws of Whir_Open in their order
// (per iteration: the two round challenges of whir_sumcheck, the l query
// positions of whir_query, update_betas' r; then the final point,
// Whir.cpp:233-249, 262-268, 327, 426-446) can be made before the
// opening starts.
struct SchedArgs {
  int T;                            // iterations
  int l[kMaxWhirIter];              // queries per iteration
  int32_t qmod[kMaxWhirIter];       // codeword length / 4 per iteration
  int lg_final;                     // log2 of the final polynomial's length
};
constexpr int kMaxDraws = kMaxWhirIter * (3 * kFieldDraws + kMaxQueries) + 8 * kFieldDraws;

// The first warp runs the generator and stores the N outputs in shared
// memory; then all threads derive the field elements (40 outputs each, a
// thread an element) and the query positions from them.  With one thread
// drawing and three deriving a launch took 17.5 us at 2^10, now 12.
__global__ void __launch_bounds__(256) k_whir_schedule(ProofState *st, SchedArgs a) {
  pdl_wait();
  __shared__ int32_t draws[kMaxDraws];
  st += blockIdx.x;
  int N = kFieldDraws * a.lg_final;
  for (int t = 0; t < a.T; t++) N += 3 * kFieldDraws + a.l[t];
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x, f0 = st->prng.f;
    const uint32_t x = prng_warp_draw(prng_warp_load(st->prng, lane), draws, N, lane);
    prng_warp_store(st->prng, x, f0, N, lane);
  }
  __syncthreads();
  // per iteration: r0, r1 (40 outputs each), l queries, update_betas' r; then the final point
  int off = 0;
  for (int t = 0; t < a.T; t++) {
    const int l = a.l[t];
    for (int i = threadIdx.x; i < l; i += blockDim.x) st->wq[t][i] = draws[off + 2 * kFieldDraws + i] % a.qmod[t];
    const int k = (int)threadIdx.x - 3 * t;
    if (k >= 0 && k < 3) {
      const int o = k < 2 ? off + kFieldDraws * k : off + 2 * kFieldDraws + l;
      const fe v = fe_make(prng_number_from(draws + o) % P, prng_number_from(draws + o + 20) % P);
      if (k < 2) st->wr[t][k] = v;
      else st->wrb[t] = v;
    }
    off += 3 * kFieldDraws + l;
  }
  for (int i = (int)blockDim.x - 1 - (int)threadIdx.x; i < a.lg_final; i += blockDim.x) {
    const int o = off + kFieldDraws * i;
    st->fin_r[i] = fe_make(prng_number_from(draws + o) % P, prng_number_from(draws + o + 20) % P);
  }
}

// update_betas of every iteration, prepared up front from the drawn query
// positions: entry base_t + i of an iteration's range holds 2 q_i,
// omega_NL^{2 q_i}, c_i = r^(i+1) and 32 powers of the root.  The beta
// updates sit on the chain of folds; with this on it they cost 2.4 us (the
// powers) and 2 us (roots and weights) more per iteration.
constexpr int kUbSlots = 1024;  // query slots of a proof (rate 2 at 2^25 uses 619)
struct UbSlots {
  fe pw[32 * kUbSlots];
  fe w[kUbSlots], c[kUbSlots];
  int32_t q2[kUbSlots];
};
static_assert(sizeof(UbSlots) <= sizeof(fe) * kUpdateBetasScratch, "update_betas scratch");
struct UbPrepArgs {
  int T;
  int base[kMaxWhirIter + 1];  // first slot of the iterations; the end
  int per[kMaxWhirIter];
  const fe *lo[kMaxWhirIter], *hi[kMaxWhirIter];  // omega_NL^e
};
__global__ void __launch_bounds__(128) k_ub_prep(const ProofState *st, UbSlots *u, uint64_t us, UbPrepArgs a) {
  pdl_wait();
  st += blockIdx.y;
  u = badv(u, us, blockIdx.y);
  const int i = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;  // a warp per query
  if (i >= a.base[a.T]) return;
  int t = 0;
  while (i >= a.base[t + 1]) t++;
  const int j = i - a.base[t];
  const uint32_t q2 = 2u * (uint32_t)st->wq[t][j];
  const fe w = pow_table(a.lo[t], a.hi[t], q2);
  u->pw[32 * i + lane] = fpow(w, (uint64_t)(lane * a.per[t]));
  if (lane == 0) {
    u->q2[i] = (int32_t)q2;
    u->w[i] = w;
    u->c[i] = fpow(st->wrb[t], (uint64_t)j + 1);
  }
}

}  // namespace

// --------------------------------------- kernels shared with the batch opening

// WHIR sumcheck round (whir_sumcheck, Whir.cpp:233-249): message h, the
// consistency check K == h(0) + h(1), challenge F::_random(), K = h(r).
__global__ void k_whir_round(const fe *partial, int blocks, ProofState *st, int i, uint8_t *tr,
                             uint64_t off_poly, uint64_t off_chal) {
  pdl_wait();
  __shared__ int32_t draws[kFieldDraws];
  __shared__ fe drawn;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x / 32 == 1) {  // the challenge, beside the sums (one thread drew for 5 of 9 us)
    const int f0 = st->prng.f;
    const uint32_t x = prng_warp_draw(prng_warp_load(st->prng, lane), draws, kFieldDraws, lane);
    const fe c = prng_warp_field(draws, lane);
    __syncwarp();
    prng_warp_store(st->prng, x, f0, kFieldDraws, lane);
    if (lane == 0) drawn = c;
  }
  fe H[3];
  sum_partials(partial, blocks, H);
  if (threadIdx.x) return;
  fe h01 = fadd(quad_eval(H[0], H[1], H[2], fe_zero()), quad_eval(H[0], H[1], H[2], fe_one()));
  if (!fe_eq(h01, st->K)) atomicOr(&st->error, 2u);
  for (int k = 0; k < 3; k++) {
    put_fe(tr, off_poly + 16 * k, H[k]);
    st->hw[i][k] = H[k];
  }
  const fe r = drawn;
  st->rw[i] = r;
  put_fe(tr, off_chal, r);
  st->K = quad_eval(H[0], H[1], H[2], r);
}

// ---- the Merkle nodes a proof reveals ------------------------------------
// create_tree_blake (merkle_tree.cpp:267-299) hashes the LEFT child twice,
// so node i of level k is G^k(leaf i 2^k) with G(h) = blake3(h || h), and
// leaf j = blake3(e[4j..4j+3]) (MT_commit_Blake, merkle_tree.cpp:195-233).
// The root and the authentication paths (open_tree_blake,
// merkle_tree.cpp:320-335) are therefore chains of compressions from single
// leaves; the prover computes only those instead of whole trees.  The same
// bytes as the full tree (gbz_merkle_commit_blake), which the transcript
// tests compare with the reference's.
__device__ __forceinline__ void leaf_hash(const fe *cw, uint64_t j, uint32_t h[8]) {
  uint32_t m[16];
  const uint4 *src = reinterpret_cast<const uint4 *>(cw + 4 * j);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint4 v = src[k];
    m[4 * k] = v.x; m[4 * k + 1] = v.y; m[4 * k + 2] = v.z; m[4 * k + 3] = v.w;
  }
  blake3_block64(m, h);
}
__device__ __forceinline__ void node_hash(uint32_t h[8]) {  // h <- blake3(h || h)
  uint32_t m[16];
#pragma unroll
  for (int k = 0; k < 8; k++) m[k] = m[8 + k] = h[k];
  blake3_block64(m, h);
}
__device__ __forceinline__ void put_hash(uint8_t *dst, const uint32_t h[8]) {  // 4-byte aligned
  uint32_t *d = reinterpret_cast<uint32_t *>(dst);
#pragma unroll
  for (int k = 0; k < 8; k++) d[k] = h[k];
}

// Root of the tree over a codeword of 4 * 2^depth elements: G^depth(leaf 0).
__device__ void merkle_root_dev(const fe *cw, int depth, uint8_t *tr, uint64_t off) {
  uint32_t h[8];
  leaf_hash(cw, 0, h);
  for (int d = 0; d < depth; d++) node_hash(h);
  put_hash(tr + off, h);
}
__global__ void k_merkle_root(const fe *cw, int depth, uint8_t *tr, uint64_t off) {
  pdl_wait();
  if (threadIdx.x) return;
  merkle_root_dev(cw, depth, tr, off);
}
// The same for a batch: proof p (grid.x) reads cw + p cws, writes tr + p trs.
__global__ void k_merkle_root_b(const fe *cw, uint64_t cws, int depth, uint8_t *tr, uint64_t trs, uint64_t off) {
  pdl_wait();
  if (threadIdx.x) return;
  merkle_root_dev(badv(cw, cws, blockIdx.x), depth, tr + trs * blockIdx.x, off);
}

// Authentication paths of the l queries: entry d of query i is the sibling
// (q >> d) ^ 1 of level d, i.e. G^d(leaf ((q >> d) ^ 1) << d).  One thread
// per entry, the deepest entries first.
__device__ __forceinline__ void path_entry(const fe *cw, int depth, int l, uint64_t t, uint8_t *tr, const int32_t *qs,
                                           uint64_t off_path) {
  if (t >= (uint64_t)l * depth) return;
  const int d = depth - 1 - (int)(t / l), i = (int)(t % l);
  const uint64_t q = (uint64_t)(uint32_t)qs[i];
  uint32_t h[8];
  leaf_hash(cw, ((q >> d) ^ 1ull) << d, h);
  for (int k = 0; k < d; k++) node_hash(h);
  put_hash(tr + off_path + 32ull * ((uint64_t)depth * i + d), h);
}
__global__ void k_whir_paths_chain(const fe *cw, uint64_t leaves, int l, uint8_t *tr, uint64_t off_q,
                                   uint64_t off_path, uint64_t cws, uint64_t trs) {
  pdl_wait();
  cw = badv(cw, cws, blockIdx.y);  // a batch: grid.y = proof
  tr += trs * blockIdx.y;
  path_entry(cw, 63 - __clzll((long long)leaves), l, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, tr,
             reinterpret_cast<const int32_t *>(tr + off_q), off_path);
}

namespace {

// whir_query (Whir.cpp:251-314) of iteration t with the drawn positions, its
// two round messages (recorded with their challenges), and the running claim
// of whir_sumcheck and update_betas: K is checked against both messages
// (K == h(0) + h(1), K = h(r)), then K += sum_i c_i y_i (Whir.cpp:383-384).
__device__ void whir_query_dev(const QueryArgs &a, int t) {
  __shared__ fe red[kOpenThreads / 32];
  ProofState *st = a.st;
  fe H[kWhirLogK][3];
  sum_partials(a.partial0, a.blocks, H[0]);
  __syncthreads();  // sum_partials' shared scratch is reused
  sum_partials(a.partial1, a.blocks, H[1]);
  const fe one = fe_one(), r0 = st->wr[t][0], r1 = st->wr[t][1];
  fe contrib = fe_zero();
  for (int i = threadIdx.x; i < a.l; i += kOpenThreads) {
    const int32_t q = st->wq[t][i];
    const uint64_t qi = (uint64_t)q;
    reinterpret_cast<int32_t *>(a.tr + a.off_q)[i] = q;
    fe seg[kWhirK];
    for (int j = 0; j < kWhirK; j++) {
      seg[j] = a.cw[qi + j * (a.L / kWhirK)];
      put_fe(a.tr, a.off_rep + 16 * (kWhirK * i + j), seg[j]);
    }
    // get_RS_multifold_segment_tensor(seg, r, L, qi) with r = the two WHIR
    // round challenges: level 0 pairs (j, j+2) with omega_L^{-(qi + j L/4)},
    // level 1 pairs (0, 1) with omega_{L/2}^{-qi} = omega_L^{-2 qi}.
    fe inv_om = pow_table(a.inv_lo, a.inv_hi, qi);
    fe part[2];
    for (int j = 0; j < 2; j++) {
      fe s = fadd(seg[j], seg[j + 2]), d = fsub(seg[j], seg[j + 2]);
      part[j] = fadd(fmul(fsub(one, r0), s), fmul(fmul(r0, inv_om), d));
      inv_om = fmul(inv_om, a.step0);
    }
    fe po = pow_table(a.inv_lo, a.inv_hi, (2 * qi) & (a.L - 1));
    fe s = fadd(part[0], part[1]), d = fsub(part[0], part[1]);
    fe y = fmul(a.len_inv, fadd(fmul(fsub(one, r1), s), fmul(r1, fmul(po, d))));
    put_fe(a.tr, a.off_ans + 16 * i, y);
    const fe c = a.u->c[a.base + i];
    put_fe(a.tr, a.off_comb + 16 * i, c);
    contrib = fadd(contrib, fmul(c, y));
  }
  for (int dd = 16; dd > 0; dd >>= 1) {
    fe v;
    v.re = __shfl_down_sync(0xffffffffu, contrib.re, dd);
    v.im = __shfl_down_sync(0xffffffffu, contrib.im, dd);
    contrib = fadd(contrib, v);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = contrib;
  __syncthreads();
  if (threadIdx.x == 0) {
    fe K = st->K;
    for (int r = 0; r < kWhirLogK; r++) {
      const fe *h = H[r], c = st->wr[t][r];
      for (int k = 0; k < 3; k++) put_fe(a.tr, a.off_poly[r] + 16 * k, h[k]);
      put_fe(a.tr, a.off_chal[r], c);
      const fe h01 = fadd(quad_eval(h[0], h[1], h[2], fe_zero()), quad_eval(h[0], h[1], h[2], fe_one()));
      if (!fe_eq(h01, K)) atomicOr(&st->error, 2u);
      K = quad_eval(h[0], h[1], h[2], c);
    }
    for (int w = 0; w < kOpenThreads / 32; w++) K = fadd(K, red[w]);
    st->K = K;
    put_fe(a.tr, a.off_K, K);
  }
}

// An iteration's work on the query stream in one launch: block 0 the root
// (a chain of depth + 1 compressions), block 1 the round messages and the
// queries, the others the authentication paths, a thread an entry.  Each is a
// serial chain of its own, so the launch takes as long as the longest; as
// three launches behind each other an iteration took 35 us at 2^18, now 13,
// and bound the opening.  Four warps a block: a compression fills the integer
// issue slots of an SM's quarter.
__global__ void __launch_bounds__(kOpenThreads) k_whir_open(QueryArgs a, int t) {
  pdl_wait();
  a.st += blockIdx.y;
  a.cw = badv(a.cw, a.cws, blockIdx.y);
  a.tr += a.trs * blockIdx.y;
  const int depth = 63 - __clzll((long long)(a.L / 4));
  if (blockIdx.x == 0) {
    if (threadIdx.x == 0) merkle_root_dev(a.cw, depth, a.tr, a.off_root);
  } else if (blockIdx.x == 1) {
    a.partial0 = badv(a.partial0, a.ps, blockIdx.y);
    a.partial1 = badv(a.partial1, a.ps, blockIdx.y);
    a.u = badv(a.u, a.us, blockIdx.y);
    whir_query_dev(a, t);
  } else {
    path_entry(a.cw, depth, a.l, (uint64_t)(blockIdx.x - 2) * kOpenThreads + threadIdx.x, a.tr, a.st->wq[t],
               a.off_path);
  }
}

}  // namespace

// The tree aggregate_commitments builds (Whir.cpp:594-605) has all-zero
// leaf hashes, so its level-d nodes all equal G^d(0): the root of a tree of
// 2^depth leaves, and every query's path entry d.
__global__ void k_zero_tree_root(int depth, uint8_t *tr, uint64_t off) {
  pdl_wait();
  if (threadIdx.x) return;
  uint32_t h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int d = 0; d < depth; d++) node_hash(h);
  put_hash(tr + off, h);
}
__global__ void k_zero_tree_paths(int depth, int l, uint8_t *tr, uint64_t off_path) {
  pdl_wait();
  const int d = blockIdx.x * blockDim.x + threadIdx.x;  // one thread per level
  if (d >= depth) return;
  uint32_t h[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int k = 0; k < d; k++) node_hash(h);
  for (int i = 0; i < l; i++) put_hash(tr + off_path + 32ull * ((uint64_t)depth * i + d), h);
}

// open_tree_blake (merkle_tree.cpp:320-335) for every query in a tree of
// `leaves` leaf hashes: sibling (pos >> d) ^ 1 of level d (levels stored back
// to back, level d starting at 2 leaves - 2 (leaves >> d)), one hash per
// thread so that all the scattered tree reads are in flight together.
__global__ void k_whir_paths(const uint8_t *tree, uint64_t leaves, int l, uint8_t *tr, uint64_t off_q,
                             uint64_t off_path) {
  pdl_wait();
  const int depth = 63 - __clzll((long long)leaves);
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (uint64_t)l * depth) return;
  const int i = (int)(t / depth), d = (int)(t % depth);
  const uint64_t q = (uint64_t)(uint32_t)reinterpret_cast<const int32_t *>(tr + off_q)[i];
  const uint64_t lvl = 2 * leaves - 2 * (leaves >> d);
  const uint4 *src = reinterpret_cast<const uint4 *>(tree + 32 * (lvl + ((q >> d) ^ 1ull)));
  const uint4 h0 = src[0], h1 = src[1];
  // transcript payloads are only 4-byte aligned
  uint32_t *dst = reinterpret_cast<uint32_t *>(tr + off_path + 32ull * ((uint64_t)depth * i + d));
  dst[0] = h0.x; dst[1] = h0.y; dst[2] = h0.z; dst[3] = h0.w;
  dst[4] = h1.x; dst[5] = h1.y; dst[6] = h1.z; dst[7] = h1.w;
}

// Final round of Whir_Open (Whir.cpp:426-446) and of Whir_Batch_Open
// (:840-869): the remaining polynomial (m <= kFinalMax entries), log2 m
// F::_random draws and evaluate_vector(b, r).  With check_K, the flag 8 is
// raised unless K equals sum arr * b (verification step 2, :848-855).
__device__ void final_dev(ProofState *st, const fe *arr, const fe *b, int m, uint8_t *tr, uint64_t off_poly,
                          uint64_t off_point, uint64_t off_eval, int check_K, const fe *point, glibc_prng &g) {
  if (m < 1 || m > kFinalMax) {
    atomicOr(&st->error, 16u);
    return;
  }
  fe Kc = st->K;
  for (int i = 0; i < m; i++) {
    put_fe(tr, off_poly + 16 * i, arr[i]);
    Kc = fsub(Kc, fmul(arr[i], b[i]));
  }
  if (check_K && !fe_eq(Kc, fe_zero())) atomicOr(&st->error, 8u);
  const int lg = 31 - __clz(m);
  fe r[8];
  if (!point) g = st->prng;
  for (int i = 0; i < lg; i++) {
    r[i] = point ? point[i] : prng_field(g);
    put_fe(tr, off_point + 16 * i, r[i]);
  }
  if (!point) st->prng = g;
  fe v[kFinalMax];
  for (int i = 0; i < m; i++) v[i] = b[i];
  for (int i = 0; i < lg; i++) {
    fe om = fsub(fe_one(), r[i]);
    int L = 1 << (lg - 1 - i);
    for (int j = 0; j < L; j++) v[j] = fadd(fmul(om, v[2 * j]), fmul(r[i], v[2 * j + 1]));
  }
  put_fe(tr, off_eval, v[0]);
}
__global__ void k_final(ProofState *st, const fe *arr, const fe *b, int m, uint8_t *tr, uint64_t off_poly,
                        uint64_t off_point, uint64_t off_eval, int check_K, const fe *point) {
  pdl_wait();
  __shared__ glibc_prng g;
  if (threadIdx.x) return;
  final_dev(st, arr, b, m, tr, off_poly, off_point, off_eval, check_K, point, g);
}
// The same for a batch of proofs whose final point was drawn up front
// (st->fin_r): proof p = grid.x, bs = strides of (arr, b, tr).
__global__ void k_final_b(ProofState *st, const fe *arr, const fe *b, int m, uint8_t *tr, uint64_t off_poly,
                          uint64_t off_point, uint64_t off_eval, BStr bs) {
  pdl_wait();
  __shared__ glibc_prng g;
  if (threadIdx.x) return;
  st += blockIdx.x;
  final_dev(st, badv(arr, bs.s[0], blockIdx.x), badv(b, bs.s[1], blockIdx.x), m, badv(tr, bs.s[2], blockIdx.x),
            off_poly, off_point, off_eval, 0, st->fin_r, g);
}

// ------------------------------------------------------------ host side

bool update_betas_by_transform(int l, uint64_t nb, uint64_t N) {
  return ilog2(N) > 13 && ilog2(N) <= kMaxNttLogN && nb <= N && (uint64_t)l * nb > 4 * N;
}

int whir_query_count(int rate) { return (int)(-100.0 / log2(sqrt(1.0 / (double)rate))); }

uint64_t Layout::rec(uint32_t tag, uint32_t count, uint32_t unit) {
  uint64_t off = len;
  if (record_headers) {
    headers.push_back({off, tag, count});
  }
  len += 8 + (uint64_t)count * unit;
  return off + 8;
}

namespace {
void graph_free(ProofGraph &g);
}
ProofPlan::~ProofPlan() {
  if (s2) cudaStreamSynchronize(s2);
  if (s3) cudaStreamSynchronize(s3);
  for (auto &g : graphs) graph_free(g);
  for (auto &kv : ntt) ntt_tables_free(kv.second);
  for (void *p : allocs) cudaFree(p);
  if (ev_in) cudaEventDestroy(ev_in);
  for (auto &e : ev_fold)
    if (e) cudaEventDestroy(e);
  for (auto &e : ev_commit)
    if (e) cudaEventDestroy(e);
  for (auto &e : ev_query)
    if (e) cudaEventDestroy(e);
  if (ev_sched) cudaEventDestroy(ev_sched);
  if (ev_root_tail) cudaEventDestroy(ev_root_tail);
  if (s2) cudaStreamDestroy(s2);
  if (s3) cudaStreamDestroy(s3);
}

void *ProofPlan::dalloc(uint64_t bytes) {
  void *p = nullptr;
  GBZ_CUDA(device_malloc(&p, bytes ? bytes : 16));
  allocs.push_back(p);
  return p;
}

NttTables &ProofPlan::tables(int lg) {
  auto it = ntt.find(lg);
  if (it != ntt.end()) return it->second;
  NttTables t;
  ntt_tables_build(t, lg);
  return ntt.emplace(lg, t).first->second;
}

// Partials of the WHIR rounds, two messages of three sums a block, of every
// iteration: they are read on the query stream while the folds move on.
static uint64_t whir_partials(uint64_t n) {
  uint64_t total = 0;
  for (uint64_t m = n; m > (uint64_t)kWhirK; m /= 4) total += 6 * (uint64_t)sc_blocks(m / 4);
  return total;
}

std::unique_ptr<ProofPlan> plan_create(int logn, int rate, int batch) {
  if (logn < 3 || logn > 25) throw ArgError("prover: log2 witness length must be in [3, 25]");
  if (rate < 2 || rate > 64 || !is_pow2((uint64_t)rate)) throw ArgError("prover: rate must be a power of two in [2, 64]");
  if (batch < 1 || batch > 65535) throw ArgError("prover: 1..65535 proofs per plan");
  const uint64_t n = 1ull << logn, L = n * (uint64_t)rate;
  if (ilog2(L) > kMaxNttLogN) throw ArgError("prover: codeword longer than 2^26");
  auto p = std::unique_ptr<ProofPlan>(new ProofPlan());
  p->logn = logn;
  p->rate = rate;
  p->n = n;
  p->L = L;
  p->B = batch;
  const uint64_t B = (uint64_t)batch;
  p->bs_w = sizeof(fe) * n;
  p->bs_cw0 = sizeof(fe) * L;
  p->bs_cw1 = sizeof(fe) * (L / 2);
  p->bs_tmp = sizeof(fe) * L;
  p->bs_tmp2 = sizeof(fe) * (L / 2);
  p->bs_v = sizeof(fe) * (n / 2);
  p->bs_arr = sizeof(fe) * (n / 2);
  p->bs_beta = sizeof(fe) * n;
  p->bs_part = sizeof(fe) * 4 * (uint64_t)sc_blocks(n / 4);
  p->bs_wpart = sizeof(fe) * whir_partials(n);
  p->bs_ub = sizeof(fe) * kUpdateBetasScratch;
  p->w = (fe *)p->dalloc(B * p->bs_w);
  p->cw[0] = (fe *)p->dalloc(B * p->bs_cw0);
  p->cw[1] = (fe *)p->dalloc(B * p->bs_cw1);
  p->tmp = (fe *)p->dalloc(B * p->bs_tmp);
  p->tmp2 = (fe *)p->dalloc(B * p->bs_tmp2);
  GBZ_CUDA(cudaStreamCreateWithFlags(&p->s2, cudaStreamNonBlocking));
  GBZ_CUDA(cudaStreamCreateWithFlags(&p->s3, cudaStreamNonBlocking));
  GBZ_CUDA(cudaEventCreateWithFlags(&p->ev_in, cudaEventDisableTiming));
  GBZ_CUDA(cudaEventCreateWithFlags(&p->ev_sched, cudaEventDisableTiming));
  GBZ_CUDA(cudaEventCreateWithFlags(&p->ev_root_tail, cudaEventDisableTiming));
  for (auto &e : p->ev_fold) GBZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  for (auto &e : p->ev_commit) GBZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  for (auto &e : p->ev_query) GBZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
  p->va[0] = (fe *)p->dalloc(B * p->bs_v);
  p->va[1] = (fe *)p->dalloc(B * p->bs_v);
  p->arr = (fe *)p->dalloc(B * p->bs_arr);
  p->vb[0] = (fe *)p->dalloc(B * p->bs_v);
  p->vb[1] = (fe *)p->dalloc(B * p->bs_v);
  p->beta = (fe *)p->dalloc(B * p->bs_beta);
  p->partial = (fe *)p->dalloc(B * p->bs_part);
  p->wpart = (fe *)p->dalloc(B * p->bs_wpart);
  p->ub_scratch = (fe *)p->dalloc(B * p->bs_ub);
  p->st = (ProofState *)p->dalloc(B * sizeof(ProofState));
  GBZ_CUDA(cudaFuncSetAttribute(k_sc_tail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)kScTailShared));
  // Build the transcript layout (record headers are constant).
  p->layout.record_headers = true;
  enqueue_proof(*p, nullptr, 1, nullptr, /*dry=*/true);  // layout and launch counts
  p->layout.record_headers = false;
  p->transcript_bytes = p->layout.len;
  p->transcript = (uint8_t *)p->dalloc(B * p->transcript_bytes);
  std::vector<uint8_t> img(p->transcript_bytes, 0);
  for (auto &h : p->layout.headers) {
    std::memcpy(&img[h.off], &h.tag, 4);
    std::memcpy(&img[h.off + 4], &h.count, 4);
  }
  for (uint64_t b = 0; b < B; b++)
    GBZ_CUDA(cudaMemcpy(p->transcript + b * p->transcript_bytes, img.data(), img.size(), cudaMemcpyHostToDevice));
  // Twiddle tables for every transform length the proof uses.
  p->tables(ilog2(L));
  for (uint64_t m = n, cur = (uint64_t)rate; m > 4; m /= 4, cur *= 2) {
    p->tables(ilog2(2 * cur * (m / 4)));
    p->tables(ilog2(cur * (m / 4)));  // the half-length update_betas transform
  }
  return p;
}

void plan_prepare_open(ProofPlan &p) {
  if (p.open_transcript) return;
  Layout saved = p.layout;
  const int launches = p.launches;
  int cat[PC_COUNT];
  for (int c = 0; c < PC_COUNT; c++) cat[c] = p.cat_launches[c];
  p.layout = Layout();
  p.layout.record_headers = true;
  OpenOnly o{};
  enqueue_proof(p, nullptr, 0, nullptr, /*dry=*/true, false, &o);
  const Layout open_layout = p.layout;
  p.layout = saved;
  p.launches = launches;
  for (int c = 0; c < PC_COUNT; c++) p.cat_launches[c] = cat[c];
  p.open_transcript_bytes = open_layout.len;
  p.open_transcript = (uint8_t *)p.dalloc(open_layout.len);
  std::vector<uint8_t> img(open_layout.len, 0);
  for (auto &h : open_layout.headers) {
    std::memcpy(&img[h.off], &h.tag, 4);
    std::memcpy(&img[h.off + 4], &h.count, 4);
  }
  GBZ_CUDA(cudaMemcpy(p.open_transcript, img.data(), img.size(), cudaMemcpyHostToDevice));
}

// Enqueue one proof.  witness: device pointer (nullptr: use plan->w).
// The dry run (dry = true) launches nothing; it fixes the transcript layout
// and counts the launches per category.
void enqueue_proof(ProofPlan &p, const fe *witness, uint32_t prng_seed, cudaStream_t s, bool dry, bool seed_in_state,
                   const OpenOnly *open, ProofPart part) {
  Layout &lay = p.layout;
  lay.len = 0;
  if (dry) {
    p.launches = 0;
    for (int c = 0; c < PC_COUNT; c++) p.cat_launches[c] = 0;
  }
  const fe *w = witness ? witness : p.w;
  const int logn = p.logn;
  uint8_t *tr = open ? p.open_transcript : p.transcript;
  ProofState *st = p.st;
  // a batch: every launch covers the plan's B proofs (per-proof strides below)
  const int B = p.B;
  if (B > 1 && (open || (witness && witness != p.w))) throw ArgError("prover: a batch reads its witnesses from the plan");
  const uint64_t trs = p.transcript_bytes, sts = sizeof(ProofState);
  const uint64_t cw_s[2] = {p.bs_cw0, p.bs_cw1};
  Profiler *prof = (!dry && p.prof && p.prof->enabled) ? p.prof : nullptr;
  // Whether what comes next is enqueued: not in the dry run, and not what
  // another part holds.
  bool go = !dry && part != PART_OPENING;
  // RUN(category, kernel launches, statement): counts in the dry run, else
  // runs the statement (bracketed by profiler events when enabled).
#define RUN_ON(strm, cat, nlaunch, ...)        \
  do {                                         \
    if (dry) {                                 \
      p.launches += (nlaunch);                 \
      p.cat_launches[cat] += (nlaunch);        \
    } else if (go) {                           \
      if (prof) prof->begin(cat, strm);        \
      __VA_ARGS__;                             \
      GBZ_CUDA(cudaGetLastError());            \
      if (prof) prof->end(strm);               \
    }                                          \
  } while (0)
#define RUN(cat, nlaunch, ...) RUN_ON(s, cat, nlaunch, __VA_ARGS__)

  // Commits go to the plan's second stream c; it starts after everything
  // the caller enqueued on s (the witness copy) and s joins it at the end.
  // With the profiler on, the commits stay on s so that the per-category
  // event times do not include waits for the other stream's kernels.
  cudaStream_t c = prof ? s : p.s2, q = prof ? s : p.s3;
  // A proof of its own seeds its generator on q, so that its three chains
  // start at once (2^18: 322 us, behind the seeding 347); the scheduler's
  // graphs, many in flight, start as one node (64 mixed proofs 4900 us, as
  // three 5090).
  const bool fork_first = !open && !seed_in_state;
  auto fork = [&]() {
    if (!go) return;
    GBZ_CUDA(cudaEventRecord(p.ev_in, s));
    GBZ_CUDA(cudaStreamWaitEvent(c, p.ev_in, 0));
    GBZ_CUDA(cudaStreamWaitEvent(q, p.ev_in, 0));
  };
  if (fork_first) fork();
  if (open) {
    RUN(PC_PROTOCOL, 1, launch_kernel(k_init_open, 1, 32, 0, s, st, open->prng, open->point, logn, open->K));
  } else {
    const cudaStream_t is = fork_first ? q : s;
    RUN_ON(is, PC_PROTOCOL, 1, launch_kernel(k_init, B, 32, 0, is, st, prng_seed, seed_in_state ? 1 : 0));
  }
  if (!fork_first) fork();
  // The records before the opening; the root's payload is written by its
  // first queries.
  uint64_t off_root[kMaxWhirIter + 1];
  off_root[0] = lay.rec(T_COMMIT_ROOT, 1, 32);
  uint64_t off = 0, m = p.n, L = p.L;
  const fe *a = w;
  int cwi = 0, iter = 0;

  auto sumcheck = [&]() {
  // 1. evaluation point and its eq table.
  off = lay.rec(T_EVAL_POINT, logn, 16);
  RUN(PC_PROTOCOL, 1, launch_kernel(k_point, B, 32, 0, s, st, logn, tr, off, trs));
  // 2. sumcheck of sum w(x) eq(z, x), two rounds a pass: w is folded by both
  //    challenges, the eq vector is represented by the shrinking tables
  //    E_{i+1} (vb ping-pong) and the prefix product epre; the last rounds
  //    (or all of a small proof) in one CTA.
  RUN(PC_BETA, 1, beta_launch(st->z + 2, logn - 2, p.vb[0], s, B, sts, p.bs_v));
  const uint64_t off_claim = lay.rec(T_CLAIM, 1, 16);
  const uint64_t off_poly0 = lay.len + 8;
  for (int r = 0; r < logn; r++) {
    const uint64_t op = lay.rec(T_SC_POLY, 3, 16), oc = lay.rec(T_SC_CHALLENGE, 1, 16);
    if (op != off_poly0 + 80ull * (uint64_t)r || oc != op + 56) throw ArgError("prover: sumcheck record layout");
  }
  off = lay.rec(T_SC_FINAL, 2, 16);
  int pp = 0, i = 0;       // va and vb ping-pong
  uint64_t as = p.bs_w;    // per-proof stride of a (the witness, then va)
  if (m > (uint64_t)kScTailMax) {
    int blocks = sc_blocks(m / 4);
    BStr rs;  // (a, E, partial)
    rs.s[0] = as;
    rs.s[1] = p.bs_v;
    rs.s[2] = p.bs_part;
    RUN(PC_SUMCHECK, 1, sc_eq_reduce_launch(a, p.vb[0], m, p.partial, blocks, s, B, rs));
    for (; m > (uint64_t)kScTailMax; i += 2, m /= 4, pp ^= 1) {
      RUN(PC_PROTOCOL, 1,
          launch_kernel(k_sc_rounds_eq, B, 256, 0, s, p.partial, blocks, st, i, tr, i == 0 ? (int64_t)off_claim : -1,
                        off_poly0 + 80ull * (uint64_t)i, p.bs_part, trs));
      blocks = sc_blocks(m / 4);
      BStr fs;  // (a, chal, a4, E, E4, partial)
      fs.s[0] = as;
      fs.s[1] = sts;
      fs.s[2] = p.bs_v;
      fs.s[3] = p.bs_v;
      fs.s[4] = p.bs_v;
      fs.s[5] = p.bs_part;
      RUN(PC_SUMCHECK, 1,
          sc_eq_fold_launch(a, p.vb[pp], m, &st->chal[i], p.va[pp], p.vb[pp ^ 1], m / 4 > (uint64_t)kScTailMax,
                            p.partial, blocks, s, B, fs));
      a = p.va[pp];
      as = p.bs_v;
    }
  }
  BStr tb;  // (a, E, tr)
  tb.s[0] = as;
  tb.s[1] = p.bs_v;
  tb.s[2] = trs;
  RUN(PC_SUMCHECK, 1,
      (launch_kernel(k_sc_tail, B, kScTailThreads, kScTailShared, s, st, a, p.vb[pp], (int)m, i, logn, tr,
                     i == 0 ? (int64_t)off_claim : -1, off_poly0 + 80ull * (uint64_t)i, off, tb)));
  };

  // The opening's randomness, drawn on the query stream while the
  // commitment and the sumcheck run, and the beta updates' powers.
  UbSlots *slots = reinterpret_cast<UbSlots *>(p.ub_scratch);
  UbPrepArgs ua{};
  auto draws = [&]() {
    SchedArgs sa{};
    uint64_t mm = p.n, LL = p.L, cc = (uint64_t)p.rate;
    for (;;) {
      if (sa.T >= kMaxWhirIter) throw ArgError("prover: too many WHIR iterations");
      mm /= 4;
      sa.l[sa.T] = whir_query_count((int)cc);
      sa.qmod[sa.T] = (int32_t)(LL / 4);
      if (sa.l[sa.T] < 1 || sa.l[sa.T] > kMaxQueries) throw ArgError("prover: query count out of range");
      sa.T++;
      LL = 2 * cc * mm;
      cc *= 2;
      if (mm <= (uint64_t)kWhirK) break;
    }
    sa.lg_final = ilog2(mm);
    RUN_ON(q, PC_PROTOCOL, 1, launch_kernel(k_whir_schedule, B, 256, 0, q, st, sa));
    ua.T = sa.T;
    LL = p.L;
    mm = p.n;
    for (int t = 0; t < sa.T; t++) {
      LL /= 2;
      mm /= 4;
      ua.base[t + 1] = ua.base[t] + sa.l[t];
      ua.per[t] = update_betas_per(mm, B);
      if (!go) continue;
      const NttTables &tnew = p.tables(ilog2(LL));
      ua.lo[t] = tnew.lo_fwd;
      ua.hi[t] = tnew.hi_fwd;
    }
    if (ua.base[sa.T] > kUbSlots) throw ArgError("prover: too many queries");
    RUN_ON(q, PC_UPDATE_BETAS, 1,
           launch_kernel(k_ub_prep, dim3((unsigned)(ua.base[sa.T] + 3) / 4, B), 128, 0, q, st, slots, p.bs_ub, ua));
    if (go) GBZ_CUDA(cudaEventRecord(p.ev_sched, q));
  };

  // 3. commitment: codeword = NTT(w padded to rate*n), Merkle tree.
  auto commit = [&]() {
  // The witness is expected in the base field (the imaginary words zero):
  // its transform is then a half-length transform of packed pairs
  // (ntt_launch_real); any other witness takes the general transform.
  if (open) {
    if (go && open->codeword != p.cw[0])
      GBZ_CUDA(cudaMemcpyAsync(p.cw[0], open->codeword, 16 * L, cudaMemcpyDeviceToDevice, c));
  } else if (B > 1 && ilog2(L) < kBatchRealLog) {
    // short codewords (launch bound): the batch's codewords as one batched
    // transform (the same values as the real-input path of a single proof)
    RUN_ON(c, PC_NTT, ntt_launch_count(ilog2(L), p.n, B),
           ntt_launch_rows(p.tables(ilog2(L)), w, p.n, p.bs_w / sizeof(fe), p.cw[0], p.bs_cw0 / sizeof(fe), B, p.tmp,
                           false, c));
  } else if (B > 1) {
    // long codewords (integer-pipe bound): the real-input transform of each
    // proof, half the multiplies of the general one
    for (int pb = 0; pb < B; pb++) {
      if (go) GBZ_CUDA(cudaMemsetAsync(&st[pb].nonreal, 0, sizeof(uint32_t), c));
      RUN_ON(c, PC_NTT, ntt_launch_real_count(ilog2(L), p.n),
             ntt_launch_real(p.tables(ilog2(L) - 1), p.tables(ilog2(L)),
                             reinterpret_cast<const fe *>(reinterpret_cast<const char *>(w) + p.bs_w * pb), p.n,
                             reinterpret_cast<fe *>(reinterpret_cast<char *>(p.cw[0]) + p.bs_cw0 * pb),
                             reinterpret_cast<fe *>(reinterpret_cast<char *>(p.tmp) + p.bs_tmp * pb), &st[pb].nonreal,
                             c));
    }
  } else {
    if (go) GBZ_CUDA(cudaMemsetAsync(&st->nonreal, 0, sizeof(uint32_t), c));
    RUN_ON(c, PC_NTT, ntt_launch_real_count(ilog2(L), p.n),
           ntt_launch_real(p.tables(ilog2(L) - 1), p.tables(ilog2(L)), w, p.n, p.cw[0], p.tmp, &st->nonreal, c));
  }
  if (go) GBZ_CUDA(cudaEventRecord(p.ev_commit[0], c));
  };

  // On one stream the order of the launches, across them the order in which a
  // graph gets going: the start alone with the sumcheck first, a whole proof
  // with its commitment first (2^24 2641 us, the sumcheck first 2705).
  if (part == PART_START) {
    sumcheck();
    draws();
    commit();
  } else {
    draws();
    commit();
    if (!open) sumcheck();
  }

  if (part == PART_START) {  // s joins the commitment and the draws
    GBZ_CUDA(cudaStreamWaitEvent(s, p.ev_commit[0], 0));
    GBZ_CUDA(cudaStreamWaitEvent(s, p.ev_sched, 0));
    lay.len = p.transcript_bytes;
    return;
  }
  if (part == PART_OPENING) {
    go = true;
    fork();
  }

  // 4. WHIR open of (v1[0], chal): b = precompute_beta(chal), arr = w.
  //    Three chains: folds and beta updates on s, commits on c, queries
  //    and the running claim K on q.  The folded polynomials are written
  //    once each (p.arr), so the commits read them while s moves on; a
  //    commit reuses a codeword/tree buffer only after the query that
  //    opened its previous content.
  // b = precompute_beta(chal) has tensor structure: for the first
  // iteration only the eq table E2 of chal[2..] is formed (a quarter of b)
  const bool eq_first = logn >= 4;
  RUN(PC_BETA, 1,
      eq_first ? beta_launch(st->chal + 2, logn - 2, p.beta, s, B, sts, p.bs_beta)
               : beta_launch(st->chal, logn, p.beta, s, B, sts, p.bs_beta));
  if (go && part == PART_ALL) GBZ_CUDA(cudaStreamWaitEvent(s, p.ev_sched, 0));  // round challenges
  a = w;
  const fe *b = p.beta;
  uint64_t ast = p.bs_w, bst = p.bs_beta;  // per-proof strides of a and b
  m = p.n;
  uint64_t cur = (uint64_t)p.rate;
  fe *arr_next = p.arr, *wpart = p.wpart;
  for (;;) {
    if (iter >= ProofPlan::kMaxIter) throw ArgError("prover: too many WHIR iterations");
    const int l = whir_query_count((int)cur);
    const uint64_t NL = 2 * cur * (m / 4);
    if (2 * NL != L) throw ArgError("prover: WHIR codeword lengths must halve");
    // both rounds in one pass over (a, b): their challenges were drawn up
    // front; arr_{t+1} goes to its own slot of p.arr, b to vb[(t + 1) mod 2]
    // (never the buffer it is read from)
    uint64_t op = lay.rec(T_WHIR_POLY, 3, 16), oc = lay.rec(T_WHIR_CHALLENGE, 1, 16);
    const uint64_t op1 = lay.rec(T_WHIR_POLY, 3, 16), oc1 = lay.rec(T_WHIR_CHALLENGE, 1, 16);
    fe *bd = p.vb[(iter + 1) & 1];
    const int blocks = sc_blocks(m / 4);
    fe *part0 = wpart, *part1 = wpart + 3 * blocks;
    wpart += 6 * blocks;
    if (iter == 0 && eq_first) {
      BStr fb;  // (a, E2, c, chal0, chal1, a4, b4, partial0, partial1)
      fb.s[0] = ast;
      fb.s[1] = bst;
      fb.s[2] = sts;
      fb.s[3] = sts;
      fb.s[4] = sts;
      fb.s[5] = p.bs_arr;
      fb.s[6] = p.bs_v;
      fb.s[7] = p.bs_wpart;
      fb.s[8] = p.bs_wpart;
      RUN(PC_SUMCHECK, 1,
          sc_fold2_eq_launch(a, b, m, st->chal, &st->wr[iter][0], &st->wr[iter][1], arr_next, bd, part0, part1,
                             blocks, s, B, fb));
    } else {
      BStr fb;  // (a, b, chal0, chal1, a4, b4, partial0, partial1)
      fb.s[0] = ast;
      fb.s[1] = bst;
      fb.s[2] = sts;
      fb.s[3] = sts;
      fb.s[4] = p.bs_arr;
      fb.s[5] = p.bs_v;
      fb.s[6] = p.bs_wpart;
      fb.s[7] = p.bs_wpart;
      RUN(PC_SUMCHECK, 1,
          sc_fold2_launch(a, b, m, &st->wr[iter][0], &st->wr[iter][1], arr_next, bd, part0, part1, blocks, s, B,
                          fb));
    }
    a = arr_next;
    b = bd;
    ast = p.bs_arr;
    bst = p.bs_v;
    m /= 4;
    arr_next += m;
    if (go) GBZ_CUDA(cudaEventRecord(p.ev_fold[iter], s));
    // commit arr_{t+1} at rate 2*cur on c, once the query that opened the
    // buffer's previous codeword (iteration t-1) is done
    const int nci = cwi ^ 1;
    off = lay.rec(T_WHIR_ROOT, 1, 32);
    if (go) {
      GBZ_CUDA(cudaStreamWaitEvent(c, p.ev_fold[iter], 0));
      if (iter > 0) GBZ_CUDA(cudaStreamWaitEvent(c, p.ev_query[iter - 1], 0));
    }
    if (B > 1) {
      RUN_ON(c, PC_NTT, ntt_launch_count(ilog2(NL), m, B),
             ntt_launch_rows(p.tables(ilog2(NL)), a, m, p.bs_arr / sizeof(fe), p.cw[nci], cw_s[nci] / sizeof(fe), B,
                             p.tmp, false, c));
    } else {
      RUN_ON(c, PC_NTT, ntt_launch_count(ilog2(NL), m),
             ntt_launch(p.tables(ilog2(NL)), a, m, p.cw[nci], p.tmp, false, c));
    }
    off_root[iter + 1] = off;
    if (go) GBZ_CUDA(cudaEventRecord(p.ev_commit[iter + 1], c));
    // queries of iteration t on q: they open the codeword of commit t,
    // record this iteration's round messages and check K against them
    const int depth = ilog2(L / 4);
    QueryArgs qa{};
    qa.st = st;
    qa.cws = cw_s[cwi];
    qa.ps = p.bs_wpart;
    qa.trs = trs;
    qa.cw = p.cw[cwi];
    qa.L = L;
    qa.l = l;
    qa.partial0 = part0;
    qa.partial1 = part1;
    qa.blocks = blocks;
    qa.tr = tr;
    qa.off_poly[0] = op;
    qa.off_chal[0] = oc;
    qa.off_poly[1] = op1;
    qa.off_chal[1] = oc1;
    qa.off_root = off_root[iter];
    qa.u = slots;
    qa.us = p.bs_ub;
    qa.base = ua.base[iter];
    qa.off_q = lay.rec(T_WHIR_QUERIES, l, 4);
    qa.off_rep = lay.rec(T_WHIR_REPLIES, l * kWhirK, 16);
    qa.off_ans = lay.rec(T_WHIR_ANSWERS, l, 16);
    qa.off_path = lay.rec(T_WHIR_PATHS, l * depth, 32);
    qa.off_comb = lay.rec(T_WHIR_COMBINE, l, 16);
    qa.off_K = lay.rec(T_WHIR_K, 1, 16);
    if (go) {
      const NttTables &told = p.tables(ilog2(L));
      qa.inv_lo = told.lo_inv;
      qa.inv_hi = told.hi_inv;
      const fe om_inv = finv(root_of_unity(ilog2(L)));
      qa.step0 = fpow(om_inv, L / kWhirK);
      qa.len_inv = finv(fe_make(kWhirK, 0));
      // the codeword it opens, and this iteration's round messages (for
      // iteration 0 also K = v1[0], set before on s)
      if (iter > 0 || part == PART_ALL) GBZ_CUDA(cudaStreamWaitEvent(q, p.ev_commit[iter], 0));
      GBZ_CUDA(cudaStreamWaitEvent(q, p.ev_fold[iter], 0));
    }
    // depth >= 2: every queried codeword has 16+ entries
    const uint64_t hashes = (uint64_t)l * depth;
    if (hashes == 0) throw ArgError("prover: empty authentication paths");
    RUN_ON(q, PC_QUERY, 1,
           launch_kernel(k_whir_open, dim3((unsigned)(2 + (hashes + kOpenThreads - 1) / kOpenThreads), B),
                         kOpenThreads, 0, q, qa, iter));
    if (go) GBZ_CUDA(cudaEventRecord(p.ev_query[iter], q));
    // update_betas on s: b[j] += sum_i c_i omega_NL^{q_i j} is the forward
    // transform of a vector with l nonzeros.  When l * |b| exceeds a few
    // transform lengths, the sparse transform is cheaper than the direct
    // sums.  The query exponents q_i * (whir_k NL / L) are even (NL = L / 2),
    // so omega_NL^{2 q_i j} = omega_{NL/2}^{q_i j}: the sparse transform runs
    // at half the codeword length on the unscaled positions.
    static_assert(kWhirK == 4, "update_betas: exponent scale 2 assumes folding by 4 with NL = L / 2");
    if (update_betas_by_transform(l, m, NL / 2)) {
      // one sparse transform per proof of a batch
      RUN(PC_UPDATE_BETAS, 2 * B, for (int pb = 0; pb < B; pb++) {
        const UbSlots *u = reinterpret_cast<const UbSlots *>(reinterpret_cast<const char *>(slots) + p.bs_ub * pb);
        ntt_sparse_accumulate(p.tables(ilog2(NL) - 1), u->q2 + ua.base[iter], u->c + ua.base[iter], l,
                              reinterpret_cast<fe *>(reinterpret_cast<char *>(bd) + p.bs_v * pb), m,
                              reinterpret_cast<fe *>(reinterpret_cast<char *>(p.tmp2) + p.bs_tmp2 * pb), s, 1);
      });
    } else {
      RUN(PC_UPDATE_BETAS, 1,
          update_betas_powers_launch(bd, m, slots->w + ua.base[iter], slots->c + ua.base[iter], l,
                                     slots->pw + 32 * ua.base[iter], s, B, p.bs_v, p.bs_ub));
    }
    cwi = nci;
    L = NL;
    cur *= 2;
    iter++;
    if (m <= (uint64_t)kWhirK) break;
  }
  uint64_t off_poly = lay.rec(T_FINAL_POLY, (uint32_t)m, 16);
  uint64_t off_point = lay.rec(T_FINAL_POINT, ilog2(m), 16);
  uint64_t off_eval = lay.rec(T_FINAL_EVAL, 1, 16);
  {
    BStr fb;  // (arr, b, tr)
    fb.s[0] = ast;
    fb.s[1] = bst;
    fb.s[2] = trs;
    RUN(PC_PROTOCOL, 1, launch_kernel(k_final_b, B, 32, 0, s, st, a, b, (int)m, tr, off_poly, off_point, off_eval, fb));
  }
  // root of the last commitment (never opened) on the query stream
  if (go) GBZ_CUDA(cudaStreamWaitEvent(q, p.ev_commit[iter], 0));
  RUN_ON(q, PC_MERKLE, 1,
         launch_kernel(k_merkle_root_b, B, 32, 0, q, p.cw[cwi], cw_s[cwi], ilog2(L / 4), tr, trs, off_root[iter]));
  if (go) {  // join the commit and query chains
    GBZ_CUDA(cudaEventRecord(p.ev_root_tail, q));
    GBZ_CUDA(cudaStreamWaitEvent(s, p.ev_commit[iter], 0));
    GBZ_CUDA(cudaStreamWaitEvent(s, p.ev_root_tail, 0));
  }
#undef RUN
#undef RUN_ON
}

void Profiler::begin(int cat, cudaStream_t s) {
  auto &v = ev[cat];
  if (used[cat] == v.size()) {
    cudaEvent_t a, b;
    GBZ_CUDA(cudaEventCreate(&a));
    GBZ_CUDA(cudaEventCreate(&b));
    v.push_back({a, b});
  }
  GBZ_CUDA(cudaEventRecord(v[used[cat]].first, s));
  open_cat = cat;
}

void Profiler::end(cudaStream_t s) {
  auto &v = ev[open_cat];
  GBZ_CUDA(cudaEventRecord(v[used[open_cat]].second, s));
  used[open_cat]++;
  open_cat = -1;
}

void Profiler::read(double ms[PC_COUNT], int counts[PC_COUNT]) {
  for (int c = 0; c < PC_COUNT; c++) {
    double t = 0;
    for (size_t i = 0; i < used[c]; i++) {
      float x = 0;
      GBZ_CUDA(cudaEventSynchronize(ev[c][i].second));
      GBZ_CUDA(cudaEventElapsedTime(&x, ev[c][i].first, ev[c][i].second));
      t += x;
    }
    ms[c] = t;
    if (counts) counts[c] = (int)used[c];
  }
}

Profiler::~Profiler() {
  for (int c = 0; c < PC_COUNT; c++)
    for (auto &e : ev[c]) {
      cudaEventDestroy(e.first);
      cudaEventDestroy(e.second);
    }
}

namespace {
__global__ void k_set_seed(ProofState *st, uint32_t seed) {
  pdl_wait();
  if (threadIdx.x == 0) st->seed_in = seed;
}
struct SeedChunk {
  uint32_t v[64];
};
__global__ void k_set_seeds(ProofState *st, SeedChunk c, int count) {
  pdl_wait();
  if ((int)threadIdx.x < count) st[threadIdx.x].seed_in = c.v[threadIdx.x];
}
}  // namespace

void set_seed_launch(ProofPlan &p, uint32_t seed, cudaStream_t s) {
  launch_kernel(k_set_seed, 1, 32, 0, s, p.st, seed);
  GBZ_CUDA(cudaGetLastError());
}

void set_seeds_launch(ProofPlan &p, const uint32_t *seeds, int count, cudaStream_t s) {
  for (int o = 0; o < count; o += 64) {
    SeedChunk c{};
    const int k = std::min(64, count - o);
    for (int i = 0; i < k; i++) c.v[i] = seeds[o + i];
    launch_kernel(k_set_seeds, 1, 64, 0, s, p.st + o, c, k);
    GBZ_CUDA(cudaGetLastError());
  }
}

namespace {
// Captures one part of a proof on s.
cudaGraph_t capture_part(ProofPlan &p, const fe *w, uint32_t prng_seed, cudaStream_t s, ProofPart part) {
  GBZ_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  cudaGraph_t g = nullptr;
  try {
    enqueue_proof(p, w, prng_seed, s, false, false, nullptr, part);
  } catch (...) {
    cudaStreamEndCapture(s, &g);
    if (g) cudaGraphDestroy(g);
    throw;
  }
  GBZ_CUDA(cudaStreamEndCapture(s, &g));
  return g;
}

void graph_free(ProofGraph &g) {
  for (cudaGraphExec_t e : g.exec)
    if (e) cudaGraphExecDestroy(e);
  for (cudaGraph_t x : g.graph)
    if (x) cudaGraphDestroy(x);
}
}  // namespace

// A launch of a graph takes about 1 us a node before its critical chain gets
// going (63 nodes at 2^18, the evaluation point 45 us late).  Up to codewords
// of 2^kSplitLog the opening is a second graph, submitted while the sumcheck
// runs (2^10 124 -> 122 us, 2^18 324 -> 313, 2^20 equal); above, where the
// commitment outlasts the sumcheck, the opening's folds would wait for it
// (2^24 2641 -> 2670).
constexpr int kSplitLog = 22;

void launch_proof_graph(ProofPlan &p, const fe *w, uint32_t prng_seed, cudaStream_t s) {
  ProofGraph *g = nullptr;
  for (auto &e : p.graphs)
    if (e.w == w) g = &e;
  if (!g) {
    constexpr size_t kMaxGraphs = 4;
    if (p.graphs.size() >= kMaxGraphs) {  // drop the least recently used
      size_t lru = 0;
      for (size_t i = 1; i < p.graphs.size(); i++)
        if (p.graphs[i].last_use < p.graphs[lru].last_use) lru = i;
      GBZ_CUDA(cudaStreamSynchronize(s));
      graph_free(p.graphs[lru]);
      p.graphs.erase(p.graphs.begin() + lru);
    }
    const bool split = ilog2(p.L) <= kSplitLog;
    ProofGraph ng;
    ng.w = w;
    try {
      ng.graph[0] = capture_part(p, w, prng_seed, s, split ? PART_START : PART_ALL);
      if (split) ng.graph[1] = capture_part(p, w, prng_seed, s, PART_OPENING);
      // the k_init node carries the seed
      size_t count = 0;
      GBZ_CUDA(cudaGraphGetNodes(ng.graph[0], nullptr, &count));
      std::vector<cudaGraphNode_t> nodes(count);
      GBZ_CUDA(cudaGraphGetNodes(ng.graph[0], nodes.data(), &count));
      for (auto nd : nodes) {
        cudaGraphNodeType ty;
        GBZ_CUDA(cudaGraphNodeGetType(nd, &ty));
        if (ty != cudaGraphNodeTypeKernel) continue;
        cudaKernelNodeParams kp{};
        GBZ_CUDA(cudaGraphKernelNodeGetParams(nd, &kp));
        if (kp.func == reinterpret_cast<void *>(k_init)) {
          ng.init_node = nd;
          ng.init_params = kp;
          break;
        }
      }
      if (!ng.init_node) throw ArgError("prover graph: initial node not found");
      for (int k = 0; k < 2; k++)
        if (ng.graph[k]) GBZ_CUDA(cudaGraphInstantiate(&ng.exec[k], ng.graph[k], 0));
    } catch (...) {
      graph_free(ng);
      throw;
    }
    p.graphs.push_back(ng);
    g = &p.graphs.back();
  }
  g->last_use = ++p.graph_tick;
  ProofState *st = p.st;
  uint32_t seed_v = prng_seed;
  int flag = 0;
  void *args[3] = {&st, &seed_v, &flag};
  cudaKernelNodeParams kp = g->init_params;
  kp.kernelParams = args;
  kp.extra = nullptr;
  GBZ_CUDA(cudaGraphExecKernelNodeSetParams(g->exec[0], g->init_node, &kp));
  GBZ_CUDA(cudaGraphLaunch(g->exec[0], s));
  if (g->exec[1]) GBZ_CUDA(cudaGraphLaunch(g->exec[1], s));
}

uint64_t plan_bytes(int logn, int rate, int batch) {
  const uint64_t n = 1ull << logn, L = n * (uint64_t)rate;
  uint64_t b = sizeof(fe) * (n + L + L / 2 + L + L / 2 + 5 * (n / 2) + n);
  b += sizeof(fe) * (4 * (uint64_t)sc_blocks(n / 4) + whir_partials(n) + kUpdateBetasScratch) + sizeof(ProofState);
  b *= (uint64_t)batch;
  b += 64ull << 20;  // transcripts, twiddle tables and allocation granularity (upper bound)
  b += (uint64_t)batch << 20;
  return b;
}

uint32_t plan_error_flags(ProofPlan &p, cudaStream_t s) {
  uint32_t e = 0;
  GBZ_CUDA(cudaMemcpyAsync(&e, &p.st->error, 4, cudaMemcpyDeviceToHost, s));
  GBZ_CUDA(cudaStreamSynchronize(s));
  return e;
}

}  // namespace gbz
