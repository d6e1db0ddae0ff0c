// The library context (gbz_ctx of include/gbz.h) and the helpers every
// translation unit with extern "C" entry points uses: device guard, error
// mapping, argument checks and host/device views of caller buffers.
#pragma once
#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "../../include/gbz.h"
#include "gbz_prover.cuh"
#include "gbz_pcs_leader.cuh"
#include "gbz_rounds.cuh"
#include "gbz_sched.cuh"

using namespace gbz;

// Device buffers of a commitment (gbz_pcs): rows, codewords, trees, roots.
struct PcsBuffers {
  void *p[4] = {nullptr, nullptr, nullptr, nullptr};
  uint64_t bytes[4] = {0, 0, 0, 0};
  uint64_t total() const { return bytes[0] + bytes[1] + bytes[2] + bytes[3]; }
  void free() {
    for (void *&q : p) {
      cudaFree(q);
      q = nullptr;
    }
  }
};

// The buffers of the last commitment that was freed, kept for the next one of
// the same sizes on the same stream: cudaMalloc and cudaFree of the 4.5 GB of
// a 16 x 2^24 commitment took 5.3 ms of a 27.4 ms commit and opening.  One
// set of at most a sixteenth of the device; anything else is freed at once.
// A set is only kept when every call on it ran on this stream, so the next
// commitment's work is ordered after it without a synchronisation.  The
// handle shares ownership: it may be freed by another thread, or after the
// context, which closes the store.
struct SpareBuffers {
  std::mutex mu;
  int device = 0;
  uint64_t limit = 0;  // a sixteenth of the device's memory
  bool closed = false;
  cudaStream_t stream = nullptr;
  PcsBuffers set;

  // true: b holds the kept set; otherwise nothing is kept any more
  bool take(PcsBuffers &b, cudaStream_t s) {
    std::lock_guard<std::mutex> lk(mu);
    if (!set.p[0]) return false;
    bool same = stream == s;
    for (int i = 0; i < 4; i++) same = same && set.bytes[i] == b.bytes[i];
    if (same) b = set;
    else set.free();
    set = PcsBuffers();
    return same;
  }
  void give(PcsBuffers &b, cudaStream_t s) {
    std::lock_guard<std::mutex> lk(mu);
    if (closed || b.total() > limit) {
      b.free();
      return;
    }
    set.free();
    set = b;
    stream = s;
  }
  uint64_t release(bool close = false) {
    std::lock_guard<std::mutex> lk(mu);
    const uint64_t n = set.p[0] ? set.total() : 0;
    set.free();
    set = PcsBuffers();
    closed = closed || close;
    return n;
  }
};
std::shared_ptr<SpareBuffers> make_spare_buffers(int device);

struct gbz_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::string last_error;
  std::map<int, std::pair<void *, uint64_t>> scratch;
  // Scratch of calls that make the same sequence of allocations for the
  // same shape (the N-party openings): keyed by the shape, buffer k of a
  // pool serves the call's k-th allocation.
  std::map<std::string, std::vector<std::pair<void *, uint64_t>>> pools;
  std::shared_ptr<SpareBuffers> spare;
  std::map<int, NttTables> ntt;
  std::map<std::pair<int, int>, std::unique_ptr<ProofPlan>> plans;
  ProofState *st = nullptr;
  fe *ub_scratch = nullptr;
  bool profiling = false;
  std::map<std::pair<int, int>, std::unique_ptr<Profiler>> profilers;
  std::unique_ptr<Scheduler> sched;
  bool graphs = true;  // gbz_prove replays captured graphs (gbz_set_graphs)
  bool group = true;   // gbz_prove_batch: proofs of one shape share launches (gbz_sched_set_grouping)
  SideStream side;     // second stream of the party sumcheck (created on first use)
  TailStreams tail;    // streams of the PCS leader's tail (created on first use)

  const SideStream &side_stream() {
    if (!side.stream) {
      GBZ_CUDA(cudaStreamCreateWithFlags(&side.stream, cudaStreamNonBlocking));
      GBZ_CUDA(cudaEventCreateWithFlags(&side.fork, cudaEventDisableTiming));
      GBZ_CUDA(cudaEventCreateWithFlags(&side.join, cudaEventDisableTiming));
    }
    return side;
  }

  const TailStreams &tail_streams() {
    for (auto &t : tail.s)
      if (!t) GBZ_CUDA(cudaStreamCreateWithFlags(&t, cudaStreamNonBlocking));
    for (auto &e : tail.ready)
      if (!e) GBZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    for (auto &e : tail.done)
      if (!e) GBZ_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return tail;
  }

  void *buf(int slot, uint64_t bytes) {
    auto &e = scratch[slot];
    if (e.second < bytes) {
      if (e.first) GBZ_CUDA(cudaFree(e.first));
      e.first = nullptr;
      e.second = 0;
      GBZ_CUDA(device_malloc(&e.first, bytes ? bytes : 16));
      e.second = bytes;
    }
    return e.first;
  }
  NttTables &tables(int lg) {
    auto it = ntt.find(lg);
    if (it != ntt.end()) return it->second;
    NttTables t;
    ntt_tables_build(t, lg);
    return ntt.emplace(lg, t).first->second;
  }
};

namespace gbz_api {

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
    if (prev != dev) GBZ_CUDA(cudaSetDevice(dev));
  }
  ~DeviceGuard() {
    int cur;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

// Device buffers of one call: allocated per call and freed at its end, or,
// with a pool, the pool's k-th buffer for the call's k-th allocation (a
// larger or new one replaces it when it is too small).
struct OpenBufs {
  std::vector<void *> owned;
  std::vector<std::pair<void *, uint64_t>> *pool = nullptr;
  size_t next = 0;
  ~OpenBufs() {
    for (void *p : owned) cudaFree(p);
  }
  template <typename T>
  T *alloc(uint64_t count) {
    const uint64_t bytes = std::max<uint64_t>(count * sizeof(T), 16);
    if (pool) {
      auto &P = *pool;
      if (next < P.size() && P[next].second >= bytes) return (T *)P[next++].first;
      void *p = nullptr;
      GBZ_CUDA(device_malloc(&p, bytes));
      if (next < P.size()) {
        cudaFree(P[next].first);
        P[next] = {p, bytes};
      } else {
        P.push_back({p, bytes});
      }
      next++;
      return (T *)p;
    }
    void *p = nullptr;
    GBZ_CUDA(device_malloc(&p, bytes));
    owned.push_back(p);
    return (T *)p;
  }
};

inline gbz_status fail(gbz_ctx *ctx, gbz_status code, const std::string &msg) {
  if (ctx) ctx->last_error = msg;
  return code;
}

#define API_BEGIN(ctx)                                    \
  if (!(ctx)) return GBZ_EINVAL;                          \
  try {                                                   \
    DeviceGuard guard_((ctx)->device);
#define API_END(ctx)                                                                    \
  }                                                                                     \
  catch (const ArgError &e) {                                                           \
    return fail(ctx, GBZ_EINVAL, e.what);                                               \
  }                                                                                     \
  catch (const CudaError &e) {                                                          \
    return fail(ctx, e.err == cudaErrorMemoryAllocation ? GBZ_ENOMEM : GBZ_ECUDA, e.what); \
  }                                                                                     \
  catch (const std::bad_alloc &) {                                                      \
    return fail(ctx, GBZ_ENOMEM, "host allocation failed");                              \
  }                                                                                     \
  return GBZ_OK;

inline void check_mem(int mem) {
  if (mem != GBZ_MEM_HOST && mem != GBZ_MEM_DEVICE) throw ArgError("mem must be GBZ_MEM_HOST or GBZ_MEM_DEVICE");
}
inline void need(const void *p, const char *what) {
  if (!p) throw ArgError(std::string("null pointer: ") + what);
}
inline void check_pow2(uint64_t n, const char *what) {
  if (!is_pow2(n)) throw ArgError(std::string(what) + " must be a power of two");
}

// Device view of a caller buffer: the pointer itself (device memory) or a
// scratch copy (host memory), copied in when `in`.
template <typename T>
T *dev_view(gbz_ctx *ctx, int slot, T *p, uint64_t bytes, int mem, bool in) {
  if (mem == GBZ_MEM_DEVICE) return p;
  T *d = (T *)ctx->buf(slot, bytes);
  if (in && bytes) GBZ_CUDA(cudaMemcpyAsync((void *)d, (const void *)p, bytes, cudaMemcpyHostToDevice, ctx->stream));
  return d;
}
// Whether kernels can load the elements where they are: 16 bytes at a time.
inline bool fe_aligned(const void *p) { return ((uintptr_t)p & 15) == 0; }
template <typename T>
void copy_out(gbz_ctx *ctx, T *host, const T *dev, uint64_t bytes, int mem) {
  if (mem == GBZ_MEM_DEVICE || !bytes) return;
  GBZ_CUDA(cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, ctx->stream));
}
inline void finish(gbz_ctx *ctx, int mem) {
  if (mem == GBZ_MEM_HOST) GBZ_CUDA(cudaStreamSynchronize(ctx->stream));
}

// coPCS Encode (coPCS.cpp:131-147) of nrows rows of 2^logrow entries
// (device) into codewords of rate * 2^logrow entries (device), on the
// context's stream; scratch slot 2 holds the intermediate.
void encode_rows_device(gbz_ctx *ctx, const fe *drows, int nrows, int logrow, int rate, int log_rate_offset,
                        fe *dout);

}  // namespace gbz_api
