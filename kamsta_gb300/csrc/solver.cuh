// solver.cuh -- host-side driver of the GB300 MSF solver (C++ over CUDA).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <functional>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

#include "../../include/kamsta_gpu.h"
#include "common.cuh"

namespace kamsta {

// Grow-only device arena.  A solve carves its buffers from it; the memory
// stays with the context between calls (the reference's analogue is the
// per-call std::vector scratch of boruvka3, re-created every call).
struct Arena {
  char* base = nullptr;
  size_t cap = 0;
  size_t off = 0;
  cudaError_t reserve(size_t bytes);
  void release();
  void reset() { off = 0; }
  template <typename T>
  T* take(size_t count) {
    const size_t bytes = (count * sizeof(T) + 255) & ~static_cast<size_t>(255);
    if (off + bytes > cap) return nullptr;
    T* p = reinterpret_cast<T*>(base + off);
    off += bytes;
    return p;
  }
};

// One block of device memory that a context keeps for its solves' scratch and
// divides on the host (best fit, neighbours merged).  The stream-ordered pool
// serves the same requests, but a solve's lists differ in size, and the pool
// then remaps physical memory for nearly each of them: 130 to 430 us of host
// time per list of a few hundred MB (G(n,m) 2^26/2^30: 23.0 -> 20.3 ms per solve
// with the heap).
// A call opens the heap for its stream (HeapScope): blocks taken and given
// back inside are reused in that stream's order only.  The block grows
// between calls to what the largest call so far had live at once, with some
// room so that it grows rarely.  It comes from the pool, which still holds what
// the call before had taken there (a context's second call on G(n,m)
// 2^26/2^30: 39.0 ms with a block of its own memory, 21.6 so; later ones
// 20.1).  The first call has none: nothing says how large it should be.
struct Heap {
  struct Region {
    size_t off, size;
  };
  char* base = nullptr;
  size_t cap = 0;
  size_t want = 0;                 // size the largest call needed
  size_t live = 0;                 // bytes out, here and in the pool, this call
  std::vector<Region> free_list;   // by offset
  std::vector<Region> used;
  std::vector<std::pair<void*, size_t>> pooled;  // this call's blocks from the pool
  cudaStream_t st = nullptr;       // the open call's stream
  int depth = 0;                   // > 0: open
  uint64_t too_large = ~0ull;      // calls of this size do not fit beside it
  bool off = false;                // the open call runs without it (heap_call)
  void* take(size_t bytes);
  bool give(void* p);              // false: not from here
  size_t room(cudaStream_t on) const {  // largest block for the open call's stream
    size_t most = 0;
    if (depth > 0 && on == st)
      for (const Region& r : free_list) most = std::max(most, r.size);
    return most;
  }
};

// Per-kernel counter block in device memory (zeroed before each round).
struct DevCounters {
  unsigned long long cnt[8];
  unsigned long long weight;
  uint32_t ticket;
  uint32_t err;
  uint32_t pad[12];
};
static_assert(sizeof(DevCounters) == 128, "counter block size");

enum CounterSlot : int { kCVertex = 0, kCEdge = 1, kCRep = 2, kCMisc = 3, kCSlots = 4 };
constexpr uint32_t kSampleCap = 4096;
constexpr uint32_t kSampleWords = kSampleCap + 16;  // the sample, then its counters
constexpr int kTimerEvents = 64;
constexpr uint32_t kCountWords = 3 * 1024;  // segment counts of a pass's outputs
constexpr size_t kHostState = 1024;  // bytes of kamsta_ctx::h_state
constexpr int kInputPieces = 16;  // host input copied in this many pieces
constexpr uint32_t kFailKinds = 3;  // KAMSTA_FAIL_*

}  // namespace kamsta

struct kamsta_ctx {
  int device = 0;
  cudaStream_t stream = nullptr;
  cudaStream_t aux = nullptr;    // second stream: small graphs of a batch wave
  cudaStream_t small_st[2] = {};  // size classes of those graphs beside it
  cudaEvent_t ev_fork = nullptr, ev_join = nullptr, ev_small[3] = {};
  // batch tuning (kamsta_batch_autotune); 0 = built-in default
  uint32_t tune_small_threads = 0;  // CTA size of the persistent small-graph kernel
  uint32_t tune_small_max_n = 0;    // largest n taken by that kernel
  // CTAs per SM of the small-graph kernels: tiny, compact by CTA size (256,
  // 512, 1024), full; 0 = not asked yet
  int small_per_sm[5] = {};
  bool found_ready = false;  // small::found_setup has run
  // single-graph tiles (kamsta_autotune_tiles); 0 = built-in default
  uint32_t tune_dir_items = 0;      // entries per thread of the first pass
  uint32_t tune_seg_items = 0;      // records per thread of the list passes
  kamsta::Arena fixed;   // vertex arrays and look-back words
  cudaMemPool_t pool = nullptr;  // scratch outside a call's heap (stream-ordered, cached)
  kamsta::Heap heap;             // scratch of the solves
  kamsta::DevCounters* d_counters = nullptr;  // kCSlots blocks
  uint32_t* d_samples = nullptr;               // weight samples (kSampleCap)
  uint32_t* d_err = nullptr;
  kamsta::DevCounters* h_counters = nullptr;  // pinned mirror
  uint32_t* h_err = nullptr;
  uint32_t* h_samples = nullptr;  // pinned: the sorted samples
  uint32_t* h_counts = nullptr;   // pinned: a pass's segment counts
  void* h_state = nullptr;        // pinned: head of the cooperative solve's state
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaEvent_t tev[kamsta::kTimerEvents] = {};  // per-phase timing events
  kamsta::Arena io;      // host-buffer entry points: device copies of in/out
  cudaEvent_t piece_ev[kamsta::kInputPieces] = {};  // host input piece k is on the device
  cudaEvent_t ev_early = nullptr;  // the first round's forest edges are written
  uint64_t mem_limit = 0;          // kamsta_ctx_set_memory_limit; 0 = none
  int solves = 0;        // nested InFlight scopes (under mu)
  uint32_t fail_in[kamsta::kFailKinds] = {};  // kamsta_ctx_fail_nth; 0 = off
  std::mutex mu;
};

namespace kamsta {

struct SolveOut {
  uint64_t count = 0;
  uint64_t weight = 0;
};

// Which reference entry point a call mirrors.
enum class Algo { kBoruvka, kFilterBoruvka };

// The host-buffer entry point overlaps its copies with the solve.  The input
// arrives in pieces on copy_stream: entries [0, piece_end[k]) are on the
// device once piece_ev[k] has completed (the events are recorded in order).
// The first pass starts on each chunk as soon as it has landed, and the
// weight sample of the class plan is drawn from the first piece.  When
// host_out is set, the forest edges that the first round writes directly
// are copied back to host_out[0, early) on copy_stream while the rest of the
// solve runs.
struct HostIo {
  int pieces = 0;
  uint64_t piece_end[kInputPieces] = {};
  const cudaEvent_t* piece_ev = nullptr;
  cudaStream_t copy_stream = nullptr;
  kamsta_wedge* host_out = nullptr;
  cudaEvent_t ev_early = nullptr;
  uint64_t early = 0;  // out
};

// Counts the contexts of this process that are solving on a device.  A
// cooperative launch takes every SM at once: it waits until the kernels of
// the other solves have drained, and they wait for it.  So a solve takes the
// cooperative rounds while at most one other context is solving, and the
// host-driven ones, whose kernels of several streams run side by side, beyond.
// Serving with 4 workers, p50 / p99 ms at 4000, 12000 and 22000 requests/s:
// always cooperative 0.35/2.0, 1.9/9.0, 6.8/27.7; only when alone 0.68/4.1,
// 1.75/6.1, 4.2/17.3; so 0.41/2.9, 1.75/6.1, 4.1/16.7.
class InFlight {
 public:
  explicit InFlight(kamsta_ctx* ctx);
  ~InFlight();
  InFlight(const InFlight&) = delete;
  InFlight& operator=(const InFlight&) = delete;
  static bool few(int device);

 private:
  kamsta_ctx* ctx_;
};

// A union of graphs read in place instead of from one array: device table in
// entry order and, per graph, whether an id was out of range (set by the
// solve).  m_directed counts the unused entries between graphs too.  Forest
// bitmap only; host-driven rounds only.
struct UnionIn {
  const UnionGraph* graphs = nullptr;
  uint32_t count = 0;
  uint32_t* err = nullptr;
};
// The smallest union read in place.  The cooperative rounds end here: they
// read an array, and win more than the copy costs (0.14 ms at 2^25 entries).
// Above, the copy only costs.
constexpr uint64_t kUnionMinMd = 1ull << 25;

// Solves one graph whose directed, (src,dst)-sorted input lies in device
// memory (or, with `uni`, in the graphs of a union; d_in is null then).
// Writes the forest to d_out (device, capacity >= n-1), or, when
// d_forest_bits is given (zeroed, one bit per input entry), sets the bit of
// the src<dst input copy of every forest edge instead (out->weight is then
// 0: the caller reads the marked entries).
kamsta_status solve_device(kamsta_ctx* ctx, Algo algo, const kamsta_wedge* d_in,
                           uint64_t m_directed, uint32_t n, const kamsta_cfg& cfg,
                           kamsta_wedge* d_out, SolveOut* out, kamsta_stats* st,
                           cudaStream_t stream, uint32_t* d_forest_bits = nullptr,
                           HostIo* io = nullptr, const UnionIn* uni = nullptr);

// Whether the operation of this kind that is about to run is the one to fail.
inline bool fail_now(kamsta_ctx* ctx, uint32_t what) {
  uint32_t& in = ctx->fail_in[what];
  return in != 0 && --in == 0;
}

void set_error(const std::string& msg);
kamsta_status cuda_status(cudaError_t e, const char* what);
// Device memory of a context under its limit (mem_limit): stream-ordered
// scratch from its pool and the growth of its arenas.  Going over the limit
// fails like a device allocation (cudaErrorMemoryAllocation -> KAMSTA_E_OOM).
uint64_t ctx_device_bytes(const kamsta_ctx* ctx);
// Scratch for work on `st`: from the heap while it is open for that stream,
// else from the pool.  ctx_free takes either back.
cudaError_t ctx_alloc(kamsta_ctx* ctx, void** p, size_t bytes, cudaStream_t st);
void ctx_free(kamsta_ctx* ctx, void* p, cudaStream_t st);
// Opens the context's heap for work on one stream until the scope ends; the
// outermost scope grows it first and, unless finished() said that the stream
// has been waited for, waits for the stream last.
class HeapScope {
 public:
  HeapScope(kamsta_ctx* ctx, cudaStream_t st);
  ~HeapScope();
  void finished() { synced_ = true; }

 private:
  kamsta_ctx* ctx_;
  cudaStream_t st_;
  bool opened_ = false, synced_ = false;
};
void heap_release(kamsta_ctx* ctx);
// Runs a call's work; when it runs out of memory while the heap holds some, the
// block is given back and the work (again = true) runs once more without one.
// bytes: an estimate of the call's device memory, for telling calls apart.
kamsta_status heap_call(kamsta_ctx* ctx, uint64_t bytes,
                        const std::function<kamsta_status(bool again)>& work);
cudaError_t ctx_reserve(kamsta_ctx* ctx, Arena& a, size_t bytes);

}  // namespace kamsta
