// rounds_coop.cuh -- all Boruvka rounds of one contraction in one cooperative
// launch.
//
// The multi-kernel rounds (kernels.cuh) cost four launches and one host read
// each: about 80 us per round whatever its size, which is most of the time of
// a graph of up to a few million edges.  Here one grid (one CTA per SM at
// most) runs every round itself; the phases of a round are separated by grid
// barriers, and nothing returns to the host until the contraction is done.
// The steps and their results are those of kernels.cuh: the same hooks, the
// same dense ids in vertex order, the same forest order.
//
//   optional prologue   relabel the source (a class list, or the directed
//                       input between two weights) by the component labels D
//   per round           hook | renumber + forest edges | label walk |
//                       relabel, drop, compact, next minimum
//   optional finalize   compose the labels, new representatives, P and D
//   optional emit       forest edges (or the batch's bitmap)
//
// What bounds it: with everything in L2 a round is a chain of dependent
// gathers and barriers, so the design cuts both.  A round over at most
// kTinyN vertices does not divide its vertex work: every CTA repeats it in
// its own shared memory, where the label map then also stays, and the only
// grid barrier left is the one after the edge phase.  Measured on one GB300,
// G(2^16, 2^20) without preprocessing, us: a barrier 1.2 to 2; the first two
// rounds' hook 3.5, renumbering 3.5, walk 2, edge phase 15 and 11 (10^6
// records: uncoalesced label and minimum accesses, about four L1 wavefronts
// per record); a tiny round 9 (vertices 3, edges 6).  The whole call 590 us
// host-driven, 214 cooperative; RGG-2D 10^6 with preprocessing 1510 / 485.
//
// Every wait is bounded: a barrier that runs out sets kErrSpin and all CTAs
// leave the kernel.  Data that other SMs write is only read after a barrier
// (whose acquire drops stale L1 lines), never through the read-only path.
#pragma once
#include <cstddef>

#include "kernels.cuh"

namespace kamsta {
namespace coop {

constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 4;            // records (vertices) per thread and step
constexpr uint32_t kTinyN = 4096;    // vertices of a round every CTA repeats
// The edge phase runs in groups of 8 warps with a segment each: their tiles
// (load, labels, rank, minima: a chain of about 3 us) overlap, where one tile
// of the whole CTA at a time left the SM waiting on that chain.
constexpr int kGroupWarps = 8;
constexpr int kGroup = kGroupWarps * 32;
constexpr int kGroups = kThreads / kGroup;
static_assert(kItems * kGroupWarps == 32, "a warp scans a tile's rows in one step");
constexpr uint32_t kMaxLaunch = 48;  // launches of one solve
constexpr uint32_t kBarStride = 32;  // u32 words: one barrier word per 128 bytes
static_assert(kMaxSeg <= kThreads, "one thread per segment builds the prefix");

// Device state of a solve, zeroed before its first launch.
struct State {
  unsigned long long msf_count;     // forest edges found
  unsigned long long direct_count;  // of those, written to the output directly
  unsigned long long weight;        // weight of the edges written so far
  unsigned long long sum_m, sum_n;  // records / vertices over all rounds
  uint32_t nreps;                   // dense labels in use
  uint32_t rounds, levels;
  uint32_t vsel;  // representatives are in Vn (1) or V (0)
  // the last launch's rounds: vertices before each, and left after the last
  uint32_t last_rounds;
  uint32_t size[kMaxRounds + 1];
  // error bits per launch: a launch that follows an error does nothing, and
  // all of its CTAs must see the same, so no launch looks at its own word
  uint32_t errs[kMaxLaunch];
  uint32_t bars[kMaxLaunch * kBarStride];
};
constexpr size_t kStateHead = offsetof(State, bars);  // what the host reads

enum class Emit : uint32_t { kNone, kEdges, kBits };

struct Args {
  // source list; null: the directed input (prologue only)
  const Rec* src;
  const uint32_t* src_count;
  uint64_t src_cap;
  uint32_t src_nseg;
  const uint32_t* in;
  uint32_t md;
  uint32_t wmin, wmax;
  uint32_t prologue;  // relabel the source by D first
  // two list buffers, kGroups segments of cap records per CTA, and their counts
  Rec* buf[2];
  uint32_t* cnt[2];
  uint32_t cap;
  uint32_t n;
  uint32_t first;   // no state yet: nr0 labels, msf0 forest edges, V as given
  uint32_t nr0;
  // earlier rounds of the same contraction (host-driven): map and
  // representative words they used, and their last representatives (or null)
  uint32_t roff0, ooff0;
  const uint32_t* orig0;
  uint64_t msf0;
  uint32_t direct;  // round 0: minima keyed by partner, edges to out
  uint32_t finalize;
  Emit emit;
  uint32_t *P, *D, *V, *Vn, *dense_of, *parent, *msfoid, *msf, *R, *orig;
  uint64_t *minA, *minB, *tiny;  // tiny: 3 * kTinyN words
  uint32_t* vcnt;                // 2 per CTA
  uint32_t *out, *bits;
  unsigned long long* weight;    // of the edges written to out
  uint32_t launch;
  State* st;
  const uint32_t* pass_err;  // error word of the passes before
  uint32_t* err;             // this launch's word in st->errs
};

struct Shared {
  uint64_t min64[kTinyN];   // a tiny round's minima, then the next round's
  uint32_t par[kTinyN];
  uint32_t map[kTinyN];
  uint32_t pre[kMaxSeg + 1];
  uint32_t rank[2 * kItems * kWarps];
  uint32_t rows[kGroups][2][32];
  uint32_t wsum[kWarps];
  uint32_t tot[2], base[2], sum[2];
  uint32_t ok;
};

// All CTAs have arrived, and what they wrote is visible.  False when the
// bounded wait ran out.
__device__ __forceinline__ bool grid_sync(Shared& s, uint32_t* bar, uint32_t& goal,
                                          uint32_t* err) {
  __syncthreads();
  if (gridDim.x == 1) return true;
  goal += gridDim.x;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
    uint32_t v, i = 0;
    for (;; ++i) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(bar) : "memory");
      if (v >= goal || i > kSpinCap) break;
    }
    if (v < goal) atomicOr(err, kErrSpin);
    s.ok = v >= goal;
  }
  __syncthreads();
  return s.ok != 0;
}

// pre[x] = records in segments < x; returns the total.
__device__ __forceinline__ uint32_t seg_prefix32(Shared& s, const uint32_t* count, uint32_t nseg) {
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
  const uint32_t c = threadIdx.x < nseg ? count[threadIdx.x] : 0u;
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= static_cast<uint32_t>(o)) incl += y;
  }
  if (lane == 31) s.wsum[warp] = incl;
  __syncthreads();
  uint32_t wv = s.wsum[lane], wi = wv;  // kWarps == 32: every warp scans the sums
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, wi, o);
    if (lane >= static_cast<uint32_t>(o)) wi += y;
  }
  const uint32_t wpre = __shfl_sync(kFull, wi - wv, warp);
  const uint32_t total = __shfl_sync(kFull, wi, 31);
  if (threadIdx.x <= nseg && threadIdx.x <= static_cast<uint32_t>(kMaxSeg))
    s.pre[threadIdx.x] = wpre + incl - c;
  if (threadIdx.x == 0) s.pre[nseg] = total;
  __syncthreads();
  return total;
}

__device__ __forceinline__ uint32_t seg_of(const uint32_t* pre, uint32_t nseg, uint32_t x) {
  uint32_t lo = 0, hi = nseg;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (pre[mid] <= x) lo = mid; else hi = mid;
  }
  return lo;
}

struct List {  // a segmented list
  const Rec* base;
  uint32_t nseg;
  uint64_t cap;
};

// Next-round minimum of a kept record.  smin (labels < smin_n) is the CTA's
// own array: with few labels every CTA would otherwise update the same words.
__device__ __forceinline__ void feed_min(uint64_t* minv, uint64_t* smin, uint32_t x, uint64_t v) {
  if (smin) {
    unsigned long long* p = reinterpret_cast<unsigned long long*>(smin + x);
    if (v < *reinterpret_cast<volatile unsigned long long*>(p))
      atomicMin(p, static_cast<unsigned long long>(v));
  } else if (v < ld_weak(&minv[x])) {
    red_min(&minv[x], v);
  }
}

// Edge phase: group q of the grid takes items [q * chunk, ...) of the m
// items, relabels them, and writes those whose labels differ to its segment
// of `out`, in order; the records feed the next minimum.  Items come from a
// segmented list (positions through s.pre) or, DIRECTED, from the input's
// src < dst entries between wmin and wmax.  label(x) maps a vertex; labels
// are < nlab.
template <bool DIRECTED, typename Label>
__device__ void edge_phase(Shared& s, const Args& a, const List& L, uint32_t m, Label label,
                           uint32_t nlab, Rec* out, uint32_t* cnt, uint64_t* minv,
                           uint64_t* smin) {
  const uint32_t lane = lane_id(), grp = threadIdx.x / kGroup, gt = threadIdx.x % kGroup;
  const uint32_t gw = gt >> 5, lt = lanemask_lt();
  const uint32_t nq = gridDim.x * kGroups, q = blockIdx.x * kGroups + grp;
  const uint32_t chunk = (m + nq - 1) / nq;
  const uint32_t lo =
      static_cast<uint32_t>(min(static_cast<uint64_t>(m), static_cast<uint64_t>(q) * chunk));
  const uint32_t hi =
      static_cast<uint32_t>(min(static_cast<uint64_t>(m), static_cast<uint64_t>(lo) + chunk));
  const uint64_t seg0 = static_cast<uint64_t>(q) * a.cap;
  uint32_t run = 0, flip = 0;
  uint32_t sg = 0;
  if (!DIRECTED && lo < hi) sg = seg_of(s.pre, L.nseg, lo);
  for (uint32_t t0 = lo; t0 < hi; t0 += kItems * kGroup, flip ^= 1) {
    Rec r[kItems];
    bool keep[kItems];
    if (!DIRECTED)
      while (t0 >= s.pre[sg + 1]) ++sg;  // the segment of the tile's first item
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const uint32_t x = t0 + j * kGroup + gt;
      keep[j] = x < hi;
      r[j] = Rec{0, 0, 0, 0};
      if (!keep[j]) continue;
      if (DIRECTED) {
        const uint32_t* e = a.in + 3ull * x;
        r[j].a = e[0];
        r[j].b = e[1];
        r[j].w = e[2];
        r[j].oid = x;
      } else {
        // nearly always in the tile's first segment or the one after it
        uint32_t g = sg;
        if (x >= s.pre[g + 1]) {
          ++g;
          if (x >= s.pre[g + 1]) g = seg_of(s.pre, L.nseg, x);
        }
        const uint4 v = *reinterpret_cast<const uint4*>(L.base + g * L.cap + (x - s.pre[g]));
        r[j] = Rec{v.x, v.y, v.z, v.w};
      }
    }
    uint32_t la[kItems], lb[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      if (DIRECTED)
        keep[j] = keep[j] && r[j].a < r[j].b && r[j].b < a.n && r[j].w >= a.wmin &&
                  r[j].w <= a.wmax;
      la[j] = lb[j] = 0;
      if (!keep[j]) continue;
      la[j] = label(r[j].a);
      lb[j] = label(r[j].b);
    }
    // stable ranks: row (j, warp) in input order, 32 rows per tile
    uint32_t* rows = s.rows[grp][flip];
    uint32_t bal[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      // a finished vertex (kNone) has no edge left in a consistent input
      keep[j] = keep[j] && la[j] != lb[j] && max(la[j], lb[j]) < nlab;
      bal[j] = __ballot_sync(kFull, keep[j]);
      if (lane == 0) rows[j * kGroupWarps + gw] = __popc(bal[j]);
    }
    asm volatile("bar.sync %0, %1;" ::"r"(grp + 1), "n"(kGroup) : "memory");
    const uint32_t c = rows[lane];
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, incl, o);
      if (lane >= static_cast<uint32_t>(o)) incl += y;
    }
    const uint32_t excl = incl - c;
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const uint32_t base = __shfl_sync(kFull, excl, j * kGroupWarps + gw);
      if (!keep[j]) continue;
      const uint32_t k = run + base + __popc(bal[j] & lt);
      if (k >= a.cap) {
        atomicOr(a.err, kErrOverflow);
        continue;
      }
      *reinterpret_cast<uint4*>(out + seg0 + k) = make_uint4(la[j], lb[j], r[j].w, r[j].oid);
      const uint64_t v = (static_cast<uint64_t>(r[j].w) << 32) | (seg0 + k);
      feed_min(minv, smin, la[j], v);
      feed_min(minv, smin, lb[j], v);
    }
    run += __shfl_sync(kFull, incl, 31);
  }
  if (gt == 0) cnt[q] = min(run, a.cap);
}

// Vertex chunk of this CTA.
__device__ __forceinline__ void vertex_range(uint32_t n, uint32_t& lo, uint32_t& hi) {
  const uint32_t chunk = (n + gridDim.x - 1) / gridDim.x;
  lo = static_cast<uint32_t>(
      min(static_cast<uint64_t>(n), static_cast<uint64_t>(blockIdx.x) * chunk));
  hi = static_cast<uint32_t>(min(static_cast<uint64_t>(n), static_cast<uint64_t>(lo) + chunk));
}

// Sums c0 / c1 over the CTA into s.sum (one barrier before the result).
__device__ __forceinline__ void block_sum2(Shared& s, uint32_t c0, uint32_t c1) {
  c0 = warp_sum(c0);
  c1 = warp_sum(c1);
  if (threadIdx.x < 2) s.sum[threadIdx.x] = 0;
  __syncthreads();
  if (lane_id() == 0) {
    if (c0) atomicAdd(&s.sum[0], c0);
    if (c1) atomicAdd(&s.sum[1], c1);
  }
  __syncthreads();
}

// s.base = counts of the CTAs before this one, s.sum = counts of all CTAs.
__device__ __forceinline__ void cta_bases(Shared& s, const uint32_t* vcnt) {
  uint32_t b0 = 0, b1 = 0, t0 = 0, t1 = 0;
  __syncthreads();
  if (threadIdx.x < 32) {
    for (uint32_t c = threadIdx.x; c < gridDim.x; c += 32) {
      const uint32_t x0 = vcnt[2 * c], x1 = vcnt[2 * c + 1];
      t0 += x0;
      t1 += x1;
      if (c < blockIdx.x) {
        b0 += x0;
        b1 += x1;
      }
    }
    b0 = warp_sum(b0);
    b1 = warp_sum(b1);
    t0 = warp_sum(t0);
    t1 = warp_sum(t1);
    if (threadIdx.x == 0) {
      s.base[0] = b0;
      s.base[1] = b1;
      s.sum[0] = t0;
      s.sum[1] = t1;
    }
  }
  __syncthreads();
}

// Hook of this CTA's vertices (k_hook); leaves its counts of live roots and
// hooked vertices in vcnt.
__device__ void hook_phase(Shared& s, const Args& a, uint32_t n, const uint64_t* minv,
                           const Rec* list, bool direct) {
  uint32_t lo, hi, c0 = 0, c1 = 0;
  vertex_range(n, lo, hi);
  for (uint32_t base = lo; base < hi; base += kItems * kThreads) {
    uint64_t val[kItems], mu[kItems];
    Rec r[kItems];
    uint32_t u[kItems];
    bool live[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t v = base + k * kThreads + threadIdx.x;
      val[k] = v < hi ? minv[v] : kInf64;
      live[k] = val[k] != kInf64;
      r[k] = Rec{0, 0, 0, 0};
    }
    if (!direct) {
#pragma unroll
      for (int k = 0; k < kItems; ++k)
        if (live[k]) r[k] = list[static_cast<uint32_t>(val[k])];
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t v = base + k * kThreads + threadIdx.x;
      mu[k] = kInf64;
      u[k] = 0;
      if (!live[k]) continue;
      u[k] = direct ? static_cast<uint32_t>(val[k]) : r[k].a ^ r[k].b ^ v;
      if (u[k] >= n || (!direct && r[k].a != v && r[k].b != v)) {
        val[k] = kInf64;  // reported, hooks nowhere
        atomicOr(a.err, kErrHook);
        continue;
      }
      mu[k] = minv[u[k]];
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      const uint32_t v = base + k * kThreads + threadIdx.x;
      if (v >= hi) continue;
      const bool mutual =
          direct ? mu[k] == ((val[k] & 0xffffffff00000000ull) | v) : mu[k] == val[k];
      if (val[k] == kInf64 || (mutual && v < u[k])) {
        a.parent[v] = v;
        a.msfoid[v] = kNone;
        c0 += live[k] ? 1u : 0u;
        continue;
      }
      // direct: v's grandparent straight away (k_hook)
      const uint32_t x = static_cast<uint32_t>(mu[k]);
      a.parent[v] = (!direct || mutual || mu[k] == kInf64 || x == v || x >= n) ? u[k] : x;
      a.msfoid[v] = r[k].oid;
      ++c1;
    }
  }
  block_sum2(s, c0, c1);
  if (threadIdx.x == 0) {
    a.vcnt[2 * blockIdx.x] = s.sum[0];
    a.vcnt[2 * blockIdx.x + 1] = s.sum[1];
  }
}

// Renumbering and forest edges of this CTA's vertices (k_vertex_write): the
// roots' parent entries become tags.  Expects s.base.
__device__ void write_phase(Shared& s, const Args& a, uint32_t n, const uint64_t* minv,
                            const uint32_t* orig_cur, uint32_t* orig_next, uint64_t* min_next,
                            uint32_t orig_cap, uint64_t msf0, bool direct) {
  uint32_t lo, hi;
  vertex_range(n, lo, hi);
  uint32_t run0 = s.base[0], run1 = s.base[1];
  uint64_t wsum = 0;
  for (uint32_t r0 = lo; r0 < hi; r0 += kItems * kThreads) {
    uint8_t cls[kItems];
    uint64_t mv[kItems];
    uint32_t par[kItems], offs[kItems], carry[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const uint32_t v = r0 + j * kThreads + threadIdx.x;
      par[j] = v < hi ? a.parent[v] : v;
      mv[j] = v < hi ? minv[v] : kInf64;
    }
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const uint32_t v = r0 + j * kThreads + threadIdx.x;
      cls[j] = v < hi ? vertex_class(v, par[j], mv[j]) : 0xff;
      offs[j] = 0;
    }
    tile_rank<2, kItems, kThreads>(cls, offs, s.rank, s.tot);
    const uint32_t tot0 = s.tot[0], tot1 = s.tot[1];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const uint32_t v = r0 + j * kThreads + threadIdx.x;
      carry[j] = cls[j] == 0 ? orig_cur[v] : (cls[j] == 1 && !direct) ? a.msfoid[v] : 0u;
    }
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
      const uint32_t v = r0 + j * kThreads + threadIdx.x;
      if (cls[j] == 0) {
        const uint32_t id = run0 + offs[j];
        if (id < orig_cap) {
          a.parent[v] = kRootTag | id;
          orig_next[id] = carry[j];
          min_next[id] = kInf64;
        } else {
          a.parent[v] = kRootTagNone;
          atomicOr(a.err, kErrHook);
        }
      } else if (cls[j] == 0xff) {
        if (v < hi) a.parent[v] = kRootTagNone;
      } else {
        const uint64_t k = msf0 + run1 + offs[j];
        if (k + 1 >= a.n) {  // a forest has at most n - 1 edges
          atomicOr(a.err, kErrHook);
        } else if (direct) {
          const uint32_t u = static_cast<uint32_t>(mv[j]), w = static_cast<uint32_t>(mv[j] >> 32);
          uint32_t* o = a.out + 3ull * k;
          o[0] = min(u, v);
          o[1] = max(u, v);
          o[2] = w;
          wsum += w;
        } else {
          a.msf[k] = carry[j];
        }
      }
    }
    run0 += tot0;
    run1 += tot1;
    __syncthreads();  // s.rank / s.tot are reused by the next step
  }
  if (direct) {
    wsum = warp_sum(wsum);
    if (lane_id() == 0 && wsum) atomicAdd(a.weight, static_cast<unsigned long long>(wsum));
  }
}

// Vertex work of a round over n <= kTinyN vertices, by every CTA in its own
// shared memory; leaves the label map in s.map.  CTA 0 writes the round's
// map, the representatives and the forest edges.  Returns the next round's
// vertex count and, in *added, the forest edges.  kPer vertices per thread.
template <int kPer>
__device__ uint32_t tiny_vertices(Shared& s, const Args& a, uint32_t n, const uint64_t* minv,
                                  const Rec* list, const uint32_t* orig_cur, uint32_t* orig_next,
                                  uint32_t* R, uint64_t msf0, uint32_t* added) {
  static_assert(kPer * kThreads <= static_cast<int>(kTinyN), "the arrays hold the round");
  uint64_t val[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t v = j * kThreads + threadIdx.x;
    val[j] = v < n ? minv[v] : kInf64;
    s.min64[v] = val[j];
  }
  Rec r[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    r[j] = Rec{0, 0, 0, 0};
    if (val[j] != kInf64) r[j] = list[static_cast<uint32_t>(val[j])];
  }
  __syncthreads();
  uint8_t cls[kPer];
  uint32_t offs[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t v = j * kThreads + threadIdx.x;
    uint32_t par = v;
    cls[j] = 0xff;
    offs[j] = 0;
    if (val[j] != kInf64) {
      const uint32_t u = r[j].a ^ r[j].b ^ v;
      cls[j] = 0;
      if (u >= n || (r[j].a != v && r[j].b != v)) {
        atomicOr(a.err, kErrHook);
      } else if (!(s.min64[u] == val[j] && v < u)) {
        par = u;
        cls[j] = 1;
      }
    }
    s.par[v] = par;
  }
  tile_rank<2, kPer, kThreads>(cls, offs, s.rank, s.tot);  // also: s.par is complete
  const uint32_t n_next = s.tot[0];
  *added = s.tot[1];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t v = j * kThreads + threadIdx.x;
    if (cls[j] == 0xff) s.map[v] = kNone;
    if (cls[j] == 0) {
      s.map[v] = offs[j];
      if (blockIdx.x == 0) orig_next[offs[j]] = orig_cur[v];
    } else if (cls[j] == 1 && blockIdx.x == 0) {
      const uint64_t k = msf0 + offs[j];
      if (k + 1 < a.n) a.msf[k] = r[j].oid;
      else atomicOr(a.err, kErrHook);
    }
  }
  // walks with halving in shared memory: entries only move to ancestors
  volatile uint32_t* par = s.par;
  uint32_t root[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t v = j * kThreads + threadIdx.x;
    uint32_t x = v, p = par[x], steps = 0;
    for (;;) {
      const uint32_t gp = par[p];
      if (gp == p) break;
      par[x] = gp;
      x = gp;
      p = par[x];
      if (++steps > 2 * kTinyN) {
        atomicOr(a.err, kErrJump);
        break;
      }
    }
    root[j] = p;
  }
  __syncthreads();  // the roots' labels are in s.map; s.min64 is free
  uint32_t lab[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) lab[j] = s.map[root[j]];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kPer; ++j) {
    const uint32_t v = j * kThreads + threadIdx.x;
    s.map[v] = lab[j];
    if (blockIdx.x == 0 && v < n) R[v] = lab[j];
    s.min64[v] = kInf64;
  }
  __syncthreads();
  return n_next;
}

__global__ void __launch_bounds__(kThreads, 1) k_rounds(const __grid_constant__ Args a) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  Shared& s = *reinterpret_cast<Shared*>(s_raw);
  __shared__ uint32_t s_size[kMaxRounds], s_roff[kMaxRounds], s_ooff[kMaxRounds + 1];
  State* st = a.st;
  uint32_t* bar = st->bars + a.launch * kBarStride;
  uint32_t goal = 0;
  // after an error of an earlier pass or launch: its lists may be incomplete
  if (__syncthreads_or(threadIdx.x == 0 ? *a.pass_err != 0
                                        : threadIdx.x <= a.launch && st->errs[threadIdx.x - 1]))
    return;
  const uint32_t tid = threadIdx.x, gtid = blockIdx.x * kThreads + tid;
  const uint32_t gsz = gridDim.x * kThreads;
  uint32_t nr = a.first ? a.nr0 : st->nreps;
  const uint32_t n0 = nr;
  const uint32_t vsel = a.first ? 0u : st->vsel;
  const uint32_t* V = vsel ? a.Vn : a.V;
  uint32_t* Vnext = vsel ? a.V : a.Vn;
  uint64_t msf_count = a.first ? a.msf0 : st->msf_count;
  unsigned long long sum_m = 0, sum_n = 0;
  for (uint32_t x = gtid; x < 3 * kTinyN; x += gsz) a.tiny[x] = kInf64;
  List cur{a.src, a.src_nseg, a.src_cap};
  const uint32_t* cur_cnt = a.src_count;
  int which = 0;  // buffer the next edge phase writes
  if (nr > 1 && a.prologue) {
    auto label = [&](uint32_t x) { return a.D[x]; };
    if (cur.base) {
      const uint32_t m = seg_prefix32(s, cur_cnt, cur.nseg);
      edge_phase<false>(s, a, cur, m, label, nr, a.buf[0], a.cnt[0], a.minA, nullptr);
    } else {
      edge_phase<true>(s, a, cur, a.md, label, nr, a.buf[0], a.cnt[0], a.minA, nullptr);
    }
    cur = List{a.buf[0], gridDim.x * kGroups, a.cap};
    cur_cnt = a.cnt[0];
    which = 1;
    if (!grid_sync(s, bar, goal, a.err)) return;
  } else if (!a.direct && nr <= kTinyN) {
    if (!grid_sync(s, bar, goal, a.err)) return;  // a.tiny is set
  }
  uint64_t* minv = a.minA;
  uint32_t tiny = 0;  // next of the three rotating arrays to receive minima
  uint32_t r = 0, roff = a.roff0, ooff = a.ooff0;
  const uint32_t* orig_cur = a.orig0 ? a.orig0 : V;
  uint32_t m = 0;
  if (nr > 1) m = seg_prefix32(s, cur_cnt, cur.nseg);
  while (m > 0) {
    // (uniform over the grid: all from counts every CTA reads alike)
    if (r >= static_cast<uint32_t>(kMaxRounds) || uint64_t(roff) + nr > 2ull * a.n + 64 ||
        uint64_t(ooff) + nr > uint64_t(a.n) + 64) {
      if (gtid == 0) atomicOr(a.err, kErrChase);
      break;
    }
    sum_m += m;
    sum_n += nr;
    uint32_t* R = a.R + roff;
    uint32_t* orig_next = a.orig + ooff;
    Rec* out = a.buf[which];
    uint32_t n_next, added;
    if (nr <= kTinyN && !(a.direct && r == 0)) {
      n_next = nr <= kThreads
                   ? tiny_vertices<1>(s, a, nr, minv, cur.base, orig_cur, orig_next, R, msf_count,
                                      &added)
                   : tiny_vertices<kTinyN / kThreads>(s, a, nr, minv, cur.base, orig_cur,
                                                      orig_next, R, msf_count, &added);
      // the array read in the round before is free again
      uint64_t* reset = a.tiny + ((tiny + 1) % 3) * kTinyN;
      for (uint32_t x = gtid; x < kTinyN; x += gsz) reset[x] = kInf64;
      minv = a.tiny + tiny * kTinyN;
      tiny = (tiny + 1) % 3;
      auto label = [&](uint32_t x) { return s.map[x]; };
      edge_phase<false>(s, a, cur, m, label, n_next, out, a.cnt[which], minv, s.min64);
      __syncthreads();
      for (uint32_t x = tid; x < n_next; x += kThreads)
        if (s.min64[x] != kInf64) red_min(&minv[x], s.min64[x]);
    } else {
      const bool direct = a.direct && r == 0;
      uint64_t* min_next = minv == a.minA ? a.minB : a.minA;
      hook_phase(s, a, nr, minv, cur.base, direct);
      if (!grid_sync(s, bar, goal, a.err)) return;
      cta_bases(s, a.vcnt);
      n_next = s.sum[0];
      added = s.sum[1];
      write_phase(s, a, nr, minv, orig_cur, orig_next, min_next, a.n + 64 - ooff, msf_count,
                  direct);
      if (!grid_sync(s, bar, goal, a.err)) return;
      label_walks<kItems>(nr, gtid, gsz, a.parent, R, a.err);
      const bool to_tiny = n_next <= kTinyN;
      if (to_tiny) {
        for (uint32_t x = tid; x < n_next; x += kThreads) s.min64[x] = kInf64;
        min_next = a.tiny + tiny * kTinyN;
        tiny = (tiny + 1) % 3;
      }
      if (!grid_sync(s, bar, goal, a.err)) return;
      minv = min_next;
      auto label = [&](uint32_t x) { return R[x]; };
      edge_phase<false>(s, a, cur, m, label, n_next, out, a.cnt[which], minv,
                        to_tiny ? s.min64 : nullptr);
      if (to_tiny) {
        __syncthreads();
        for (uint32_t x = tid; x < n_next; x += kThreads)
          if (s.min64[x] != kInf64) red_min(&minv[x], s.min64[x]);
      }
      if (direct && gtid == 0) st->direct_count = added;
    }
    if (tid == 0) {
      s_size[r] = nr;
      s_roff[r] = roff;
      s_ooff[r + 1] = ooff;
    }
    msf_count += added;
    roff += nr;
    ooff += n_next;
    orig_cur = orig_next;
    nr = n_next;
    cur = List{out, gridDim.x * kGroups, a.cap};
    cur_cnt = a.cnt[which];
    which ^= 1;
    ++r;
    if (!grid_sync(s, bar, goal, a.err)) return;
    m = seg_prefix32(s, cur_cnt, cur.nseg);
  }
  __syncthreads();
  uint32_t nreps = n0;
  if (r > 0 && a.finalize) {
    // labels composed backwards over the round maps (k_compose); runs of
    // small maps by CTA 0 alone
    bool synced = true;  // the maps written so far are visible to every CTA
    for (int k = static_cast<int>(r) - 1; k >= 1; --k) {
      const uint32_t nk = s_size[k];
      uint32_t* Rk = a.R + s_roff[k];
      const uint32_t* next = k + 1 == static_cast<int>(r) ? a.orig + s_ooff[r]
                                                          : a.R + s_roff[k + 1];
      const uint32_t* ok = a.orig + s_ooff[k];
      if (nk <= 4 * kThreads) {
        if (blockIdx.x == 0)
          for (uint32_t x = tid; x < nk; x += kThreads) {
            const uint32_t y = Rk[x];
            Rk[x] = y == kNone ? ok[x] : next[y];
          }
        __syncthreads();
        synced = false;
        continue;
      }
      if (!synced && !grid_sync(s, bar, goal, a.err)) return;
      for (uint32_t x = gtid; x < nk; x += gsz) {
        const uint32_t y = Rk[x];
        Rk[x] = y == kNone ? ok[x] : next[y];
      }
      synced = false;
    }
    if (!synced && !grid_sync(s, bar, goal, a.err)) return;
    {
      const uint32_t* next = r == 1 ? a.orig + s_ooff[1] : a.R + s_roff[1];
      uint32_t lo, hi, c0 = 0;
      vertex_range(n0, lo, hi);
      for (uint32_t base = lo + tid; base < hi; base += kItems * kThreads) {
        uint32_t y[kItems], o[kItems];
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
          const uint32_t x = base + k * kThreads;
          y[k] = x < hi ? a.R[x] : kNone;
          o[k] = x < hi ? V[x] : 0u;
        }
#pragma unroll
        for (int k = 0; k < kItems; ++k)
          if (y[k] != kNone) y[k] = next[y[k]];
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
          if (base + k * kThreads >= hi) continue;
          const uint32_t f = y[k] == kNone ? o[k] : y[k];
          a.P[o[k]] = f;
          c0 += f == o[k] ? 1u : 0u;
        }
      }
      block_sum2(s, c0, 0);
      if (tid == 0) {
        a.vcnt[2 * blockIdx.x] = s.sum[0];
        a.vcnt[2 * blockIdx.x + 1] = 0;
      }
    }
    if (!grid_sync(s, bar, goal, a.err)) return;
    cta_bases(s, a.vcnt);
    nreps = s.sum[0];
    {
      uint32_t lo, hi, run = s.base[0];
      vertex_range(n0, lo, hi);
      for (uint32_t r0 = lo; r0 < hi; r0 += kItems * kThreads) {
        uint8_t cls[kItems];
        uint32_t v[kItems], offs[kItems];
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
          const uint32_t i = r0 + j * kThreads + tid;
          v[j] = i < hi ? V[i] : 0u;
        }
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
          const uint32_t i = r0 + j * kThreads + tid;
          cls[j] = i < hi && a.P[v[j]] == v[j] ? 0 : 0xff;
          offs[j] = 0;
        }
        tile_rank<1, kItems, kThreads>(cls, offs, s.rank, s.tot);
        const uint32_t tot = s.tot[0];
#pragma unroll
        for (int j = 0; j < kItems; ++j) {
          if (cls[j] != 0) continue;
          const uint32_t k = run + offs[j];
          Vnext[k] = v[j];
          a.dense_of[v[j]] = k;
        }
        run += tot;
        __syncthreads();
      }
    }
    if (!grid_sync(s, bar, goal, a.err)) return;
    for (uint64_t base = gtid; base < a.n; base += uint64_t(kItems) * gsz) {
      uint32_t p[kItems], d[kItems];
#pragma unroll
      for (int k = 0; k < kItems; ++k)
        p[k] = base + uint64_t(k) * gsz < a.n ? a.P[base + uint64_t(k) * gsz] : 0u;
#pragma unroll
      for (int k = 0; k < kItems; ++k) p[k] = a.P[p[k]];
#pragma unroll
      for (int k = 0; k < kItems; ++k) d[k] = a.dense_of[p[k]];
#pragma unroll
      for (int k = 0; k < kItems; ++k) {
        const uint64_t x = base + uint64_t(k) * gsz;
        if (x >= a.n) continue;
        a.P[x] = p[k];
        a.D[x] = d[k];
      }
    }
  }
  if (a.finalize) {  // the next contraction's minima
    for (uint32_t x = gtid; x < nreps; x += gsz) a.minA[x] = kInf64;
  }
  if (a.emit != Emit::kNone) {
    const uint64_t k0 = a.emit == Emit::kBits ? 0ull
                        : (a.direct && r > 0) ? st->direct_count
                        : a.first             ? 0ull
                                              : st->direct_count;
    uint64_t local = 0;
    msf_count = min(msf_count, static_cast<uint64_t>(a.n) - 1);
    for (uint64_t base = k0 + gtid; base < msf_count; base += uint64_t(kItems) * gsz) {
      uint32_t o[kItems], e0[kItems], e1[kItems], e2[kItems];
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const uint64_t k = base + uint64_t(j) * gsz;
        o[j] = k < msf_count ? min(a.msf[k], a.md - 1) : 0u;
      }
      if (a.emit == Emit::kBits) {
#pragma unroll
        for (int j = 0; j < kItems; ++j)
          if (base + uint64_t(j) * gsz < msf_count)
            atomicOr(&a.bits[o[j] >> 5], 1u << (o[j] & 31));
        continue;
      }
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const uint32_t* e = a.in + 3ull * o[j];
        e0[j] = e[0];
        e1[j] = e[1];
        e2[j] = e[2];
      }
#pragma unroll
      for (int j = 0; j < kItems; ++j) {
        const uint64_t k = base + uint64_t(j) * gsz;
        if (k >= msf_count) continue;
        uint32_t* q = a.out + 3 * k;
        q[0] = min(e0[j], e1[j]);
        q[1] = max(e0[j], e1[j]);
        q[2] = e2[j];
        local += e2[j];
      }
    }
    local = warp_sum(local);
    if (lane_id() == 0 && local) atomicAdd(a.weight, static_cast<unsigned long long>(local));
  }
  // (a launch that is not the solve's first has passed a barrier after its
  // prologue, and with it every CTA's reads of the state)
  if (gtid == 0 && (a.first || (n0 > 1 && a.prologue))) {
    st->msf_count = msf_count;
    st->nreps = nreps;
    st->rounds += r;
    st->levels += 1;
    st->sum_m += sum_m;
    st->sum_n += sum_n;
    st->last_rounds = r;
    for (uint32_t k = 0; k < r; ++k) st->size[k] = s_size[k];
    st->size[r] = nr;
    if (r > 0 && a.finalize) st->vsel = vsel ^ 1u;
  }
}

}  // namespace coop
}  // namespace kamsta
