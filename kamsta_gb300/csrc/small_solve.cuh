// small_solve.cuh -- the whole MSF solve of a small graph inside one CTA.
//
// Used by kamsta_mst_boruvka_noalloc (one CTA, a static scratch array) and by
// the batched path (persistent kernels whose CTAs take small graphs from a
// work queue, each CTA with its own scratch slot).  The rounds are those of
// the multi-kernel solver -- hook along the minimum edge (of a mutual pair the
// lower label stays root), renumbering of live roots, label walk, relabel +
// self-loop removal with the next round's minimum -- and so is the tie-break:
// (w, position of the src < dst copy) orders edges by (w, min, max).
//
// What bounds it: one SM's instruction issue and the chain of phases.  So
//  - minima, hooks and the label map live in shared memory (16-bit labels);
//    an edge costs two shared gathers and two shared compares a round;
//  - an edge is (labels, key) with key = w << bits | input position.  When
//    the weights leave room for the position in 32 bits, the key is one
//    word, an edge 8 bytes and its minimum a native 32-bit shared atomic;
//    otherwise key and atomic are 64-bit;
//  - the position in the key identifies the edge, so the edge list needs no
//    order: survivors are appended behind one shared counter per 128 edges,
//    where keeping the order took two block barriers per THREADS edges;
//  - a round has four block barriers whatever its size, and a list occupies
//    one warp per 128 edges;
//  - dense graphs contract their light edges first (see `split`).
// Measured on one GB300 against the ordered lists in L2 that this replaced:
// 1024 graphs of 2^8..2^12 vertices (24.9 M entries) in one batch call 1554
// -> 322 us, the allocation-free call on 1000 vertices and 8000 entries 85 ->
// 43 us.  A graph of 4000 vertices and 64000 entries takes 89 us on 512
// threads: 27 us its first pass (0.9 us per 2048 entries, the latency of the
// entries read one step ahead), 10 us the heavy edges, 12 us the output, the
// rest rounds of 3 to 6 us.
#pragma once
#include <cstddef>

#include "common.cuh"

namespace kamsta {
namespace small {

constexpr uint32_t kMaxN = 1u << 15;
constexpr uint64_t kMaxMd = 1ull << 18;
constexpr uint32_t kMaxRounds = 40;
// Size classes of the batch: a graph that needs little shared memory and has
// little work goes to a small CTA, several of which share an SM.
enum class Size { kTiny, kCompact, kFull };
constexpr uint32_t max_n(Size c) {
  return c == Size::kTiny ? 1u << 10 : c == Size::kCompact ? 1u << 12 : kMaxN;
}
constexpr uint32_t max_md(Size c) {
  return c == Size::kTiny ? 1u << 14 : c == Size::kCompact ? 1u << 16
                                                           : static_cast<uint32_t>(kMaxMd);
}
// Beyond kSharedN vertices the composite labels (and 64-bit minima) stay in
// the scratch slot: 128 KB of 32-bit minima and 64 KB of hooks are what an SM
// holds.
constexpr uint32_t kSharedN = 1u << 14;

// Shared bytes of a CTA whose graphs have at most n vertices.
constexpr size_t shared_bytes(uint32_t n) {
  n = (n + 3) & ~3u;
  return n <= kSharedN ? size_t(n) * (8 + 2 + 2) : size_t(n) * (4 + 2);
}
constexpr size_t kSharedFull =
    shared_bytes(kSharedN) > shared_bytes(kMaxN) ? shared_bytes(kSharedN) : shared_bytes(kMaxN);
constexpr size_t shared_bytes(Size c) {
  return c == Size::kFull ? kSharedFull : shared_bytes(max_n(c));
}

// Scratch layout (bytes, 256-aligned) for graphs of up to md entries.
struct Slot {
  size_t l0, l1, gmin, lab, msf, flags, bytes;
};
constexpr Slot slot_layout(uint64_t md, uint32_t n) {
  Slot s{};
  // (an input that lists edges in one direction only may overflow it: kErrOverflow)
  const size_t mu = md / 2 < 256 ? 256 : md / 2;
  s.l0 = 256;                                     // Result
  s.l1 = s.l0 + mu * 16;
  s.gmin = s.l1 + mu * 16;
  s.lab = s.gmin + size_t(n) * 8;
  s.msf = s.lab + size_t(n) * 2;
  s.flags = s.msf + size_t(n) * 4;  // one bit per input entry
  s.bytes = (s.flags + md / 8 + 4 + 255) & ~size_t(255);
  return s;
}
constexpr Slot slot_layout(Size c) { return slot_layout(max_md(c), max_n(c)); }
constexpr size_t kScratchBytes = slot_layout(Size::kFull).bytes;

struct Result {
  unsigned long long count;
  unsigned long long weight;
  uint32_t err;
  uint32_t rounds;
};

// Output order of the forest.
enum class Out {
  kFound,   // in the order the rounds find the edges
  kSorted,  // sorted by (src, dst): the input order of the src<dst copies
};

template <typename Key>
struct Edge;
template <>
struct __align__(8) Edge<uint32_t> {
  uint32_t ab, key;  // labels a | b << 16
};
template <>
struct __align__(16) Edge<unsigned long long> {
  uint32_t ab, pad;
  unsigned long long key;
};

constexpr uint32_t kTag = 0x8000u;   // a root's entry: kTag | its new label
constexpr uint32_t kDone = 0xffffu;  // a finished root
constexpr uint32_t kGone = 0x7fffu;  // label of a finished vertex

// Weight samples of the light / heavy split.
constexpr uint32_t kSamples = 128;
// Smallest graph that is split: below, a round costs its barriers, and the
// split adds rounds.
constexpr uint32_t kSplitMd = 1u << 13;

// Shared counters and buffers of a solve besides its arrays.
template <int THREADS>
struct Counters {
  uint32_t w[2 * (THREADS / 32)];
  uint32_t edges[2];  // list lengths, by round parity; before the rounds
                      // light and heavy edges
  uint32_t pivot;     // largest light weight
  uint32_t sample[kSamples];
  uint32_t roots[2];
  uint32_t forest;
  uint32_t err;
  unsigned long long weight;
};

// Stable block-wide ranks of this thread's item for two flags (one item per
// thread, items in thread order): r = rank among the block's items with
// the same flag, t = block totals.
template <int THREADS>
__device__ __forceinline__ void block_rank2(bool f0, bool f1, uint32_t& r0, uint32_t& r1,
                                            uint32_t& t0, uint32_t& t1, uint32_t* s_w) {
  constexpr int kWarps = THREADS / 32;
  const uint32_t lane = lane_id(), warp = threadIdx.x >> 5, lt = lanemask_lt();
  const uint32_t b0 = __ballot_sync(kFull, f0), b1 = __ballot_sync(kFull, f1);
  if (lane == 0) {
    s_w[warp] = __popc(b0);
    s_w[kWarps + warp] = __popc(b1);
  }
  __syncthreads();
  uint32_t p0 = 0, p1 = 0, a0 = 0, a1 = 0;
#pragma unroll 8
  for (int w = 0; w < kWarps; ++w) {
    const uint32_t x0 = s_w[w], x1 = s_w[kWarps + w];
    if (static_cast<uint32_t>(w) < warp) {
      p0 += x0;
      p1 += x1;
    }
    a0 += x0;
    a1 += x1;
  }
  __syncthreads();
  r0 = p0 + __popc(b0 & lt);
  r1 = p1 + __popc(b1 & lt);
  t0 = a0;
  t1 = a1;
}

// Slots behind two shared counters for a warp's kept items (kU per lane, at
// most one of f / g each): one atomic instruction, lane 0's on the first
// counter and lane 1's on the second, which lies behind it.
template <int kU>
__device__ __forceinline__ void append_slots2(const bool (&f)[kU], const bool (&g)[kU],
                                              uint32_t* counters, uint32_t (&slot)[kU]) {
  const uint32_t lt = lanemask_lt();
  uint32_t tf = 0, tg = 0;
#pragma unroll
  for (int j = 0; j < kU; ++j) {
    const uint32_t bf = __ballot_sync(kFull, f[j]), bg = __ballot_sync(kFull, g[j]);
    slot[j] = f[j] ? tf + __popc(bf & lt) : tg + __popc(bg & lt);
    tf += __popc(bf);
    tg += __popc(bg);
  }
  uint32_t base = 0;
  if (lane_id() < 2) base = atomicAdd(counters + lane_id(), lane_id() ? tg : tf);
  const uint32_t base_f = __shfl_sync(kFull, base, 0), base_g = __shfl_sync(kFull, base, 1);
#pragma unroll
  for (int j = 0; j < kU; ++j) slot[j] += f[j] ? base_f : base_g;
}

// Slots behind a shared counter for a warp's kept items (kU per lane).
template <int kU>
__device__ __forceinline__ void append_slots(const bool (&keep)[kU], uint32_t* counter,
                                             uint32_t (&slot)[kU]) {
  const uint32_t lt = lanemask_lt();
  uint32_t tot = 0;
#pragma unroll
  for (int j = 0; j < kU; ++j) {
    const uint32_t b = __ballot_sync(kFull, keep[j]);
    slot[j] = tot + __popc(b & lt);
    tot += __popc(b);
  }
  uint32_t base = 0;
  if (lane_id() == 0 && tot) base = atomicAdd(counter, tot);
  base = __shfl_sync(kFull, base, 0);
#pragma unroll
  for (int j = 0; j < kU; ++j) slot[j] += base;
}

__device__ __forceinline__ void lower_to(uint32_t* p, uint32_t v) { atomicMin(p, v); }
__device__ __forceinline__ void lower_to(unsigned long long* p, unsigned long long v) {
  atomicMin(p, v);
}

// Minima of both endpoints of a thread's kept edges.  All current values are
// read before the first compare (other edges read entry 0), and only smaller
// keys go to the atomics: one shared-memory latency per step, not one per
// endpoint.
template <int kU, typename Key>
__device__ __forceinline__ void feed_minima(Key* mn, const bool (&keep)[kU],
                                            const uint32_t (&a)[kU], const uint32_t (&b)[kU],
                                            const Key (&key)[kU]) {
  Key ca[kU], cb[kU];
#pragma unroll
  for (int j = 0; j < kU; ++j) {
    ca[j] = *static_cast<volatile Key*>(mn + (keep[j] ? a[j] : 0u));
    cb[j] = *static_cast<volatile Key*>(mn + (keep[j] ? b[j] : 0u));
  }
#pragma unroll
  for (int j = 0; j < kU; ++j) {
    if (keep[j] && key[j] < ca[j]) lower_to(mn + a[j], key[j]);
    if (keep[j] && key[j] < cb[j]) lower_to(mn + b[j], key[j]);
  }
}

// The solve with one key type; BIG: more than kSharedN vertices.  False when
// the weights do not fit 32-bit keys (nothing is written then).  The caller's
// threads are synchronised on return.
template <int THREADS, Out OUT, typename Key, bool BIG>
__device__ bool solve_keys(const uint32_t* __restrict__ in, uint32_t md, uint32_t n,
                           unsigned char* scratch, const Slot& lay, uint32_t mu_cap,
                           uint32_t* __restrict__ out, Result* res, unsigned char* s_raw,
                           Counters<THREADS>& c, bool check_ids, bool check_order) {
  constexpr bool kWide = sizeof(Key) == 8;
  constexpr bool kGmin = BIG && kWide;
  constexpr Key kInf = static_cast<Key>(~Key(0));
  // (minima in global memory are updated in the L2)
  auto min_of = [](const Key* p) { return kGmin ? __ldcg(p) : *p; };
  // A step covers THREADS * kU items, kU * 32 consecutive ones per warp (item
  // j of a lane is w0 + j * 32 past the step's base), so that a short list
  // occupies few warps and the others skip the step.
  constexpr int kU = 4;
  const uint32_t tid = threadIdx.x;
  const uint32_t wfirst = (tid >> 5) * (32 * kU), w0 = wfirst + lane_id();
  const uint32_t bits = kWide ? 32u : (md > 1 ? 32u - __clz(md - 1) : 1u);
  const uint32_t wlimit = kWide ? 0xffffffffu : (0xffffffffu >> bits) - 1u;  // key < kInf
  const uint32_t pmask = kWide ? 0xffffffffu : (1u << bits) - 1u;
  Edge<Key>* L[2] = {reinterpret_cast<Edge<Key>*>(scratch + lay.l0),
                     reinterpret_cast<Edge<Key>*>(scratch + lay.l1)};
  Key* mn;
  unsigned char* at = s_raw;
  if constexpr (kGmin) {
    mn = reinterpret_cast<Key*>(scratch + lay.gmin);
  } else {
    mn = reinterpret_cast<Key*>(at);
    at += sizeof(Key) * ((n + 3) & ~3u);
  }
  volatile uint16_t* par = reinterpret_cast<uint16_t*>(at);
  at += sizeof(uint16_t) * ((n + 3) & ~3u);
  uint16_t* lab;
  if constexpr (BIG) lab = reinterpret_cast<uint16_t*>(scratch + lay.lab);
  else lab = reinterpret_cast<uint16_t*>(at);
  uint32_t* msf = reinterpret_cast<uint32_t*>(scratch + lay.msf);
  uint32_t* flags = reinterpret_cast<uint32_t*>(scratch + lay.flags);
  // Error bits this thread raised.  Every break decision is taken with
  // __syncthreads_or over these, so all threads leave the rounds together;
  // c.err only collects the codes for the result.
  uint32_t terr = 0;
  auto flag_err = [&](uint32_t code) {
    terr |= code;
    atomicOr(&c.err, code);
  };
  if (tid == 0) {
    c.err = 0;
    c.weight = 0;
    c.forest = 0;
    c.edges[0] = c.edges[1] = 0;
    c.roots[0] = c.roots[1] = 0;
    c.pivot = 0xffffffffu;
  }
  // Light edges first (kSorted, whose output order is the input's): with at
  // least four edges per vertex, the rounds run on the lightest part, about
  // two edges per vertex, and one pass over the others then drops those
  // inside a component -- nearly all, where ids follow no geometry, and each
  // of them would have been read in every round.
  bool split = false;
  if (OUT == Out::kSorted && md >= 8ull * n && md >= kSplitMd) {
    split = true;
    uint32_t w = 0;
    if (tid < kSamples) {
      w = in[3ull * (mix64(tid) % md) + 2];
      c.sample[tid] = w;
    }
    __syncthreads();
    if (tid < kSamples) {
      uint32_t rank = 0;
#pragma unroll 8
      for (uint32_t k = 0; k < kSamples; ++k)
        rank += c.sample[k] < w || (c.sample[k] == w && k < tid) ? 1u : 0u;
      if (rank == static_cast<uint32_t>(4ull * n * kSamples / md)) c.pivot = w;
    }
  }
  for (uint32_t v = tid; v < n; v += THREADS) {
    mn[v] = kInf;
    lab[v] = static_cast<uint16_t>(v);
  }
  if (tid < 4 && n + tid < ((n + 3) & ~3u)) lab[n + tid] = 0;  // (updated with the others)
  const uint32_t words = (md + 31) / 32;
  if (OUT == Out::kSorted)
    for (uint32_t k = tid; k < words; k += THREADS) flags[k] = 0;
  __syncthreads();
  // first pass: the src<dst copies; heavy ones fill l1 from its end
  const uint32_t pivot = c.pivot;
  Edge<Key>* const H = L[1] + mu_cap;  // heavy edge k is H[-1 - k]
  // (the next step's entries are on their way while a step is handled: one
  // CTA has no other work to hide their latency behind; the light edges'
  // minima are fed afterwards from their list, an eighth to a half as long)
  uint32_t ns[kU], nd[kU], nw[kU];
  auto fetch = [&](uint32_t base) {
    const uint32_t* e = in + 3ull * (base + w0);
    if (base + THREADS * kU <= md) {
#pragma unroll
      for (int j = 0; j < kU; ++j) {
        ns[j] = e[96 * j];
        nd[j] = e[96 * j + 1];
        nw[j] = e[96 * j + 2];
      }
      return;
    }
#pragma unroll
    for (int j = 0; j < kU; ++j) {
      ns[j] = nd[j] = nw[j] = 0;  // a self loop: not kept
      if (base + w0 + 32 * j < md) {
        ns[j] = e[96 * j];
        nd[j] = e[96 * j + 1];
        nw[j] = e[96 * j + 2];
      }
    }
  };
  uint32_t id_max = 0, w_max = 0;
  fetch(0);
  for (uint32_t base = 0; base + wfirst < md; base += THREADS * kU) {
    uint32_t s[kU], d[kU], slot[kU];
    bool keep[kU], heavy[kU];
    Edge<Key> e[kU];
#pragma unroll
    for (int j = 0; j < kU; ++j) {
      s[j] = ns[j];
      d[j] = nd[j];
      const uint32_t w = nw[j];
      id_max = max(id_max, max(s[j], d[j]));
      w_max = max(w_max, w);
      keep[j] = s[j] < d[j] && d[j] < n;
      heavy[j] = keep[j] && w > pivot;
      keep[j] = keep[j] && !heavy[j];
      e[j].ab = s[j] | (d[j] << 16);
      e[j].key = static_cast<Key>((static_cast<Key>(w) << bits) | (base + w0 + 32 * j));
    }
    fetch(base + THREADS * kU);
    append_slots2<kU>(keep, heavy, &c.edges[0], slot);
#pragma unroll
    for (int j = 0; j < kU; ++j) {
      if ((keep[j] || heavy[j]) && slot[j] < mu_cap)
        *(heavy[j] ? H - 1 - slot[j] : L[0] + slot[j]) = e[j];
    }
  }
  // (without entries id_max is no id: an empty graph of no vertices is valid)
  if (check_ids && md != 0 && id_max >= n) flag_err(kErrRange);
  if (check_order)
    for (uint32_t i = tid + 1; i < md; i += THREADS) {
      const uint32_t* p = in + 3ull * (i - 1);
      if (p[3] < p[0] || (p[3] == p[0] && p[4] <= p[1])) flag_err(kErrOrder);
    }
  const bool wide_w = w_max > wlimit;
  if (__syncthreads_or(!kWide && wide_w)) return false;
  uint32_t m = c.edges[0], nr = n, cur = 0, round = 0, found = 0;
  const uint32_t mh = c.edges[1];
  // light lists grow from the front of l0 / l1 and never reach the heavy part
  if (m + mh > mu_cap) flag_err(kErrOverflow);  // (the same in every thread)
  unsigned long long wsum = 0;
  Edge<Key> ne[kU];  // the next step's edges: list[step * i], i < count
  auto fetch_edges = [&](uint32_t base, uint32_t count, const Edge<Key>* list, int step) {
#pragma unroll
    for (int j = 0; j < kU; ++j) {
      const uint32_t i = base + w0 + 32 * j;
      if (i < count) ne[j] = list[static_cast<ptrdiff_t>(i) * step];
      else ne[j].ab = 0, ne[j].key = kInf;
    }
  };
  // round-0 minima (m is at most mu_cap, or the rounds do not start)
  if (m <= mu_cap) {
    fetch_edges(0, m, L[0], 1);
    for (uint32_t base = 0; base + wfirst < m; base += THREADS * kU) {
      uint32_t a[kU], b[kU];
      bool keep[kU];
      Key key[kU];
#pragma unroll
      for (int j = 0; j < kU; ++j) {
        keep[j] = base + w0 + 32 * j < m;
        a[j] = ne[j].ab & 0xffffu;
        b[j] = ne[j].ab >> 16;
        key[j] = ne[j].key;
      }
      fetch_edges(base + THREADS * kU, m, L[0], 1);
      feed_minima<kU, Key>(mn, keep, a, b, key);
    }
  }
  __syncthreads();
  for (;;) {
    if (m == 0) {
      if (!split) break;
      // the light edges are contracted (every component still has a label,
      // and all minima are unset): the heavy ones that join two components
      split = false;
      if (__syncthreads_or((terr & ~kErrRange) != 0)) break;
      cur = 0;
      uint32_t* cnt = &c.edges[round & 1];  // zero: it counted the last round's survivors
      fetch_edges(0, mh, H - 1, -1);
      for (uint32_t base = 0; base + wfirst < mh; base += THREADS * kU) {
        Edge<Key> e[kU];
        uint32_t a[kU], b[kU], slot[kU];
        bool keep[kU];
#pragma unroll
        for (int j = 0; j < kU; ++j) {
          keep[j] = base + w0 + 32 * j < mh;
          e[j] = ne[j];
        }
        fetch_edges(base + THREADS * kU, mh, H - 1, -1);
#pragma unroll
        for (int j = 0; j < kU; ++j) {  // (an edge past the end is 0, 0)
          a[j] = lab[e[j].ab & 0xffffu];
          b[j] = lab[e[j].ab >> 16];
        }
#pragma unroll
        for (int j = 0; j < kU; ++j) keep[j] = keep[j] && a[j] != b[j];
        append_slots<kU>(keep, cnt, slot);
        Key key[kU];
#pragma unroll
        for (int j = 0; j < kU; ++j) {
          key[j] = e[j].key;
          e[j].ab = a[j] | (b[j] << 16);
          if (keep[j]) L[0][slot[j]] = e[j];
        }
        feed_minima<kU, Key>(mn, keep, a, b, key);
      }
      __syncthreads();
      m = *cnt;
      continue;
    }
    if (__syncthreads_or((terr & ~kErrRange) != 0)) break;
    if (round >= kMaxRounds) {  // round is the same in every thread
      terr |= kErrChase;
      if (tid == 0) c.err |= kErrChase;
      break;
    }
    // hook along the minimum edge and number the live roots
    const uint32_t rp = round & 1;
    uint32_t n_next = 0;
    constexpr int kH = OUT == Out::kSorted ? kU : 1;  // vertices per thread and step
    constexpr bool kSkip = OUT == Out::kSorted;  // (kFound ranks with block barriers)
    for (uint32_t vb = 0; vb + (kSkip ? wfirst : 0u) < nr; vb += THREADS * kH) {
      Key key[kH];
      uint32_t u[kH], oid[kH], es[kH], ed[kH], slot[kH];
      bool root[kH], hooked[kH];
#pragma unroll
      for (int j = 0; j < kH; ++j) {
        const uint32_t v = vb + (kSkip ? w0 + 32 * j : tid);
        key[j] = v < nr ? min_of(mn + v) : kInf;
        oid[j] = static_cast<uint32_t>(key[j]) & pmask;
        es[j] = ed[j] = 0;
        if (key[j] != kInf) {
          es[j] = in[3ull * oid[j]];
          ed[j] = in[3ull * oid[j] + 1];
        }
      }
#pragma unroll
      for (int j = 0; j < kH; ++j) {
        const uint32_t v = vb + (kSkip ? w0 + 32 * j : tid);
        u[j] = v;
        // before the heavy edges a vertex without light ones keeps a label
        root[j] = split && v < nr;
        hooked[j] = false;
        if (key[j] != kInf) {
          const uint32_t a = lab[es[j]], b = lab[ed[j]];
          u[j] = a ^ b ^ v;
          root[j] = true;
          if ((a != v && b != v) || u[j] >= nr) {
            flag_err(kErrHook);
          } else if (!(min_of(mn + u[j]) == key[j] && v < u[j])) {
            root[j] = false;
            hooked[j] = true;
          }
        }
      }
      if constexpr (OUT == Out::kFound) {
        uint32_t r0, r1, t0, t1;
        block_rank2<THREADS>(root[0], hooked[0], r0, r1, t0, t1, c.w);
        slot[0] = n_next + r0;
        if (hooked[0]) {
          if (found + r1 < n) msf[found + r1] = oid[0];
          else flag_err(kErrOverflow);
        }
        n_next += t0;
        found += t1;
      } else {
        append_slots<kH>(root, &c.roots[rp], slot);
#pragma unroll
        for (int j = 0; j < kH; ++j) {
          if (!hooked[j]) continue;
          atomicOr(&flags[oid[j] >> 5], 1u << (oid[j] & 31));
          wsum += key[j] >> bits;
          ++found;
        }
      }
#pragma unroll
      for (int j = 0; j < kH; ++j) {
        const uint32_t v = vb + (kSkip ? w0 + 32 * j : tid);
        if (v < nr)
          par[v] = static_cast<uint16_t>(hooked[j] ? u[j] : root[j] ? (kTag | slot[j]) : kDone);
      }
    }
    __syncthreads();
    if (OUT == Out::kSorted) n_next = c.roots[rp];
    for (uint32_t v = tid; v < n_next; v += THREADS) mn[v] = kInf;
    if (tid == 0) c.edges[rp ^ 1] = 0;
    // label walk: an entry with kTag is a label (a root's, or one that a walk
    // has already found); a thread writes only its own vertices' entries,
    // nearer ancestors or labels, so walks shorten one another
    for (uint32_t it = 0;; ++it) {
      bool more = false;
      for (uint32_t v = tid; v < nr; v += THREADS) {
        uint32_t p = par[v];
        if (p & kTag) continue;
#pragma unroll 1
        for (int k = 0; k < 8 && !(p & kTag); ++k) p = par[p];
        par[v] = static_cast<uint16_t>(p);
        more |= !(p & kTag);
      }
      if (!__syncthreads_or(more)) break;
      if (it > kMaxRounds) {  // (a cycle; it is the same in every thread)
        flag_err(kErrJump);
        break;
      }
    }
    if (tid == 0) c.roots[rp ^ 1] = 0;
    // labels of the original vertices (an edge's endpoints in the next hook),
    // four at a time
    for (uint32_t x = tid; x < (n + 3) / 4; x += THREADS) {
      ushort4 l = reinterpret_cast<ushort4*>(lab)[x];
      auto next = [&](uint16_t y) -> uint16_t {
        return round == 0 || y != kGone ? static_cast<uint16_t>(par[y] & kGone) : y;
      };
      l.x = next(l.x);
      l.y = next(l.y);
      l.z = next(l.z);
      l.w = next(l.w);
      reinterpret_cast<ushort4*>(lab)[x] = l;
    }
    // relabel, drop self loops, feed the next minimum
    const Edge<Key>* from = L[cur];
    Edge<Key>* to = L[cur ^ 1];
    fetch_edges(0, m, from, 1);
    for (uint32_t base = 0; base + wfirst < m; base += THREADS * kU) {
      Edge<Key> e[kU];
      uint32_t a[kU], b[kU], slot[kU];
      bool keep[kU];
#pragma unroll
      for (int j = 0; j < kU; ++j) {
        keep[j] = base + w0 + 32 * j < m;
        e[j] = ne[j];
      }
      fetch_edges(base + THREADS * kU, m, from, 1);
#pragma unroll
      for (int j = 0; j < kU; ++j) {  // (an edge past the end is 0, 0)
        a[j] = par[e[j].ab & 0xffffu] & kGone;
        b[j] = par[e[j].ab >> 16] & kGone;
      }
#pragma unroll
      for (int j = 0; j < kU; ++j) keep[j] = keep[j] && a[j] != b[j];
      append_slots<kU>(keep, &c.edges[rp ^ 1], slot);
      Key key[kU];
#pragma unroll
      for (int j = 0; j < kU; ++j) {
        key[j] = e[j].key;
        e[j].ab = a[j] | (b[j] << 16);
        if (keep[j]) to[slot[j]] = e[j];
      }
      feed_minima<kU, Key>(mn, keep, a, b, key);
    }
    __syncthreads();
    m = c.edges[rp ^ 1];
    nr = n_next;
    cur ^= 1;
    ++round;
  }
  // forest output: the src<dst input copy of every forest edge
  const bool ok = !__syncthreads_or((terr & ~kErrRange) != 0);
  if (OUT == Out::kFound) {
    if (ok) {
#pragma unroll 8
      for (uint32_t k = tid; k < 3 * found; k += THREADS) {
        const uint32_t x = in[3ull * msf[k / 3] + k % 3];
        out[k] = x;
        if (k % 3 == 2) wsum += x;
      }
    }
  } else if (ok) {
    // the marked input positions in input order, listed first so that their
    // entries are then gathered side by side
    constexpr uint32_t kW = 4;  // words per thread and step
    uint32_t written = 0;
    for (uint32_t wb = 0; wb < words; wb += THREADS * kW) {
      const uint32_t k0 = wb + tid * kW;
      uint32_t f[kW], cnt = 0;
#pragma unroll
      for (uint32_t j = 0; j < kW; ++j) {
        f[j] = k0 + j < words ? __ldcg(flags + k0 + j) : 0u;
        cnt += __popc(f[j]);
      }
      // exclusive prefix of the set bits over the block's words
      uint32_t incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane_id() >= static_cast<uint32_t>(o)) incl += y;
      }
      if (lane_id() == 31) c.w[threadIdx.x >> 5] = incl;
      __syncthreads();
      uint32_t wpre = 0, tot = 0;
#pragma unroll 8
      for (int w = 0; w < THREADS / 32; ++w) {
        const uint32_t x = c.w[w];
        if (static_cast<uint32_t>(w) < (threadIdx.x >> 5)) wpre += x;
        tot += x;
      }
      __syncthreads();
      uint32_t o = written + wpre + incl - cnt;
#pragma unroll
      for (uint32_t j = 0; j < kW; ++j)
        for (uint32_t x = f[j]; x; x &= x - 1, ++o)
          if (o < n) msf[o] = (k0 + j) * 32 + (__ffs(x) - 1);
      written += tot;
    }
    __syncthreads();
#pragma unroll 8
    for (uint32_t k = tid; k < 3 * written; k += THREADS)
      out[k] = in[3ull * msf[k / 3] + k % 3];
    uint32_t mine = warp_sum(found);
    if (lane_id() == 0 && mine) atomicAdd(&c.forest, mine);
  }
  wsum = warp_sum(wsum);
  if (lane_id() == 0 && wsum) atomicAdd(&c.weight, wsum);
  __syncthreads();
  if (tid == 0) {
    res->count = !ok ? 0 : OUT == Out::kFound ? found : c.forest;
    res->weight = ok ? c.weight : 0;
    res->err = c.err;
    res->rounds = round;
  }
  __syncthreads();
  return true;
}

// The whole solve by the calling CTA (THREADS threads) of a graph of at most
// the size class, in shared_bytes(CLASS) of shared memory and
// slot_layout(CLASS).bytes of scratch.  check_ids: entries with an id >= n set
// kErrRange (they are skipped either way); check_order: entries not strictly
// (src, dst)-increasing set kErrOrder.
template <int THREADS, Out OUT, Size CLASS>
__device__ void solve(const uint32_t* __restrict__ in, uint32_t md, uint32_t n,
                      unsigned char* scratch, uint32_t* __restrict__ out, Result* res,
                      unsigned char* s_raw, bool check_ids, bool check_order = false) {
  __shared__ Counters<THREADS> c;
  constexpr Slot lay = slot_layout(CLASS);
  constexpr uint32_t cap = max_md(CLASS) / 2;
  if (CLASS != Size::kFull || n <= kSharedN) {
    if (solve_keys<THREADS, OUT, uint32_t, false>(in, md, n, scratch, lay, cap, out, res, s_raw, c,
                                                  check_ids, check_order))
      return;
    solve_keys<THREADS, OUT, unsigned long long, false>(in, md, n, scratch, lay, cap, out, res,
                                                        s_raw, c, check_ids, check_order);
    return;
  }
  if constexpr (CLASS == Size::kFull) {
    if (solve_keys<THREADS, OUT, uint32_t, true>(in, md, n, scratch, lay, cap, out, res, s_raw, c,
                                                 check_ids, check_order))
      return;
    solve_keys<THREADS, OUT, unsigned long long, true>(in, md, n, scratch, lay, cap, out, res,
                                                       s_raw, c, check_ids, check_order);
  }
}

}  // namespace small
}  // namespace kamsta
