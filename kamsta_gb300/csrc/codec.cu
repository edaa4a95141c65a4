// codec.cu -- 7-bit varint difference encoding of the directed input
// (Compression::SEVEN_BIT_DIFF_ENCODING, algorithm_configurations.hpp:18-25).
//
// Per edge the reference stores varint(src - prev_src), varint(dst),
// varint(w) (DifferenceEncodedGraph::encode_edges,
// difference_encoded_graph.hpp:175-205) with its 7-bit little-endian
// varint, continuation bit 0x80 (encode_value / decode_value,
// variable_length_encoding.hpp:6-167); the edge list is cut into chunks, each
// starting with a raw first edge and a byte offset.  The byte stream of a
// chunk here is exactly that; chunks are small (<= 4096 edges) so that the
// device decodes one chunk per CTA:
//   1. the chunk's bytes go to shared memory;
//   2. a block scan over the counts of "last byte of a value" gives every
//      value its index, and its end goes to a list;
//   3. each lane fetches its edge's values between their ends; scans over the
//      src deltas restore src; edges are written out.
// The host encoder runs on all host cores.  A decoded input feeds the normal
// solver, so a compressed graph costs about half the bytes to keep resident
// or to copy to the device.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>
#include <vector>

#include "codec.cuh"
#include "common.cuh"
#include "solver.cuh"

namespace kamsta {

namespace {

constexpr int kDecBlock = 512;

inline uint32_t varint_len(uint64_t v) {
  uint32_t n = 1;
  while (v >= 128) {
    v >>= 7;
    ++n;
  }
  return n;
}

inline uint8_t* varint_put(uint64_t v, uint8_t* o) {
  while (v >= 128) {
    *o++ = static_cast<uint8_t>((v & 0x7f) | 0x80);
    v >>= 7;
  }
  *o++ = static_cast<uint8_t>(v);
  return o;
}

// Block-wide exclusive scan of one u32 per thread; returns the total.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* excl, uint32_t* s_warp) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(kFull, incl, o);
    if (lane >= static_cast<uint32_t>(o)) incl += y;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    const uint32_t wv = lane < kDecBlock / 32 ? s_warp[lane] : 0u;
    uint32_t wi = wv;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, wi, o);
      if (lane >= static_cast<uint32_t>(o)) wi += y;
    }
    if (lane < kDecBlock / 32) s_warp[lane] = wi - wv;
    if (lane == kDecBlock / 32 - 1) s_warp[kDecBlock / 32] = wi;
  }
  __syncthreads();
  *excl = s_warp[warp] + incl - v;
  const uint32_t total = s_warp[kDecBlock / 32];
  __syncthreads();
  return total;
}

// Terminator bits (bit 7 clear, one per byte at bit 7) of a window word.
__device__ __forceinline__ uint32_t terminators(uint32_t word) { return ~word & 0x80808080u; }

// The varint in window bytes [q, q + len): its first five groups of 7 bits
// (ids and weights are 32-bit, so later groups fall away mod 2^32).  Two byte
// dot products put four groups together.
__device__ __forceinline__ uint32_t varint_at(const uint32_t* w, uint32_t q, uint32_t len) {
  const uint32_t a = w[q >> 2], b = w[(q >> 2) + 1];
  uint32_t lo = __funnelshift_r(a, b, 8 * q), mask;  // (the shift counts mod 32)
  asm("bmsk.clamp.b32 %0, 0, %1;" : "=r"(mask) : "r"(8 * len));
  lo &= mask & 0x7f7f7f7fu;
  uint32_t v = __dp4a(lo, 0x00008001u, 0u) + (__dp4a(lo, 0x80010000u, 0u) << 14);
  if (len > 4) v |= (b >> ((8 * q) & 31)) << 28;
  return v;
}

// One chunk per CTA step:
//   1. its bytes into shared memory (16-byte loads for the aligned middle);
//   2. each thread counts the value terminators (bytes without bit 7) in its
//      run of 4-byte words, a block scan numbers the values, and each thread
//      writes the end of every value that ends in its words to a list;
//   3. a warp takes 32 consecutive edges per step: each lane fetches its
//      edge's three values from the window between their ends (two words and
//      a funnel shift each, the same work in every lane), and the srcs come
//      from warp scans of the deltas;
//   4. after the warps' delta sums have been exchanged, the edges go through
//      a 384-byte warp buffer to coalesced stores.
// What bounded the decoder before was step 3 as one serial, diverging walk
// over each thread's bytes, with its values scattered over shared memory:
// 2^25 entries (184 MB encoded) 308 -> 263 us, now at 70% of the shared-memory
// wavefronts an SM can issue.
constexpr int kDecWarps = kDecBlock / 32;
constexpr int kDecEdges = kMaxChunkEdges / kDecBlock;  // per thread
constexpr size_t dec_ends_bytes(uint32_t C) { return (6ull * C + 2 + 15) & ~15ull; }
constexpr size_t dec_smem_bytes(uint32_t C) { return dec_ends_bytes(C) + 15ull * C + 64; }

__global__ void __launch_bounds__(kDecBlock, 2)
    k_decode_7bit(const uint64_t* __restrict__ chunk_off, const kamsta_wedge* __restrict__ first,
                  const uint8_t* __restrict__ data, uint64_t m, uint32_t C, uint64_t nchunks,
                  uint32_t* __restrict__ out, uint32_t* err) {
  extern __shared__ __align__(16) unsigned char smem[];
  // ends[v]: window byte behind value v - 1 (ends[0]: the chunk's first byte);
  // at most 15 * C + 16 bytes, so 16 bits hold it
  uint16_t* ends = reinterpret_cast<uint16_t*>(smem);
  // the chunk's bytes, placed as in a window that starts at the 16-byte
  // boundary at or below the chunk's first byte (<= 15 * C + 16 bytes)
  uint8_t* win = smem + dec_ends_bytes(C);
  const uint32_t* wwin = reinterpret_cast<const uint32_t*>(win);
  __shared__ uint32_t s_warp[kDecBlock / 32 + 1];
  __shared__ uint32_t s_delta[2][kDecWarps];
  __shared__ uint32_t s_out[kDecWarps][96];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t le = lanemask_lt() | (1u << lane);
  int flip = 0;
  for (uint64_t c = blockIdx.x; c < nchunks; c += gridDim.x, flip ^= 1) {
    const uint64_t e0 = c * C;
    const uint32_t ce = static_cast<uint32_t>(m - e0 < C ? m - e0 : C);  // edges in chunk
    const uint64_t b0 = chunk_off[c];
    const uint32_t nb = static_cast<uint32_t>(chunk_off[c + 1] - b0);
    const kamsta_wedge f = first[c];
    const uint32_t nv = 3 * (ce - 1);
    if (nb > 15u * C) {  // cannot come from sorted 32-bit input
      if (threadIdx.x == 0) atomicOr(err, kErrRange);
      continue;
    }
    // 16-byte loads for the aligned middle of the byte range, single bytes
    // for its ragged ends; every load lies inside [b0, b0 + nb)
    const uint64_t b1 = b0 + nb, a0 = b0 & ~15ull;
    const uint64_t m0 = (b0 + 15) & ~15ull, m1 = b1 & ~15ull;
    if (m0 < m1) {
      const uint4* src = reinterpret_cast<const uint4*>(data + m0);
      uint4* dst = reinterpret_cast<uint4*>(win + (m0 - a0));
#pragma unroll 4
      for (uint32_t q = threadIdx.x; q < static_cast<uint32_t>((m1 - m0) / 16); q += kDecBlock)
        dst[q] = __ldcs(src + q);
      for (uint64_t x = b0 + threadIdx.x; x < m0; x += kDecBlock) win[x - a0] = data[x];
      for (uint64_t x = m1 + threadIdx.x; x < b1; x += kDecBlock) win[x - a0] = data[x];
    } else {
      for (uint64_t x = b0 + threadIdx.x; x < b1; x += kDecBlock) win[x - a0] = data[x];
    }
    const uint32_t skip = static_cast<uint32_t>(b0 - a0), wend = skip + nb;
    const uint32_t nw = (wend + 3) / 4;
    // window bytes around the chunk's end no value
    if (threadIdx.x < skip) win[threadIdx.x] = 0x80;
    if (threadIdx.x < 4 * nw - wend) win[wend + threadIdx.x] = 0x80;
    __syncthreads();
    // (odd: the threads' words lie on distinct banks)
    const uint32_t perw = ((nw + kDecBlock - 1) / kDecBlock) | 1u;
    const uint32_t w_lo = min(nw, threadIdx.x * perw), w_hi = min(nw, w_lo + perw);
    uint32_t cnt = 0;
    for (uint32_t q = w_lo; q < w_hi; ++q) cnt += __popc(terminators(wwin[q]));
    uint32_t v = 0;
    const uint32_t total = block_excl_scan(cnt, &v, s_warp);
    if (total != nv) {
      if (threadIdx.x == 0) atomicOr(err, kErrRange);
      continue;
    }
    if (threadIdx.x == 0) ends[0] = static_cast<uint16_t>(skip);
    for (uint32_t q = w_lo; q < w_hi; ++q) {
      const uint32_t t = terminators(wwin[q]);
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j)
        if (t & (0x80u << (8 * j))) ends[++v] = static_cast<uint16_t>(4 * q + j + 1);
    }
    __syncthreads();
    // warp w: edges [1 + w * steps * 32, ...), 32 per step
    const uint32_t steps = (ce - 1 + kDecBlock - 1) / kDecBlock;  // <= kDecEdges
    const uint32_t a = 1 + warp * steps * 32 + lane;
    uint32_t src[kDecEdges], dst[kDecEdges], wt[kDecEdges];
    uint32_t run = 0;
#pragma unroll
    for (int k = 0; k < kDecEdges; ++k) {
      src[k] = dst[k] = wt[k] = 0;
      if (k >= static_cast<int>(steps)) break;
      const uint32_t e = a + k * 32;
      if (e < ce) {
        const uint16_t* p = ends + 3 * (e - 1);
        const uint32_t p0 = p[0], p1 = p[1], p2 = p[2], p3 = p[3];
        src[k] = varint_at(wwin, p0, p1 - p0);
        dst[k] = varint_at(wwin, p1, p2 - p1);
        wt[k] = varint_at(wwin, p2, p3 - p2);
      }
      // prefix sum of the deltas: one ballot while they are 0 or 1, as they are
      // but where ids without edges are skipped
      if (!__any_sync(kFull, src[k] > 1)) {
        const uint32_t ones = __ballot_sync(kFull, src[k] != 0);
        src[k] = run + __popc(ones & le);
        run += __popc(ones);
      } else {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(kFull, src[k], o);
          if (lane >= static_cast<uint32_t>(o)) src[k] += y;
        }
        src[k] += run;
        run = __shfl_sync(kFull, src[k], 31);
      }
    }
    if (lane == 0) s_delta[flip][warp] = run;
    __syncthreads();  // also: the window and the list are free
    uint32_t base = f.src;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w)
      if (static_cast<uint32_t>(w) < warp) base += s_delta[flip][w];
    // the chunk's entries: its raw first edge, then the decoded ones
    uint32_t* o = out + 3 * e0;
    if (threadIdx.x < 3)
      o[threadIdx.x] = threadIdx.x == 0 ? f.src : threadIdx.x == 1 ? f.dst : f.w;
    uint32_t* buf = s_out[warp];
#pragma unroll
    for (int k = 0; k < kDecEdges; ++k) {
      if (k >= static_cast<int>(steps)) break;
      const uint32_t g0 = 1 + warp * steps * 32 + k * 32;  // the step's first edge
      if (g0 >= ce) break;
      buf[3 * lane] = base + src[k];
      buf[3 * lane + 1] = dst[k];
      buf[3 * lane + 2] = wt[k];
      __syncwarp();
      const uint32_t nwords = 3 * min(32u, ce - g0);
      uint32_t* og = o + 3 * g0;
#pragma unroll
      for (uint32_t j = 0; j < 3; ++j)
        if (j * 32 + lane < nwords) __stcs(og + j * 32 + lane, buf[j * 32 + lane]);
      __syncwarp();
    }
  }
}

}  // namespace

kamsta_status encode_7bit(const kamsta_wedge* e, uint64_t m, uint32_t C, uint64_t* off,
                          kamsta_wedge* first, uint8_t* data, uint64_t cap, uint64_t* bytes) {
  *bytes = 0;
  if (C == 0 || C > kMaxChunkEdges) {
    set_error("encode_7bit: chunk_edges must be in [1, 4096]");
    return KAMSTA_E_INPUT;
  }
  const uint64_t nch = (m + C - 1) / C;
  std::vector<uint64_t> len(nch, 0);
  const unsigned hw = std::max(1u, std::min(32u, std::thread::hardware_concurrency()));
  auto par = [&](auto&& fn) {
    std::vector<std::thread> th;
    for (unsigned t = 0; t < hw; ++t)
      th.emplace_back([&, t] {
        for (uint64_t c = nch * t / hw; c < nch * (t + 1) / hw; ++c) fn(c);
      });
    for (auto& x : th) x.join();
  };
  std::atomic<bool> bad{false};
  par([&](uint64_t c) {
    uint64_t l = 0;
    const uint64_t a = c * C, z = std::min<uint64_t>(m, a + C);
    for (uint64_t i = a + 1; i < z; ++i) {
      if (e[i].src < e[i - 1].src) bad = true;  // deltas must be non-negative
      l += varint_len(static_cast<uint64_t>(e[i].src) - e[i - 1].src) + varint_len(e[i].dst) +
           varint_len(e[i].w);
    }
    len[c] = l;
  });
  if (bad) {
    set_error("encode_7bit: input must be sorted by src");
    return KAMSTA_E_INPUT;
  }
  uint64_t total = 0;
  for (uint64_t c = 0; c < nch; ++c) {
    if (off) off[c] = total;
    total += len[c];
  }
  if (off) off[nch] = total;
  *bytes = total;
  if (!data) return KAMSTA_OK;
  if (!off || !first) {
    set_error("encode_7bit: chunk_offset and chunk_first are required");
    return KAMSTA_E_INPUT;
  }
  if (total > cap) {
    set_error("encode_7bit: data capacity too small (required bytes in data_bytes)");
    return KAMSTA_E_INPUT;
  }
  par([&](uint64_t c) {
    const uint64_t a = c * C, z = std::min<uint64_t>(m, a + C);
    first[c] = e[a];
    uint8_t* o = data + off[c];
    for (uint64_t i = a + 1; i < z; ++i) {
      o = varint_put(static_cast<uint64_t>(e[i].src) - e[i - 1].src, o);
      o = varint_put(e[i].dst, o);
      o = varint_put(e[i].w, o);
    }
  });
  return KAMSTA_OK;
}

kamsta_status decode_7bit(const kamsta_cgraph& g, kamsta_wedge* d_out, uint32_t* d_err,
                          cudaStream_t st) {
  if (g.m_directed == 0) return KAMSTA_OK;
  if (g.chunk_edges == 0 || g.chunk_edges > kMaxChunkEdges ||
      g.num_chunks != (g.m_directed + g.chunk_edges - 1) / g.chunk_edges) {
    set_error("decode_7bit: inconsistent chunk layout");
    return KAMSTA_E_INPUT;
  }
  const size_t smem = dec_smem_bytes(g.chunk_edges);
  cudaError_t e = cudaFuncSetAttribute(k_decode_7bit, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       static_cast<int>(smem));
  if (e != cudaSuccess) return cuda_status(e, "cudaFuncSetAttribute(k_decode_7bit)");
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const uint64_t grid = std::min<uint64_t>(g.num_chunks, uint64_t(sms) * 8);
  k_decode_7bit<<<static_cast<uint32_t>(grid), kDecBlock, smem, st>>>(
      g.chunk_offset, g.chunk_first, g.data, g.m_directed, g.chunk_edges, g.num_chunks,
      reinterpret_cast<uint32_t*>(d_out), d_err);
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e, "k_decode_7bit");
  return KAMSTA_OK;
}

}  // namespace kamsta
