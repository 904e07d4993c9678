// Batched Mutations: many filters per pass over the vertical index and the missing-interval events.
//
// The plain path streams every container once per query. Here the filters of a batch are
// transposed into 16-bit query masks per row (bit q of group g = row in filter 16 g + q) and every
// container element and event is read once per pass of up to 256 queries. Both passes count
// 32 queries per lane in bit-sliced counters. Results are bit-identical to the single-query kernels.
//
//   transpose_kernel       filter row sets -> masks, pass-major rows (32 B per row and pass)
//   mut_ctr_batch_kernel   container pass, one warp per (position, chunk range) unit: |F_q ∩ c|
//                          for every container c (reference: mutations_node.cpp:138-190)
//   mut_ctr_narrow_kernel  the same for a pass of at most 32 queries, masks in shared memory; its run
//   mut_runs_narrow_kernel containers apart, the filters' words in shared memory
//   mut_cov_batch_kernel   missing-interval and coverage boundary events (reference:
//                          mutations_node.cpp:51-136)
//   mut_final_batch_kernel prefix sums and reference counts per query
//   mut_select_kernel      splits the slots by their filter's cardinality: none for empty filters,
//                          the row-index pass for filters of at most sparse_max rows, the dense
//                          passes above (over a compacted slot list) for the others
//   mut_sparse_batch_kernel the row-index pass of the sparse slots
#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <string>

#include "device.h"
#include "mutations_common.cuh"
#include "rows_rule.cuh"

namespace rhygpu {

constexpr uint32_t MUT_GROUP = 16;   // queries per 16-bit mask
constexpr uint32_t PASS_GROUPS = 16;  // groups per mask pass (256 queries, one 32-byte sector per row)

namespace {

constexpr uint32_t BT = 256;

// Mask layout: pass p (queries 256 p ..) holds rows x wp(p) u32, wp(p) = min(8, nqc - 8 p) with
// nqc = ceil(nq / 32); u32 c of a row holds groups 2c (low half) and 2c + 1 (high half) of the pass.
// Every pass but the last is rows x 8 u32, so pass p starts at u16 offset p * rows * 16.
__device__ __forceinline__ uint32_t pass_width_u32(uint32_t nqc, uint32_t pass) {
   return nqc - 8 * pass < 8 ? nqc - 8 * pass : 8u;
}

// A warp turns four words of every filter into 128 row masks: per 32 filters, lane l reads the four words of
// filter l, four transposes give lane l those filters' bits of its four rows, and a row's mask words of a pass
// are stored together. Bound by the latency of the filter reads (16 bytes of 32 filters each). 2M rows, 263
// queries: 48 us; 215 with 32 ballots per word and the masks staged in shared memory for the stores.
constexpr uint32_t TR_WORDS = 4 * (BT / 32);  // filter words per CTA
static_assert(CHUNK_WORDS % TR_WORDS == 0, "whole CTAs per chunk");
__global__ void __launch_bounds__(BT) transpose_kernel(const uint32_t* __restrict__ tiles,
                                                       const uint32_t* __restrict__ lists, uint32_t nq_max,
                                                       uint32_t nchunks, uint32_t* __restrict__ R) {
   const uint32_t nq = lists[2 * nq_max];  // dense slots: lists[0 .. nq)
   const uint32_t lane = threadIdx.x & 31;
   const size_t words = static_cast<size_t>(nchunks) * CHUNK_WORDS, rows = 32 * words;
   const uint32_t nqc = (nq + 31) / 32;
   const uint32_t w = blockIdx.x * TR_WORDS + 4 * (threadIdx.x >> 5);
   for (uint32_t pass = 0; 8 * pass < nqc; ++pass) {
      const uint32_t wp = pass_width_u32(nqc, pass);
      uint32_t m[4][8];
#pragma unroll
      for (uint32_t c = 0; c < 8; ++c) {
         if (c >= wp) break;
         const uint32_t q = 256 * pass + 32 * c + lane;
         uint4 x = make_uint4(0, 0, 0, 0);
         if (q < nq) x = __ldg(reinterpret_cast<const uint4*>(tiles + lists[q] * words + w));
         m[0][c] = warp_transpose32(x.x, lane);
         m[1][c] = warp_transpose32(x.y, lane);
         m[2][c] = warp_transpose32(x.z, lane);
         m[3][c] = warp_transpose32(x.w, lane);
      }
      uint32_t* dst = R + pass * rows * 8 + (32 * static_cast<size_t>(w) + lane) * wp;
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k, dst += 32 * wp) {
         if (wp == 8) {
            reinterpret_cast<uint4*>(dst)[0] = make_uint4(m[k][0], m[k][1], m[k][2], m[k][3]);
            reinterpret_cast<uint4*>(dst)[1] = make_uint4(m[k][4], m[k][5], m[k][6], m[k][7]);
         } else {
#pragma unroll
            for (uint32_t c = 0; c < 7; ++c)
               if (c < wp) dst[c] = m[k][c];
         }
      }
   }
}

// Per-lane counters of the 32 queries of one mask word, as bit planes: bit q of p[k] is bit k of query q's
// count. Rows are added eight at a time by a Harley-Seal tree of carry-save adders (one LOP3 for the sum
// and one for the carry of three words), or two at a time, and the carry word ripples through the planes
// above (two LOP3 each). The passes that count rows are bound by issue slots: byte counters for the
// multiples of eight took 40 instructions a block, the planes take 16. At most COUNT_MAX rows a lane.
struct BitCounter {
   static constexpr uint32_t PLANES = 11, COUNT_MAX = (1u << PLANES) - 1;
   uint32_t p[PLANES];
   uint32_t rows;

   __device__ __forceinline__ void clear() {
#pragma unroll
      for (uint32_t k = 0; k < PLANES; ++k) p[k] = 0;
      rows = 0;
   }
   __device__ __forceinline__ static void csa(uint32_t& carry, uint32_t& sum, uint32_t a, uint32_t b, uint32_t c) {
      const uint32_t u = a ^ b;
      carry = (a & b) | (u & c);
      sum = u ^ c;
   }
   template <uint32_t FROM>
   __device__ __forceinline__ void ripple(uint32_t carry) {
#pragma unroll
      for (uint32_t k = FROM; k < PLANES; ++k) {
         const uint32_t t = p[k] & carry;
         p[k] ^= carry;
         carry = t;
      }
   }
   __device__ __forceinline__ void add8(const uint32_t (&m)[8]) {
      uint32_t twos_a, twos_b, fours_a, fours_b, eights;
      csa(twos_a, p[0], p[0], m[0], m[1]);
      csa(twos_b, p[0], p[0], m[2], m[3]);
      csa(fours_a, p[1], p[1], twos_a, twos_b);
      csa(twos_a, p[0], p[0], m[4], m[5]);
      csa(twos_b, p[0], p[0], m[6], m[7]);
      csa(fours_b, p[1], p[1], twos_a, twos_b);
      csa(eights, p[2], p[2], fours_a, fours_b);
      ripple<3>(eights);
      rows += 8;
   }
   __device__ __forceinline__ void add2(uint32_t m0, uint32_t m1) {
      uint32_t twos;
      csa(twos, p[0], p[0], m0, m1);
      ripple<1>(twos);
      rows += 2;
   }
   __device__ __forceinline__ bool full() const { return rows > COUNT_MAX - 8; }
};

// How a warp shares out the mask words of a pass that has wp of them per row: lane (g, w) takes word w
// of every G-th row of a window of 8 G rows, w < W the smallest power of two >= wp, G = 32 / W. A pass of
// 225 to 256 queries has 8 words (4 rows at a time), one of at most 32 queries one word (32 rows).
struct LaneSplit {
   uint32_t wsh, g, w, G;
   __device__ __forceinline__ LaneSplit(uint32_t wp, uint32_t lane) {
      wsh = wp > 4 ? 3u : wp > 2 ? 2u : wp > 1 ? 1u : 0u;
      g = lane >> wsh;
      w = lane & ((1u << wsh) - 1u);
      G = 32u >> wsh;
   }
};

// Adds the rows row_of(t), t < cnt, of a window to the counters: every lane reads its word of each of its
// rows' masks (Rw: word l.w of row 0; zero past wp) and adds the words. A window of at most two rows per
// lane, as most arrays are in a pass of one word, takes the shorter addition.
template <typename RowOf>
__device__ __forceinline__ void count_window_bits(BitCounter& k, const LaneSplit& l, uint32_t cnt,
                                                  const uint32_t* __restrict__ Rw, uint32_t wp, RowOf&& row_of) {
   const uint32_t n = l.w < wp ? cnt : 0u;
   if (cnt <= 2 * l.G) {
      uint32_t m[2];
#pragma unroll
      for (uint32_t i = 0; i < 2; ++i) {
         const uint32_t t = l.G * i + l.g, e = row_of(t);
         m[i] = t < n ? __ldg(Rw + static_cast<size_t>(e) * wp) : 0u;
      }
      k.add2(m[0], m[1]);
      return;
   }
   uint32_t m[8];
#pragma unroll
   for (uint32_t i = 0; i < 8; ++i) {
      const uint32_t t = l.G * i + l.g, e = row_of(t);
      m[i] = t < n ? __ldg(Rw + static_cast<size_t>(e) * wp) : 0u;
   }
   k.add8(m);
}

// Sums the warp's counters over the row groups, clears them and calls put(i, q, count) for the queries that
// this lane ends up with: query q of the mask word l.w, i counting the lane's queries (at most 8, the same
// ones each time). The counts leave the planes as pairs of 16 bits (32 lanes of COUNT_MAX fit), and each
// exchange between row groups halves the pairs a lane holds. qn: the queries a mask word can have.
template <uint32_t N, uint32_t M>
__device__ __forceinline__ void halve_words(uint32_t (&W)[M], uint32_t off) {
   const bool up = threadIdx.x & off;
#pragma unroll
   for (uint32_t i = 0; i < N; ++i) {
      const uint32_t keep = up ? W[i + N] : W[i], send = up ? W[i] : W[i + N];
      W[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, off);
   }
}
// Four queries' (4 j .. 4 j + 3) sums over the planes [B, E), at most 7 of them, one byte each.
template <uint32_t B, uint32_t E>
__device__ __forceinline__ uint32_t plane_bytes(const BitCounter& k, uint32_t j) {
   uint32_t x = 0;
#pragma unroll
   for (uint32_t b = B; b < E; ++b) x += ((((k.p[b] >> (4 * j)) & 0xFu) * 0x00204081u) & 0x01010101u) << (b - B);
   return x;
}
template <uint32_t B, uint32_t E>
__device__ __forceinline__ void add_planes(const BitCounter& k, uint32_t (&W)[16], uint32_t qn) {
#pragma unroll
   for (uint32_t j = 0; j < 8; ++j) {
      if (4 * j >= qn) continue;
      const uint32_t x = plane_bytes<B, E>(k, j);
      W[2 * j] += (x & 0x00FF00FFu) << B;
      W[2 * j + 1] += ((x >> 8) & 0x00FF00FFu) << B;
   }
}
// FEW: a flush follows few rows (an event pass's position: 16 rows a lane and less), so that the upper planes
// are mostly empty and it is worth a look, and narrow passes skip the queries they don't have. The container
// pass flushes after hundreds of rows, and the tests and the registers they hold cost it 5%.
template <bool FEW, typename Put>
__device__ __forceinline__ void take_counts(BitCounter& k, const LaneSplit& l, uint32_t qn, Put&& put) {
   const uint32_t lane = threadIdx.x & 31;
   constexpr uint32_t P = BitCounter::PLANES;
   const uint32_t high = k.p[7] | k.p[8] | k.p[9] | k.p[10];
   uint32_t W[16];  // W[2 j + h]: queries 4 j + h and, in the upper half, 4 j + 2 + h
   if (FEW) {
#pragma unroll
      for (uint32_t j = 0; j < 16; ++j) W[j] = 0;
      add_planes<0, 3>(k, W, qn);
      if (__any_sync(0xFFFFFFFFu, (k.p[3] | k.p[4] | k.p[5] | k.p[6] | high) != 0u)) add_planes<3, 7>(k, W, qn);
   } else {
#pragma unroll
      for (uint32_t j = 0; j < 8; ++j) {
         const uint32_t x = plane_bytes<0, 7>(k, j);
         W[2 * j] = x & 0x00FF00FFu;
         W[2 * j + 1] = (x >> 8) & 0x00FF00FFu;
      }
   }
   if (__any_sync(0xFFFFFFFFu, high != 0u)) add_planes<7, P>(k, W, 32);
   k.clear();
   halve_words<8>(W, 16);
   halve_words<4>(W, 8);
   uint32_t first = (lane & 16 ? 8u : 0u) + (lane & 8 ? 4u : 0u), n = 4;
   if (l.wsh < 3) {
      halve_words<2>(W, 4);
      first += lane & 4 ? 2u : 0u;
      n = 2;
   }
   if (l.wsh < 2) {
      halve_words<1>(W, 2);
      first += lane & 2 ? 1u : 0u;
      n = 1;
   }
   if (l.wsh < 1) {
      W[0] += __shfl_xor_sync(0xFFFFFFFFu, W[0], 1);
      if (lane & 1) n = 0;
   }
#pragma unroll
   for (uint32_t i = 0; i < 4; ++i) {
      if (i >= n) continue;
      const uint32_t word = first + i, q = 4 * (word >> 1) + (word & 1u);
      put(2 * i, q, W[i] & 0xFFFFu);
      put(2 * i + 1, q + 2, W[i] >> 16);
   }
}

// One warp per (unit, pass): for every symbol present at the unit's position, the containers of the
// unit's chunks are counted for all queries of the pass. The lanes split the pass's mask words and the
// rows of a window between them (LaneSplit) and add the words into bit-sliced counters; the row
// groups' counts are summed with shuffles and added to counts once per symbol. Bitset containers are
// expanded 1024 rows at a time into a per-warp row list in shared memory.
// Bound: issue slots (60% of them taken) and the latency of the mask gathers; loading the next containers'
// descriptors and rows ahead cost 10%, and three CTAs per SM in place of four 20%. 2M rows and 263 queries
// (256 and 7): 1.11 ms, 1.26 with byte counters; 0.75 without the 7 (mut_ctr_narrow_kernel).
__global__ void __launch_bounds__(BT, 4) mut_ctr_batch_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                           const CtrUnit* __restrict__ units, uint32_t n_units,
                                                           const uint16_t* __restrict__ R,
                                                           const uint32_t* __restrict__ lists, uint32_t nq_max,
                                                           uint32_t* __restrict__ counts) {
   __shared__ uint16_t list[BT / 32][1024];
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const uint32_t u = blockIdx.x * (BT / 32) + warp;
   const uint32_t nq = lists[2 * nq_max];  // dense slots: lists[0 .. nq)
   if (u >= n_units || blockIdx.y * PASS_GROUPS * MUT_GROUP >= nq) return;  // the whole warp leaves
   if (pass_width_u32((nq + 31) / 32, blockIdx.y) == 1) return;              // mut_ctr_narrow_kernel's
   const DevSeqCol* cs = &tab->seq[col];
   const uint32_t L = cs->L;
   const size_t per_query = static_cast<size_t>(cs->nsym) * L;
   const CtrDesc* __restrict__ ctrs = cs->ctrs;
   const uint16_t* __restrict__ payload = cs->payload;
   const uint32_t pass = blockIdx.y;
   const uint32_t nqc = (nq + 31) / 32;
   const size_t rows = static_cast<size_t>(tab->nchunks) * CHUNK_ROWS;
   const uint32_t wp = pass_width_u32(nqc, pass);  // mask words per row in this pass
   const LaneSplit ls(wp, lane);
   const uint32_t WIN = 8 * ls.G;
   const uint32_t* Rp = reinterpret_cast<const uint32_t*>(R + static_cast<size_t>(pass) * rows * 16);

   const CtrUnit unit = units[u];
   const uint32_t p = unit.pos, v0 = unit.v0, nv = unit.v1 - unit.v0;
   uint32_t cb = 0, ce = 0;  // lane i: the containers of chunk v0 + i at p
   if (lane < nv) {
      cb = __ldg(cs->off + static_cast<size_t>(v0 + lane) * L + p);
      ce = __ldg(cs->off + static_cast<size_t>(v0 + lane) * L + p + 1);
   }
   uint32_t symmask = 0;
   for (uint32_t i = cb; i < ce; ++i) symmask |= 1u << __ldg(&ctrs[i].sym);
   symmask = __reduce_or_sync(0xFFFFFFFFu, symmask);
   uint16_t* wl = list[warp];
   while (symmask) {
      const uint32_t s = __ffs(symmask) - 1;
      symmask &= symmask - 1;
      uint32_t idx = 0xFFFFFFFFu;
      for (uint32_t i = cb; i < ce; ++i)
         if (__ldg(&ctrs[i].sym) == s) idx = i;
      uint32_t have = __ballot_sync(0xFFFFFFFFu, idx != 0xFFFFFFFFu);
      BitCounter k;
      k.clear();
      // adds the counts to the query tables (at the end of a symbol, or before the planes could overflow)
      auto flush = [&]() {
         take_counts<false>(k, ls, 32, [&](uint32_t, uint32_t q, uint32_t c) {
            const uint32_t slot = 256 * pass + 32 * ls.w + q;
            if (c && slot < nq)
               atomicAdd(counts + static_cast<size_t>(lists[slot]) * per_query + static_cast<size_t>(s) * L + p, c);
         });
      };
      auto window = [&](uint32_t cnt, const uint32_t* Rw, auto&& row_of) {
         count_window_bits(k, ls, cnt, Rw, wp, row_of);
         if (k.full()) flush();
      };
      while (have) {
         const uint32_t j = __ffs(have) - 1;
         have &= have - 1;
         const uint32_t ci = __shfl_sync(0xFFFFFFFFu, idx, j);
         const uint4 raw = __ldg(reinterpret_cast<const uint4*>(ctrs) + ci);
         const CtrDesc d = *reinterpret_cast<const CtrDesc*>(&raw);
         const uint32_t* Rw = Rp + static_cast<size_t>(v0 + j) * CHUNK_ROWS * wp + ls.w;
         if (d.type == CT_BITSET) {
            const uint32_t* bits = reinterpret_cast<const uint32_t*>(payload + d.payload);
            for (uint32_t wb = 32u * unit.w0; wb < 32u * unit.w1; wb += 32) {
               uint32_t x = __ldcs(bits + wb + lane);
               const uint32_t c = __popc(x);
               uint32_t incl = c;
#pragma unroll
               for (uint32_t o = 1; o < 32; o <<= 1) {
                  const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                  if (lane >= o) incl += y;
               }
               const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
               uint32_t at = incl - c;
               while (x) {
                  const uint32_t b = __ffs(x) - 1;
                  x &= x - 1;
                  wl[at++] = static_cast<uint16_t>(32 * (wb + lane) + b);
               }
               __syncwarp();
               for (uint32_t base = 0; base < total; base += WIN)
                  window(total - base, Rw, [&](uint32_t t) { return base + t < total ? wl[base + t] : 0u; });
               __syncwarp();
            }
         } else if (unit.w0 != 0) {
            continue;  // a later part of a heavy chunk: its bitset words only
         } else if (d.type == CT_ARRAY) {
            const uint32_t n = d.card_m1 + 1u;
            const uint16_t* a = payload + d.payload;
            // container payloads stream through once: read them evict-first so that the masks the
            // gathers reuse stay in L2
            if (ls.wsh == 3) {
               uint32_t next = lane < n ? __ldcs(a + lane) : 0u;
               for (uint32_t base = 0; base < n; base += 32) {
                  const uint32_t x = next;
                  next = base + 32 + lane < n ? __ldcs(a + base + 32 + lane) : 0u;
                  window(n - base, Rw, [&](uint32_t t) { return __shfl_sync(0xFFFFFFFFu, x, t); });
               }
            } else {
               for (uint32_t base = 0; base < n; base += WIN)
                  window(n - base, Rw, [&](uint32_t t) { return base + t < n ? static_cast<uint32_t>(__ldcs(a + base + t)) : 0u; });
            }
         } else {
            const uint16_t* r = payload + d.payload;
            for (uint32_t i = 0; i < d.nruns; ++i) {
               const uint32_t s0 = __ldg(r + 2 * i), n = __ldg(r + 2 * i + 1) + 1u;
               for (uint32_t base = 0; base < n; base += WIN)
                  window(n - base, Rw, [&](uint32_t t) { return s0 + base + t; });
            }
         }
      }
      if (k.rows) flush();
   }
}

// Container pass of a pass of one mask word (blockIdx.y: its first or second 16 queries). A CTA stages the
// 16-bit masks of a chunk's rows in shared memory and counts its share of the chunk's containers, 32 at a time
// per warp: arrays of up to NARROW_LIGHT rows four at a time, eight lanes each; longer arrays with the whole
// warp; bitsets by population counts with the filters' own words; run containers: mut_runs_narrow_kernel. Two rows' masks make a word whose
// bits are added to nibble counters (nibble k of nib[j]: query j + 4 (k % 4)); their bytes are summed over
// the lanes. Bound by issue slots, then by the gathers (one of 32 banks each): a mask from L2 takes a sector,
// and the wide pass, whose lanes then are all on different rows, took 350 us at 2M rows and 7 queries,
// 137 us so; 107 and 46 us at 500,000 rows and 12 queries. A pass of two words stays with the wide pass: 400 us
// at 2M rows against four times 130.
constexpr uint32_t NARROW_T = 1024, NARROW_LIGHT = 240;  // 15 additions of 16 rows to a nibble
constexpr uint32_t NARROW_SMEM = CHUNK_ROWS * 2;

// the 16 queries' counts of a lane's nibbles: byte k of E[j] is query j + 8 (k & 1) + 4 (k >> 1)
__device__ __forceinline__ void nibble_bytes(const uint32_t (&nib)[4], uint32_t (&E)[4]) {
#pragma unroll
   for (uint32_t j = 0; j < 4; ++j) {
      const uint32_t a = nib[j] & 0x0F0F0F0Fu, b = (nib[j] >> 4) & 0x0F0F0F0Fu;
      E[j] = __byte_perm(a + (a >> 16), b + (b >> 16), 0x5410);
   }
}
// adds rows row_of(t) < CHUNK_ROWS for the t below n among t0 + stride * i, i < 2 U
template <uint32_t U, typename RowOf>
__device__ __forceinline__ void add_masks(uint32_t (&nib)[4], const uint16_t* masks, uint32_t t0, uint32_t stride, uint32_t n,
                                          RowOf&& row_of) {
   uint32_t row[2 * U];
#pragma unroll
   for (uint32_t i = 0; i < 2 * U; ++i) row[i] = t0 + stride * i < n ? row_of(t0 + stride * i) : 0xFFFFFFFFu;
#pragma unroll
   for (uint32_t i = 0; i < 2 * U; i += 2) {
      const uint32_t m0 = row[i] < CHUNK_ROWS ? masks[row[i]] : 0u, m1 = row[i + 1] < CHUNK_ROWS ? masks[row[i + 1]] : 0u;
      const uint32_t w = m0 | (m1 << 16);
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) nib[j] += (w >> j) & 0x11111111u;
   }
}

__global__ void __launch_bounds__(NARROW_T, 1) mut_ctr_narrow_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                                     const uint32_t* __restrict__ filters,
                                                                     const uint16_t* __restrict__ R,
                                                                     const uint32_t* __restrict__ lists, uint32_t nq_max,
                                                                     uint32_t per_chunk, uint32_t* __restrict__ counts) {
   extern __shared__ __align__(16) uint16_t masks[];
   __shared__ uint32_t next;
   const uint32_t nq = lists[2 * nq_max];  // dense slots: lists[0 .. nq)
   const uint32_t nqc = (nq + 31) / 32, pass = (nqc + 7) / 8 - 1, q0 = 256 * pass + 16 * blockIdx.y;
   if (nq == 0 || pass_width_u32(nqc, pass) != 1 || q0 >= nq) return;
   const DevSeqCol* cs = &tab->seq[col];
   const uint32_t L = cs->L, lane = threadIdx.x & 31;
   const uint32_t v = blockIdx.x / per_chunk, part = blockIdx.x % per_chunk;
   const size_t words = static_cast<size_t>(tab->nchunks) * CHUNK_WORDS, rows = 32 * words;
   const size_t per_query = static_cast<size_t>(cs->nsym) * L;
   {
      const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint32_t*>(R) + pass * rows * 8 +
                                                        static_cast<size_t>(v) * CHUNK_ROWS);
      const uint32_t half = blockIdx.y ? 0x7632u : 0x5410u;
      uint2* dst = reinterpret_cast<uint2*>(masks);
#pragma unroll 8
      for (uint32_t i = threadIdx.x; i < CHUNK_ROWS / 4; i += NARROW_T) {
         const uint4 x = __ldg(src + i);
         dst[i] = make_uint2(__byte_perm(x.x, x.y, half), __byte_perm(x.z, x.w, half));
      }
   }
   if (threadIdx.x == 0) next = 0;
   const CtrDesc* __restrict__ ctrs = cs->ctrs;
   const uint16_t* __restrict__ payload = cs->payload;
   const uint32_t a = __ldg(cs->off + static_cast<size_t>(v) * L), n_all = __ldg(cs->off + static_cast<size_t>(v) * L + L) - a;
   const uint32_t c0 = a + static_cast<uint32_t>(static_cast<uint64_t>(n_all) * part / per_chunk);
   const uint32_t c1 = a + static_cast<uint32_t>(static_cast<uint64_t>(n_all) * (part + 1) / per_chunk);
   // the count tables of the queries this lane adds to: two of a light array, one of the others
   auto table_of = [&](uint32_t q) { return q0 + q < nq ? counts + lists[q0 + q] * per_query : nullptr; };
   const uint32_t qa = ((lane >> 1) & 3u) + 4 * (lane & 1u);
   const uint32_t qh = (lane >> 3) + 8 * ((lane >> 2) & 1u) + 4 * (lane & 1u);  // of the lanes with bit 1 clear
   uint32_t* const ta = table_of(qa);
   uint32_t* const tb = table_of(qa + 8);
   uint32_t* const th = table_of(qh);
   __syncthreads();
   for (;;) {
      uint32_t c = 0;
      if (lane == 0) c = atomicAdd(&next, 32u);
      c = c0 + __shfl_sync(0xFFFFFFFFu, c, 0);
      if (c >= c1) break;
      const bool have = c + lane < c1;
      uint4 raw = make_uint4(0, 0, 0, 0);
      if (have) raw = __ldg(reinterpret_cast<const uint4*>(ctrs) + c + lane);
      const CtrDesc mine = *reinterpret_cast<const CtrDesc*>(&raw);
      const uint32_t card = have ? mine.card_m1 + 1u : 0u;
      const bool light = have && mine.type == CT_ARRAY && card <= NARROW_LIGHT;
      const uint32_t n_light = light ? card : 0u, cell = mine.sym * L + mine.key;  // below 2^32: nsym * L is
#pragma unroll 1
      for (uint32_t k = 0; k < 8; ++k) {
         const uint32_t j = 4 * k + (lane >> 3);
         const uint32_t n = __shfl_sync(0xFFFFFFFFu, n_light, j), at = __shfl_sync(0xFFFFFFFFu, cell, j);
         const uint16_t* p = payload + __shfl_sync(0xFFFFFFFFu, mine.payload, j);
         const uint32_t n_max = __reduce_max_sync(0xFFFFFFFFu, n);
         if (n_max == 0) continue;
         uint32_t nib[4] = {0, 0, 0, 0}, E[4];
#pragma unroll 1
         for (uint32_t t = 0; t < n_max; t += 64)
            add_masks<4>(nib, masks, t + (lane & 7u), 8, n, [&](uint32_t i) { return static_cast<uint32_t>(__ldcs(p + i)); });
         nibble_bytes(nib, E);
         halve_words<2>(E, 4);
         halve_words<1>(E, 2);
         E[0] += __shfl_xor_sync(0xFFFFFFFFu, E[0], 1);
         const uint32_t x = E[0] >> (lane & 1u ? 16 : 0);  // queries qa and qa + 8
         if (ta && (x & 0xFFu)) atomicAdd(ta + at, x & 0xFFu);
         if (tb && ((x >> 8) & 0xFFu)) atomicAdd(tb + at, (x >> 8) & 0xFFu);
      }
      uint32_t heavy = __ballot_sync(0xFFFFFFFFu, have && !light && mine.type != CT_RUN);
      while (heavy) {
         const uint32_t j = __ffs(heavy) - 1;
         heavy &= heavy - 1;
         const uint4 dr = make_uint4(__shfl_sync(0xFFFFFFFFu, raw.x, j), __shfl_sync(0xFFFFFFFFu, raw.y, j),
                                     __shfl_sync(0xFFFFFFFFu, raw.z, j), __shfl_sync(0xFFFFFFFFu, raw.w, j));
         const CtrDesc d = *reinterpret_cast<const CtrDesc*>(&dr);
         const uint16_t* p = payload + d.payload;
         const uint32_t at = d.sym * L + d.key;
         // counts rows row_of(t), t < n <= 61,440: the pairs' sums fit 16 bits
         auto count_rows = [&](uint32_t n, auto&& row_of) {
            uint32_t acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
            for (uint32_t b = 0; b < n; b += 960) {  // 15 additions of 64 rows to a nibble
               uint32_t nib[4] = {0, 0, 0, 0}, E[4];
#pragma unroll 1
               for (uint32_t t = b; t < min(b + 960, n); t += 320)
                  add_masks<5>(nib, masks, t + lane, 32, n, row_of);
               nibble_bytes(nib, E);
#pragma unroll
               for (uint32_t i = 0; i < 4; ++i) {
                  acc[2 * i] += E[i] & 0x00FF00FFu;
                  acc[2 * i + 1] += (E[i] >> 8) & 0x00FF00FFu;
               }
            }
            halve_words<4>(acc, 16);
            halve_words<2>(acc, 8);
            halve_words<1>(acc, 4);
            acc[0] += __shfl_xor_sync(0xFFFFFFFFu, acc[0], 2);
            acc[0] += __shfl_xor_sync(0xFFFFFFFFu, acc[0], 1);
            const uint32_t x = lane & 1u ? acc[0] >> 16 : acc[0] & 0xFFFFu;
            if (!(lane & 2u) && th && x) atomicAdd(th + at, x);
         };
         if (d.type == CT_ARRAY) {
            count_rows(d.card_m1 + 1u, [&](uint32_t i) { return static_cast<uint32_t>(__ldcs(p + i)); });
         } else {
            const uint4* bits = reinterpret_cast<const uint4*>(p);
#pragma unroll 1
            for (uint32_t q = 0; q < 16 && q0 + q < nq; ++q) {
               const uint4* f = reinterpret_cast<const uint4*>(filters + lists[q0 + q] * words + static_cast<size_t>(v) * CHUNK_WORDS);
               uint32_t k = 0;
#pragma unroll 4
               for (uint32_t i = lane; i < CHUNK_WORDS / 4; i += 32) {
                  const uint4 x = __ldg(bits + i), y = __ldg(f + i);
                  k += __popc(x.x & y.x) + __popc(x.y & y.y) + __popc(x.z & y.z) + __popc(x.w & y.w);
               }
               k = __reduce_add_sync(0xFFFFFFFFu, k);
               if (lane == 0 && k) atomicAdd(counts + lists[q0 + q] * per_query + at, k);
            }
         }
      }
   }
}

// The run containers of such a pass, by population counts with the filters' words of the chunk, which a CTA stages in
// shared memory, 16 filters at a time; a warp takes a container, 32 runs of it at once: each lane the words of its
// own run, and the words of a run of more than NARROW_RUN rows the whole warp. One of many long runs is read as
// the bitset that filters have of it. Bound by the shared-memory reads, one per word and filter. 16 queries over 64
// sites of 1,800 runs each at 70,000 rows: 51 us; 760 us as a part of the kernel above, which took their rows
// from the masks and reduced the counts once per run.
constexpr uint32_t NARROW_RUN = 96;
__global__ void __launch_bounds__(NARROW_T, 1) mut_runs_narrow_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                                      const uint32_t* __restrict__ filters,
                                                                      const uint32_t* __restrict__ lists, uint32_t nq_max,
                                                                      uint32_t per_chunk, uint32_t* __restrict__ counts) {
   extern __shared__ __align__(16) uint32_t words_of[];  // 16 filters x CHUNK_WORDS
   static_assert(NARROW_SMEM == 16 * CHUNK_WORDS * 4, "16 filters of a chunk");
   __shared__ uint32_t next;
   const uint32_t nq = lists[2 * nq_max];  // dense slots: lists[0 .. nq)
   const uint32_t nqc = (nq + 31) / 32, pass = (nqc + 7) / 8 - 1, q0 = 256 * pass + 16 * blockIdx.y;
   if (nq == 0 || pass_width_u32(nqc, pass) != 1 || q0 >= nq) return;
   const DevSeqCol* cs = &tab->seq[col];
   const uint32_t v = blockIdx.x / per_chunk, part = blockIdx.x % per_chunk, lane = threadIdx.x & 31;
   const uint32_t a = __ldg(cs->run_off + v), n = __ldg(cs->run_off + v + 1) - a;
   const uint32_t r0 = a + static_cast<uint32_t>(static_cast<uint64_t>(n) * part / per_chunk);
   const uint32_t r1 = a + static_cast<uint32_t>(static_cast<uint64_t>(n) * (part + 1) / per_chunk);
   if (r0 == r1) return;
   const size_t words = static_cast<size_t>(tab->nchunks) * CHUNK_WORDS, per_query = static_cast<size_t>(cs->nsym) * cs->L;
   for (uint32_t i = threadIdx.x; i < 16 * CHUNK_WORDS / 4; i += NARROW_T) {
      const uint32_t q = i / (CHUNK_WORDS / 4), w = i % (CHUNK_WORDS / 4);
      uint4 x = make_uint4(0, 0, 0, 0);
      if (q0 + q < nq) x = __ldg(reinterpret_cast<const uint4*>(filters + lists[q0 + q] * words + static_cast<size_t>(v) * CHUNK_WORDS) + w);
      reinterpret_cast<uint4*>(words_of)[i] = x;
   }
   if (threadIdx.x == 0) next = r0;
   __syncthreads();
   for (;;) {
      uint32_t r = 0;
      if (lane == 0) r = atomicAdd(&next, 1u);
      r = __shfl_sync(0xFFFFFFFFu, r, 0);
      if (r >= r1) break;
      const uint32_t c = __ldg(cs->run_ctrs + r);
      const uint4 raw = __ldg(reinterpret_cast<const uint4*>(cs->fctrs) + c);
      const CtrDesc d = *reinterpret_cast<const CtrDesc*>(&raw);
      uint32_t sum[16];
#pragma unroll
      for (uint32_t q = 0; q < 16; ++q) sum[q] = 0;
      auto add_word = [&](uint32_t w, uint32_t m) {  // the rows of mask m in word w
#pragma unroll
         for (uint32_t q = 0; q < 16; ++q) sum[q] += __popc(words_of[q * CHUNK_WORDS + w] & m);
      };
      auto mask = [](uint32_t w, uint32_t s, uint32_t e) {  // the rows [s, e) in word w, which holds one of them
         const uint32_t b = 32 * w;
         return (s > b ? 0xFFFFFFFFu << (s - b) : 0xFFFFFFFFu) & (e < b + 32 ? 0xFFFFFFFFu >> (b + 32 - e) : 0xFFFFFFFFu);
      };
      if (d.type == CT_BITSET) {
         const uint32_t* bits = reinterpret_cast<const uint32_t*>(cs->payload + d.payload) + lane;
         constexpr uint32_t U = 8;  // loads in flight
#pragma unroll 1
         for (uint32_t w = 0; w < CHUNK_WORDS; w += 32 * U) {
            uint32_t x[U];
#pragma unroll
            for (uint32_t k = 0; k < U; ++k) x[k] = __ldg(bits + w + 32 * k);
#pragma unroll
            for (uint32_t k = 0; k < U; ++k) add_word(w + 32 * k + lane, x[k]);
         }
      } else {
         const uint16_t* p = cs->payload + d.payload;
#pragma unroll 1
         for (uint32_t i0 = 0; i0 < d.nruns; i0 += 32) {
            uint32_t s = 0, e = 0;
            if (i0 + lane < d.nruns) {
               s = __ldg(p + 2 * (i0 + lane));
               e = s + __ldg(p + 2 * (i0 + lane) + 1) + 1u;
            }
            uint32_t wide = __ballot_sync(0xFFFFFFFFu, e - s > NARROW_RUN);
            if (s < e && e - s <= NARROW_RUN)
#pragma unroll 1
               for (uint32_t w = s >> 5; w <= (e - 1) >> 5; ++w) add_word(w, mask(w, s, e));
            __syncwarp();
#pragma unroll 1
            for (; wide; wide &= wide - 1) {
               const uint32_t j = __ffs(wide) - 1, x = __shfl_sync(0xFFFFFFFFu, s, j), z = __shfl_sync(0xFFFFFFFFu, e, j);
#pragma unroll 1
               for (uint32_t w = (x >> 5) + lane; w <= (z - 1) >> 5; w += 32) add_word(w, mask(w, x, z));
            }
         }
      }
      uint32_t mine = 0;  // lane q: query q
#pragma unroll
      for (uint32_t q = 0; q < 16; ++q) {
         const uint32_t k = __reduce_add_sync(0xFFFFFFFFu, sum[q]);
         if (lane == q) mine = k;
      }
      if (mine) atomicAdd(counts + lists[q0 + lane] * per_query + static_cast<size_t>(d.sym) * cs->L + d.key, mine);
   }
}

// One CTA per event item and pass of up to 256 queries (blockIdx.y), a warp per slice of the item's
// position-sorted events. The events of a position are counted like the rows of a container: 32 at a time,
// the lanes splitting the pass's mask words and the events between them (LaneSplit), and the counts are
// added to each query's difference array (missing events: +1 start, -1 end) or boundary histogram (coverage
// events) when the position changes, and once per segment to the segment totals. Bound by issue slots and
// the latency of the mask gathers. 2M rows and 263 queries: 0.32 ms; 0.80 ms with one event at a time and
// 16 queries a lane in nibble counters (335M instructions, and half of the lanes idle at 17 groups).
__global__ void __launch_bounds__(BT, 3) mut_cov_batch_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                              const EvItem* __restrict__ items,
                                                              const uint16_t* __restrict__ R,
                                                              const uint32_t* __restrict__ lists, uint32_t nq_max,
                                                              uint32_t* __restrict__ scratch) {
   const uint32_t nq = lists[2 * nq_max];  // dense slots: lists[0 .. nq)
   const uint32_t pass = blockIdx.y;
   if (pass * PASS_GROUPS * MUT_GROUP >= nq) return;
   const DevSeqCol* cs = &tab->seq[col];
   const uint32_t L = cs->L, nseg = mut_nseg(L);
   const size_t per_query = mut_scratch_words(L);
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nsub = blockDim.x >> 5;
   const size_t rows = static_cast<size_t>(tab->nchunks) * CHUNK_ROWS;
   const uint32_t wp = pass_width_u32((nq + 31) / 32, pass);  // mask words per row in this pass
   const LaneSplit ls(wp, lane);
   const uint32_t* Rw = reinterpret_cast<const uint32_t*>(R + static_cast<size_t>(pass) * rows * 16) + ls.w;
   const EvItem it = items[blockIdx.x];
   const uint32_t n = it.end - it.begin;
   const uint32_t s0 = it.begin + static_cast<uint32_t>(static_cast<uint64_t>(n) * warp / nsub);
   const uint32_t s1 = it.begin + static_cast<uint32_t>(static_cast<uint64_t>(n) * (warp + 1) / nsub);

   const bool missing = it.list <= EV_MEND;
   const uint32_t* mev = it.list == EV_MSTART ? cs->mstart : cs->mend;
   const uint2* cev = reinterpret_cast<const uint2*>(it.list == EV_CSTART ? cs->cstart : cs->cend);
   const uint32_t pbase = missing ? it.block * NBLOCK : 0u;
   const uint32_t hist = missing ? 2 * (L + 1) : (it.list == EV_CSTART ? 0u : L + 1);
   const uint32_t segb = 3 * (L + 1) + (missing ? 2 * nseg : (it.list == EV_CSTART ? 0u : nseg));
   const uint32_t sign = it.list == EV_MEND ? 0xFFFFFFFFu : 1u;  // multiplier modulo 2^32
   const uint32_t slot0 = 256 * pass + 32 * ls.w, qn = min(nq - 256 * pass, 32u);
   auto sc_of = [&](uint32_t q) { return scratch + static_cast<size_t>(lists[slot0 + q]) * per_query; };

   constexpr uint32_t NONE = 0xFFFFFFFFu;
   BitCounter k;
   k.clear();
   uint32_t seg[8], segq[8];  // the lane's queries of take_counts
#pragma unroll
   for (uint32_t i = 0; i < 8; ++i) seg[i] = segq[i] = 0;
   uint32_t cur = NONE, curseg = NONE;
   auto flush_seg = [&]() {
#pragma unroll
      for (uint32_t i = 0; i < 8; ++i) {
         if (seg[i]) atomicAdd(sc_of(segq[i]) + segb + curseg, seg[i] * sign);
         seg[i] = 0;
      }
   };
   auto flush_pos = [&]() {
      take_counts<true>(k, ls, qn, [&](uint32_t i, uint32_t q, uint32_t c) {
         if (c == 0 || slot0 + q >= nq) return;
         atomicAdd(sc_of(q) + hist + cur, c * sign);
         seg[i] += c;
         segq[i] = q;
      });
   };
   auto event = [&](uint32_t i, uint32_t& row, uint32_t& pos) {
      row = 0;
      pos = NONE;
      if (i >= s1) return;
      if (missing) {
         const uint32_t e = __ldg(mev + i);
         row = e >> 8;
         pos = pbase + (e & 0xFFu);
      } else {
         const uint2 e = __ldg(cev + i);
         row = e.x;
         pos = e.y;
      }
      if (pos > L) pos = NONE;  // past the genome: not counted
   };
   uint32_t nrow, npos;
   event(s0 + lane, nrow, npos);
   for (uint32_t i = s0; i < s1; i += 32) {  // 32 events at a time, one position's after the other's
      const uint32_t row = nrow, pos = npos;
      event(i + 32 + lane, nrow, npos);
      uint32_t left = __ballot_sync(0xFFFFFFFFu, pos != NONE);
      while (left) {
         const uint32_t b = __ffs(left) - 1, p = __shfl_sync(0xFFFFFFFFu, pos, b);
         const uint32_t other = ~(__ballot_sync(0xFFFFFFFFu, pos == p) >> b);  // the run of p from lane b on
         const uint32_t cnt = other ? __ffs(other) - 1u : 32u;
         left &= cnt + b < 32 ? 0xFFFFFFFFu << (cnt + b) : 0u;
         if (p != cur) {
            if (k.rows) flush_pos();
            cur = p;
            if (p / MUT_SEG != curseg) {
               if (curseg != NONE) flush_seg();
               curseg = p / MUT_SEG;
            }
         }
         count_window_bits(k, ls, cnt, Rw, wp,
                           [&](uint32_t t) { return __shfl_sync(0xFFFFFFFFu, row, (b + t) & 31u); });
         if (k.full()) flush_pos();
      }
   }
   if (k.rows) flush_pos();
   if (curseg != NONE) flush_seg();
}

// One CTA: the dense slot list, the sparse slot list and their lengths, in slot order.
__global__ void __launch_bounds__(1024) mut_select_kernel(const unsigned long long* __restrict__ fcounts,
                                                          const uint32_t* __restrict__ slot_query, uint32_t nq,
                                                          unsigned long long sparse_max, uint32_t* __restrict__ lists) {
   __shared__ uint32_t wd[32], wsp[32];
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
   uint32_t nd = 0, ns = 0;  // the same in every thread
   for (uint32_t q0 = 0; q0 < nq; q0 += blockDim.x) {
      const uint32_t q = q0 + threadIdx.x;
      const unsigned long long fc = q < nq ? fcounts[slot_query[q]] : 0ull;
      const bool dense = fc > sparse_max, sparse = fc > 0 && fc <= sparse_max;
      const uint32_t bd = __ballot_sync(0xFFFFFFFFu, dense), bs = __ballot_sync(0xFFFFFFFFu, sparse);
      if (lane == 0) {
         wd[warp] = __popc(bd);
         wsp[warp] = __popc(bs);
      }
      __syncthreads();
      uint32_t pd = 0, ps = 0, td = 0, ts = 0;
      for (uint32_t w = 0; w < nw; ++w) {
         pd += w < warp ? wd[w] : 0u;
         ps += w < warp ? wsp[w] : 0u;
         td += wd[w];
         ts += wsp[w];
      }
      const uint32_t below = (1u << lane) - 1u;
      if (dense) lists[nd + pd + __popc(bd & below)] = q;
      if (sparse) lists[nq + ns + ps + __popc(bs & below)] = q;
      nd += td;
      ns += ts;
      __syncthreads();
   }
   if (threadIdx.x == 0) {
      lists[2 * nq] = nd;
      lists[2 * nq + 1] = ns;
   }
}

// grid (CTAs per slot, nq): the row-index pass of sparse slot blockIdx.y, if there is one.
__global__ void __launch_bounds__(BT) mut_sparse_batch_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                              const uint32_t* __restrict__ filters,
                                                              const uint32_t* __restrict__ lists, uint32_t nq,
                                                              uint32_t* counts, uint32_t* scratch) {
   __shared__ uint32_t list[BT / 32][1024];
   if (blockIdx.y >= lists[2 * nq + 1]) return;
   const uint32_t slot = lists[nq + blockIdx.y];
   const DevSeqCol* cs = &tab->seq[col];
   const uint32_t words = tab->nchunks * CHUNK_WORDS;
   const uint32_t warp = threadIdx.x >> 5, nwarps = gridDim.x * (BT / 32);
   const uint32_t* F = filters + static_cast<size_t>(slot) * words;
   uint32_t* cnt = counts + static_cast<size_t>(slot) * cs->nsym * cs->L;
   uint32_t* sc = scratch + static_cast<size_t>(slot) * mut_scratch_words(cs->L);
   for (uint32_t w = (blockIdx.x * (BT / 32) + warp) * 32; w < words; w += nwarps * 32)
      row_index_pass32(cs, F, w, words, cnt, sc, list[warp]);
}

// grid (ceil(L / MUT_SEG), nq): reference counts of slot blockIdx.y. With out.blk (the Mutations rows are
// wanted), the CTA also makes the output rows of its MUT_SEG (= ROWS_BLOCK) positions under the slot's
// minimum proportion from the counts it has just read: their number goes to out.blk[slot *
// gridDim.x + blockIdx.x] and the rows, where they fit, to the next free part of out.stage, which the
// write pass copies into their final order (see rows.cu). A count is so read once; the write pass that
// made the rows from the count tables took 0.46 ms for the 2,048-query batch, the copy takes 0.11.
__global__ void __launch_bounds__(MUT_SEG, 2) mut_final_batch_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                                     const unsigned long long* __restrict__ fcounts,
                                                                     const uint32_t* __restrict__ slot_query,
                                                                     uint32_t* counts,
                                                                     const uint32_t* __restrict__ scratch, RowsOut out) {
   static_assert(MUT_SEG == ROWS_BLOCK, "a final CTA covers one block of the row counts");
   __shared__ uint32_t wtot[MUT_SEG / 32], base_sh;
   const DevSeqCol* cs = &tab->seq[col];
   const uint32_t q = blockIdx.y, L = cs->L;
   const uint32_t total = static_cast<uint32_t>(fcounts[slot_query[q]]);
   const size_t bi = static_cast<size_t>(q) * gridDim.x + blockIdx.x;
   if (total == 0) {  // an empty filter: its counts stay zero and it has no rows
      if (out.blk != nullptr && threadIdx.x == 0) out.blk[bi] = 0;
      return;
   }
   uint32_t* cnt = counts + static_cast<size_t>(q) * cs->nsym * L;
   const FinalCount f = final_position_counts(cs, total, cnt, scratch + static_cast<size_t>(q) * mut_scratch_words(L));
   if (out.blk == nullptr) return;
   const uint32_t p = blockIdx.x * MUT_SEG + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const uint32_t syms = p < L ? cs->valid_mask & (cs->syms[p] | 1u << f.local) : 0u;
   auto count = [&](uint32_t k) { return k == f.local ? f.count : cnt[static_cast<size_t>(k) * L + p]; };
   const PosRows r = position_rows(cs, p, syms, out.min_prop[q], count);
   uint32_t incl = r.n;
#pragma unroll
   for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
   }
   if (lane == 31) wtot[warp] = incl;
   __syncthreads();
   const uint32_t w = wtot[lane];
   const uint32_t sum = __reduce_add_sync(0xFFFFFFFFu, w), before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? w : 0u);
   if (threadIdx.x == 0) {
      out.blk[bi] = sum;
      base_sh = sum ? atomicAdd(out.cursor, sum) : 0u;
      out.base[bi] = base_sh;
   }
   if (sum == 0) return;
   __syncthreads();
   if (base_sh + sum > out.cap || r.n == 0) return;  // the write pass makes the rows of a block that did not fit
   DevMutationRow* o = out.stage + base_sh + before + incl - r.n;
   for (uint32_t m = syms & ~(1u << r.ref); m; m &= m - 1) {
      const uint32_t k = __ffs(m) - 1, n = count(k);
      if (n > r.thr) *o++ = mutation_row(cs, p, r, k, n);
   }
}
static_assert(MUT_SEG / 32 == 32, "one lane per warp's total");

}  // namespace

void mutations_batch_setup() {
   cudaError_t e =
      cudaFuncSetAttribute(mut_ctr_narrow_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(NARROW_SMEM));
   if (e == cudaSuccess)
      e = cudaFuncSetAttribute(mut_runs_narrow_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(NARROW_SMEM));
   if (e != cudaSuccess)
      throw std::runtime_error(std::string("shared memory of the narrow container pass: ") + cudaGetErrorString(e));
}

size_t mutations_batch_mask_bytes(uint32_t nq, uint32_t nchunks) {
   const uint32_t nqc = (nq + 31) / 32;
   return static_cast<size_t>(nqc) * nchunks * CHUNK_ROWS * 4;
}

void launch_mutations_batch(const DevTable* d_table, const DevSeqCol& col_host, uint32_t col, uint32_t nchunks, uint32_t sms,
                            const uint32_t* d_filters, uint32_t nq, const unsigned long long* d_fcounts,
                            const uint32_t* d_slot_query, const EvItem* d_ev, uint32_t n_ev, const CtrUnit* d_units,
                            uint32_t n_units, uint16_t* d_masks, uint32_t* d_counts, uint32_t* d_scratch,
                            uint32_t* d_lists, uint64_t sparse_max, void* stream, uint32_t parts, const RowsOut& rows) {
   if (nq == 0) return;
   cudaStream_t s = static_cast<cudaStream_t>(stream);
   const uint32_t ngroups = (nq + MUT_GROUP - 1) / MUT_GROUP;  // grids for the largest dense list
   // the slot lists are made with the transpose part, which every timed part follows; the split
   // does not depend on which parts run (without the row-index part its slots stay uncounted)
   if (parts & BMUT_PART_TRANSPOSE) {
      mut_select_kernel<<<1, 1024, 0, s>>>(d_fcounts, d_slot_query, nq, static_cast<unsigned long long>(sparse_max),
                                           d_lists);
      transpose_kernel<<<nchunks * CHUNK_WORDS / TR_WORDS, BT, 0, s>>>(d_filters, d_lists, nq, nchunks,
                                                                       reinterpret_cast<uint32_t*>(d_masks));
   }
   if ((parts & BMUT_PART_CTR) && n_units > 0) {
      const dim3 grid((n_units + BT / 32 - 1) / (BT / 32), (ngroups + PASS_GROUPS - 1) / PASS_GROUPS);
      mut_ctr_batch_kernel<<<grid, BT, 0, s>>>(d_table, col, d_units, n_units, d_masks, d_lists, nq, d_counts);
      const uint32_t per_chunk = std::max(1u, sms / nchunks);  // one CTA per SM
      mut_ctr_narrow_kernel<<<dim3(nchunks * per_chunk, nq > 16 ? 2 : 1), NARROW_T, NARROW_SMEM, s>>>(
         d_table, col, d_filters, d_masks, d_lists, nq, per_chunk, d_counts);
      if (col_host.n_run_ctrs > 0) {  // a container per warp at least
         const uint32_t ctas = std::clamp(col_host.n_run_ctrs / nchunks / (NARROW_T / 32), 1u, per_chunk);
         mut_runs_narrow_kernel<<<dim3(nchunks * ctas, nq > 16 ? 2 : 1), NARROW_T, NARROW_SMEM, s>>>(
            d_table, col, d_filters, d_lists, nq, ctas, d_counts);
      }
   }
   if ((parts & BMUT_PART_COV) && n_ev > 0)
      mut_cov_batch_kernel<<<dim3(n_ev, (ngroups + PASS_GROUPS - 1) / PASS_GROUPS), BT, 0, s>>>(d_table, col, d_ev, d_masks, d_lists, nq,
                                                                          d_scratch);
   if ((parts & BMUT_PART_SPARSE) && sparse_max > 0) {
      const uint32_t per_slot = std::max(1u, std::min(nchunks * CHUNK_WORDS / 32 / (BT / 32), 64u));
      mut_sparse_batch_kernel<<<dim3(per_slot, nq), BT, 0, s>>>(d_table, col, d_filters, d_lists, nq, d_counts,
                                                                d_scratch);
   }
   if (parts & BMUT_PART_FINAL) {
      dim3 fin((col_host.L + MUT_SEG - 1) / MUT_SEG, nq);
      mut_final_batch_kernel<<<fin, MUT_SEG, 0, s>>>(d_table, col, d_fcounts, d_slot_query, d_counts, d_scratch, rows);
   }
}

}  // namespace rhygpu
