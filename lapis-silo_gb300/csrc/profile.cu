// MutationProfile row sets (reference: src/rhydb/query_engine/scalar_expressions/mutation_profile.cpp:198-257).
//
// The reference rewrites a profile into Not(NOf(distance + 1, one SymbolInSet per position)), a
// threshold over up to a genome's length of children. Here every row counts its differences from
// the row index in one pass. A covered row holding the local reference everywhere has `base`
// differences. Each row-index entry then corrects that count on its own:
//   own symbol s at p       + [s is a difference at p] - [the local reference is]
//   covered region from s   + diff[s]                  (positions [0, s) hold the missing symbol)
//   covered region up to e  + diff[L] - diff[e]        (positions [e, L))
//   missing interval [a, z) - diff[a] ... + diff[z]    (one term per event)
// where diff[p] counts, over positions < p, the missing symbol's differences minus the local
// reference's. Null rows match no SymbolInSet, so they count no difference. A row is in the set
// when its count is at most the distance.
//
// A profile that differs from the local reference at few positions (a list of mutations, a sequence of which
// little is missing) needs none of that: profile_delta_kernel starts from every row's stored distance to the
// local reference and corrects the rows in the lists of those positions. A row's sequence with 20
// substitutions differs at 300 to 1,350 positions, most of them in its missing runs (every missing position
// is a difference: 7% of the genome are too many): 50 us for 1,344 positions at 2M rows, 133 us for the
// whole row index.
//
// The row index otherwise. One warp per 32 consecutive rows. Their entries are one contiguous range of
// the row index, read in windows of 256: each lane loads 8 consecutive entries as two 16-byte loads
// (the range is widened down to a 16-byte boundary, entries outside it count 0), looks up their terms
// and sums them locally; one warp scan over the lane sums places every entry's exclusive prefix in
// shared memory, where each row reads the prefix at its first entry. A row's count is the prefix at
// the next row's first entry minus the prefix at its own.
//   profile_staged_kernel  genomes up to 32,767 positions: the terms (mask u32, diff i16 per
//                          position, 6 bytes) staged in shared memory, one CTA of 1,024 threads
//                          per SM walking the row words;
//   profile_kernel         longer genomes: 8-byte terms read through L1/L2.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "device.h"

namespace rhygpu {

namespace cg = cooperative_groups;

namespace {

constexpr uint32_t PT = 256;           // threads of profile_kernel
constexpr uint32_t ST = 1024;          // threads of profile_staged_kernel
constexpr uint32_t PU = 8;             // entries per lane per window
constexpr uint32_t PW = 32 * PU;       // entries per window
constexpr uint32_t STAGE_MAX_L = 32767;  // diff fits 16 bits

__device__ __forceinline__ int32_t event_term(uint32_t code, int32_t d, int32_t diff_L) {
   if (code == ROW_COV_START) return d;
   if (code == ROW_COV_END) return diff_L - d;
   if (code == ROW_MISS_START) return -d;
   return d;  // ROW_MISS_END
}

// Terms read from the interleaved global array.
struct GlobalTerms {
   const uint2* __restrict__ t;
   int32_t diff_L;
   __device__ __forceinline__ int32_t operator()(uint32_t ent) const {
      const uint32_t code = ent & 31u;
      const uint2 v = __ldg(t + (ent >> 5));
      if (code < ROW_COV_START) return static_cast<int32_t>((v.x >> code) & 1u) - static_cast<int32_t>(v.x >> 31);
      return event_term(code, static_cast<int32_t>(v.y), diff_L);
   }
};

// Terms read from shared memory.
struct StagedTerms {
   const uint32_t* mask;
   const int16_t* diff;
   int32_t diff_L;
   __device__ __forceinline__ int32_t operator()(uint32_t ent) const {
      const uint32_t code = ent & 31u, p = ent >> 5;
      if (code < ROW_COV_START) {
         const uint32_t m = mask[p];
         return static_cast<int32_t>((m >> code) & 1u) - static_cast<int32_t>(m >> 31);
      }
      return event_term(code, diff[p], diff_L);
   }
};

// Whole warp: the aux word of rows 32 w .. 32 w + 31. The row index holds 8 entries of readable
// tail past its end.
template <class Terms>
__device__ __forceinline__ void profile_word(const DevTable* __restrict__ tab, const DevSeqCol* __restrict__ cs,
                                             const DevProfile& pr, const Terms& terms, uint32_t w, int32_t* lp,
                                             uint32_t* __restrict__ aux_word) {
   const uint32_t lane = threadIdx.x & 31;
   const uint32_t r = 32 * w + lane;
   const uint32_t b0 = __ldg(cs->hrow_off + 32 * w);
   const uint32_t a0 = b0 & ~3u;  // 16-byte aligned start
   const uint32_t lo = b0 - a0, hi = lo + (__ldg(cs->hrow_off + 32 * w + 32) - b0);  // valid [lo, hi)
   const uint32_t f = lo + (__ldg(cs->hrow_off + r) - b0);  // this row's first entry
   const uint4* __restrict__ src = reinterpret_cast<const uint4*>(cs->hent + a0);
   int32_t S = 0;         // terms of the entries before the window
   int32_t at_first = 0;  // terms of the entries before this row's first
   for (uint32_t j0 = 0; j0 < hi; j0 += PW) {
      const uint32_t j = j0 + PU * lane;
      uint32_t ent[PU];
      if (j < hi) {
         const uint4 x = __ldg(src + j / 4), y = __ldg(src + j / 4 + 1);
         ent[0] = x.x, ent[1] = x.y, ent[2] = x.z, ent[3] = x.w, ent[4] = y.x, ent[5] = y.y, ent[6] = y.z, ent[7] = y.w;
      }
      int32_t c[PU], sum = 0;
#pragma unroll
      for (uint32_t u = 0; u < PU; ++u) {
         c[u] = (j + u >= lo && j + u < hi) ? terms(ent[u]) : 0;
         sum += c[u];
      }
      int32_t incl = sum;
#pragma unroll
      for (uint32_t o = 1; o < 32; o <<= 1) {
         const int32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
         if (lane >= o) incl += v;
      }
      int32_t run = S + incl - sum;
      int32_t ex[PU];
#pragma unroll
      for (uint32_t u = 0; u < PU; ++u) {
         ex[u] = run;
         run += c[u];
      }
      reinterpret_cast<int4*>(lp)[2 * lane] = make_int4(ex[0], ex[1], ex[2], ex[3]);
      reinterpret_cast<int4*>(lp)[2 * lane + 1] = make_int4(ex[4], ex[5], ex[6], ex[7]);
      __syncwarp();
      if (f >= j0 && f < j0 + PW) at_first = lp[f - j0];
      S += __shfl_sync(0xFFFFFFFFu, incl, 31);
      __syncwarp();
   }
   if (f >= hi) at_first = S;  // rows without entries at the end of the range
   const int32_t next = __shfl_down_sync(0xFFFFFFFFu, at_first, 1);
   const int32_t n = static_cast<int32_t>(pr.base) + (lane == 31 ? S : next) - at_first;
   const bool null_row = (__ldg(cs->null_tiles + w) >> lane) & 1u;
   const bool valid = (r & (CHUNK_ROWS - 1)) < __ldg(tab->chunk_sizes + (r >> 16));
   const bool in = valid && (null_row || n <= static_cast<int32_t>(min(pr.distance, 0x7FFFFFFFu)));
   const uint32_t bits = __ballot_sync(0xFFFFFFFFu, in);
   if (lane == 0) *aux_word = bits;
}

// grid (row words / 8, profiles)
__global__ void __launch_bounds__(PT) profile_kernel(const DevTable* __restrict__ tab,
                                                     const DevProfile* __restrict__ profiles,
                                                     uint32_t* __restrict__ aux) {
   __shared__ __align__(16) int32_t prefix[PT / 32][PW];
   const DevProfile pr = profiles[blockIdx.y];
   if (pr.terms == nullptr) return;  // counted from its differences
   const DevSeqCol* cs = &tab->seq[pr.col];
   const uint32_t words = tab->nchunks * CHUNK_WORDS;
   const uint32_t w = (blockIdx.x * PT + threadIdx.x) >> 5;
   if (w >= words) return;  // the whole warp leaves
   const GlobalTerms terms{pr.terms, static_cast<int32_t>(__ldg(pr.terms + cs->L).y)};
   profile_word(tab, cs, pr, terms, w, prefix[threadIdx.x >> 5], aux + static_cast<size_t>(blockIdx.y) * words + w);
}

// grid (SMs, profiles), one CTA per SM; dynamic shared memory: the prefix windows, then mask[L],
// then diff[L + 1] as int16.
__global__ void __launch_bounds__(ST, 1) profile_staged_kernel(const DevTable* __restrict__ tab,
                                                               const DevProfile* __restrict__ profiles,
                                                               uint32_t* __restrict__ aux) {
   extern __shared__ __align__(16) int32_t sm_prefix[];
   const DevProfile pr = profiles[blockIdx.y];
   if (pr.terms == nullptr) return;  // counted from its differences
   const DevSeqCol* cs = &tab->seq[pr.col];
   const uint32_t L = cs->L;
   uint32_t* mask = reinterpret_cast<uint32_t*>(sm_prefix + (ST / 32) * PW);
   int16_t* diff = reinterpret_cast<int16_t*>(mask + L);
   for (uint32_t p = threadIdx.x; p <= L; p += ST) {
      const uint2 v = __ldg(pr.terms + p);
      if (p < L) mask[p] = v.x;
      diff[p] = static_cast<int16_t>(static_cast<int32_t>(v.y));
   }
   __syncthreads();
   const StagedTerms terms{mask, diff, diff[L]};
   const uint32_t words = tab->nchunks * CHUNK_WORDS;
   int32_t* lp = sm_prefix + (threadIdx.x >> 5) * PW;
   uint32_t* out = aux + static_cast<size_t>(blockIdx.y) * words;
   for (uint32_t w = blockIdx.x * (ST / 32) + (threadIdx.x >> 5); w < words; w += gridDim.x * (ST / 32))
      profile_word(tab, cs, pr, terms, w, lp, out + w);
}

// A cluster of CTAs per chunk: each CTA takes a share of the positions and keeps what they add to every row
// of the chunk in shared memory (16-bit halves of a word: at most PROFILE_DELTA_MAX positions of 2), and the
// CTAs then add the shares of a part of the rows each, from one another's shared memory, to the stored
// distances. The rows of a position's containers and those not covered there get the profile's terms in place
// of the local reference's. A warp looks up to 32 positions up at once, then their containers, numbered across
// the warp, and reads the rows of four containers at a time. Bound: latency, about ten dependent loads per 32
// positions (a missing run of the profile is hundreds of positions with a few containers each), and the
// home distances (4 bytes per row). 1,344 positions at 2M rows: 50 us; 72 with a CTA per 16,384 rows, which
// read the rows of a chunk's containers for a quarter of them (of the 50: staging and the sums' exchange 14,
// containers 14, bitsets 17, rows not covered 5; bitsets by whole warps alone made it 90). 1,024 threads leave 64
// registers each, and 60 bytes of a thread are spilled.
// Runs of up to a whole chunk (a table sorted by lineage holds them at the lineages' positions) add once per
// SPAN rows they cover, and the spans are added to their rows at the end: a count of the rows within 30 of the
// reference over 400,000 rows sorted by lineage takes 0.11 ms, and took 0.65 with an atomic per row of one lane.
constexpr uint32_t DT = 1024, DELTA_BITSETS = 512, DELTA_SMEM = CHUNK_ROWS * 2;
constexpr uint32_t SPAN = 64, RUN_OWN = 16;  // a run of at most RUN_OWN rows is its own lane's
static_assert(2 * PROFILE_DELTA_MAX < 32768, "a row's sum fits 16 bits");
// what two rows' sums in one word are: the lower half is signed, and its borrow is in the upper one
__device__ __forceinline__ int32_t delta_half(uint32_t x, uint32_t upper) {
   const int32_t lo = static_cast<int16_t>(x);
   return upper ? static_cast<int16_t>((x - static_cast<uint32_t>(lo)) >> 16) : lo;
}
__global__ void __launch_bounds__(DT) profile_delta_kernel(const DevTable* __restrict__ tab,
                                                           const DevProfile* __restrict__ profiles,
                                                           uint32_t* __restrict__ aux) {
   extern __shared__ __align__(16) uint32_t cnt[];
   __shared__ uint16_t runs[PROFILE_DELTA_MAX];    // first differences of this CTA's position blocks
   __shared__ int16_t sums[DT / 32][NBLOCK + 4];   // per warp: the uncovered rows' terms of positions below q
   __shared__ uint2 bitsets[DELTA_BITSETS];        // bitset containers: payload, term
   __shared__ int32_t spans[CHUNK_ROWS / SPAN];    // what run containers add to every row of SPAN rows
   __shared__ uint32_t n_runs, n_bitsets, any_span;
   const DevProfile pr = profiles[blockIdx.y];
   if (pr.terms != nullptr) return;  // counted from the row index
   const DevSeqCol* cs = &tab->seq[pr.col];
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const cg::cluster_group cluster = cg::this_cluster();
   const uint32_t parts = cluster.num_blocks(), part = cluster.block_rank(), v = blockIdx.x / parts;
   const size_t g0 = static_cast<size_t>(v) * CHUNK_ROWS;
   for (uint32_t i = threadIdx.x; i < CHUNK_ROWS / 8; i += DT) reinterpret_cast<uint4*>(cnt)[i] = make_uint4(0, 0, 0, 0);
   auto add = [&](uint32_t row, int32_t a) { atomicAdd(cnt + (row >> 1), static_cast<uint32_t>(a) << (16 * (row & 1u))); };
   if (threadIdx.x < CHUNK_ROWS / SPAN) spans[threadIdx.x] = 0;
   static_assert(CHUNK_ROWS / SPAN <= DT, "one span per thread");
   if (threadIdx.x == 0) n_runs = n_bitsets = any_span = 0;
   __syncthreads();
   // rows [x, y), x < y, by lane l of n: two of a word at a time
   auto add_rows = [&](uint32_t x, uint32_t y, int32_t a, uint32_t l, uint32_t n) {
      for (uint32_t w = (x >> 1) + l; w <= (y - 1) >> 1; w += n)
         atomicAdd(cnt + w, ((2 * w >= x ? 1u : 0u) | (2 * w + 1 < y ? 0x10000u : 0u)) * static_cast<uint32_t>(a));
   };
   const uint32_t missing = cs->nsym - 1;  // the missing symbol is the last one
   // what a row with symbol s at the position adds beyond d_ref
   auto term = [](uint32_t mask, uint32_t home, int32_t d_ref, uint32_t s) {
      return static_cast<int32_t>((mask >> s) & 1u) - static_cast<int32_t>((home >> s) & 1u) - d_ref;
   };
   constexpr uint32_t PIECE = 256, PIECES = CHUNK_WORDS / PIECE;  // words of a bitset that a warp takes at a time
   auto add_bitset = [&](uint32_t payload, uint32_t piece, int32_t a) {
      const uint32_t* words = reinterpret_cast<const uint32_t*>(cs->payload + payload);
      constexpr uint32_t U = PIECE / 32;  // loads in flight
      const uint32_t w0 = PIECE * piece + lane;
      uint32_t y[U];
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) y[u] = __ldg(words + w0 + 32 * u);
#pragma unroll
      for (uint32_t u = 0; u < U; ++u)
         for (uint32_t k = 0; k < 16; ++k) {  // two words at a time, a lane per pair of their rows
            const uint32_t j = 2 * k + (lane >> 4), bits = (__shfl_sync(0xFFFFFFFFu, y[u], j) >> (2 * (lane & 15u))) & 3u;
            if (bits) atomicAdd(cnt + 16 * (w0 - lane + 32 * u + j) + (lane & 15u), ((bits | (bits << 15)) & 0x10001u) * static_cast<uint32_t>(a));
         }
   };
   // positions per warp and step: at most 32, the same for every warp and step
   for (uint32_t i = threadIdx.x; i < pr.n_delta; i += DT) {
      const uint32_t blk = __ldg(&pr.delta[i].x) / NBLOCK;
      if (blk % parts == part && (i == 0 || __ldg(&pr.delta[i - 1].x) / NBLOCK != blk))
         runs[atomicAdd(&n_runs, 1u)] = static_cast<uint16_t>(i);
   }
   const uint32_t nd = (pr.n_delta - part + parts - 1) / parts;  // this CTA's positions: part, part + parts, ...
   const uint32_t steps = (nd + DT - 1) / DT, per = steps ? (nd + steps * (DT / 32) - 1) / (steps * (DT / 32)) : 1u;
   for (uint32_t i0 = warp * per; i0 < nd; i0 += per * (DT / 32)) {
      const uint32_t np = min(per, nd - i0);
      uint4 d = make_uint4(0, 0, 0, 0);  // lane l < np: position l and its containers
      uint32_t c0 = 0, nc = 0;
      if (lane < np) {
         d = __ldg(pr.delta + (i0 + lane) * parts + part);
         const size_t slot = static_cast<size_t>(v) * cs->L + d.x;
         c0 = __ldg(cs->off + slot);
         nc = __ldg(cs->off + slot + 1) - c0;
      }
      uint32_t first = nc;  // containers before this position's, after the scan
#pragma unroll
      for (uint32_t o = 1; o < 32; o <<= 1) {
         const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, first, o);
         if (lane >= o) first += y;
      }
      const uint32_t total = __shfl_sync(0xFFFFFFFFu, first, 31);
      first -= nc;
      for (uint32_t t0 = 0; t0 < total; t0 += 32) {
         const uint32_t t = t0 + lane;
         uint32_t l = 0;  // the last lane whose first container is <= t holds container t
#pragma unroll
         for (uint32_t step = 16; step > 0; step >>= 1)
            if (__shfl_sync(0xFFFFFFFFu, first, l + step) <= t) l += step;
         const uint32_t cl = __shfl_sync(0xFFFFFFFFu, c0, l), fl = __shfl_sync(0xFFFFFFFFu, first, l);
         const uint32_t dy = __shfl_sync(0xFFFFFFFFu, d.y, l), dz = __shfl_sync(0xFFFFFFFFu, d.z, l),
                        dw = __shfl_sync(0xFFFFFFFFu, d.w, l);
         uint4 raw = make_uint4(0, 0, 0, 0);
         int32_t a = 0;
         if (t < total) {
            raw = __ldg(reinterpret_cast<const uint4*>(cs->fctrs) + cl + (t - fl));
            const CtrDesc* x = reinterpret_cast<const CtrDesc*>(&raw);
            a = term(dy, dz, static_cast<int32_t>(dw), x->sym);
            if (a != 0 && x->type == CT_BITSET) {  // shared out over the warps afterwards
               const uint32_t at = atomicAdd(&n_bitsets, 1u);
               if (at < DELTA_BITSETS) {
                  bitsets[at] = make_uint2(x->payload, static_cast<uint32_t>(a));
                  a = 0;
               }
            }
         }
         uint32_t todo = __ballot_sync(0xFFFFFFFFu, a != 0);
         while (todo) {
            constexpr uint32_t U = 4;  // containers whose first rows are in flight together
            CtrDesc x[U];
            int32_t ax[U];
            uint32_t row[U][2];  // an array's rows lane and lane + 32 (arrays of up to 64 rows)
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
               const uint32_t j = todo ? __ffs(todo) - 1 : 0u;
               const uint4 y = make_uint4(__shfl_sync(0xFFFFFFFFu, raw.x, j), 0, __shfl_sync(0xFFFFFFFFu, raw.z, j),
                                          __shfl_sync(0xFFFFFFFFu, raw.w, j));
               x[u] = *reinterpret_cast<const CtrDesc*>(&y);
               ax[u] = todo ? __shfl_sync(0xFFFFFFFFu, a, j) : 0;
               todo &= todo - 1;
               const bool small = ax[u] != 0 && x[u].type == CT_ARRAY && x[u].card_m1 < 64;
#pragma unroll
               for (uint32_t h = 0; h < 2; ++h)
                  row[u][h] = small && lane + 32 * h <= x[u].card_m1
                                 ? static_cast<uint32_t>(__ldg(cs->payload + x[u].payload + 32 * h + lane))
                                 : 0xFFFFFFFFu;
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
               if (row[u][0] < CHUNK_ROWS) add(row[u][0], ax[u]);
               if (row[u][1] < CHUNK_ROWS) add(row[u][1], ax[u]);
               if (ax[u] == 0 || (x[u].type == CT_ARRAY && x[u].card_m1 < 64)) continue;
               if (x[u].type == CT_ARRAY) {  // 8 rows per lane and load
                  const uint32_t lead = x[u].payload & 7u, end = lead + x[u].card_m1 + 1u;
                  const uint4* src = reinterpret_cast<const uint4*>(cs->payload + (x[u].payload - lead));
                  for (uint32_t k = 8 * lane; k < end; k += 256) {
                     const uint4 y = __ldg(src + k / 8);
                     const uint32_t w[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                     for (uint32_t q = 0; q < 8; ++q) {
                        if (k + q >= lead && k + q < end) add((w[q >> 1] >> (16 * (q & 1))) & 0xFFFFu, ax[u]);
                     }
                  }
               } else if (x[u].type == CT_BITSET) {
                  for (uint32_t k = 0; k < PIECES; ++k) add_bitset(x[u].payload, k, ax[u]);
               } else {
                  // 32 runs at a time: a short one by its own lane, the others by the warp, whole spans once
                  const uint16_t* p = cs->payload + x[u].payload;
                  for (uint32_t k0 = 0; k0 < x[u].nruns; k0 += 32) {
                     uint32_t s = 0, e = 0;
                     if (k0 + lane < x[u].nruns) {
                        s = __ldg(p + 2 * (k0 + lane));
                        e = min(s + __ldg(p + 2 * (k0 + lane) + 1) + 1u, CHUNK_ROWS);
                     }
                     uint32_t wide = __ballot_sync(0xFFFFFFFFu, e - s > RUN_OWN);
                     if (s < e && e - s <= RUN_OWN) add_rows(s, e, ax[u], 0, 1);
                     for (; wide; wide &= wide - 1) {
                        const uint32_t j = __ffs(wide) - 1, a = __shfl_sync(0xFFFFFFFFu, s, j), z = __shfl_sync(0xFFFFFFFFu, e, j);
                        const uint32_t b0 = (a + SPAN - 1) / SPAN, b1 = z / SPAN;
                        if (b0 >= b1) {
                           add_rows(a, z, ax[u], lane, 32);
                           continue;
                        }
                        if (a < b0 * SPAN) add_rows(a, b0 * SPAN, ax[u], lane, 32);
                        for (uint32_t b = b0 + lane; b < b1; b += 32) atomicAdd(spans + b, ax[u]);
                        if (lane == 0) any_span = 1;
                        if (b1 * SPAN < z) add_rows(b1 * SPAN, z, ax[u], lane, 32);
                     }
                  }
               }
            }
         }
      }
   }
   __syncthreads();
   if (any_span)
      for (uint32_t i = threadIdx.x; i < CHUNK_ROWS / 2; i += DT) {
         const int32_t a = spans[2 * i / SPAN];
         if (a != 0) atomicAdd(cnt + i, 0x10001u * static_cast<uint32_t>(a));
      }
   for (uint32_t i = warp; i < min(n_bitsets, DELTA_BITSETS) * PIECES; i += DT / 32)
      add_bitset(bitsets[i / PIECES].x, i % PIECES, static_cast<int32_t>(bitsets[i / PIECES].y));
   // The rows not covered, a warp per block of positions: the terms of the block's differences (sorted by
   // position) are summed below each position, so that an interval, read once, adds the sum over its
   // positions (a missing run of the profile is hundreds of differences in a few blocks).
   for (uint32_t i = warp; i < n_runs; i += DT / 32) {
      const uint32_t first = runs[i], blk = __ldg(&pr.delta[first].x) / NBLOCK;
      int16_t* P = sums[warp];
      for (uint32_t q = lane; q < NBLOCK; q += 32) P[q] = 0;
      __syncwarp();
      for (uint32_t k = first + lane;; k += 32) {
         uint4 d = make_uint4(0, 0, 0, 0);
         const bool in = k < pr.n_delta && (d = __ldg(pr.delta + k)).x / NBLOCK == blk;
         if (in) P[d.x % NBLOCK] = static_cast<int16_t>(term(d.y, d.z, static_cast<int32_t>(d.w), missing));
         if (!__all_sync(0xFFFFFFFFu, in)) break;
      }
      __syncwarp();
      int32_t t[4], sum = 0;  // exclusive sums: lane l has the positions 4 l .. 4 l + 3
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) {
         t[j] = sum;
         sum += P[4 * lane + j];
      }
      int32_t incl = sum;
#pragma unroll
      for (uint32_t o = 1; o < 32; o <<= 1) {
         const int32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
         if (lane >= o) incl += y;
      }
      const int32_t all = __shfl_sync(0xFFFFFFFFu, incl, 31);
      __syncwarp();
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j) P[4 * lane + j] = static_cast<int16_t>(incl - sum + t[j]);
      if (lane == 0) P[NBLOCK] = static_cast<int16_t>(all);
      const bool any = __any_sync(0xFFFFFFFFu, sum != 0 || t[1] != 0 || t[2] != 0 || t[3] != 0);
      __syncwarp();
      if (!any) continue;  // the missing symbol counts as the local reference does at all of them
      const size_t b = static_cast<size_t>(blk) * tab->nchunks + v;
      const uint32_t* toff = cs->nblk_toff + b * TOFF_N;
      const uint32_t m0 = __ldg(toff), m1 = __ldg(toff + TOFF_N - 1);
      const uint4 g = __ldg(cs->cov_rng + b);
      constexpr uint32_t U = 4;  // loads in flight; four intervals each (0: none)
      for (uint32_t k0 = m0 / 4 + lane; k0 < (m1 + 3) / 4; k0 += 32 * U) {
         uint4 x[U];
#pragma unroll
         for (uint32_t u = 0; u < U; ++u)
            x[u] = k0 + 32 * u < (m1 + 3) / 4 ? __ldg(reinterpret_cast<const uint4*>(cs->nblk) + k0 + 32 * u) : make_uint4(0, 0, 0, 0);
#pragma unroll
         for (uint32_t u = 0; u < U; ++u) {
            const uint32_t w[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
               const int32_t a = P[min(w[j] >> 24, NBLOCK)] - P[min((w[j] >> 16) & 0xFFu, NBLOCK)];
               if (a != 0) add(w[j] & 0xFFFFu, a);
            }
         }
      }
      const uint32_t p0 = blk * NBLOCK;
      for (uint32_t k = lane; k < g.y + g.w; k += 32) {  // positions before a late start, or from an early end on
         const bool late = k < g.y;
         const CovBound e = late ? cs->cov_late[g.x + k] : cs->cov_early[g.z + (k - g.y)];
         const int32_t below = P[e.bound <= p0 ? 0u : min(e.bound - p0, NBLOCK)], a = late ? below : all - below;
         if (a != 0) add(e.row, a);
      }
      __syncwarp();  // P is read until here
   }
   cluster.sync();
   const uint32_t csize = __ldg(tab->chunk_sizes + v);
   const int32_t limit = static_cast<int32_t>(min(pr.distance, 0x7FFFFFFFu));
   uint32_t* out = aux + static_cast<size_t>(blockIdx.y) * tab->nchunks * CHUNK_WORDS + g0 / 32;
   // four rows a lane, four words a warp and step
   const uint32_t r1 = CHUNK_ROWS / parts * (part + 1), base = pr.base;
#pragma unroll 2
   for (uint32_t r = CHUNK_ROWS / parts * part + 4 * threadIdx.x; r < r1; r += 4 * DT) {
      const uint32_t null4 = __ldg(cs->null_tiles + (g0 + r) / 32) >> (r & 31u);
      const int4 h = __ldg(reinterpret_cast<const int4*>(cs->home + g0 + r));
      int32_t n[4] = {h.x, h.y, h.z, h.w};
#pragma unroll 4
      for (uint32_t k = 0; k < parts; ++k) {
         const uint2 x = *reinterpret_cast<const uint2*>(cluster.map_shared_rank(cnt, k) + r / 2);
         n[0] += delta_half(x.x, 0);
         n[1] += delta_half(x.x, 1);
         n[2] += delta_half(x.y, 0);
         n[3] += delta_half(x.y, 1);
      }
      uint32_t bits = 0;
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j)
         if (r + j < csize && (((null4 >> j) & 1u) || n[j] + static_cast<int32_t>(base) <= limit)) bits |= 1u << j;
      bits <<= r & 31u;
#pragma unroll
      for (uint32_t o = 1; o < 8; o <<= 1) bits |= __shfl_xor_sync(0xFFFFFFFFu, bits, o);
      if ((lane & 7u) == 0) out[r / 32] = bits;
   }
   cluster.sync();  // the others read this CTA's sums until then
}

__global__ void __launch_bounds__(PT) profile_home_kernel(const DevTable* __restrict__ tab, uint32_t col, uint32_t rows,
                                                          const uint2* __restrict__ t, uint32_t base, int32_t* home) {
   const uint32_t r = blockIdx.x * PT + threadIdx.x;
   if (r >= rows) return;
   const DevSeqCol* cs = &tab->seq[col];
   const GlobalTerms terms{t, static_cast<int32_t>(__ldg(t + cs->L).y)};
   int32_t n = static_cast<int32_t>(base);
   for (uint32_t i = __ldg(cs->hrow_off + r); i < __ldg(cs->hrow_off + r + 1); ++i) n += terms(__ldg(cs->hent + i));
   home[r] = n;
}

}  // namespace

cudaError_t launch_profile_home(const DevTable* d_table, uint32_t col, uint32_t nchunks, const uint2* d_terms, uint32_t base,
                                int32_t* d_home, void* stream) {
   const uint32_t rows = nchunks * CHUNK_ROWS;
   profile_home_kernel<<<(rows + PT - 1) / PT, PT, 0, static_cast<cudaStream_t>(stream)>>>(d_table, col, rows, d_terms, base,
                                                                                         d_home);
   return cudaGetLastError();
}

// prefix windows, mask, diff (see profile_staged_kernel)
static size_t staged_smem(uint32_t L) { return (ST / 32) * PW * 4 + static_cast<size_t>(L) * 4 + (static_cast<size_t>(L) + 1) * 2; }

void profile_setup() {
   const auto allow = [](const void* kernel, size_t bytes) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
      if (e != cudaSuccess) throw std::runtime_error(std::string("shared memory of the profile kernels: ") + cudaGetErrorString(e));
   };
   allow(reinterpret_cast<const void*>(profile_delta_kernel), DELTA_SMEM);
   allow(reinterpret_cast<const void*>(profile_staged_kernel), staged_smem(STAGE_MAX_L));
}

void launch_profiles(const DevTable* d_table, uint32_t nchunks, uint32_t sms, const DevProfile* d_profiles, uint32_t n,
                     bool any_delta, uint32_t max_L, uint32_t* d_aux, void* stream) {
   const uint32_t words = nchunks * CHUNK_WORDS;
   const cudaStream_t s = static_cast<cudaStream_t>(stream);
   if (any_delta) {
      for (uint32_t k = 0; k < n; k += 65535) {  // grid.y is at most 65535
         const uint32_t m = n - k < 65535 ? n - k : 65535;
         // CTAs per chunk: eight (the most that every device takes) while they find an SM each, else four
         const uint32_t parts = static_cast<uint64_t>(nchunks) * m * 8 <= sms ? 8 : 4;
         cudaLaunchAttribute attr{};
         attr.id = cudaLaunchAttributeClusterDimension;
         attr.val.clusterDim.x = parts;
         attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
         cudaLaunchConfig_t cfg{};
         cfg.gridDim = dim3(nchunks * parts, m);
         cfg.blockDim = DT;
         cfg.dynamicSmemBytes = DELTA_SMEM;
         cfg.stream = s;
         cfg.attrs = &attr;
         cfg.numAttrs = 1;
         cudaLaunchKernelEx(&cfg, profile_delta_kernel, d_table, d_profiles + k, d_aux + static_cast<size_t>(k) * words);
      }
   }
   if (max_L == 0) return;
   const size_t smem = staged_smem(max_L);
   const bool staged = max_L <= STAGE_MAX_L;
   for (uint32_t k = 0; k < n; k += 65535) {  // grid.y is at most 65535
      const uint32_t m = n - k < 65535 ? n - k : 65535;
      if (staged)
         profile_staged_kernel<<<dim3(sms, m), ST, smem, s>>>(d_table, d_profiles + k, d_aux + static_cast<size_t>(k) * words);
      else
         profile_kernel<<<dim3((words + PT / 32 - 1) / (PT / 32), m), PT, 0, s>>>(d_table, d_profiles + k,
                                                                                 d_aux + static_cast<size_t>(k) * words);
   }
}

}  // namespace rhygpu
