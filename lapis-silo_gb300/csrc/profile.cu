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
// A profile that differs from the local reference at few positions (a sequence of the data set, a list of
// mutations) needs none of that: profile_delta_kernel starts from every row's stored distance to the
// local reference and corrects the rows in the lists of those positions. A row's sequence with 20
// substitutions differs at 300 to 1,350 positions, most of them in its missing runs: 72 us for 1,344
// positions at 2M rows, 133 us for the whole row index.
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
#include <cuda_runtime.h>

#include "device.h"

namespace rhygpu {

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

// One CTA per 16,384 rows: their counts in shared memory, the positions shared out over the warps. The
// rows of a position's containers and those not covered there get the profile's terms in place of the
// local reference's. A warp looks up to 32 positions up at once, then their containers, numbered across
// the warp, and reads the rows of four containers at a time. Bound: the home distances (4 bytes per
// row) and latency, about ten dependent loads per 32 positions (a missing run of the profile is
// hundreds of positions with a few containers each).
constexpr uint32_t DT = 1024, DELTA_TILE = 16384, DELTA_BITSETS = 512;
__global__ void __launch_bounds__(DT) profile_delta_kernel(const DevTable* __restrict__ tab,
                                                           const DevProfile* __restrict__ profiles,
                                                           uint32_t* __restrict__ aux) {
   extern __shared__ __align__(16) int32_t cnt[];
   __shared__ uint16_t listed[PROFILE_DELTA_MAX];  // positions whose uncovered rows count differently
   __shared__ uint2 bitsets[DELTA_BITSETS];        // bitset containers: payload, term
   __shared__ uint32_t n_listed, n_bitsets;
   const DevProfile pr = profiles[blockIdx.y];
   if (pr.terms != nullptr) return;  // counted from the row index
   const DevSeqCol* cs = &tab->seq[pr.col];
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   constexpr uint32_t T = CHUNK_ROWS / DELTA_TILE;
   const uint32_t v = blockIdx.x / T, row0 = blockIdx.x % T * DELTA_TILE;
   const size_t g0 = static_cast<size_t>(v) * CHUNK_ROWS + row0;
   const int4* home = reinterpret_cast<const int4*>(cs->home + g0);
   const int32_t base = static_cast<int32_t>(pr.base);
   for (uint32_t i = threadIdx.x; i < DELTA_TILE / 4; i += DT) {
      const int4 h = __ldg(home + i);
      reinterpret_cast<int4*>(cnt)[i] = make_int4(h.x + base, h.y + base, h.z + base, h.w + base);
   }
   if (threadIdx.x == 0) n_listed = n_bitsets = 0;
   __syncthreads();
   const uint32_t missing = cs->nsym - 1;  // the missing symbol is the last one
   // what a row with symbol s at the position adds beyond d_ref
   auto term = [](uint32_t mask, uint32_t home, int32_t d_ref, uint32_t s) {
      return static_cast<int32_t>((mask >> s) & 1u) - static_cast<int32_t>((home >> s) & 1u) - d_ref;
   };
   auto add_bitset = [&](uint32_t payload, int32_t a) {
      const uint32_t* words = reinterpret_cast<const uint32_t*>(cs->payload + payload) + (row0 >> 5);
      constexpr uint32_t U = 8;  // loads in flight
      for (uint32_t w0 = lane; w0 < DELTA_TILE / 32; w0 += 32 * U) {
         uint32_t y[U];
#pragma unroll
         for (uint32_t u = 0; u < U; ++u) y[u] = __ldg(words + w0 + 32 * u);
#pragma unroll
         for (uint32_t u = 0; u < U; ++u)
            for (uint32_t z = y[u]; z; z &= z - 1) atomicAdd(cnt + 32 * (w0 + 32 * u) + (__ffs(z) - 1), a);
      }
   };
   // positions per warp and step: at most 32, the same for every warp and step
   const uint32_t steps = (pr.n_delta + DT - 1) / DT, per = steps ? (pr.n_delta + steps * (DT / 32) - 1) / (steps * (DT / 32)) : 1u;
   for (uint32_t i0 = warp * per; i0 < pr.n_delta; i0 += per * (DT / 32)) {
      const uint32_t np = min(per, pr.n_delta - i0);
      uint4 d = make_uint4(0, 0, 0, 0);  // lane l < np: position l and its containers
      uint32_t c0 = 0, nc = 0;
      if (lane < np) {
         d = __ldg(pr.delta + i0 + lane);
         const size_t slot = static_cast<size_t>(v) * cs->L + d.x;
         c0 = __ldg(cs->off + slot);
         nc = __ldg(cs->off + slot + 1) - c0;
         if (term(d.y, d.z, static_cast<int32_t>(d.w), missing) != 0)
            listed[atomicAdd(&n_listed, 1u)] = static_cast<uint16_t>(i0 + lane);
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
                                 ? static_cast<uint32_t>(__ldg(cs->payload + x[u].payload + 32 * h + lane)) - row0
                                 : 0xFFFFFFFFu;
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
               if (row[u][0] < DELTA_TILE) atomicAdd(cnt + row[u][0], ax[u]);
               if (row[u][1] < DELTA_TILE) atomicAdd(cnt + row[u][1], ax[u]);
               if (ax[u] == 0 || (x[u].type == CT_ARRAY && x[u].card_m1 < 64)) continue;
               if (x[u].type == CT_ARRAY) {  // 8 rows per lane and load
                  const uint32_t lead = x[u].payload & 7u, end = lead + x[u].card_m1 + 1u;
                  const uint4* src = reinterpret_cast<const uint4*>(cs->payload + (x[u].payload - lead));
                  for (uint32_t k = 8 * lane; k < end; k += 256) {
                     const uint4 y = __ldg(src + k / 8);
                     const uint32_t w[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                     for (uint32_t q = 0; q < 8; ++q) {
                        const uint32_t e = ((w[q >> 1] >> (16 * (q & 1))) & 0xFFFFu) - row0;
                        if (k + q >= lead && k + q < end && e < DELTA_TILE) atomicAdd(cnt + e, ax[u]);
                     }
                  }
               } else if (x[u].type == CT_BITSET) {
                  add_bitset(x[u].payload, ax[u]);
               } else {
                  const uint16_t* p = cs->payload + x[u].payload;
                  for (uint32_t k = lane; k < x[u].nruns; k += 32) {
                     const uint32_t s = __ldg(p + 2 * k), e = s + __ldg(p + 2 * k + 1) + 1u;
                     for (uint32_t y = max(s, row0); y < min(e, row0 + DELTA_TILE); ++y) atomicAdd(cnt + (y - row0), ax[u]);
                  }
               }
            }
         }
      }
   }
   __syncthreads();
   for (uint32_t i = warp; i < min(n_bitsets, DELTA_BITSETS); i += DT / 32)
      add_bitset(bitsets[i].x, static_cast<int32_t>(bitsets[i].y));
   for (uint32_t i = warp; i < n_listed; i += DT / 32) {  // a warp per position again
      const uint4 d = __ldg(pr.delta + listed[i]);
      const uint32_t pos = d.x, q = pos % NBLOCK;
      const int32_t a = term(d.y, d.z, static_cast<int32_t>(d.w), missing);
      const size_t b = static_cast<size_t>(pos / NBLOCK) * tab->nchunks + v;
      const uint32_t* toff = cs->nblk_toff + b * TOFF_N;
      const uint32_t m0 = __ldg(toff + row0 / TOFF_ROWS), m1 = __ldg(toff + (row0 + DELTA_TILE) / TOFF_ROWS);
      const uint4 g = __ldg(cs->cov_rng + b);
      constexpr uint32_t U = 4;  // loads in flight; four intervals each, rows outside the tile drop out
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
               const uint32_t r = (w[j] & 0xFFFFu) - row0;
               if (r < DELTA_TILE && ((w[j] >> 16) & 0xFFu) <= q && q < (w[j] >> 24)) atomicAdd(cnt + r, a);
            }
         }
      }
      for (uint32_t k = lane; k < g.y + g.w; k += 32) {
         const bool late = k < g.y;
         const CovBound e = late ? cs->cov_late[g.x + k] : cs->cov_early[g.z + (k - g.y)];
         const uint32_t r = e.row - row0;
         if (r < DELTA_TILE && (e.bound > pos) == late) atomicAdd(cnt + r, a);
      }
   }
   __syncthreads();
   const uint32_t csize = __ldg(tab->chunk_sizes + v);
   const int32_t limit = static_cast<int32_t>(min(pr.distance, 0x7FFFFFFFu));
   uint32_t* out = aux + static_cast<size_t>(blockIdx.y) * tab->nchunks * CHUNK_WORDS + g0 / 32;
   for (uint32_t w = warp; w < DELTA_TILE / 32; w += DT / 32) {
      const uint32_t r = 32 * w + lane;
      const bool null_row = (__ldg(cs->null_tiles + g0 / 32 + w) >> lane) & 1u;
      const uint32_t bits = __ballot_sync(0xFFFFFFFFu, row0 + r < csize && (null_row || cnt[r] <= limit));
      if (lane == 0) out[w] = bits;
   }
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

void launch_profiles(const DevTable* d_table, uint32_t nchunks, const DevProfile* d_profiles, uint32_t n,
                     bool any_delta, uint32_t max_L, uint32_t* d_aux, void* stream) {
   const uint32_t words = nchunks * CHUNK_WORDS;
   const cudaStream_t s = static_cast<cudaStream_t>(stream);
   if (any_delta) {
      cudaFuncSetAttribute(profile_delta_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DELTA_TILE * 4);
      for (uint32_t k = 0; k < n; k += 65535)  // grid.y is at most 65535
         profile_delta_kernel<<<dim3(nchunks * (CHUNK_ROWS / DELTA_TILE), n - k < 65535 ? n - k : 65535), DT, DELTA_TILE * 4, s>>>(
            d_table, d_profiles + k, d_aux + static_cast<size_t>(k) * words);
   }
   if (max_L == 0) return;
   const size_t smem = (ST / 32) * PW * 4 + static_cast<size_t>(max_L) * 4 + (static_cast<size_t>(max_L) + 1) * 2;
   int dev = 0, sms = 0, optin = 0;
   bool staged = max_L <= STAGE_MAX_L && cudaGetDevice(&dev) == cudaSuccess &&
                 cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
                 cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess &&
                 smem <= static_cast<size_t>(optin) &&
                 cudaFuncSetAttribute(profile_staged_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(smem)) == cudaSuccess;
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
