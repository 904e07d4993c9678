// Grouped counts of a filter's rows (BitmapAggregation, reference:
// src/rhydb/query_engine/operators/bitmap_aggregation_node.cpp:51-140).
//
//  agg_keys_kernel   a CTA per 8,192 rows: the filtered rows' group in every dimension, combined into
//                    one mixed-radix key (dimension 0 most significant), counted in a dense array.
//  agg_nonzero_kernel / agg_write_kernel
//                    the nonzero keys in key order, which is the reference's depth-first order
//                    over the dimensions' groups.
//
// A sequence dimension's groups are the column's symbols in alphabet order and then the null
// group. A row's symbol at the position is that of the container holding it, else the missing symbol
// where the row is not covered or inside a missing interval, else the local reference symbol; null
// rows form the null group. This is the partition compileSymbolInSet(column, position, {symbol})
// makes for each symbol, with the null rows added last (bitmap_aggregation_node.cpp:51-84). A
// dictionary dimension's groups are its values in string order and then the null group (:237-259).
#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

#include "aggregate.h"

namespace rhygpu {

namespace {

constexpr uint32_t AT = 256;

constexpr uint32_t AGG_TILE = 8192;  // rows per CTA
constexpr uint32_t RUN_OWN = 16;     // a run of at most so many rows is its own lane's

// The symbol of every row of the tile at a position, one byte per row: the local reference, then the
// missing symbol where the row is not covered, then the symbols of the position's containers (no row is
// in two of these lists, null rows apart).
__device__ __forceinline__ void tile_symbols(uint8_t* sym, const DevTable* __restrict__ tab,
                                             const DevSeqCol* __restrict__ cs, uint32_t v, uint32_t row0, uint32_t pos) {
   const uint32_t ref = __ldg(cs->local_ref + pos) * 0x01010101u;
   for (uint32_t i = threadIdx.x; i < AGG_TILE / 4; i += AT) reinterpret_cast<uint32_t*>(sym)[i] = ref;
   __syncthreads();
   const uint8_t missing = static_cast<uint8_t>(cs->nsym - 1);  // the missing symbol is the last one
   const size_t b = static_cast<size_t>(pos / NBLOCK) * tab->nchunks + v;
   const uint4 rng = __ldg(cs->cov_rng + b);
   for (uint32_t i = threadIdx.x; i < rng.y + rng.w; i += AT) {
      const bool late = i < rng.y;
      const CovBound e = late ? cs->cov_late[rng.x + i] : cs->cov_early[rng.z + (i - rng.y)];
      const uint32_t r = e.row - row0;
      if (r < AGG_TILE && (e.bound > pos) == late) sym[r] = missing;
   }
   const uint32_t* toff = cs->nblk_toff + b * TOFF_N;
   const uint32_t q = pos % NBLOCK;
   for (uint32_t i = __ldg(toff + row0 / TOFF_ROWS) + threadIdx.x; i < __ldg(toff + (row0 + AGG_TILE) / TOFF_ROWS); i += AT) {
      const uint32_t e = __ldg(cs->nblk + i), r = (e & 0xFFFFu) - row0;
      if (r < AGG_TILE && ((e >> 16) & 0xFFu) <= q && q < (e >> 24)) sym[r] = missing;
   }
   const size_t slot = static_cast<size_t>(v) * cs->L + pos;
   const uint32_t lane = threadIdx.x & 31;
   for (uint32_t c = __ldg(cs->off + slot) + (threadIdx.x >> 5); c < __ldg(cs->off + slot + 1); c += AT / 32) {  // a warp each
      const uint4 raw = __ldg(reinterpret_cast<const uint4*>(cs->fctrs) + c);
      const CtrDesc d = *reinterpret_cast<const CtrDesc*>(&raw);
      const uint16_t* p = cs->payload + d.payload;
      if (d.type == CT_BITSET) {
         const uint32_t* words = reinterpret_cast<const uint32_t*>(p) + (row0 >> 5);
         for (uint32_t w = lane; w < AGG_TILE / 32; w += 32)
            for (uint32_t x = __ldg(words + w); x; x &= x - 1) sym[32 * w + (__ffs(x) - 1)] = d.sym;
      } else if (d.type == CT_ARRAY) {
         for (uint32_t i = lane; i <= d.card_m1; i += 32) {
            const uint32_t r = static_cast<uint32_t>(__ldg(p + i)) - row0;
            if (r < AGG_TILE) sym[r] = d.sym;
         }
      } else {
         // 32 runs at a time: a short one by its own lane, the others by the warp, four rows a store (two
         // positions of 400,000 rows in long runs: a call 252 us with a lane per run, 79 us so)
         for (uint32_t i0 = 0; i0 < d.nruns; i0 += 32) {
            uint32_t a = 0, b = 0;  // this lane's run in the tile: [a, b)
            if (i0 + lane < d.nruns) {
               const uint32_t s = __ldg(p + 2 * (i0 + lane)), e = s + __ldg(p + 2 * (i0 + lane) + 1) + 1u;
               a = max(s, row0) - row0;
               b = max(min(e, row0 + AGG_TILE), row0) - row0;
            }
            uint32_t wide = __ballot_sync(0xFFFFFFFFu, a < b && b - a > RUN_OWN);
            if (a < b && b - a <= RUN_OWN)
               for (uint32_t r = a; r < b; ++r) sym[r] = d.sym;
            for (; wide; wide &= wide - 1) {
               const uint32_t j = __ffs(wide) - 1, x = __shfl_sync(0xFFFFFFFFu, a, j), y = __shfl_sync(0xFFFFFFFFu, b, j);
               for (uint32_t w = x / 4 + lane; w <= (y - 1) / 4; w += 32) {
                  if (4 * w >= x && 4 * w + 4 <= y) {
                     reinterpret_cast<uint32_t*>(sym)[w] = d.sym * 0x01010101u;
                  } else {
                     for (uint32_t r = max(4 * w, x); r < min(4 * w + 4, y); ++r) sym[r] = d.sym;
                  }
               }
            }
         }
      }
   }
   __syncthreads();
}

// Dynamic shared memory: a key and a symbol per row of the tile, then (hist) a counter per key.
// Bound: the lists of one position per sequence dimension (a few KB per chunk) and 4 bytes per row and
// dictionary dimension. It replaced a lane per filtered row that walked the row's whole row-index
// entry list (31.5 on average) for each sequence dimension and added to global counters: 184 us per
// query at 2M rows, 613 us for 900,000 filtered rows.
__global__ void __launch_bounds__(AT) agg_keys_kernel(const DevTable* __restrict__ tab, const uint32_t* __restrict__ F,
                                                      const AggDim* __restrict__ dims, uint32_t nd, uint32_t keys,
                                                      bool hist, uint32_t* __restrict__ counters) {
   extern __shared__ __align__(16) uint32_t agg_smem[];
   uint32_t* key = agg_smem;
   uint8_t* sym = reinterpret_cast<uint8_t*>(agg_smem + AGG_TILE);
   uint32_t* local = agg_smem + AGG_TILE + AGG_TILE / 4;
   constexpr uint32_t T = CHUNK_ROWS / AGG_TILE, TW = AGG_TILE / 32;
   const uint32_t v = blockIdx.x / T, row0 = blockIdx.x % T * AGG_TILE;
   const uint32_t* Ft = F + static_cast<size_t>(v) * CHUNK_WORDS + (row0 >> 5);
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   // warp w owns the 32 row words from 32 w on, lane l holds the l-th; a step takes four of them, so that
   // their loads are in flight together
   static_assert(TW == AT, "one row word per thread");
   const uint32_t Fw = __ldg(Ft + threadIdx.x);
   const uint32_t busy = __ballot_sync(0xFFFFFFFFu, Fw != 0);
   if (!__syncthreads_or(busy != 0)) return;
   if (hist)
      for (uint32_t k = threadIdx.x; k < keys; k += AT) local[k] = 0;
   for (uint32_t d = 0; d < nd; ++d) {
      const AggDim dim = dims[d];
      const uint32_t stride = static_cast<uint32_t>(dim.stride);
      const DevSeqCol* cs = &tab->seq[dim.col];  // of a sequence dimension
      if (dim.kind == AGG_SEQUENCE) tile_symbols(sym, tab, cs, v, row0, dim.pos);
      const uint32_t r0 = 1024 * warp + lane, g0 = v * CHUNK_ROWS + row0 + r0;
      const uint32_t nulls = dim.kind == AGG_SEQUENCE ? __ldg(cs->null_tiles + (v * CHUNK_ROWS + row0) / 32 + threadIdx.x) : 0u;
      for (uint32_t j0 = 0; j0 < 32; j0 += 4) {
         if (!((busy >> j0) & 15u)) continue;  // four words without rows
         uint32_t g[4];
         bool in[4];
#pragma unroll
         for (uint32_t j = 0; j < 4; ++j) {
            in[j] = (__shfl_sync(0xFFFFFFFFu, Fw, j0 + j) >> lane) & 1u;
            const uint32_t null_word = __shfl_sync(0xFFFFFFFFu, nulls, j0 + j);
            if (dim.kind == AGG_SEQUENCE) g[j] = ((null_word >> lane) & 1u) ? cs->nsym : sym[r0 + 32 * (j0 + j)];
            else g[j] = in[j] ? __ldg(dim.ids + g0 + 32 * (j0 + j)) : 0xFFFFFFFFu;
         }
         if (dim.kind != AGG_SEQUENCE) {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) g[j] = g[j] == 0xFFFFFFFFu ? dim.ngroups - 1 : __ldg(dim.rank + g[j]);
         }
#pragma unroll
         for (uint32_t j = 0; j < 4; ++j) {
            uint32_t& k = key[r0 + 32 * (j0 + j)];
            if (in[j]) k = (d ? k : 0u) + g[j] * stride;
         }
      }
      __syncthreads();  // sym is rewritten by the next dimension
   }
   for (uint32_t j = 0; j < 32; ++j)
      if ((__shfl_sync(0xFFFFFFFFu, Fw, j) >> lane) & 1u)
         atomicAdd((hist ? local : counters) + key[1024 * warp + 32 * j + lane], 1u);
   if (!hist) return;
   __syncthreads();
   for (uint32_t k = threadIdx.x; k < keys; k += AT)
      if (local[k]) atomicAdd(counters + k, local[k]);
}

// Nonzero counters per block of AGG_BLOCK keys.
__global__ void __launch_bounds__(AT) agg_nonzero_kernel(const uint32_t* __restrict__ counters, uint64_t keys,
                                                         uint32_t* __restrict__ block_nonzero) {
   __shared__ uint32_t red[AT / 32];
   const uint64_t k0 = static_cast<uint64_t>(blockIdx.x) * AGG_BLOCK;
   uint32_t n = 0;
   for (uint32_t i = threadIdx.x; i < AGG_BLOCK; i += AT) n += (k0 + i < keys && counters[k0 + i] != 0u) ? 1u : 0u;
   n = __reduce_add_sync(0xFFFFFFFFu, n);
   if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = n;
   __syncthreads();
   if (threadIdx.x == 0) {
      uint32_t s = 0;
      for (uint32_t w = 0; w < AT / 32; ++w) s += red[w];
      block_nonzero[blockIdx.x] = s;
   }
}

// (key, count) of the nonzero counters of each block, at the block's offset, in key order.
__global__ void __launch_bounds__(AT) agg_write_kernel(const uint32_t* __restrict__ counters, uint64_t keys,
                                                       const uint32_t* __restrict__ block_off, AggCount* __restrict__ out) {
   __shared__ uint32_t wsum[AT / 32];
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const uint64_t k0 = static_cast<uint64_t>(blockIdx.x) * AGG_BLOCK;
   uint32_t base = block_off[blockIdx.x];
   for (uint32_t i0 = 0; i0 < AGG_BLOCK; i0 += AT) {
      const uint64_t k = k0 + i0 + threadIdx.x;
      const uint32_t c = k < keys ? counters[k] : 0u;
      const uint32_t m = __ballot_sync(0xFFFFFFFFu, c != 0u);
      if (lane == 0) wsum[warp] = __popc(m);
      __syncthreads();
      uint32_t before = 0, all = 0;
      for (uint32_t w = 0; w < AT / 32; ++w) {
         before += w < warp ? wsum[w] : 0u;
         all += wsum[w];
      }
      if (c) out[base + before + __popc(m & ((1u << lane) - 1u))] = AggCount{k, c};
      base += all;
      __syncthreads();
   }
}

}  // namespace

void aggregate_setup() {
   const cudaError_t e = cudaFuncSetAttribute(agg_keys_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              static_cast<int>(AGG_TILE * 5 + AGG_DENSE * 4));
   if (e != cudaSuccess) throw std::runtime_error(std::string("shared memory of the aggregation: ") + cudaGetErrorString(e));
}

cudaError_t launch_agg_keys(const DevTable* d_table, uint32_t nchunks, const uint32_t* d_filter, const AggDim* d_dims,
                            uint32_t nd, uint64_t keys, uint32_t* d_counters, void* stream) {
   const bool hist = keys <= AGG_DENSE;  // a tile's counters in shared memory: up to 32 KiB beside its 40 KiB
   const size_t smem = AGG_TILE * 5 + (hist ? keys * 4 : 0);
   agg_keys_kernel<<<nchunks * (CHUNK_ROWS / AGG_TILE), AT, smem, static_cast<cudaStream_t>(stream)>>>(
      d_table, d_filter, d_dims, nd, static_cast<uint32_t>(keys), hist, d_counters);
   return cudaGetLastError();
}

void launch_agg_nonzero(const uint32_t* d_counters, uint64_t keys, uint32_t* d_block_nonzero, void* stream) {
   const uint32_t blocks = static_cast<uint32_t>((keys + AGG_BLOCK - 1) / AGG_BLOCK);
   agg_nonzero_kernel<<<blocks, AT, 0, static_cast<cudaStream_t>(stream)>>>(d_counters, keys, d_block_nonzero);
}

void launch_agg_write(const uint32_t* d_counters, uint64_t keys, const uint32_t* d_block_off, AggCount* d_out,
                      void* stream) {
   const uint32_t blocks = static_cast<uint32_t>((keys + AGG_BLOCK - 1) / AGG_BLOCK);
   agg_write_kernel<<<blocks, AT, 0, static_cast<cudaStream_t>(stream)>>>(d_counters, keys, d_block_off, d_out);
}

}  // namespace rhygpu
