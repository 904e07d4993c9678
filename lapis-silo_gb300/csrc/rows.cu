// Output rows of the Mutations action on the device (reference: mutations_node.cpp:292-366).
//
// For every query slot and position: total = sum of the counts of the valid mutation symbols;
// positions with total 0 are skipped; threshold = (min_proportion == 0) ? 0
// : u32(ceil(total * min_proportion) - 1); every valid symbol other than the global reference
// symbol whose count exceeds the threshold yields (position + 1, from, to, count, coverage = total,
// proportion = count / total). The double operations are single IEEE operations (a product, ceil,
// a quotient), so the values equal the host's bit for bit.
//
// Three steps keep the output packed and in (slot, position, symbol) order:
//   the batched final pass (mut_final_batch_kernel) makes the rows per block of ROWS_BLOCK positions of
//                      every slot from the counts it has just completed, and stages them
//   rows_scan_kernel   exclusive prefix over all (slot, block) counts; the total follows them
//   rows_write_kernel  copies each block's staged rows to their offsets; a block whose rows did not fit
//                      the staging buffer is made again from its counts
#include <cuda_runtime.h>

#include <cmath>

#include "device.h"
#include "rows_rule.cuh"

namespace rhygpu {

namespace {

constexpr uint32_t RT = ROWS_BLOCK;  // one thread per position

__device__ __forceinline__ uint32_t block_scan_excl(uint32_t x, uint32_t* wsum, uint32_t* total) {
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
   uint32_t incl = x;
#pragma unroll
   for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
      if (lane >= o) incl += y;
   }
   if (lane == 31) wsum[warp] = incl;
   __syncthreads();
   uint32_t before = 0, all = 0;
   for (uint32_t w = 0; w < nw; ++w) {
      const uint32_t v = wsum[w];
      before += w < warp ? v : 0u;
      all += v;
   }
   *total = all;
   return before + incl - x;
}

// One CTA: exclusive prefix sum over n entries in place, the total written to blk[n].
__global__ void __launch_bounds__(RT) rows_scan_kernel(uint32_t* blk, uint32_t n) {
   __shared__ uint32_t wsum[RT / 32];
   const uint32_t per = (n + RT - 1) / RT;
   const uint32_t b = threadIdx.x * per, e = min(b + per, n);
   uint32_t s = 0;
   for (uint32_t i = b; i < e; ++i) s += blk[i];
   uint32_t total;
   uint32_t run = block_scan_excl(s, wsum, &total);
   for (uint32_t i = b; i < e; ++i) {
      const uint32_t x = blk[i];
      blk[i] = run;
      run += x;
   }
   if (threadIdx.x == 0) blk[n] = total;
}

__global__ void __launch_bounds__(RT) rows_write_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                        const uint32_t* __restrict__ counts,
                                                        RowsOut out, DevMutationRow* rows) {
   __shared__ uint32_t wsum[RT / 32];
   const size_t bi = static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x;
   const uint32_t at0 = out.blk[bi], n = out.blk[bi + 1] - at0;
   if (n == 0) return;  // a block without rows (the scan's next entry, or its total, is equal)
   const uint32_t base = out.base[bi];
   if (base + n <= out.cap) {
      const uint2* src = reinterpret_cast<const uint2*>(out.stage + base);
      uint2* dst = reinterpret_cast<uint2*>(rows + at0);
      for (uint32_t i = threadIdx.x; i < n * (sizeof(DevMutationRow) / 8); i += RT) dst[i] = src[i];
      return;
   }
   const DevSeqCol* cs = &tab->seq[col];
   const uint32_t q = blockIdx.y, p = blockIdx.x * RT + threadIdx.x;
   const uint32_t L = cs->L;
   const uint32_t* c = counts + static_cast<size_t>(q) * cs->nsym * L;
   const uint32_t syms = p < L ? cs->valid_mask & (cs->syms[p] | 1u << cs->local_ref[p]) : 0u;
   auto count = [&](uint32_t k) { return __ldg(c + static_cast<size_t>(k) * L + p); };
   const PosRows r = position_rows(cs, p, syms, out.min_prop[q], count);
   uint32_t total;
   uint32_t at = at0 + block_scan_excl(r.n, wsum, &total);
   if (r.n == 0) return;
   for (uint32_t m = syms & ~(1u << r.ref); m; m &= m - 1) {
      const uint32_t k = __ffs(m) - 1, n = count(k);
      if (n > r.thr) rows[at++] = mutation_row(cs, p, r, k, n);
   }
}

}  // namespace

uint32_t rows_blocks(uint32_t L) { return (L + RT - 1) / RT; }

void launch_rows_scan(uint32_t* d_blk, uint32_t n, void* stream) {
   rows_scan_kernel<<<1, RT, 0, static_cast<cudaStream_t>(stream)>>>(d_blk, n);
}

void launch_rows_write(const DevTable* d_table, const DevSeqCol& col_host, uint32_t col, const uint32_t* d_counts,
                       uint32_t nq, const RowsOut& out, DevMutationRow* d_rows, void* stream) {
   if (nq == 0) return;
   rows_write_kernel<<<dim3(rows_blocks(col_host.L), nq), RT, 0, static_cast<cudaStream_t>(stream)>>>(d_table, col, d_counts,
                                                                                                    out, d_rows);
}

}  // namespace rhygpu
