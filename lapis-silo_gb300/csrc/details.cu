// Details action on the device: the first k row ids of a filter in ascending order (reference:
// TableScanNode, exec_node/table_scan.h:42-104, which walks the row set from its smallest id).
//
// One CTA per query scans the dense row set in windows of FK_T x 4 words: a block prefix sum of the
// words' population counts gives each thread's first output slot, every thread writes the ids of its
// words that fall below k, and the scan stops at the window that reaches k. Bound: the chain of windows
// (load, scan, two barriers each); 1,024 threads of four words make 16 of them at 2M rows, where 256
// threads of one word made 244 (175 us for a set with fewer than k rows).
#include <cuda_runtime.h>

#include "device.h"

namespace rhygpu {

namespace {

constexpr uint32_t FK_T = 1024;

__global__ void __launch_bounds__(FK_T) first_k_kernel(const uint32_t* __restrict__ tiles, uint32_t words,
                                                       const uint32_t* __restrict__ k_of,
                                                       const uint32_t* __restrict__ out_off, uint32_t* __restrict__ ids,
                                                       uint32_t* __restrict__ n_out) {
   __shared__ uint32_t wsum[2][FK_T / 32];
   const uint32_t q = blockIdx.x, k = k_of[q];
   const uint4* t = reinterpret_cast<const uint4*>(tiles + static_cast<size_t>(q) * words);  // words is a multiple of 2048
   uint32_t* out = ids + out_off[q];
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, words4 = words / 4;
   uint32_t have = 0;
   uint4 next = threadIdx.x < words4 ? __ldg(t + threadIdx.x) : make_uint4(0, 0, 0, 0);
   for (uint32_t w0 = 0, b = 0; w0 < words4 && have < k; w0 += FK_T, b ^= 1) {
      const uint4 x = next;
      const uint32_t w = w0 + threadIdx.x;
      next = w + FK_T < words4 ? __ldg(t + w + FK_T) : make_uint4(0, 0, 0, 0);  // in flight during the scan
      const uint32_t c = __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
      uint32_t incl = c;
#pragma unroll
      for (uint32_t o = 1; o < 32; o <<= 1) {
         const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
         if (lane >= o) incl += y;
      }
      if (lane == 31) wsum[b][warp] = incl;
      __syncthreads();  // the windows alternate between the two rows of totals
      const uint32_t s = wsum[b][lane];
      const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? s : 0u);
      uint32_t at = have + before + incl - c;
      have += __reduce_add_sync(0xFFFFFFFFu, s);
      const uint32_t v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (uint32_t j = 0; j < 4; ++j)
         for (uint32_t y = v[j]; y && at < k; y &= y - 1) out[at++] = (4 * w + j) * 32 + (__ffs(y) - 1);
   }
   if (threadIdx.x == 0) n_out[q] = have < k ? have : k;
}
static_assert(FK_T / 32 == 32, "one lane per warp's total");

}  // namespace

void launch_first_k(const uint32_t* d_tiles, uint32_t nq, uint32_t nchunks, const uint32_t* d_k,
                    const uint32_t* d_out_off, uint32_t* d_ids, uint32_t* d_n, void* stream) {
   if (nq == 0) return;
   first_k_kernel<<<nq, FK_T, 0, static_cast<cudaStream_t>(stream)>>>(d_tiles, nchunks * CHUNK_WORDS, d_k, d_out_off, d_ids,
                                                                       d_n);
}

}  // namespace rhygpu
