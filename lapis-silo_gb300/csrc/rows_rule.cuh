// The row rule of the Mutations output for one position (reference: mutations_node.cpp:292-366),
// shared by the row kernels and the batched final pass, which counts the rows of its positions
// while it has their counts at hand.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

#include "device.h"

namespace rhygpu {

struct PosRows {
   uint32_t n;      // rows of this position
   uint32_t total;  // coverage
   uint32_t thr;    // counts above it are reported
   uint32_t ref;    // global reference symbol
};

// Sum of count(s) over the symbols of the mask, four loads in flight.
template <typename CountOf>
__device__ __forceinline__ uint32_t sum_counts(uint32_t m, CountOf&& count) {
   uint32_t sum = 0;
   while (m) {
      uint32_t c[4];
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
         c[k] = m ? count(__ffs(m) - 1) : 0u;
         m &= m - 1;
      }
      sum += c[0] + c[1] + c[2] + c[3];
   }
   return sum;
}

// total = sum of the counts of the valid symbols (0: no rows); threshold = (min_prop == 0) ? 0 :
// u32(ceil(total * min_prop) - 1); a row for every valid symbol other than the global reference
// whose count exceeds the threshold. count(s) returns the count of symbol s at p; syms: the valid
// symbols whose counts can be other than zero.
template <typename CountOf>
__device__ __forceinline__ PosRows position_rows(const DevSeqCol* __restrict__ cs, uint32_t p, uint32_t syms,
                                                 double min_prop, CountOf&& count) {
   PosRows r{0, 0, 0, 0};
   r.total = sum_counts(syms, count);
   if (r.total == 0) return r;
   r.thr = min_prop == 0.0 ? 0u : static_cast<uint32_t>(ceil(static_cast<double>(r.total) * min_prop) - 1.0);
   r.ref = __ldg(cs->global_ref + p);
   const uint32_t thr = r.thr;
   r.n = sum_counts(syms & ~(1u << r.ref), [&](uint32_t s) { return count(s) > thr ? 1u : 0u; });
   return r;
}

__device__ __forceinline__ DevMutationRow mutation_row(const DevSeqCol* __restrict__ cs, uint32_t p, const PosRows& r,
                                                       uint32_t symbol, uint32_t count) {
   DevMutationRow o;
   o.position = p + 1;
   o.from = cs->chars[r.ref];
   o.to = cs->chars[symbol];
   o.pad = 0;
   o.count = count;
   o.coverage = r.total;
   o.proportion = static_cast<double>(count) / static_cast<double>(r.total);
   return o;
}

}  // namespace rhygpu
