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

// total = sum of the counts of the valid symbols (0: no rows); threshold = (min_prop == 0) ? 0 :
// u32(ceil(total * min_prop) - 1); a row for every valid symbol other than the global reference
// whose count exceeds the threshold. count(s) returns the count of symbol s at p.
template <typename CountOf>
__device__ __forceinline__ PosRows position_rows(const DevSeqCol* __restrict__ cs, uint32_t p, double min_prop,
                                                 CountOf&& count) {
   PosRows r{0, 0, 0, 0};
   const uint32_t nsym = cs->nsym, valid = cs->valid_mask;
   for (uint32_t s = 0; s < nsym; ++s)
      if ((valid >> s) & 1u) r.total += count(s);
   if (r.total == 0) return r;
   r.thr = min_prop == 0.0 ? 0u : static_cast<uint32_t>(ceil(static_cast<double>(r.total) * min_prop) - 1.0);
   r.ref = __ldg(cs->global_ref + p);
   for (uint32_t s = 0; s < nsym; ++s)
      if (((valid >> s) & 1u) && s != r.ref && count(s) > r.thr) ++r.n;
   return r;
}

// The same with the position's counts in registers (`valid`: the column's valid symbols, 0 for no rows).
template <uint32_t NS>
__device__ __forceinline__ PosRows position_rows(const DevSeqCol* __restrict__ cs, uint32_t p, uint32_t valid,
                                                 double min_prop, const uint32_t (&c)[NS]) {
   PosRows r{0, 0, 0, 0};
#pragma unroll
   for (uint32_t s = 0; s < NS; ++s)
      if ((valid >> s) & 1u) r.total += c[s];
   if (r.total == 0) return r;
   r.thr = min_prop == 0.0 ? 0u : static_cast<uint32_t>(ceil(static_cast<double>(r.total) * min_prop) - 1.0);
   r.ref = __ldg(cs->global_ref + p);
#pragma unroll
   for (uint32_t s = 0; s < NS; ++s)
      if (((valid >> s) & 1u) && s != r.ref && c[s] > r.thr) ++r.n;
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
