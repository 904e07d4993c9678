// Mutations action kernels of the plain single-query path.
//
//  mut_ring_kernel   every vertical container once: |F ∩ container| against the filter tile of its
//                    chunk staged in shared memory; integer counts per (symbol, position)
//                    (reference: mutations_node.cpp:139-189). A producer warp bulk-copies units of
//                    at most WU array elements into a shared-memory ring that consumer warps count.
//  mut_cov_kernel    rows of F outside their covered region and inside missing intervals, as
//                    differences over positions (reference: mutations_node.cpp:51-136).
//  mut_final_kernel  prefix sums and the local-reference count per position
//                    (reference: mutations_node.cpp:192-203).
//                    Filters of few rows: each row of F adds its row-index entries, the same counts
//                    this and the container pass add for it (the reference's mixed path walks the
//                    filtered rows for coverage the same way, mutations_node.cpp:111-136).
// The filter count decides on the device between the full path (|F| == rows: stored
// cardinalities, reference: mutations_node.cpp:240-266), the empty path and the mixed path.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <stdexcept>
#include <string>

#include "device.h"
#include "mutations_common.cuh"

namespace rhygpu {

namespace {

constexpr uint32_t MT = 256;
constexpr uint32_t NW = MT / 32;

// The pass is a chain of short kernels (2M rows: clearing 2 us, coverage 18, containers 36, prefix sums 6),
// launched as programmatic dependents: each starts while the one before still runs, as soon as every CTA of
// that has called pdl_trigger, and waits with pdl_wait for its completion where it needs its results. The
// order is clear, coverage (waits after staging its filter words), containers (needs only the cleared
// counts, which the coverage pass waited for before its trigger; fills the SMs beside it and waits for its
// end before its own), prefix sums (waits at once). Both calls do nothing in a kernel launched otherwise. What a
// kernel of the chain writes is not read-only while the next one runs, so no parameter that points there is
// __restrict__: the compiler could otherwise take its loads through the read-only path and above the wait.
// One pass over a resident filter at 2M rows: 74 us as seven operations in a row, 57 so.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Shared-memory ring of the container pass.
constexpr uint32_t RING_SLOTS = 16;
constexpr uint32_t RING_CONSUMERS = 8;                 // consumer warps per CTA; warp 0 is the producer
constexpr uint32_t RING_T = 32 * (RING_CONSUMERS + 1);
constexpr uint32_t SLOT_HDR = 16;                      // e0, c0, n | tile << 15 | nd << 16, unit ordinal
constexpr uint32_t SLOT_PAY = 2 * WU;                  // the unit's payload (u16 row ids)
constexpr uint32_t SLOT_BYTES = SLOT_HDR + SLOT_PAY + 16 * WU_DESC;  // then its first WU_DESC descriptors
static_assert(SLOT_BYTES % 16 == 0, "slots start on 16-byte boundaries");
struct Ring {
   uint32_t F[2][CHUNK_WORDS];             // filter tiles of the range's chunks v0 and v1
   uint8_t slot[RING_SLOTS][SLOT_BYTES];
   uint64_t full[RING_SLOTS];              // a slot's copies landed (one arrival + bytes)
   uint64_t empty[RING_SLOTS];             // a slot's unit was counted (one arrival)
   uint64_t tile[2];
   uint32_t next_arr, next_oth, abort_flag;
   uint32_t issued[RING_SLOTS];            // rounds of copies issued into each slot
};
constexpr size_t RING_SMEM = sizeof(Ring);

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
   const uint32_t b = static_cast<uint32_t>(__cvta_generic_to_shared(bar));
   asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(b) : "memory");
}

// Waits for the phase of `bar` with the given parity to complete. It polls without a suspend hint
// and sleeps between polls (backing off up to max_sleep_ns), so that a warp waiting on the ring
// takes few issue slots from the warps that count. Bounded by limit_ns on the global timer and by
// 2^26 polls; false if it gave up.
__device__ __forceinline__ bool ring_wait(uint64_t* bar, uint32_t parity, uint32_t max_sleep_ns, uint64_t limit_ns) {
   const uint32_t b = static_cast<uint32_t>(__cvta_generic_to_shared(bar));
   uint64_t t0 = 0;
   uint32_t ns = 16;
   for (uint32_t i = 0; i < (1u << 26); ++i) {
      uint32_t done;
      asm volatile(
         "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
         : "=r"(done)
         : "r"(b), "r"(parity)
         : "memory");
      if (done) return true;
      const uint64_t now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > limit_ns) return false;
      __nanosleep(ns);
      ns = min(2 * ns, max_sleep_ns);
   }
   return false;
}

// Non-blocking test of the phase of `bar` with the given parity.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
   const uint32_t b = static_cast<uint32_t>(__cvta_generic_to_shared(bar));
   uint32_t done;
   asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(done)
      : "r"(b), "r"(parity)
      : "memory");
   return done != 0;
}

// One arrival on a ring slot's full barrier that announces `bytes` of bulk copies. No proxy fence
// is needed here: the slot's previous contents were only read by generic loads of the consumer that
// released it through the empty barrier this thread waited on, and the header that this thread
// writes with generic stores is read only by generic loads.
__device__ __forceinline__ void ring_expect(uint64_t* bar, uint32_t bytes) {
   const uint32_t b = static_cast<uint32_t>(__cvta_generic_to_shared(bar));
   asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}\n" ::"r"(b), "r"(bytes)
                : "memory");
}

// Waits until the producer has written unit ordinal k into a slot header (bounded by limit_ns).
// A consumer that runs a whole ring ahead sees the previous round's ordinal until then; checking
// the ordinal first keeps its barrier wait from matching the previous round's phase.
__device__ __forceinline__ bool wait_slot_unit(const uint32_t* hdr, uint32_t k, uint64_t limit_ns) {
   uint64_t t0 = 0;
   for (uint32_t i = 0; i < (1u << 26); ++i) {
      if (*reinterpret_cast<const volatile uint32_t*>(hdr + 3) == k) return true;
      const uint64_t now = global_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > limit_ns) return false;
      __nanosleep(64);
   }
   return false;
}

// Testing the failure path of the container pass's bounded waits: while set (on the current
// device), the producer announces each unit's copy bytes on the slot's barrier but never issues the
// copies, so the consumers' waits give up (after 1 ms) and the pass sets DEVERR_WAIT_MUTATIONS. No
// copy is left in flight: the withheld copies never start. Off by default; set only through
// set_ring_withholding.
__device__ uint32_t g_withhold_ring_copies = 0;

// Membership bits of a unit's row ids in the filter tile F: W[it] holds the two u16 row ids of
// elements 64 it + 2 lane and 64 it + 2 lane + 1, whose bits land at 2 it and 2 it + 1. The bit of
// row r is bit r & 31 of word r >> 5; rotating that word right by (r - k) & 31 brings it to bit k
// (the rotation takes its amount modulo 32, so neither half of W needs masking).
__device__ __forceinline__ uint32_t unit_members(const uint32_t (&W)[WU / 64], const uint32_t* __restrict__ F) {
   uint32_t m = 0;
#pragma unroll
   for (uint32_t it = 0; it < WU / 64; ++it) {
      const uint32_t w = W[it], hi = w >> 16;
      const uint32_t f0 = F[(w >> 5) & 0x7FFu], f1 = F[hi >> 5];
      m |= __funnelshift_r(f0, f0, w - 2 * it) & (1u << (2 * it));
      m |= __funnelshift_r(f1, f1, hi - (2 * it + 1)) & (2u << (2 * it));
   }
   return m;
}

// Container pass of the Mutations action (reference: mutations_node.cpp:139-190, full path
// :240-266): |F ∩ c| for every container c of the column, added to counts[symbol][position].
// One CTA per host-built range (array units and bitset / run units of at most two chunks):
//   warp 0 (producer) bulk-copies the filter tiles of the range's chunks; then its lane j keeps
//     ring slot j busy: it copies the payload (row ids, WU at most) and the first WU_DESC
//     descriptors of units j, j + RING_SLOTS, ... into the slot, each as soon as the slot's previous
//     unit was released (full / empty mbarrier pair per slot), so that up to RING_SLOTS units are in
//     flight while earlier ones are counted;
//   warps 1..8 (consumers) first count the bitset and run units straight from global memory, then
//     claim array units in order; a claimed unit moves into registers and its slot is released.
//     Lane l holds elements 64 it + 2l and 64 it + 2l + 1 of step it and sets their membership bits
//     (bits 2 it and 2 it + 1); a warp bit transpose gives lane 2q the bits of the even and lane
//     2q + 1 those of the odd elements of [64q, 64q + 64), and a prefix sum over the lanes turns
//     every descriptor's |F ∩ c| into the difference of two prefix values (a container cut by a
//     unit boundary adds two partial counts).
// Full filters (|F| == rows) add the stored cardinalities: only descriptors are copied. Every wait
// is bounded; one that gives up sets DEVERR_WAIT_MUTATIONS in *err and ends the CTA's work.
__global__ void __launch_bounds__(RING_T, RING_CTAS_PER_SM) mut_ring_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                          const uint32_t* __restrict__ filter,
                                                          const unsigned long long* __restrict__ fcount,
                                                          unsigned long long sparse_max, uint32_t* counts, int* err) {
   extern __shared__ __align__(128) uint8_t ring_raw[];
   Ring& R = *reinterpret_cast<Ring*>(ring_raw);
   pdl_trigger();
   const unsigned long long fc = *fcount;
   if (fc == 0 || fc <= sparse_max) {  // empty, or counted by the row-index pass
      pdl_wait();
      return;
   }
   const bool full = fc == tab->n_rows;
   const DevSeqCol* cs = &tab->seq[col];
   const StreamRange rg = cs->ranges[blockIdx.x];
   const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, L = cs->L;
   const uint32_t na = rg.a1 - rg.a0, no = rg.o1 - rg.o0;
   const bool two = rg.v1 != rg.v0;
   const bool withhold = *static_cast<volatile uint32_t*>(&g_withhold_ring_copies) != 0;
   const uint64_t limit = withhold ? WAIT_LIMIT_TEST_NS : WAIT_LIMIT_NS;
   if (tid == 0) {
      for (uint32_t s = 0; s < RING_SLOTS; ++s) {
         mbar_init(&R.full[s]);
         mbar_init(&R.empty[s]);
      }
      mbar_init(&R.tile[0]);
      mbar_init(&R.tile[1]);
      R.next_arr = 0;
      R.next_oth = 0;
      R.abort_flag = 0;
   }
   if (tid < RING_SLOTS) {
      reinterpret_cast<uint32_t*>(R.slot[tid])[3] = 0xFFFFFFFFu;  // no unit yet
      R.issued[tid] = 0;
   }
   __syncthreads();
   const CtrDesc* __restrict__ ctrs = cs->ctrs;
   volatile uint32_t* abort_flag = &R.abort_flag;
   if (warp == 0) {
      // ---------------- producer ----------------
      if (lane == 0 && !full) {
         mbar_expect(&R.tile[0], CHUNK_WORDS * 4);
         bulk_copy_g2s_tx(R.F[0], filter + static_cast<size_t>(rg.v0) * CHUNK_WORDS, CHUNK_WORDS * 4, &R.tile[0]);
         if (two) {
            mbar_expect(&R.tile[1], CHUNK_WORDS * 4);
            bulk_copy_g2s_tx(R.F[1], filter + static_cast<size_t>(rg.v1) * CHUNK_WORDS, CHUNK_WORDS * 4, &R.tile[1]);
         }
      }
      // lane j < RING_SLOTS owns slot j and issues the units j, j + RING_SLOTS, ... into it, each as
      // soon as the consumer of the slot's previous unit has released it: one pass of the warp
      // refills every free slot
      bool ok = true;
      const uint4* recs = reinterpret_cast<const uint4*>(cs->au) + rg.a0;
      uint32_t kj = lane;  // this lane's next unit
      uint4 rec = lane < RING_SLOTS && kj < na ? __ldg(recs + kj) : make_uint4(0, 0, 0, 0);
      uint64_t t_idle = 0;
      uint32_t ns = 32;
      for (;;) {
         const bool mine = lane < RING_SLOTS && kj < na;
         if (!__any_sync(0xFFFFFFFFu, mine)) break;
         if (*abort_flag) {
            ok = false;
            break;
         }
         const uint32_t round = kj / RING_SLOTS;
         const bool ready = mine && (round == 0 || mbar_test(&R.empty[lane], (round - 1) & 1u));
         if (ready) {
            const uint32_t n = rec.z & 0xFFFFu, nd = rec.z >> 16;
            uint32_t* h = reinterpret_cast<uint32_t*>(R.slot[lane]);
            const uint32_t pay = full ? 0u : (2 * n + 15) & ~15u;
            const uint32_t dsc = 16 * min(nd, WU_DESC);
            h[0] = rec.x;
            h[1] = rec.y;
            h[2] = n | ((rec.w == rg.v0 ? 0u : 1u) << 15) | (nd << 16);
            *reinterpret_cast<volatile uint32_t*>(h + 3) = kj;
            ring_expect(&R.full[lane], pay + dsc);
            if (!withhold) {
               if (pay) bulk_copy_g2s_tx(R.slot[lane] + SLOT_HDR, cs->payload + rec.x, pay, &R.full[lane]);
               bulk_copy_g2s_tx(R.slot[lane] + SLOT_HDR + SLOT_PAY, ctrs + rec.y, dsc, &R.full[lane]);
            }
            R.issued[lane] = round + 1;
            kj += RING_SLOTS;
            rec = kj < na ? __ldg(recs + kj) : make_uint4(0, 0, 0, 0);  // in flight until the slot frees
         }
         if (__any_sync(0xFFFFFFFFu, ready)) {
            t_idle = 0;
            ns = 32;
            continue;
         }
         // no slot free: back off, bounded by the time since the last copy was issued
         const uint64_t now = global_ns();
         if (t_idle == 0) t_idle = now;
         else if (now - t_idle > limit) {
            ok = false;
            break;
         }
         __nanosleep(ns);
         ns = min(2 * ns, 256u);
      }
      if (!ok && lane == 0) {
         *abort_flag = 1;
         if (err) atomicExch(err, DEVERR_WAIT_MUTATIONS);
      }
   } else {
      // ---------------- consumers ----------------
      bool ok = full || (ring_wait(&R.tile[0], 0, 256, limit) && (!two || ring_wait(&R.tile[1], 0, 256, limit)));
      ok = __all_sync(0xFFFFFFFFu, ok);
      // bitset and run units first, straight from global memory, while the producer fills the ring
      while (ok && *abort_flag == 0) {
         uint32_t u = 0;
         if (lane == 0) u = atomicAdd(&R.next_oth, 1u);
         u = __shfl_sync(0xFFFFFFFFu, u, 0);
         if (u >= no) break;
         const uint4 uraw = __ldg(reinterpret_cast<const uint4*>(cs->ou) + rg.o0 + u);
         const OtherUnit U = *reinterpret_cast<const OtherUnit*>(&uraw);
         const uint32_t* F = R.F[U.v == rg.v0 ? 0 : 1];
         const uint4 raw = __ldg(reinterpret_cast<const uint4*>(ctrs) + U.c);
         const CtrDesc d = *reinterpret_cast<const CtrDesc*>(&raw);
         uint32_t k = 0;
         if (full) {
            k = lane == 0 ? d.card_m1 + 1u : 0u;
         } else if (U.kind == SU_BITSET) {
            const uint4* f4 = reinterpret_cast<const uint4*>(F);
            const uint4* p4 = reinterpret_cast<const uint4*>(cs->payload + U.e0);
            constexpr uint32_t BV = CHUNK_WORDS / 4 / 32, BB = 8;  // uint4 per lane; loads in flight
#pragma unroll
            for (uint32_t j0 = 0; j0 < BV; j0 += BB) {
               uint4 a[BB];
#pragma unroll
               for (uint32_t j = 0; j < BB; ++j) a[j] = __ldg(p4 + lane + 32 * (j0 + j));
#pragma unroll
               for (uint32_t j = 0; j < BB; ++j) {
                  const uint4 y = f4[lane + 32 * (j0 + j)];
                  k += __popc(a[j].x & y.x) + __popc(a[j].y & y.y) + __popc(a[j].z & y.z) + __popc(a[j].w & y.w);
               }
            }
         } else {
            const uint16_t* r = cs->payload + d.payload;
            for (uint32_t i = lane; i < d.nruns; i += 32) {
               const uint32_t s0 = __ldg(r + 2 * i);
               k += count_range(F, s0, s0 + __ldg(r + 2 * i + 1) + 1u);
            }
         }
         k = __reduce_add_sync(0xFFFFFFFFu, k);
         if (lane == 0 && k) atomicAdd(&counts[static_cast<size_t>(d.sym) * L + d.key], k);
      }
      // array units from the ring, in order of claim: the unit moves into registers and its slot is
      // released before it is counted
      while (ok && *abort_flag == 0) {
         uint32_t k = 0;
         if (lane == 0) k = atomicAdd(&R.next_arr, 1u);
         k = __shfl_sync(0xFFFFFFFFu, k, 0);
         if (k >= na) break;
         const uint32_t s = k % RING_SLOTS, round = k / RING_SLOTS;
         const uint8_t* slot = R.slot[s];
         const uint32_t* h = reinterpret_cast<const uint32_t*>(slot);
         ok = __all_sync(0xFFFFFFFFu, wait_slot_unit(h, k, limit) && ring_wait(&R.full[s], round & 1u, 128, limit));
         if (!ok) break;
         const uint32_t e0 = h[0], c0 = h[1], w2 = h[2];
         const uint32_t n = w2 & 0x7FFFu, nd = w2 >> 16, tile = (w2 >> 15) & 1u;
         uint32_t W[WU / 64];
         if (!full) {
            const uint32_t* pw = reinterpret_cast<const uint32_t*>(slot + SLOT_HDR) + lane;
#pragma unroll
            for (uint32_t it = 0; it < WU / 64; ++it) W[it] = pw[32 * it];
         }
         const uint4* dsl = reinterpret_cast<const uint4*>(slot + SLOT_HDR + SLOT_PAY);
         const uint32_t nds = min(nd, WU_DESC);
         uint4 D[WU_DESC / 32];
#pragma unroll
         for (uint32_t g = 0; g < WU_DESC / 32; ++g) D[g] = 32 * g + lane < nds ? dsl[32 * g + lane] : make_uint4(0, 0, 0, 0);
         __syncwarp();
         if (lane == 0) mbar_arrive(&R.empty[s]);
         // lane l bit 2 it + h: element 64 it + 2 l + h is in F; after the transpose lane 2q holds the
         // bits of the even and lane 2q + 1 those of the odd elements of [64q, 64q + 64)
         uint32_t T = 0, pb = 0, total = 0;
         if (!full) {
            uint32_t m = tile ? unit_members(W, R.F[1]) : unit_members(W, R.F[0]);
            if (n < WU) {  // elements past the unit's end hold stale slot contents
               uint32_t valid = 0;
#pragma unroll
               for (uint32_t it = 0; it < WU / 64; ++it) {
                  const uint32_t idx = 64 * it + 2 * lane;
                  valid |= (idx < n ? 1u : 0u) << (2 * it);
                  valid |= (idx + 1 < n ? 2u : 0u) << (2 * it);
               }
               m &= valid;
            }
            T = warp_transpose32(m, lane);
            const uint32_t c = __popc(T);
            uint32_t incl = c;
#pragma unroll
            for (uint32_t o = 1; o < 32; o <<= 1) {
               const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
               if (lane >= o) incl += y;
            }
            pb = incl - c;  // lane 2q: members before element 64q
            total = __shfl_sync(0xFFFFFFFFu, incl, 31);
         }
         auto prefix = [&](uint32_t i) -> uint32_t {  // members among the unit's elements [0, i), i <= n
            const uint32_t q = (i >> 6) & 15u, l = (i >> 1) & 31u;
            const uint32_t base = __shfl_sync(0xFFFFFFFFu, pb, 2 * q);
            const uint32_t e = __shfl_sync(0xFFFFFFFFu, T, 2 * q), o = __shfl_sync(0xFFFFFFFFu, T, 2 * q + 1);
            const uint32_t m = (1u << l) - 1u;
            const uint32_t v = base + __popc(e & m) + __popc(o & m) + ((i & 1u) ? ((e >> l) & 1u) : 0u);
            return i >= WU ? total : v;
         };
         auto count_desc = [&](const uint4& raw, uint32_t j) {  // descriptor j of the unit (lane-varying)
            uint32_t a = 0, b = 0, sym = 0, key = 0;
            if (j < nd) {
               const CtrDesc d = *reinterpret_cast<const CtrDesc*>(&raw);
               if (d.type == CT_ARRAY) {
                  const uint32_t x = max(d.payload, e0), y = min(d.payload + d.card_m1 + 1u, e0 + n);
                  if (x < y) {
                     a = x - e0;
                     b = y - e0;
                     sym = d.sym;
                     key = d.key;
                  }
               }
            }
            const uint32_t cnt = full ? b - a : prefix(b) - prefix(a);
            if (cnt) atomicAdd(&counts[static_cast<size_t>(sym) * L + key], cnt);
         };
#pragma unroll
         for (uint32_t g = 0; g < WU_DESC / 32; ++g)
            if (32 * g < nd) count_desc(D[g], 32 * g + lane);
         for (uint32_t j0 = WU_DESC; j0 < nd; j0 += 32) {  // descriptors past the slot's copy
            const uint32_t j = j0 + lane;
            count_desc(j < nd ? __ldg(reinterpret_cast<const uint4*>(ctrs) + c0 + j) : make_uint4(0, 0, 0, 0), j);
         }
      }
      if (!ok && lane == 0) {
         *abort_flag = 1;
         if (err) atomicExch(err, DEVERR_WAIT_MUTATIONS);
      }
   }
   __syncthreads();
   if (tid == 0 && *abort_flag) {
      // after a wait gave up: let the copies still in flight land before the CTA's shared memory is
      // released (the last round issued into each slot; bounded like every other wait)
      for (uint32_t s = 0; s < RING_SLOTS; ++s)
         if (R.issued[s] && !ring_wait(&R.full[s], (R.issued[s] - 1) & 1u, 256, limit)) break;
      if (!full) {
         ring_wait(&R.tile[0], 0, 256, limit);
         if (two) ring_wait(&R.tile[1], 0, 256, limit);
      }
   }
   pdl_wait();  // the coverage pass, so that what follows this kernel follows both
}

// Coverage of the filter per position, as differences over positions (reference:
// mutations_node.cpp:51-136). The first CTAs take COV_BLOCKS x COV_CHUNKS buckets of missing-interval
// boundaries each: the chunks' filter tiles are staged in shared memory, a warp reads a bucket and adds
// +1 (first positions) or -1 (positions after the last) of the intervals whose row is in F to a shared
// histogram. The others count the rows of F whose covered region starts (ends) at each position, one
// event per thread.
// Bound: 4 bytes and about 14 instructions per boundary (31 MB at 2M rows) and 8 KiB of filter per CTA and
// chunk. Before, the same boundaries sorted by position over all chunks each tested a filter bit in L2:
// 58.8 us at 2M rows and 400,000 filtered rows, one 32-byte sector per boundary.
//
// Filters of 1..sparse_max rows take the row-index pass here instead (one warp per 32 filter words at a
// time, any grid), in the same shared memory: a kernel of its own cost every other filter a launch.
constexpr uint32_t COV_BLOCKS = 4, COV_CHUNKS = 4;
__global__ void __launch_bounds__(MT) mut_cov_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                     const uint32_t* __restrict__ filter,
                                                     const unsigned long long* __restrict__ fcount,
                                                     unsigned long long sparse_max, bool coverage, uint32_t* counts,
                                                     uint32_t* scratch) {
   __shared__ __align__(16) uint32_t F[COV_CHUNKS][CHUNK_WORDS];
   __shared__ int hist[COV_BLOCKS][NBLOCK];
   const unsigned long long fc = *fcount;
   const DevSeqCol* cs = &tab->seq[col];
   if (fc <= sparse_max || !coverage) {
      pdl_wait();
      pdl_trigger();
      if (fc == 0 || fc > sparse_max) return;
      static_assert(sizeof(F) >= NW * 1024 * sizeof(uint32_t), "the rows of 32 words per warp");
      const uint32_t words = tab->nchunks * CHUNK_WORDS, nwarps = gridDim.x * NW, w0 = threadIdx.x >> 5;
      for (uint32_t w = (blockIdx.x * NW + w0) * 32; w < words; w += nwarps * 32)
         row_index_pass32(cs, filter, w, words, counts, scratch, F[0] + 1024 * w0);
      return;
   }
   const uint32_t L = cs->L, nseg = mut_nseg(L), nchunks = tab->nchunks, nblocks = cs->nblocks_ev;
   uint32_t* start_hist = scratch;
   uint32_t* ndiff = scratch + 2 * (L + 1);  // (the ends' histogram lies between)
   uint32_t* seg_s = scratch + 3 * (L + 1);
   uint32_t* seg_n = seg_s + 2 * nseg;
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
   const uint32_t gv = (nchunks + COV_CHUNKS - 1) / COV_CHUNKS, gb = (nblocks + COV_BLOCKS - 1) / COV_BLOCKS;
   if (blockIdx.x < gb * gv) {
      const uint32_t b0 = blockIdx.x / gv * COV_BLOCKS, v0 = blockIdx.x % gv * COV_CHUNKS;
      const uint32_t nv = min(COV_CHUNKS, nchunks - v0), nb = min(COV_BLOCKS, nblocks - b0);
      const uint4* src = reinterpret_cast<const uint4*>(filter + static_cast<size_t>(v0) * CHUNK_WORDS);
      for (uint32_t i = threadIdx.x; i < nv * (CHUNK_WORDS / 4); i += MT) reinterpret_cast<uint4*>(F[0])[i] = __ldg(src + i);
      for (uint32_t i = threadIdx.x; i < COV_BLOCKS * NBLOCK; i += MT) hist[0][i] = 0;
      pdl_wait();
      pdl_trigger();
      __syncthreads();
      for (uint32_t j = warp; j < nb * nv; j += NW) {
         const uint32_t bl = j / nv, v = j % nv;
         const uint32_t* off = cs->mev_off + static_cast<size_t>(b0 + bl) * nchunks + v0 + v;
         const uint32_t e0 = __ldg(off) / 4, e1 = __ldg(off + 1) / 4;
         const uint4* ev = reinterpret_cast<const uint4*>(cs->mev);
         constexpr uint32_t U = 4;  // loads in flight per lane: about 270 boundaries per bucket
         for (uint32_t i0 = e0; i0 < e1; i0 += 32 * U) {
            uint4 x[U];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
               const uint32_t i = i0 + 32 * u + lane;
               x[u] = i < e1 ? __ldg(ev + i) : make_uint4(MEV_NONE, MEV_NONE, MEV_NONE, MEV_NONE);
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
               if (i0 + 32 * u >= e1) break;
               const uint32_t w[4] = {x[u].x, x[u].y, x[u].z, x[u].w};
#pragma unroll
               for (uint32_t k = 0; k < 4; ++k) {
                  const uint32_t in = F[v][(w[k] & 0xFFFFu) >> 5] >> (w[k] & 31u);
                  const uint32_t p = (w[k] >> 16) & 0xFFu;
                  if ((in & 1u) && p < NBLOCK) atomicAdd(&hist[bl][p], (w[k] >> 31) ? 1 : -1);
               }
            }
         }
      }
      __syncthreads();
      const uint32_t seg = b0 * NBLOCK / MUT_SEG;  // COV_BLOCKS * NBLOCK divides MUT_SEG
      for (uint32_t i = threadIdx.x; i < COV_BLOCKS * NBLOCK; i += MT) {
         const int x = hist[0][i];
         const uint32_t p = b0 * NBLOCK + i;  // at most L where x is not 0
         if (x != 0) atomicAdd(&ndiff[p], static_cast<uint32_t>(x));
         const int s = __reduce_add_sync(0xFFFFFFFFu, x);
         if (lane == 0 && s) atomicAdd(&seg_n[seg], static_cast<uint32_t>(s));
      }
   } else {
      const uint32_t ns = cs->n_cstart, n = ns + cs->n_cend;
      const uint32_t i = (blockIdx.x - gb * gv) * MT + threadIdx.x;  // one event per thread
      const bool start = i < ns;
      pdl_wait();
      pdl_trigger();
      const uint2 e = i < n ? __ldg(reinterpret_cast<const uint2*>(start ? cs->cstart + i : cs->cend + (i - ns))) : make_uint2(0, 0);
      const bool in = i < n && ((__ldg(filter + (e.x >> 5)) >> (e.x & 31)) & 1u);
      // events are sorted by position: the lanes of a position, and those of a segment, add once
      const uint32_t at = in ? (start ? 0u : L + 1) + e.y : 0xFFFFFFFFu;
      const uint32_t same = __match_any_sync(0xFFFFFFFFu, at);
      if (in && lane == static_cast<uint32_t>(__ffs(same) - 1)) atomicAdd(start_hist + at, static_cast<uint32_t>(__popc(same)));
      const uint32_t key = in ? (start ? 0u : nseg) + e.y / MUT_SEG : 0xFFFFFFFFu;
      const uint32_t segm = __match_any_sync(0xFFFFFFFFu, key);
      if (in && lane == static_cast<uint32_t>(__ffs(segm) - 1)) atomicAdd(seg_s + key, static_cast<uint32_t>(__popc(segm)));
   }
}
static_assert(MUT_SEG % (COV_BLOCKS * NBLOCK) == 0, "a CTA's positions lie in one segment");

__global__ void __launch_bounds__(1024) mut_clear_kernel(uint32_t* counts, uint32_t n_counts, uint32_t* scratch,
                                                         uint32_t n_scratch, int* status) {
   pdl_trigger();
   const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
   for (uint32_t i = i0; i < n_counts; i += step) counts[i] = 0;
   for (uint32_t i = i0; i < n_scratch; i += step) scratch[i] = 0;
   if (status && i0 == 0) *status = 0;
}

__global__ void __launch_bounds__(MUT_SEG, 2) mut_final_kernel(const DevTable* __restrict__ tab, uint32_t col,
                                                            const unsigned long long* __restrict__ fcount,
                                                            uint32_t* counts, const uint32_t* scratch) {
   pdl_wait();
   final_position_counts(&tab->seq[col], static_cast<uint32_t>(*fcount), counts, scratch);
}

}  // namespace

void set_ring_withholding(bool on) {
   const uint32_t v = on ? 1u : 0u;
   const cudaError_t e = cudaMemcpyToSymbol(g_withhold_ring_copies, &v, sizeof(v));
   if (e != cudaSuccess) throw std::runtime_error(std::string("set_ring_withholding: ") + cudaGetErrorString(e));
}

void mutations_setup() {
   const cudaError_t e = cudaFuncSetAttribute(mut_ring_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              static_cast<int>(RING_SMEM));
   if (e != cudaSuccess)
      throw std::runtime_error(std::string("shared memory of the Mutations container pass: ") + cudaGetErrorString(e));
}

void launch_mutations(const DevTable* d_table, const DevSeqCol& col_host, uint32_t col, uint32_t nchunks, uint32_t sms,
                      const uint32_t* d_filter,
                      const unsigned long long* d_filter_count, uint32_t* d_counts, uint32_t* d_scratch, int* d_err,
                      void* stream, uint32_t parts, uint64_t sparse_max, int* d_err_clear) {
   cudaStream_t s = static_cast<cudaStream_t>(stream);
   if (!(parts & MUT_PART_SPARSE)) sparse_max = 0;  // the dense passes count every filter
   // a dependent only of a kernel of this pass launched just before it, in the order above
   auto launch = [&](auto* kernel, uint32_t grid, uint32_t threads, size_t smem, bool dependent, auto... args) {
      cudaLaunchAttribute attr{};
      attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr.val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = grid;
      cfg.blockDim = threads;
      cfg.dynamicSmemBytes = smem;
      cfg.stream = s;
      cfg.attrs = &attr;
      cfg.numAttrs = dependent ? 1 : 0;
      cudaLaunchKernelEx(&cfg, kernel, args...);  // errors are read by the caller
   };
   const unsigned long long limit = sparse_max;
   const bool clear = parts & MUT_PART_CLEAR;
   if (clear) {
      const uint32_t words = col_host.nsym * col_host.L;
      launch(mut_clear_kernel, std::min((words + 1023) / 1024, sms), 1024, 0, false, d_counts, words, d_scratch,
             static_cast<uint32_t>(mut_scratch_words(col_host.L)), d_err_clear);
   }
   const bool coverage = parts & MUT_PART_COV;
   const bool first = coverage || sparse_max > 0;
   if (first) {
      const uint32_t buckets =
         ((nchunks + COV_CHUNKS - 1) / COV_CHUNKS) * ((col_host.nblocks_ev + COV_BLOCKS - 1) / COV_BLOCKS);
      const uint32_t events = (col_host.n_cstart + col_host.n_cend + MT - 1) / MT;
      const uint32_t groups = nchunks * CHUNK_WORDS / 32;  // 32-word groups, one per warp and step
      const uint32_t sparse_ctas = sparse_max ? std::max(1u, std::min(groups / NW, 2048u)) : 1u;
      launch(mut_cov_kernel, std::max(coverage ? buckets + events : 1u, sparse_ctas), MT, 0, clear, d_table, col, d_filter,
             d_filter_count, limit, coverage, d_counts, d_scratch);
   }
   const bool ring = (parts & MUT_PART_CTR) && col_host.nranges > 0;
   if (ring) launch(mut_ring_kernel, col_host.nranges, RING_T, RING_SMEM, first, d_table, col, d_filter, d_filter_count, limit,
                    d_counts, d_err);
   if (parts & MUT_PART_FINAL)
      launch(mut_final_kernel, (col_host.L + MUT_SEG - 1) / MUT_SEG, MUT_SEG, 0, ring, d_table, col, d_filter_count, d_counts,
             static_cast<const uint32_t*>(d_scratch));
}

}  // namespace rhygpu
