// sm_103a kernels of the filter and Count path (the Mutations kernels are in mutations.cu and
// batch.cu, the output rows in rows.cu, Details in details.cu).
//
//  filter_kernel        one CTA per (chunk, tile of W rows): runs the postorder filter program over a
//                       stack of W-bit tiles in shared memory; writes the row-set tile and/or adds
//                       its popcount (Count action, reference: copy_on_write_bitmap.cpp:108-118).
//                       With a trace buffer it records every instruction's cycles and result size
//                       (planner training).
//  filter_batch_kernel  persistent variant: CTAs pull (query, tile) work items from a counter.
//
// What bounds them: issue slots and latency, not bytes (a container holds 36 rows on average, a tile is
// 8 KiB). Hence a leaf followed by the operator that consumes it is one instruction (fuse_leaves),
// whose rows go straight into the top tile or the counter planes; leaves whose order does not
// matter are applied together, a warp each (group_leaves); arrays and run containers of DENSE_MIN rows and
// more are stored a second time as bitsets (or read as the few runs they are), combined word by word by
// the threads that own the words.
// Measured (2M rows, 4,096 trees of 1-64 leaves, one launch): 34.5 ms with a tile per leaf, 20.8 ms
// this way; the benchmark's 2,048 queries 3.28 -> 2.83 ms. 128 threads per CTA instead of 256: 25.6
// and 2.9 ms (the trees wait on latency, and more warps hide it).
// All arithmetic is integer; results are bit-exact with the CPU operators.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>

#include "device.h"

namespace rhygpu {

namespace {

constexpr uint32_t FT = 256;  // threads per filter CTA (the single-query kernel takes fewer for narrow tiles)

__device__ __forceinline__ uint32_t valid_word(uint32_t w, uint32_t nvalid) {
   const uint32_t b = w * 32;
   if (b + 32 <= nvalid) return 0xFFFFFFFFu;
   if (b >= nvalid) return 0u;
   return (1u << (nvalid - b)) - 1u;
}

struct TileCtx {
   const DevTable* __restrict__ tab;
   uint32_t v;
   uint32_t row0;
   uint32_t W;
   uint32_t nvalid;
   const uint32_t* aux;  // the query's precomputed row sets (PUSH_AUX), nchunks * CHUNK_WORDS words each
};

// Per-item staging for the chunk and row range of the current tile:
//  - the program's first LC_CODE instructions;
//  - container leaves (PUSH_SCAN / PUSH_DICT, c = ordinal + 1): the slot offsets of all leaves are
//    read in one round of loads and their descriptors in a second; every container whose symbol the
//    leaf ORs becomes an entry, so a leaf costs no dependent loads when the program reaches it;
//  - coverage leaves (PUSH_COVERED, c = ordinal + 1): the tile's ranges of uncovered rows and missing
//    intervals.
// Array payloads are copied into shared memory by TMA bulk copies while they fit; every other staged
// payload and range is handed to the TMA engine as a bulk L2 prefetch.
constexpr uint32_t LC_LEAVES = 128;
constexpr uint32_t LC_ENTS = 256;
constexpr uint32_t LC_COV = 64;
constexpr uint32_t LC_CODE = INLINE_CODE;
constexpr uint16_t LC_NONE = 0xFFFF;
constexpr uint32_t LC_PAY = 3072;      // u16 of array payloads copied into shared memory per item
constexpr uint32_t LC_BIG = 0x80000000u;
constexpr uint32_t LC_OWNER_MAX = 64;  // leaves of at most this many copied rows are set by their words' owners

// A container of a staged leaf: y = kind << 28 | rows (runs for E_RUN), x = where its payload is. Bitsets and the
// containers of few long runs (E_SPANS) have no rows to go through one by one.
// E_COPIED: x = byte offset in shared memory, else u16 offset in the arena. E_SPANS: runs << 24 in place of rows; x = the
// run (first row | rows - 1 << 16) of a container of one.
enum : uint32_t { E_COPIED = 0, E_ARRAY = 1, E_BITSET = 2, E_RUN = 3, E_SPANS = 4 };
constexpr uint32_t E_COUNT = 0x00FFFFFFu;

struct LeafCache {
   uint4 code[LC_CODE];
   uint4 pay4[LC_PAY / 8];        // array payloads (TMA bulk copies, 16-byte aligned runs)
   uint4 cov[LC_COV];             // a coverage leaf's late and early rows
   uint2 covm[LC_COV];            // and its missing intervals
   uint2 ent[LC_ENTS];            // leaf k's entries: arrays and runs from beg[k] up, bitsets and spans from beg[k] + n[k] down
   const uint4* src[LC_LEAVES];   // the leaf's descriptors
   const uint16_t* pay[LC_LEAVES];
   uint32_t symmask[LC_LEAVES];   // symbols the leaf ORs (every container for dictionary leaves)
   uint32_t cnt[LC_LEAVES];       // its array and run entries, bitset and span entries << 16
   uint32_t tot[LC_LEAVES];       // rows of the leaf's copied arrays; LC_BIG: it has other arrays or runs
   uint16_t n[LC_LEAVES];         // descriptors of the leaf's slot
   uint16_t beg[LC_LEAVES];       // LC_NONE: not staged (the leaf reads its descriptors from global memory)
   uint8_t dleaf[LC_ENTS];        // leaf (0-based) of staged descriptor i
   uint64_t bar;                  // completes the item's payload copies
   uint32_t nstaged;              // staged descriptors: the staged leaves are a prefix of the leaves
   uint32_t pay_used;             // u16 of pay4 reserved by this item's copies
   uint32_t ext_used;             // u16 of the program's free stack tiles reserved by this item's copies
   uint32_t next_item;
};
static_assert(sizeof(LeafCache) % 16 == 0, "tiles follow the leaf cache");

// Bulk prefetch of global bytes [a, b) into L2; a is rounded down and b up to 16 bytes, so the
// caller guarantees the rounded range stays inside the allocation.
__device__ __forceinline__ void prefetch_l2(const void* a, const void* b) {
   const uintptr_t s = reinterpret_cast<uintptr_t>(a) & ~static_cast<uintptr_t>(15);
   const uintptr_t e = (reinterpret_cast<uintptr_t>(b) + 15) & ~static_cast<uintptr_t>(15);
   if (e <= s) return;
   const uint32_t n = static_cast<uint32_t>(min(e - s, static_cast<uintptr_t>(32768)));
   asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(s), "r"(n) : "memory");
}

// Once per CTA, before the first item: the barrier of the payload copies.
__device__ __forceinline__ void init_leaves(LeafCache& lc) {
   if (threadIdx.x == 0) {
      const uint32_t b = static_cast<uint32_t>(__cvta_generic_to_shared(&lc.bar));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
   }
}

// What a coverage leaf at pos reads for the tile: rng = its late and early rows of the chunk
// (DevSeqCol::cov_rng), miss = its range in the missing-interval bucket of pos (sorted by row;
// TOFF_ROWS divides every tile boundary or is divided by it).
struct CoverRange {
   uint4 rng;
   uint2 miss;
};
__device__ __forceinline__ CoverRange cover_ranges(const DevTable* __restrict__ tab, const DevSeqCol* __restrict__ col,
                                                   uint32_t v, uint32_t row0, uint32_t W, uint32_t pos) {
   const uint32_t k0 = row0 / TOFF_ROWS, k1 = (row0 + W + TOFF_ROWS - 1) / TOFF_ROWS;
   const size_t b = static_cast<size_t>(pos / NBLOCK) * tab->nchunks + v;
   const uint32_t* no = col->nblk_toff + b * TOFF_N;
   return CoverRange{__ldg(col->cov_rng + b), make_uint2(__ldg(no + k0), __ldg(no + k1))};
}

// Testing the failure path of the bounded waits: while set (on the current device), the threads that
// stage leaf payloads announce their bytes on the item's barrier but never issue the bulk copies,
// so the item's wait gives up (after 1 ms) and the kernel sets error 6 (DEVERR_WAIT_FILTER). No
// copy is left in flight: the withheld copies never start. Off by default; set only through
// set_copy_withholding.
__device__ uint32_t g_withhold_leaf_copies = 0;

// Waits for phase `parity` of the copies' barrier, bounded by `limit_ns` on the GPU's global timer
// (2 s: a copy lands in microseconds) and, as a second bound, by 2^26 polls of at most about 1 us
// each; false if it gave up.
__device__ __forceinline__ bool wait_copies(LeafCache& lc, uint32_t parity, uint64_t limit_ns) {
   const uint32_t b = static_cast<uint32_t>(__cvta_generic_to_shared(&lc.bar));
   uint64_t t0 = 0;
#pragma unroll 1
   for (uint32_t i = 0; i < (1u << 26); ++i) {
      uint32_t done;
      asm volatile(
         "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
         : "=r"(done)
         : "r"(b), "r"(parity), "r"(1000u)
         : "memory");
      if (done) return true;
      uint64_t now;
      asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      else if (now - t0 > limit_ns) return false;
   }
   return false;
}

// Stages the item's instructions and leaves (see LeafCache). Array containers are also copied into
// shared memory by TMA bulk copies, into pay4 or into the ext_cap u16 at ext (the stack tiles the
// item's program leaves free): each issuing thread announces its bytes on the barrier (expect_tx)
// before starting its copy, and one thread arrives after every announcement, so the phase completes
// when the last copy lands. `phase` is the parity of this item's wait, flipped when copies were
// made. With next_item, thread 0 claims the CTA's next work item into lc.next_item while the copies
// are in flight. Returns false (error flag set) if the copies did not land. The caller has reset
// pay_used and ext_used and passed a barrier since the previous item.
__device__ bool stage_leaves(LeafCache& lc, const TileCtx& c, const Instr* __restrict__ code, uint32_t ncode,
                             uint32_t nl, uint32_t ncov, uint16_t* ext, uint32_t ext_cap, uint32_t& phase,
                             uint32_t* next_item, int* err) {
   const DevTable* __restrict__ tab = c.tab;
   const bool withhold = *static_cast<volatile uint32_t*>(&g_withhold_leaf_copies) != 0;
#pragma unroll 1
   for (uint32_t i = threadIdx.x; i < LC_ENTS; i += blockDim.x) lc.ent[i] = make_uint2(0, 0);  // E_COPIED, no rows
#pragma unroll 1
   for (uint32_t i = threadIdx.x; i < ncode; i += blockDim.x) {
      const uint4 raw = reinterpret_cast<const uint4*>(code)[i];  // global memory or the kernel's parameters
      if (i < LC_CODE) lc.code[i] = raw;
      const Instr in = *reinterpret_cast<const Instr*>(&raw);
      if (in.op == OP_PUSH_COVERED) {
         if (in.c == 0 || in.c > ncov) continue;
         const DevSeqCol* col = &tab->seq[in.col];
         const CoverRange r = cover_ranges(tab, col, c.v, c.row0, c.W, in.a);
         lc.cov[in.c - 1] = r.rng;
         lc.covm[in.c - 1] = r.miss;
         prefetch_l2(col->cov_late + r.rng.x, col->cov_late + r.rng.x + r.rng.y);
         prefetch_l2(col->cov_early + r.rng.z, col->cov_early + r.rng.z + r.rng.w);
         prefetch_l2(col->nblk + r.miss.x, col->nblk + r.miss.y);
         continue;
      }
      if ((in.op != OP_PUSH_SCAN && in.op != OP_PUSH_DICT) || in.c == 0 || in.c > nl) continue;
      const CtrDesc* ctrs;
      const uint32_t* off;
      const uint16_t* payload;
      size_t slot;
      if (in.op == OP_PUSH_SCAN) {
         const DevSeqCol* col = &tab->seq[in.col];
         ctrs = col->fctrs;
         off = col->off;
         payload = col->payload;
         slot = static_cast<size_t>(c.v) * col->L + in.a;
      } else {
         const DevDictCol* col = &tab->dict[in.col];
         ctrs = col->fctrs;
         off = col->off;
         payload = col->payload;
         slot = static_cast<size_t>(c.v) * col->nkeys + in.a;
      }
      const uint32_t b = __ldg(off + slot), e = __ldg(off + slot + 1), k = in.c - 1;
      lc.src[k] = reinterpret_cast<const uint4*>(ctrs) + b;
      lc.pay[k] = payload;
      lc.n[k] = static_cast<uint16_t>(e - b);
      lc.symmask[k] = in.op == OP_PUSH_SCAN ? in.b : 0xFFFFFFFFu;
      lc.cnt[k] = 0;
      lc.tot[k] = 0;
   }
   __syncthreads();
   if (threadIdx.x < 32) {  // exclusive scan of the counts; leaves that do not fit stay unstaged
      const uint32_t lane = threadIdx.x;
      uint32_t carry = 0, staged = 0;
#pragma unroll 1
      for (uint32_t k0 = 0; k0 < nl; k0 += 32) {
         const uint32_t k = k0 + lane;
         const uint32_t x = k < nl ? lc.n[k] : 0u;
         uint32_t incl = x;
#pragma unroll
         for (uint32_t o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if (lane >= o) incl += y;
         }
         const uint32_t ex = carry + incl - x;
         const bool fits = ex + x <= LC_ENTS;  // the leaves that fit are a prefix of them
         if (k < nl) lc.beg[k] = fits ? static_cast<uint16_t>(ex) : LC_NONE;
         if (fits) {
#pragma unroll 1
            for (uint32_t i = 0; i < x; ++i) lc.dleaf[ex + i] = static_cast<uint8_t>(k);
         }
         staged = max(staged, __reduce_max_sync(0xFFFFFFFFu, fits ? ex + x : 0u));
         carry += __shfl_sync(0xFFFFFFFFu, incl, 31);
      }
      if (lane == 0) lc.nstaged = staged;
   }
   __syncthreads();
   // one staged descriptor per thread: its load, and the copy or prefetch of its payload
   const uint32_t bar = static_cast<uint32_t>(__cvta_generic_to_shared(&lc.bar));
   const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(&lc));
#pragma unroll 1
   for (uint32_t j = threadIdx.x; j < lc.nstaged; j += blockDim.x) {
      const uint32_t k = lc.dleaf[j];
      const uint4 raw = __ldg(lc.src[k] + (j - lc.beg[k]));
      const CtrDesc d = *reinterpret_cast<const CtrDesc*>(&raw);
      if (!((lc.symmask[k] >> d.sym) & 1u)) continue;  // a symbol the leaf does not OR
      const uint32_t card = d.card_m1 + 1u;
      uint32_t at_ent;
      if (d.type == CT_BITSET || d.type == CT_SPANS) at_ent = lc.beg[k] + lc.n[k] - 1 - (atomicAdd(&lc.cnt[k], 0x10000u) >> 16);
      else at_ent = lc.beg[k] + (atomicAdd(&lc.cnt[k], 1u) & 0xFFFFu);
      // the arena ends with 16 spare bytes, so rounding the end up stays inside it
      const uint16_t* p = lc.pay[k] + d.payload;
      if (d.type == CT_ARRAY) {
         const uintptr_t a = reinterpret_cast<uintptr_t>(p);
         const uintptr_t a0 = a & ~static_cast<uintptr_t>(15);
         const uint32_t bytes = static_cast<uint32_t>(((a + 2u * card + 15) & ~static_cast<uintptr_t>(15)) - a0);
         uint32_t dst = 0;
         if (bytes <= 2 * LC_PAY) {
            const uint32_t at = atomicAdd(&lc.pay_used, bytes / 2);
            if (at + bytes / 2 <= LC_PAY) dst = static_cast<uint32_t>(__cvta_generic_to_shared(lc.pay4)) + 2 * at;
         }
         if (dst == 0 && ext_cap) {
            const uint32_t at = atomicAdd(&lc.ext_used, bytes / 2);
            if (at + bytes / 2 <= ext_cap) dst = static_cast<uint32_t>(__cvta_generic_to_shared(ext)) + 2 * at;
         }
         if (dst != 0) {
            lc.ent[at_ent] = make_uint2(dst - base + static_cast<uint32_t>(a - a0), (E_COPIED << 28) | card);
            atomicAdd(&lc.tot[k], card);
            asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
            if (!withhold)
               asm volatile(
                  "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                  "l"(a0), "r"(bytes), "r"(bar)
                  : "memory");
            continue;
         }
         lc.ent[at_ent] = make_uint2(d.payload, (E_ARRAY << 28) | card);
         atomicOr(&lc.tot[k], LC_BIG);
         prefetch_l2(p, p + card);
      } else if (d.type == CT_BITSET) {
         lc.ent[at_ent] = make_uint2(d.payload, static_cast<uint32_t>(E_BITSET) << 28);
         prefetch_l2(p + (c.row0 >> 4), p + ((c.row0 + c.W) >> 4));
      } else if (d.type == CT_SPANS) {
         const uint32_t x = d.nruns == 1 ? __ldg(p) | static_cast<uint32_t>(__ldg(p + 1)) << 16 : d.payload;
         lc.ent[at_ent] = make_uint2(x, (E_SPANS << 28) | static_cast<uint32_t>(d.nruns) << 24);
         if (d.nruns > 1) prefetch_l2(p, p + 2u * d.nruns);
      } else {
         lc.ent[at_ent] = make_uint2(d.payload, (E_RUN << 28) | d.nruns);
         atomicOr(&lc.tot[k], LC_BIG);
         prefetch_l2(p, p + 2u * d.nruns);
      }
   }
   __syncthreads();
   uint32_t claimed = 0;
   if (next_item && threadIdx.x == 0) claimed = atomicAdd(next_item, 1u);
   bool ok = true;
   if (lc.pay_used != 0 || lc.ext_used != 0) {  // otherwise no copies this item
      if (threadIdx.x == 0)
         asm volatile("{\n .reg .b64 st;\n mbarrier.arrive.shared::cta.b64 st, [%0];\n}\n" ::"r"(bar) : "memory");
      const uint64_t limit = withhold ? 1000000ull : 2000000000ull;
      ok = wait_copies(lc, phase, limit);
      if (!ok) ok = wait_copies(lc, phase, limit);  // once more before giving up with copies possibly in flight
      phase ^= 1u;
      ok = __syncthreads_and(ok);
      if (!ok && threadIdx.x == 0) atomicExch(err, DEVERR_WAIT_FILTER);
   }
   if (next_item && threadIdx.x == 0) lc.next_item = claimed;  // read after the caller's next barrier
   return ok;
}

// Every tile has one fixed mapping: thread t owns the uint4 words t, t + blockDim.x, ... of every tile.
// Operators on whole tiles therefore need no barrier; only row lists write words that a thread does
// not own.
__device__ __forceinline__ uint4 valid4(uint32_t w4, const TileCtx& c) {
   if (c.nvalid == c.W) return make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
   return make_uint4(valid_word(4 * w4, c.nvalid), valid_word(4 * w4 + 1, c.nvalid), valid_word(4 * w4 + 2, c.nvalid),
                     valid_word(4 * w4 + 3, c.nvalid));
}
__device__ __forceinline__ uint4 and4(uint4 a, uint4 b) { return make_uint4(a.x & b.x, a.y & b.y, a.z & b.z, a.w & b.w); }
__device__ __forceinline__ uint4 andnot4(uint4 a, uint4 b) {
   return make_uint4(a.x & ~b.x, a.y & ~b.y, a.z & ~b.z, a.w & ~b.w);
}
__device__ __forceinline__ uint4 xor4(uint4 a, uint4 b) { return make_uint4(a.x ^ b.x, a.y ^ b.y, a.z ^ b.z, a.w ^ b.w); }
__device__ __forceinline__ uint4 or4(uint4 a, uint4 b) { return make_uint4(a.x | b.x, a.y | b.y, a.z | b.z, a.w | b.w); }
__device__ __forceinline__ bool any4(uint4 a) { return (a.x | a.y | a.z | a.w) != 0u; }
__device__ __forceinline__ bool ne4(uint4 a, uint4 b) {
   return ((a.x ^ b.x) | (a.y ^ b.y) | (a.z ^ b.z) | (a.w ^ b.w)) != 0u;
}


// ---- applying a leaf ----
//
// A leaf's rows are applied one by one where its value is consumed: set in or removed from the top
// tile, or added to the counter planes, with shared-memory atomics. Leaves are sparse (36 rows per
// container on average), so this takes a fraction of the instructions of building the leaf's tile
// and combining it word by word.

// The rows of the masks b0 at word q0 and b1 at word q1 of a tile (A_ADD: of the P counter planes there,
// WW words apart), their atomics in flight together; an empty mask touches nothing. Additions commute, also when
// threads add to one row at a time: each plane's exchange returns the old bits as the carries, so a plane
// receives half as many carries at a row as the one below it received bits, in any order; the top plane
// only ever gets set.
__device__ __forceinline__ void apply_masks(uint32_t* q0, uint32_t b0, uint32_t* q1, uint32_t b1, uint32_t WW, uint32_t P,
                                            uint32_t A) {
   if (A == A_ADD) {
#pragma unroll 1
      for (uint32_t i = 0; i + 1 < P && (b0 | b1); ++i, q0 += WW, q1 += WW) {
         uint32_t o0 = 0, o1 = 0;
         if (b0) o0 = atomicXor(q0, b0);
         if (b1) o1 = atomicXor(q1, b1);
         b0 &= o0;
         b1 &= o1;
      }
   }
   if (A == A_ANDNOT) {
      if (b0) atomicAnd(q0, ~b0);
      if (b1) atomicAnd(q1, ~b1);
   } else {
      if (b0) atomicOr(q0, b0);
      if (b1) atomicOr(q1, b1);
   }
}
// Rows r0 (with `one`) and r1 (with `two`) of the tile at T.
__device__ __forceinline__ void apply_rows(uint32_t* T, uint32_t WW, uint32_t P, uint32_t A, uint32_t r0, bool one,
                                           uint32_t r1, bool two) {
   apply_masks(T + (r0 >> 5), one ? 1u << (r0 & 31) : 0u, T + (r1 >> 5), two ? 1u << (r1 & 31) : 0u, WW, P, A);
}
__device__ __forceinline__ void apply_row(uint32_t* T, uint32_t WW, uint32_t P, uint32_t A, uint32_t r) {
   apply_rows(T, WW, P, A, r, true, 0, false);
}

// The value v of uint4 word w4 meets the target: stored, combined with the tile at T4, or (FUSE_THR_ADD)
// added to the P counter planes at T4.
__device__ __forceinline__ void put_word(uint4* T4, uint32_t W4, uint32_t P, uint32_t f, uint32_t w4, uint4 v) {
   uint4* q = T4 + w4;
   if (f == FUSE_THR_ADD) {
#pragma unroll 1
      for (uint32_t i = 0; i + 1 < P && any4(v); ++i, q += W4) {  // ripple carry
         const uint4 p = *q;
         *q = make_uint4(p.x ^ v.x, p.y ^ v.y, p.z ^ v.z, p.w ^ v.w);
         v = and4(v, p);
      }
      if (any4(v)) *q = or4(*q, v);
   } else if (f == FUSE_NONE) {
      *q = v;
   } else {
      const uint4 x = *q;
      *q = f == FUSE_AND ? and4(x, v) : f == FUSE_OR ? or4(x, v) : andnot4(x, v);
   }
}

// Thread t of nt: its share of the rows of an array in global memory, read 8 at a time (the arena ends
// with 16 spare bytes).
__device__ __forceinline__ void apply_array(uint32_t* T, uint32_t P, uint32_t A, const TileCtx& c,
                                            const uint16_t* __restrict__ p, uint32_t n, uint32_t t, uint32_t nt) {
   const uint32_t lead = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p) & 15u) / 2;
   const uint4* a = reinterpret_cast<const uint4*>(p - lead);
#pragma unroll 1
   for (uint32_t i = 8 * t; i < lead + n; i += 8 * nt) {
      uint4 v = __ldg(a + (i >> 3));
#pragma unroll 1
      for (uint32_t j = i; j < i + 8; j += 2) {
         const uint32_t r0 = (v.x & 0xFFFFu) - c.row0, r1 = (v.x >> 16) - c.row0;
         apply_rows(T, c.W >> 5, P, A, r0, j >= lead && j < lead + n && r0 < c.W, r1,
                    j + 1 >= lead && j + 1 < lead + n && r1 < c.W);
         v = make_uint4(v.y, v.z, v.w, 0);
      }
   }
}
// Runs that are not in one of the other forms (fewer than DENSE_MIN rows, or a leaf that was not staged). Whole
// warps (thread t of nt): 32 runs at a time, each lane the first and the last word of its own run and, where they
// are few, the words between them; the words inside a longer run go to the whole warp. Applied row by row by one
// thread a run, a count over a column that the rows are sorted by (runs of up to a whole chunk) took 780 us
// at 400,000 rows, and 18 us so; NOf of 30 such sites 27.4 ms, and 0.11.
constexpr uint32_t RUN_OWN = 4;  // words inside a run that its own lane takes
__device__ __forceinline__ void apply_runs(uint32_t* T, uint32_t P, uint32_t A, const TileCtx& c,
                                           const uint16_t* __restrict__ p, uint32_t n, uint32_t t, uint32_t nt) {
   const uint32_t lane = t & 31, WW = c.W >> 5;
   constexpr uint32_t NO_RUN = 0xFFFFFFFFu;  // first row | rows - 1 << 16
   auto load = [&](uint32_t i) { return i < n ? __ldg(p + 2 * i) | static_cast<uint32_t>(__ldg(p + 2 * i + 1)) << 16 : NO_RUN; };
   uint32_t next = load(t);
#pragma unroll 1
   for (uint32_t i = t; i - lane < n; i += nt) {
      const uint32_t run = next;
      next = load(i + nt);
      uint32_t a = 0, b = 0;  // this lane's run in the tile: [a, b)
      if (run != NO_RUN) {
         const uint32_t s = run & 0xFFFFu, e = s + (run >> 16) + 1u;
         a = max(s, c.row0) - c.row0;
         b = max(min(e, c.row0 + c.W), c.row0) - c.row0;
      }
      uint32_t w = 0, last = 0;
      if (a < b) {
         w = a >> 5;
         last = (b - 1) >> 5;
         const uint32_t head = 0xFFFFFFFFu << (a & 31), tail = 0xFFFFFFFFu >> (31 - ((b - 1) & 31));
         apply_masks(T + w, w == last ? head & tail : head, T + last, w == last ? 0u : tail, WW, P, A);
      }
      const bool wide = last - w > RUN_OWN + 1;
      uint32_t todo = __ballot_sync(0xFFFFFFFFu, wide);
      if (!wide)
#pragma unroll 1
         for (++w; w < last; w += 2) apply_masks(T + w, 0xFFFFFFFFu, T + w + 1, w + 1 < last ? 0xFFFFFFFFu : 0u, WW, P, A);
      __syncwarp();
#pragma unroll 1
      for (; todo; todo &= todo - 1) {
         const uint32_t l = __ffs(todo) - 1, e = __shfl_sync(0xFFFFFFFFu, last, l);
#pragma unroll 1
         for (uint32_t x = __shfl_sync(0xFFFFFFFFu, w, l) + 1 + lane; x < e; x += 64)
            apply_masks(T + x, 0xFFFFFFFFu, T + x + 32, x + 32 < e ? 0xFFFFFFFFu : 0u, WW, P, A);
      }
   }
}

// Bits below n (0 .. 32) of a word.
__device__ __forceinline__ uint32_t low_bits(int32_t n) { return ~__funnelshift_lc(0u, 0xFFFFFFFFu, static_cast<uint32_t>(min(max(n, 0), 32))); }

// The n <= SPAN_RUNS runs of a container (x: the run itself if it is one, else where they are in the arena) meet
// the target as a bitset's words do, each combined by the thread that owns it: no atomics, no barrier. A warp
// passes over the runs that miss its 4,096 rows.
__device__ __forceinline__ void put_spans(uint4* T4, uint32_t P, uint32_t f, const TileCtx& c,
                                          const uint16_t* __restrict__ payload, uint32_t x, uint32_t n) {
   const uint32_t lane = threadIdx.x & 31, W4 = c.W >> 7;
   uint32_t mine = x;  // lane j: run j
   if (n > 1 && lane < n) {
      const uint16_t* p = payload + x + 2 * lane;
      mine = __ldg(p) | static_cast<uint32_t>(__ldg(p + 1)) << 16;
   }
#pragma unroll 1
   for (uint32_t b4 = threadIdx.x - lane; b4 < W4; b4 += blockDim.x) {  // the warp's 32 words
      const int32_t r0 = static_cast<int32_t>(c.row0 + 128 * b4), r = r0 + 128 * static_cast<int32_t>(lane);
      uint4 v = make_uint4(0, 0, 0, 0);
#pragma unroll 1
      for (uint32_t j = 0; j < n; ++j) {
         const uint32_t run = __shfl_sync(0xFFFFFFFFu, mine, j);
         const int32_t s = static_cast<int32_t>(run & 0xFFFFu), e = s + static_cast<int32_t>(run >> 16) + 1;
         if (e <= r0 || s >= r0 + 4096) continue;  // the same in every lane
         v.x |= low_bits(e - r) & ~low_bits(s - r);
         v.y |= low_bits(e - r - 32) & ~low_bits(s - r - 32);
         v.z |= low_bits(e - r - 64) & ~low_bits(s - r - 64);
         v.w |= low_bits(e - r - 96) & ~low_bits(s - r - 96);
      }
      if (b4 + lane < W4 && any4(v)) put_word(T4, W4, P, f, b4 + lane, v);
   }
}

// A container leaf that was not staged, from its descriptors; every thread takes part, with barriers.
__device__ __noinline__ void apply_unstaged(uint32_t* T, uint32_t P, uint32_t A, const Instr& in, const TileCtx& c) {
   const CtrDesc* ctrs;
   const uint16_t* payload;
   const uint32_t* off;
   size_t slot;
   uint32_t mask = 0xFFFFFFFFu;
   if (in.op == OP_PUSH_SCAN) {
      const DevSeqCol* col = &c.tab->seq[in.col];
      ctrs = col->fctrs, payload = col->payload, off = col->off, mask = in.b;
      slot = static_cast<size_t>(c.v) * col->L + in.a;
   } else {
      const DevDictCol* col = &c.tab->dict[in.col];
      ctrs = col->fctrs, payload = col->payload, off = col->off;
      slot = static_cast<size_t>(c.v) * col->nkeys + in.a;
   }
   const uint32_t b = __ldg(off + slot), e = __ldg(off + slot + 1), W4 = c.W >> 7;
   const uint32_t f = A == A_OR ? FUSE_OR : A == A_ANDNOT ? FUSE_ANDNOT : FUSE_THR_ADD;
   __syncthreads();
#pragma unroll 1
   for (uint32_t i = b; i < e; ++i) {
      const uint4 raw = __ldg(reinterpret_cast<const uint4*>(ctrs) + i);
      const CtrDesc d = *reinterpret_cast<const CtrDesc*>(&raw);
      if (!((mask >> d.sym) & 1u)) continue;
      const uint16_t* p = payload + d.payload;
      if (d.type == CT_BITSET) {
         const uint4* src = reinterpret_cast<const uint4*>(p) + (c.row0 >> 7);
#pragma unroll 1
         for (uint32_t w4 = threadIdx.x; w4 < W4; w4 += blockDim.x)
            put_word(reinterpret_cast<uint4*>(T), W4, P, f, w4, __ldg(src + w4));
      } else if (d.type == CT_ARRAY) {
         apply_array(T, P, A, c, p, d.card_m1 + 1u, threadIdx.x, blockDim.x);
      } else {
         apply_runs(T, P, A, c, p, d.nruns, threadIdx.x, blockDim.x);
      }
      __syncthreads();
   }
}

// Applies the rows not covered at pos: those whose covered region starts after pos or ends before it, and
// those with a missing interval over pos (intervals lie inside the covered region, so no row comes
// twice). All threads share the lists.
__device__ __forceinline__ void apply_uncovered(uint32_t* T, uint32_t P, uint32_t A, const TileCtx& c,
                                                const DevSeqCol* __restrict__ col, uint32_t pos, const CoverRange& r) {
   const uint32_t WW = c.W >> 5, nb = r.rng.y + r.rng.w;
#pragma unroll 1
   for (uint32_t i = threadIdx.x; i < nb; i += blockDim.x) {
      const bool late = i < r.rng.y;
      const uint2 e = __ldg(reinterpret_cast<const uint2*>(late ? col->cov_late + r.rng.x + i : col->cov_early + r.rng.z + (i - r.rng.y)));
      const uint32_t row = e.x - c.row0;
      if (row < c.W && (e.y > pos) == late) apply_row(T, WW, P, A, row);
   }
   // four intervals per load: 256 threads read a chunk's bucket of a 128-position block (about 540) at once
   const uint32_t q = pos % NBLOCK;
   const uint4* nblk = reinterpret_cast<const uint4*>(col->nblk);
#pragma unroll 1
   for (uint32_t i = r.miss.x / 4 + threadIdx.x; i < (r.miss.y + 3) / 4; i += blockDim.x) {
      uint4 e = __ldg(nblk + i);
#pragma unroll 1
      for (uint32_t k = 0; k < 2; ++k) {
         const uint32_t r0 = (e.x & 0xFFFFu) - c.row0, r1 = (e.y & 0xFFFFu) - c.row0;
         apply_rows(T, WW, P, A, r0, r0 < c.W && ((e.x >> 16) & 0xFFu) <= q && q < (e.x >> 24), r1,
                    r1 < c.W && ((e.y >> 16) & 0xFFu) <= q && q < (e.y >> 24));
         e = make_uint4(e.z, e.w, 0, 0);
      }
   }
}

__device__ __forceinline__ Instr fetch(const Instr* __restrict__ code, uint32_t pc, const LeafCache& lc) {
   const uint4 raw = pc < LC_CODE ? lc.code[pc] : __ldg(reinterpret_cast<const uint4*>(code) + pc);
   return *reinterpret_cast<const Instr*>(&raw);
}

// Applies row-list leaves to one target (the tile, scratch tile or counter planes at T): mc container
// leaves with ordinals k0 + 1 .., their instructions from pc on, then mv coverage leaves. Bitsets
// first, each owner its own words; then, between two barriers, the staged entries and the coverage
// lists. A group's entries are shared out over the warps, so that a leaf costs one warp a few
// instructions per 32 rows instead of every warp its control work; a lone leaf's rows over all
// threads; a lone leaf of at most LC_OWNER_MAX rows goes to the warps that own its words (every warp
// reads every row), with no CTA barrier.
__device__ __forceinline__ void apply_leaves(uint32_t* T, uint32_t P, uint32_t A, const Instr* __restrict__ code,
                                             uint32_t pc, uint32_t k0, uint32_t mc, uint32_t mv, const TileCtx& c,
                                             const LeafCache& lc, uint32_t nl, uint32_t ncov) {
   const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W4 = c.W >> 7;
   bool owner = false;
   if (mc > 0 && (k0 + mc > nl || lc.beg[k0 + mc - 1] == LC_NONE)) {
#pragma unroll 1
      for (uint32_t i = 0; i < mc; ++i) apply_unstaged(T, P, A, fetch(code, pc + i, lc), c);
      if (mv == 0) return;
   } else {
      if (mc > 0) {
         // bitsets, three at a time: their loads in flight together, and a full adder in front of the planes (a
         // word at a time: unrolled by two, the code cost the 4,096 trees of 1-64 leaves 2% in instruction fetches)
         const uint32_t f = A == A_OR ? FUSE_OR : A == A_ANDNOT ? FUSE_ANDNOT : FUSE_THR_ADD;
         uint32_t l = k0, nb = lc.cnt[k0] >> 16;
#pragma unroll 1
         for (;;) {
            const uint4 *p0 = nullptr, *p1 = nullptr, *p2 = nullptr;
            uint32_t have = 0;
#pragma unroll 1
            while (have < 3) {
               if (nb == 0) {
                  if (++l >= k0 + mc) break;
                  nb = lc.cnt[l] >> 16;
                  continue;
               }
               const uint2 en = lc.ent[lc.beg[l] + lc.n[l] - nb];
               --nb;
               if (en.y >> 28 == E_SPANS) {
                  put_spans(reinterpret_cast<uint4*>(T), P, f, c, lc.pay[l], en.x, (en.y >> 24) & 15u);
                  continue;
               }
               const uint4* p = reinterpret_cast<const uint4*>(lc.pay[l] + en.x) + (c.row0 >> 7);
               if (have == 0) p0 = p;
               else if (have == 1) p1 = p;
               else p2 = p;
               ++have;
            }
            if (have == 0) break;
#pragma unroll 1
            for (uint32_t w4 = threadIdx.x; w4 < W4; w4 += blockDim.x) {
               uint4* T4 = reinterpret_cast<uint4*>(T);
               const uint4 zero = make_uint4(0, 0, 0, 0);
               const uint4 x = __ldg(p0 + w4), y = have > 1 ? __ldg(p1 + w4) : zero, z = have > 2 ? __ldg(p2 + w4) : zero;
               if (f == FUSE_THR_ADD && P > 1) {
                  const uint4 u = xor4(x, y), carry = or4(and4(x, y), and4(u, z));
                  put_word(T4, W4, P, f, w4, xor4(u, z));
                  if (any4(carry)) put_word(T4 + W4, W4, P - 1, f, w4, carry);
               } else {
                  put_word(T4, W4, P, f, w4, or4(or4(x, y), z));
               }
            }
            if (l >= k0 + mc) break;
         }
         if (mc == 1 && mv == 0) {
            const uint32_t tot = lc.tot[k0];
            if (tot == 0) return;  // bitsets only, or nothing
            owner = tot <= LC_OWNER_MAX;
         }
      }
      if (owner) __syncwarp();
      else __syncthreads();
      if (mc > 0) {
         const bool lone = mc == 1;
         const uint32_t j0 = lone && !owner ? threadIdx.x : lane, js = lone && !owner ? blockDim.x : 32u;
         const uint32_t wmask = owner ? (blockDim.x >> 5) - 1u : 0u, wsel = owner ? warp : 0u;
         const uint32_t e = lc.beg[k0 + mc - 1] + lc.n[k0 + mc - 1];
         uint32_t turn = lone ? 0u : warp;  // entries to pass over before this warp's next
#pragma unroll 1
         for (uint32_t i0 = lc.beg[k0]; i0 < e; i0 += 32) {
            const uint2 mine = i0 + lane < e ? lc.ent[i0 + lane] : make_uint2(0, 0);
            uint32_t todo = __ballot_sync(0xFFFFFFFFu, (mine.y & E_COUNT) != 0u);  // bitsets and spans have no count
#pragma unroll 1
            for (; todo; todo &= todo - 1) {
               if (turn) {
                  --turn;
                  continue;
               }
               turn = lone ? 0u : (blockDim.x >> 5) - 1u;
               const uint32_t l = __ffs(todo) - 1;
               const uint32_t x = __shfl_sync(0xFFFFFFFFu, mine.x, l), y = __shfl_sync(0xFFFFFFFFu, mine.y, l);
               const uint32_t kind = y >> 28, n = y & E_COUNT;
               if (kind == E_COPIED) {
                  const uint16_t* sp = reinterpret_cast<const uint16_t*>(reinterpret_cast<const uint8_t*>(&lc) + x);
#pragma unroll 1
                  for (uint32_t j = j0; j < n; j += 2 * js) {
                     const uint32_t r0 = static_cast<uint32_t>(sp[j]) - c.row0;
                     const uint32_t r1 = j + js < n ? static_cast<uint32_t>(sp[j + js]) - c.row0 : 0xFFFFFFFFu;
                     apply_rows(T, c.W >> 5, P, A, r0, r0 < c.W && ((r0 >> 12) & wmask) == wsel, r1,
                                r1 < c.W && ((r1 >> 12) & wmask) == wsel);
                  }
               } else if (kind == E_ARRAY) {
                  apply_array(T, P, A, c, lc.pay[lc.dleaf[i0 + l]] + x, n, j0, js);
               } else {
                  apply_runs(T, P, A, c, lc.pay[lc.dleaf[i0 + l]] + x, n, j0, js);
               }
               __syncwarp();
            }
         }
      }
   }
#pragma unroll 1
   for (uint32_t i = 0; i < mv; ++i) {
      const Instr in = fetch(code, pc + mc + i, lc);
      const DevSeqCol* col = &c.tab->seq[in.col];
      const CoverRange r = (in.c >= 1 && in.c <= ncov) ? CoverRange{lc.cov[in.c - 1], lc.covm[in.c - 1]}
                                                       : cover_ranges(c.tab, col, c.v, c.row0, c.W, in.a);
      apply_uncovered(T, P, A, c, col, in.a, r);
   }
   if (owner) __syncwarp();
   else __syncthreads();
}

// Rows whose date lies in [lo, hi] (outside it: flags & 2); null dates match with flags & 1. Every
// comparison of the date predicates and the two-sided DateBetween reduce to this form: dates up to
// hi but not up to lo - 1, read from the range-encoded index (DevDateCol).
struct DateLeaf {
   const uint4* planes;
   const uint4* nulls;
   size_t stride4;
   uint32_t ndig, width, last;
   uint32_t hi, below;           // offsets from the index's base; below = lo - 1
   bool none, all_up, no_below;  // no date in [lo, hi]; hi at or past the last date; lo at or before the first
   uint32_t flags;
};
__device__ __forceinline__ DateLeaf date_leaf(const TileCtx& c, const DevDateCol* __restrict__ col, int32_t lo, int32_t hi,
                                              uint32_t flags) {
   DateLeaf d;
   const int64_t l = static_cast<int64_t>(lo) - col->base, h = static_cast<int64_t>(hi) - col->base, span = col->span;
   d.none = lo > hi || h < 0 || l > span;
   d.all_up = h >= span;
   d.no_below = l <= 0;
   d.hi = static_cast<uint32_t>(h);
   d.below = static_cast<uint32_t>(l - 1);
   d.ndig = col->ndig;
   d.width = col->width;
   d.last = col->last;
   d.stride4 = static_cast<size_t>(c.tab->nchunks) * (CHUNK_WORDS / 4);
   const size_t base4 = (static_cast<size_t>(c.v) * CHUNK_WORDS + (c.row0 >> 5)) / 4;
   d.planes = reinterpret_cast<const uint4*>(col->planes) + base4;
   d.nulls = reinterpret_cast<const uint4*>(col->nulls) + base4;
   d.flags = flags;
   return d;
}
// The rows whose date offset is at most v, from the lowest digit up.
__device__ __forceinline__ uint4 date_upto(const DateLeaf& d, uint32_t v, uint32_t w4) {
   const uint4* p = d.planes + w4;
   const uint32_t m = (1u << d.width) - 1u;
   uint4 acc = __ldg(p + (v & m) * d.stride4);
#pragma unroll 1
   for (uint32_t i = 1; i < d.ndig; ++i) {
      const uint32_t g = (i << d.width) + ((v >> (d.width * i)) & m);
      const uint4 x = __ldg(p + g * d.stride4);
      const uint4 y = (g & m) ? __ldg(p + (g - 1) * d.stride4) : make_uint4(0, 0, 0, 0);
      acc = or4(y, and4(x, acc));
   }
   return acc;
}
__device__ __forceinline__ uint4 date_word(const DateLeaf& d, uint32_t w4) {
   uint4 in = make_uint4(0, 0, 0, 0);
   if (!d.none) {
      in = d.all_up ? __ldg(d.planes + d.last * d.stride4 + w4) : date_upto(d, d.hi, w4);
      if (!d.no_below) in = andnot4(in, date_upto(d, d.below, w4));
   }
   if (d.flags & 2) in = andnot4(__ldg(d.planes + d.last * d.stride4 + w4), in);
   if (d.flags & 1) in = or4(in, __ldg(d.nulls + w4));
   return in;
}

// Runs a filter program for one tile over a stack of `cap` tiles at stk4; the result is left in tile 0,
// complete for the thread that owns each word. X4 is the scratch tile: zero between leaves, it holds
// the rows of the few leaves whose operator needs all of them at once (AND of a row list, and the
// operators that take its complement). Returns false on a malformed program (the error flag is set).
// With TRACE (the single-query kernel's trace mode, for planner training) every executed instruction pc
// stores trace[2 pc] = its cycles (first thread, between barriers around the instruction) and
// trace[2 pc + 1] = the population count of the top of the stack after it.
// Every part of the interpreter exists once in the code, and its loops are not unrolled far: the
// warps of an SM are in different instructions, and a first version specialised by tile width and
// operator (575 KB of code) spent most of its time on instruction fetches.
template <bool TRACE>
__device__ __forceinline__ bool run_program(const TileCtx& c, const Instr* __restrict__ code, uint32_t ncode,
                                            uint4* stk4, uint32_t cap, uint4* X4, const LeafCache& lc, uint32_t nl,
                                            uint32_t ncov, int* err, uint32_t* trace) {
   const uint32_t W4 = c.W >> 7;
   uint32_t sp = 0;
   uint32_t steps = 0;
   int bad = 0;
#pragma unroll 1
   for (uint32_t pc = 0; pc < ncode;) {
      if (++steps > 4u * MAX_PROGRAM) {  // jumps only go forward; this bounds a corrupted program
         bad = 3;
         break;
      }
      long long t_start = 0;
      if (TRACE) {
         __syncthreads();
         t_start = clock64();
      }
      const Instr in = fetch(code, pc, lc);
      uint32_t next = pc + 1;
      // what combines with the target word by word, if anything does
      enum : uint32_t { S_NONE, S_ZERO, S_FULL, S_SET, S_DATE, S_SCRATCH, S_TILE };
      uint32_t src = S_NONE, f = FUSE_NONE, P = 0;
      const uint4* from = nullptr;
      bool negate = false;
      uint4* T4 = stk4;
      if (is_leaf(in.op) || in.op == OP_GROUP) {
         const bool group = in.op == OP_GROUP;
         const bool list = group || in.op == OP_PUSH_SCAN || in.op == OP_PUSH_DICT || in.op == OP_PUSH_COVERED;
         P = leaf_planes(in.flags);
         bool add, push;
         uint32_t A = in.flags & 3u;
         if (group) {
            add = A == A_ADD;
            push = in.flags & GROUP_PUSH;
            next = pc + 1 + in.a;
            if (next > ncode) bad = 4;
         } else {
            f = leaf_fused(in.flags);
            add = f == FUSE_THR_ADD || f == FUSE_THR_ADD_NOT;
            push = f == FUSE_NONE;
         }
         if (push) {
            if (sp >= cap) bad = 1;
            ++sp;
         } else if (sp < (add ? P : 1u)) {
            bad = 2;
         }
         if (bad) break;
         T4 = stk4 + (sp - (add ? P : 1u)) * W4;  // the new tile, the top tile, or the counter's planes
         if (list) {
            bool scratch = false;
            if (!group) {
               // the leaf is a list of rows, or (comp) all valid rows but those listed
               const bool comp = in.op == OP_PUSH_COVERED && !(in.flags & 1);
               if (f == (comp ? FUSE_THR_ADD_NOT : FUSE_THR_ADD)) {
                  A = A_ADD;
               } else if (comp ? (push || f == FUSE_AND) : f == FUSE_ANDNOT) {
                  A = A_ANDNOT;
               } else {
                  A = A_OR;
                  scratch = comp || (!push && f != FUSE_OR);
               }
               if (scratch) {  // then the scratch tile, or its complement, meets the target
                  src = S_SCRATCH;
                  negate = add || f == FUSE_OR;
                  if (add) f = FUSE_THR_ADD;
                  else if (f == FUSE_ANDNOT) f = FUSE_AND;  // not (valid but X): X
               }
            }
            if (push) {
#pragma unroll 1
               for (uint32_t w4 = threadIdx.x; w4 < W4; w4 += blockDim.x)
                  T4[w4] = A == A_ANDNOT ? valid4(w4, c) : make_uint4(0, 0, 0, 0);
            }
            const uint32_t mc = group ? in.b >> 16 : in.op != OP_PUSH_COVERED, mv = group ? in.c >> 16 : mc ^ 1u;
            apply_leaves(reinterpret_cast<uint32_t*>(scratch ? X4 : T4), P, A, code, group ? pc + 1 : pc,
                         (group ? in.b & 0xFFFFu : in.c) - 1, mc, mv, c, lc, nl, ncov);
         } else {
            if (f == FUSE_THR_ADD_NOT) {
               negate = true;
               f = FUSE_THR_ADD;
            }
            src = in.op == OP_PUSH_DATE ? S_DATE : in.op == OP_PUSH_FULL ? S_FULL : in.op == OP_PUSH_EMPTY ? S_ZERO : S_SET;
            if (src == S_SET) {
               const uint32_t* set = in.op == OP_PUSH_NULLS ? c.tab->seq[in.col].null_tiles : c.aux;
               if (set == nullptr) {
                  bad = 5;
                  break;
               }
               if (in.op == OP_PUSH_AUX) set += static_cast<size_t>(in.a) * c.tab->nchunks * CHUNK_WORDS;
               from = reinterpret_cast<const uint4*>(set + static_cast<size_t>(c.v) * CHUNK_WORDS + (c.row0 >> 5));
            }
         }
      } else if (in.op == OP_AND || in.op == OP_ANDNOT || in.op == OP_OR || in.op == OP_THR_ADD) {
         const bool add = in.op == OP_THR_ADD;
         P = add ? in.a : 1u;
         if (sp < P + 1) {
            bad = 2;
            break;
         }
         --sp;
         src = S_TILE;
         from = stk4 + sp * W4;
         T4 = stk4 + (sp - P) * W4;
         f = in.op == OP_AND ? FUSE_AND : in.op == OP_OR ? FUSE_OR : add ? FUSE_THR_ADD : FUSE_ANDNOT;
         negate = add && (in.flags & 1);
      } else if (in.op == OP_NOT) {
         if (sp < 1) {
            bad = 2;
            break;
         }
         src = S_TILE;
         from = T4 = stk4 + (sp - 1) * W4;
         negate = true;
      } else if (in.op == OP_THR_BEGIN) {
         if (sp + in.a > cap) {
            bad = 1;
            break;
         }
#pragma unroll 1
         for (uint32_t i = sp; i < sp + in.a; ++i)
#pragma unroll 1
            for (uint32_t w4 = threadIdx.x; w4 < W4; w4 += blockDim.x) stk4[i * W4 + w4] = make_uint4(0, 0, 0, 0);
         sp += in.a;
      } else if (in.op == OP_THR_END) {
         const uint32_t n = in.b;
         P = in.a;
         if (sp < P) {
            bad = 2;
            break;
         }
         sp -= P;
#pragma unroll 1
         for (uint32_t w4 = threadIdx.x; w4 < W4; w4 += blockDim.x) {  // compare with n from the top plane down
            uint4 gt = make_uint4(0, 0, 0, 0), eq = make_uint4(~0u, ~0u, ~0u, ~0u);
#pragma unroll 2
            for (int i = static_cast<int>(P) - 1; i >= 0; --i) {
               const uint4 p = stk4[(sp + i) * W4 + w4];
               if ((n >> i) & 1u) {
                  eq = and4(eq, p);
               } else {
                  gt = or4(gt, and4(eq, p));
                  eq = andnot4(eq, p);
               }
            }
            if (n >> P) eq = gt = make_uint4(0, 0, 0, 0);  // n does not fit: more than the children
            stk4[sp * W4 + w4] = and4((in.flags & 1) ? eq : or4(gt, eq), valid4(w4, c));
         }
         ++sp;
      } else if (in.op == OP_JZ || in.op == OP_JFULL) {
         if (sp < 1) {
            bad = 2;
            break;
         }
         const uint4* x4 = stk4 + (sp - 1) * W4;
         int differs = 0;
#pragma unroll 1
         for (uint32_t w4 = threadIdx.x; w4 < W4; w4 += blockDim.x)
            differs |= ne4(x4[w4], in.op == OP_JZ ? make_uint4(0, 0, 0, 0) : valid4(w4, c));
         if (!__syncthreads_or(differs)) {
            next = in.a;
            if (in.a <= pc || in.a > ncode) {
               bad = 4;
               break;
            }
         }
      } else {
         bad = 5;
         break;
      }
      if (src != S_NONE) {
         DateLeaf d;
         if (src == S_DATE)
            d = date_leaf(c, &c.tab->date[in.col], static_cast<int32_t>(in.a), static_cast<int32_t>(in.b), in.flags);
#pragma unroll 1
         for (uint32_t w4 = threadIdx.x; w4 < W4; w4 += blockDim.x) {
            uint4 v = make_uint4(0, 0, 0, 0);
            if (src == S_TILE) {
               v = from[w4];
            } else if (src == S_SCRATCH) {
               v = X4[w4];
               X4[w4] = make_uint4(0, 0, 0, 0);
            } else if (src == S_SET) {
               v = __ldg(from + w4);
            } else if (src == S_DATE) {
               v = and4(date_word(d, w4), valid4(w4, c));
            } else if (src == S_FULL) {
               v = valid4(w4, c);
            }
            if (negate) v = andnot4(valid4(w4, c), v);
            put_word(T4, W4, P, f, w4, v);
         }
         if (src == S_SCRATCH) __syncwarp();  // the cleared words before the next leaf's rows
      }
      if (TRACE) {
         __shared__ uint32_t tred[FT / 32];
         __syncthreads();
         const long long t_end = clock64();
         uint32_t n = 0;
         if (sp >= 1) {
#pragma unroll 1
            for (uint32_t w4 = threadIdx.x; w4 < W4; w4 += blockDim.x) {
               const uint4 x = stk4[(sp - 1) * W4 + w4];
               n += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
            }
         }
         n = __reduce_add_sync(0xFFFFFFFFu, n);
         if ((threadIdx.x & 31) == 0) tred[threadIdx.x >> 5] = n;
         __syncthreads();
         if (threadIdx.x == 0) {
            uint32_t s = 0;
#pragma unroll 1
            for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) s += tred[w];
            const long long dt = t_end - t_start;
            trace[2 * pc] = static_cast<uint32_t>(dt < 1 ? 1 : (dt > 0xFFFFFFFFll ? 0xFFFFFFFFll : dt));
            trace[2 * pc + 1] = s;
         }
         __syncthreads();
      }
      pc = next;
   }
   if (!bad && sp != 1) bad = 2;
   if (bad && threadIdx.x == 0) atomicExch(err, bad);
   return !bad;
}

// One tile: runs the program, adds the result's population count to *count and copies it to dst
// (both optional). A tile without rows has an empty result.
template <bool TRACE>
__device__ __forceinline__ bool run_tile(const TileCtx& c, const Instr* __restrict__ code, uint32_t ncode, uint4* stk4,
                                         uint32_t cap, uint4* X4, const LeafCache& lc, uint32_t nl, uint32_t ncov,
                                         uint32_t* dst, unsigned long long* count, int* err, uint32_t* trace = nullptr) {
   if (c.nvalid && !run_program<TRACE>(c, code, ncode, stk4, cap, X4, lc, nl, ncov, err, trace)) return false;
   uint32_t pc = 0;
#pragma unroll 1
   for (uint32_t w4 = threadIdx.x; w4 < (c.W >> 7); w4 += blockDim.x) {
      const uint4 x = c.nvalid ? stk4[w4] : make_uint4(0, 0, 0, 0);
      pc += __popc(x.x) + __popc(x.y) + __popc(x.z) + __popc(x.w);
      if (dst) reinterpret_cast<uint4*>(dst)[w4] = x;
   }
   if (count) {
      pc = __reduce_add_sync(0xFFFFFFFFu, pc);
      if ((threadIdx.x & 31) == 0 && pc) atomicAdd(count, static_cast<unsigned long long>(pc));
   }
   return true;
}

// Dynamic shared memory of both kernels: the leaf cache, the scratch tile (of the widest tile), the stack tiles.
constexpr size_t LC_BYTES = sizeof(LeafCache);

// The CTA's part of a call's end (see CallEnd): the last CTA delivers the count and the error flag.
__device__ __forceinline__ void end_call(const CallEnd& end, unsigned long long* count, int* err) {
   __syncthreads();  // the count's additions of every warp
   if (threadIdx.x != 0) return;
   __threadfence();
   if (atomicAdd(end.ticket, 1u) != gridDim.x - 1) return;
   __threadfence();
   const unsigned long long total = atomicExch(end.acc, 0ull);
   *end.ticket = 0;  // for the next call
   *count = total;
   end.host->count = total;
   end.host->err = atomicAdd(err, 0);
}

// The program comes in the kernel's parameters (ic, at most INLINE_CODE instructions) or, with code, from
// global memory. With end.host the count goes through end.acc and the call's end is delivered.
template <bool TRACE>
__global__ void __launch_bounds__(FT) filter_kernel(const DevTable* __restrict__ tab, const Instr* gcode,
                                                    uint32_t ncode, uint32_t n_leaves, uint32_t tile_bits, uint32_t cap,
                                                    uint32_t* __restrict__ out_tiles, unsigned long long* count, int* err,
                                                    uint32_t* trace, const uint32_t* __restrict__ aux, const CallEnd end,
                                                    const __grid_constant__ InlineCode ic) {
   extern __shared__ __align__(16) uint8_t smem[];
   const Instr* code = gcode ? gcode : ic.code;
   LeafCache& lc = *reinterpret_cast<LeafCache*>(smem);
   const uint32_t T = CHUNK_ROWS / tile_bits;
   TileCtx c;
   c.tab = tab;
   c.v = blockIdx.x / T;
   c.W = tile_bits;
   c.row0 = (blockIdx.x % T) * tile_bits;
   c.aux = aux;
   const uint32_t csize = __ldg(tab->chunk_sizes + c.v);
   c.nvalid = csize > c.row0 ? min(tile_bits, csize - c.row0) : 0u;
   const uint32_t nl = min(n_leaves & 0xFFFFu, LC_LEAVES), ncov = min(n_leaves >> 16, LC_COV);
   uint4* X4 = reinterpret_cast<uint4*>(smem + LC_BYTES);
   uint4* stk4 = X4 + (tile_bits >> 7);
   if (c.nvalid) {
      init_leaves(lc);
      if (threadIdx.x == 0) lc.pay_used = lc.ext_used = 0;
#pragma unroll 1
      for (uint32_t w4 = threadIdx.x; w4 < (tile_bits >> 7); w4 += blockDim.x) X4[w4] = make_uint4(0, 0, 0, 0);
      __syncthreads();
      uint32_t phase = 0;
      if (!stage_leaves(lc, c, code, ncode, nl, ncov, nullptr, 0, phase, nullptr, err)) {
         if (end.host) end_call(end, count, err);
         return;
      }
   }
   uint32_t* dst = out_tiles ? out_tiles + static_cast<size_t>(c.v) * CHUNK_WORDS + (c.row0 >> 5) : nullptr;
   run_tile<TRACE>(c, code, ncode, stk4, cap, X4, lc, nl, ncov, dst, end.host ? end.acc : count, err,
                   TRACE ? trace + static_cast<size_t>(blockIdx.x) * ncode * 2 : nullptr);
   if (end.host) end_call(end, count, err);
}

// launch bounds: three CTAs per SM (at most 85 registers a thread; 64 for four cost 17%).
__global__ void __launch_bounds__(FT, 3) filter_batch_kernel(const DevTable* __restrict__ tab, const Instr* __restrict__ code,
                                                          const QueryDesc* __restrict__ queries,
                                                          const WorkItem* __restrict__ items, uint32_t n_items,
                                                          uint32_t scratch_bytes, uint32_t stack_bytes,
                                                          uint32_t* __restrict__ out_tiles, unsigned long long* counts,
                                                          uint32_t* next_item, int* err,
                                                          const uint32_t* __restrict__ aux) {
   extern __shared__ __align__(16) uint8_t smem[];
   LeafCache& lc = *reinterpret_cast<LeafCache*>(smem);
   const size_t per_query = static_cast<size_t>(tab->nchunks) * CHUNK_WORDS;
   uint4* X4 = reinterpret_cast<uint4*>(smem + LC_BYTES);
   uint8_t* stack = smem + LC_BYTES + scratch_bytes;
   init_leaves(lc);
#pragma unroll 1
   for (uint32_t i = threadIdx.x; i < scratch_bytes / 16; i += FT) X4[i] = make_uint4(0, 0, 0, 0);
   uint32_t phase = 0;
   if (threadIdx.x == 0) lc.next_item = atomicAdd(next_item, 1u);
#pragma unroll 1
   for (;;) {
      // this thread's earlier shared-memory accesses (stack tiles, staged payloads of the previous
      // item) are ordered before the bulk copies into the same memory issued after the barrier
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      if (threadIdx.x == 0) lc.pay_used = lc.ext_used = 0;
      __syncthreads();
      const uint32_t it = lc.next_item;
      if (it >= n_items) return;
      const WorkItem wi = items[it];
      const QueryDesc q = queries[wi.query];
      const uint32_t tile_bits = q.tile_bits, T = CHUNK_ROWS / tile_bits;
      // the program uses q.depth - 1 stack tiles; the CTA's other tiles take this item's payloads
      const uint32_t cap = stack_bytes / (tile_bits >> 3);
      const uint32_t tiles = min(max(q.depth, 2u) - 1u, cap);
      uint16_t* ext = reinterpret_cast<uint16_t*>(stack + static_cast<size_t>(tiles) * (tile_bits >> 3));
      const uint32_t ext_cap = (cap - tiles) * (tile_bits / 16);
      const uint32_t nl = min(q.n_leaves & 0xFFFFu, LC_LEAVES), ncov = min(q.n_leaves >> 16, LC_COV);
      TileCtx c;
      c.tab = tab;
      c.v = wi.tile / T;
      c.W = tile_bits;
      c.row0 = (wi.tile % T) * tile_bits;
      c.aux = aux ? aux + static_cast<size_t>(q.aux_base) * per_query : nullptr;
      const uint32_t csize = __ldg(tab->chunk_sizes + c.v);
      c.nvalid = csize > c.row0 ? min(tile_bits, csize - c.row0) : 0u;
      const Instr* prog = code + q.code_off;
      if (c.nvalid) {
         if (!stage_leaves(lc, c, prog, q.code_len, nl, ncov, ext, ext_cap, phase, next_item, err)) return;
      } else {
         __syncthreads();  // every thread has read lc.next_item
         if (threadIdx.x == 0) lc.next_item = atomicAdd(next_item, 1u);
      }
      uint32_t* dst = q.out_tiles ? out_tiles + static_cast<size_t>(q.out_tiles - 1) * per_query +
                                       static_cast<size_t>(c.v) * CHUNK_WORDS + (c.row0 >> 5)
                                  : nullptr;
      unsigned long long* count = counts + wi.query;
      uint4* stk4 = reinterpret_cast<uint4*>(stack);
      // the stack may not grow past the program's tiles into the staged payloads
      const bool ok = run_tile<false>(c, prog, q.code_len, stk4, tiles, X4, lc, nl, ncov, dst, count, err);
      if (!ok) return;
   }
}

// Planes of a date column: one warp per word of 32 rows, a ballot per plane.
__global__ void __launch_bounds__(256) date_index_kernel(const int32_t* __restrict__ days, uint32_t n, uint32_t words,
                                                         const DevDateCol col, uint32_t* planes, uint32_t* nulls) {
   const uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
   if (w >= words) return;  // the whole warp leaves
   const uint32_t g = 32 * w + lane;
   const int32_t day = g < n ? days[g] : INT32_MIN;
   const bool has = day != INT32_MIN;
   const uint32_t x = has ? static_cast<uint32_t>(day - col.base) : 0u, m = (1u << col.width) - 1u;
#pragma unroll 1
   for (uint32_t k = 0; k <= col.last; ++k) {
      const uint32_t digit = (x >> (col.width * (k >> col.width))) & m;
      const uint32_t b = __ballot_sync(0xFFFFFFFFu, has && digit <= (k & m));
      if (lane == 0) planes[static_cast<size_t>(k) * words + w] = b;
   }
   const uint32_t b = __ballot_sync(0xFFFFFFFFu, g < n && !has);
   if (lane == 0) nulls[w] = b;
}

// Dense forms of the filter path: one CTA per array of at least DENSE_MIN rows, or run container of as many in
// more than SPAN_RUNS runs, writes its bitset.
__global__ void __launch_bounds__(256) dense_forms_kernel(uint16_t* arena, const DenseJob* __restrict__ jobs) {
   __shared__ uint4 tile[CHUNK_WORDS / 4];
   const DenseJob j = jobs[blockIdx.x];
#pragma unroll 1
   for (uint32_t i = threadIdx.x; i < CHUNK_WORDS / 4; i += blockDim.x) tile[i] = make_uint4(0, 0, 0, 0);
   __syncthreads();
   uint32_t* t = reinterpret_cast<uint32_t*>(tile);
#pragma unroll 1
   for (uint32_t i = threadIdx.x; i < j.rows; i += blockDim.x) {
      const uint32_t r = arena[j.src + i];
      atomicOr(&t[r >> 5], 1u << (r & 31));
   }
   for (uint32_t i = threadIdx.x; i < j.runs; i += blockDim.x) {
      const uint32_t s = arena[j.src + 2 * i], e = s + arena[j.src + 2 * i + 1];  // [s, e]
      for (uint32_t w = s >> 5; w <= e >> 5; ++w)
         atomicOr(&t[w], (w == s >> 5 ? 0xFFFFFFFFu << (s & 31) : 0xFFFFFFFFu) & (w == e >> 5 ? 0xFFFFFFFFu >> (31 - (e & 31)) : 0xFFFFFFFFu));
   }
   __syncthreads();
   uint4* dst = reinterpret_cast<uint4*>(arena + j.dst);
#pragma unroll 1
   for (uint32_t i = threadIdx.x; i < CHUNK_WORDS / 4; i += blockDim.x) dst[i] = tile[i];
}
}  // namespace

// ------------------------------------------------------------------------------------------------
// launchers

static_assert(LC_BYTES + CHUNK_ROWS / 8 + TILES_BYTES <= 227 * 1024, "shared memory of a CTA");
void filter_setup() {
   const auto allow = [](const void* kernel, size_t bytes) {
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes));
      if (e != cudaSuccess) throw std::runtime_error(std::string("shared memory of the filter kernels: ") + cudaGetErrorString(e));
   };
   allow(reinterpret_cast<const void*>(filter_kernel<false>), LC_BYTES + TILES_BYTES);
   allow(reinterpret_cast<const void*>(filter_kernel<true>), LC_BYTES + TILES_BYTES);
   allow(reinterpret_cast<const void*>(filter_batch_kernel), LC_BYTES + CHUNK_ROWS / 8 + TILES_BYTES);
}

cudaError_t launch_filter(const DevTable* d_table, uint32_t nchunks, const Instr* d_code, uint32_t ncode,
                          uint32_t n_leaves, uint32_t tile_bits, uint32_t stack_tiles, uint32_t* d_out_tiles, unsigned long long* d_count,
                          int* d_err, void* stream, uint32_t* d_trace, const uint32_t* d_aux, const CallEnd& end,
                          const Instr* inline_code) {
   InlineCode ic;
   if (inline_code) {
      if (ncode > INLINE_CODE) return cudaErrorInvalidValue;
      std::memcpy(ic.code, inline_code, ncode * sizeof(Instr));
   }
   const uint32_t grid = nchunks * (CHUNK_ROWS / tile_bits);
   const uint32_t threads = std::max(32u, std::min(FT, tile_bits / 128));
   const size_t smem = LC_BYTES + static_cast<size_t>(std::max(stack_tiles, 1u)) * (tile_bits / 8);
   const auto kernel = d_trace ? filter_kernel<true> : filter_kernel<false>;
   kernel<<<grid, threads, smem, static_cast<cudaStream_t>(stream)>>>(d_table, inline_code ? nullptr : d_code, ncode, n_leaves, tile_bits,
                                                                      stack_tiles - 1, d_out_tiles, d_count, d_err, d_trace,
                                                                      d_aux, end, ic);
   return cudaGetLastError();
}

int filter_batch_blocks_per_sm(size_t scratch_bytes, size_t stack_bytes) {
   const size_t smem = LC_BYTES + scratch_bytes + stack_bytes;
   int n = 0;
   if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, filter_batch_kernel, FT, smem) != cudaSuccess) {
      cudaGetLastError();
      return 1;
   }
   return n > 0 ? n : 1;
}

cudaError_t launch_filter_batch(const DevTable* d_table, const Instr* d_code, const QueryDesc* d_queries,
                         const WorkItem* d_items, uint32_t n_items, uint32_t scratch_bytes, uint32_t stack_bytes,
                         uint32_t* d_out_tiles, unsigned long long* d_counts, uint32_t* d_next, uint32_t grid, int* d_err,
                         void* stream, const uint32_t* d_aux) {
   const size_t smem = LC_BYTES + scratch_bytes + stack_bytes;
   filter_batch_kernel<<<grid, FT, smem, static_cast<cudaStream_t>(stream)>>>(
      d_table, d_code, d_queries, d_items, n_items, scratch_bytes, stack_bytes, d_out_tiles, d_counts, d_next, d_err, d_aux);
   return cudaGetLastError();
}

cudaError_t launch_date_index(const int32_t* d_days, uint32_t n, uint32_t words, const DevDateCol& col, void* stream) {
   date_index_kernel<<<(words + 7) / 8, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      d_days, n, words, col, const_cast<uint32_t*>(col.planes), const_cast<uint32_t*>(col.nulls));
   return cudaGetLastError();
}

cudaError_t launch_dense_forms(uint16_t* d_arena, const DenseJob* d_jobs, uint32_t n, void* stream) {
   if (n == 0) return cudaSuccess;
   dense_forms_kernel<<<n, 256, 0, static_cast<cudaStream_t>(stream)>>>(d_arena, d_jobs);
   return cudaGetLastError();
}

void set_copy_withholding(bool on) {
   const uint32_t v = on ? 1u : 0u;
   const cudaError_t e = cudaMemcpyToSymbol(g_withhold_leaf_copies, &v, sizeof(v));
   if (e != cudaSuccess) throw std::runtime_error(std::string("set_copy_withholding: ") + cudaGetErrorString(e));
}

}  // namespace rhygpu
