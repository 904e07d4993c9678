// The planner's network on the GPU: 24 -> 64 -> 64 -> 2 with ReLU, BF16 weights, FP32 arithmetic.
//
//   mlp_forward_kernel   one thread per sample; the BF16 weights are widened once per CTA into
//                        shared memory; the second hidden layer is folded into the output as it
//                        is produced, so only the first hidden layer lives in registers. Bound by
//                        the chains of dependent additions (30,000 samples put two warps on an SM's
//                        scheduler), so four units of the second layer go at a time, each in the
//                        order of its inputs. The planner's form takes raw features and returns
//                        selectivity and cost.
//   mlp_grad_kernel      forward + backward of the mean squared error for 128 samples per CTA, the
//                        hidden layers' products on the tensor cores (tcgen05.mma, accumulators in
//                        tensor memory), FP32 operands entering as split BF16 parts.
//   mlp_adam_kernel      Adam on the FP32 master weights; writes the BF16 copy the other kernels use.
// The gradient is taken with respect to the BF16 weights the forward pass used and applied to the
// master weights.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>

#include "mlp.h"

namespace rhygpu {

namespace {

constexpr uint32_t FWD_T = 128;

__device__ __forceinline__ void load_weights(const __nv_bfloat16* __restrict__ w, float* sw) {
   for (uint32_t i = threadIdx.x; i < MLP_NPARAM; i += blockDim.x) sw[i] = __bfloat162float(w[i]);
   __syncthreads();
}

template <bool PLAN>
__global__ void __launch_bounds__(FWD_T) mlp_forward_kernel(const __nv_bfloat16* __restrict__ w,
                                                            const float* __restrict__ X, uint32_t n,
                                                            float* __restrict__ Y, const MlpScale scale,
                                                            double* __restrict__ sel, double* __restrict__ cost) {
   extern __shared__ float sw[];
   load_weights(w, sw);
   const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
   if (s >= n) return;
   const float* W1 = sw + MLP_W1;
   const float* B1 = sw + MLP_B1;
   const float* W2 = sw + MLP_W2;
   const float* B2 = sw + MLP_B2;
   const float* W3 = sw + MLP_W3;
   const float* B3 = sw + MLP_B3;
   float x[MLP_IN];
#pragma unroll
   for (uint32_t i = 0; i < MLP_IN; ++i) x[i] = X[static_cast<size_t>(s) * MLP_IN + i];
   const float x0 = x[0], x1 = x[1], x8 = x[8];
   if (PLAN) {
#pragma unroll
      for (uint32_t i = 0; i < MLP_IN; ++i) x[i] = __fdiv_rn(__fsub_rn(x[i], scale.mean[i]), scale.std[i]);
   }
   float h1[MLP_H];
#pragma unroll
   for (uint32_t j = 0; j < MLP_H; ++j) {
      float a = B1[j];
#pragma unroll
      for (uint32_t i = 0; i < MLP_IN; ++i) a = fmaf(W1[j * MLP_IN + i], x[i], a);
      h1[j] = fmaxf(a, 0.0f);
   }
   float y0 = B3[0], y1 = B3[1];
   constexpr uint32_t U = 4;
#pragma unroll 1
   for (uint32_t j = 0; j < MLP_H; j += U) {
      float a[U];
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) a[u] = B2[j + u];
#pragma unroll
      for (uint32_t i = 0; i < MLP_H; ++i) {
#pragma unroll
         for (uint32_t u = 0; u < U; ++u) a[u] = fmaf(W2[(j + u) * MLP_H + i], h1[i], a[u]);
      }
#pragma unroll
      for (uint32_t u = 0; u < U; ++u) {
         const float h = fmaxf(a[u], 0.0f);
         y0 = fmaf(W3[j + u], h, y0);
         y1 = fmaf(W3[MLP_H + j + u], h, y1);
      }
   }
   if (PLAN) {
      const double rule = static_cast<double>(x8) * -scale.min_log_sel;
      const double ls = x0 > 0.5f || x1 > 0.5f ? rule : rule + static_cast<double>(y0) * scale.tstd[0] + scale.tmean[0];
      const double m = ls < 0.0 ? ls : 0.0;  // also for a NaN
      sel[s] = exp(scale.min_log_sel < m ? m : scale.min_log_sel);
      cost[s] = exp(static_cast<double>(y1) * scale.tstd[1] + scale.tmean[1]);
   } else {
      Y[2 * static_cast<size_t>(s)] = y0;
      Y[2 * static_cast<size_t>(s) + 1] = y1;
   }
}

// ---- gradient on the tensor cores ----
//
// One CTA of 512 threads per 128 samples (the MMA's M): sample r is row r of every accumulator in tensor
// memory (TMEM lane r), and its four threads take 16 of the 64 units each (a warp reads the 32 TMEM lanes of
// its index modulo 4). The kernel is bound by the latency of its phases, one CTA per SM: with one thread per
// sample, 2-byte stores of every operand element and one atomic per gradient element and thread a CTA took
// 60 us, so operand rows are stored 16 bytes at a time, the partial gradients are put in order in shared
// memory and added 16 bytes at a time, and the sums over a warp's samples are taken for 32 values at once
// (30,011 samples: 128 -> 25 us). The products run as tcgen05.mma (kind::f16,
// BF16 operands, FP32 accumulation) issued by one thread, operands in shared memory in the
// no-swizzle K-major layout (8 x 16-byte core matrices), accumulators in TMEM:
//   phase 0  Z1 = X W1^T                     (M 128, N 64, K 32: the 24 features and zeros)
//   phase 1  Z2 = H1 W2^T                    (N 64, K 64)
//   phase 2  G1 = D2 W2                      (N 64, K 64)
//            [D2_hi^T; D2_lo^T] [H1^T; 1]^T  (N 80, K 128 samples): dW2 and, from the ones row, db2
//   phase 3  [D1_hi^T; D1_lo^T] [X^T; 1]^T   (N 32, K 128 samples): dW1 and db1
// The network keeps FP32 arithmetic: an FP32 operand v enters as two BF16 parts, hi = bf16(v) and
// lo = bf16(v - hi), and the products add the parts' MMAs (the weights are BF16 already, so a
// forward product takes two MMAs; a weight gradient takes all four combinations, the lo rows of
// its A operand giving the second half of the accumulator rows, which are added when the
// gradient is written out). That leaves a relative error near 2^-16 per product. The output layer,
// dW3 and db3 (two outputs) stay on the CUDA cores with warp reductions.
constexpr uint32_t TC_S = 128, TC_T = 512;
// byte offset of element (r, k) in a K-major operand of kc 16-byte chunks along K
__device__ __forceinline__ uint32_t cm_off(uint32_t r, uint32_t k, uint32_t kc) {
   return ((((r >> 3) * kc) + (k >> 3)) << 7) + ((r & 7) << 4) + ((k & 7) << 1);
}
// shared memory of the gradient kernel (bytes)
constexpr uint32_t SO_XA_HI = 0;           // X [128 x 32], hi / lo
constexpr uint32_t SO_XA_LO = 8192;
constexpr uint32_t SO_XB_HI = 16384;       // [X^T; 1; 0] [32 x 128], hi / lo
constexpr uint32_t SO_XB_LO = 24576;
constexpr uint32_t SO_W1 = 32768;          // W1 [64 x 32]
constexpr uint32_t SO_W2 = 36864;          // W2 [64 x 64]
constexpr uint32_t SO_W2T = 45056;         // W2^T [64 x 64]
constexpr uint32_t SO_A_HI = 53248;        // H1 [128 x 64] hi / lo; then D2 hi / lo; then [D1_hi^T; D1_lo^T]
constexpr uint32_t SO_A_LO = 69632;
constexpr uint32_t SO_H1B_HI = 86016;      // [H1^T; 1; 0] [80 x 128], hi / lo
constexpr uint32_t SO_H1B_LO = 106496;
constexpr uint32_t SO_D2T = 126976;        // [D2_hi^T; D2_lo^T] [128 x 128]
constexpr uint32_t SO_F32 = 159744;        // W3 (128), b1 (64), b2 (64), b3 (2) as floats
constexpr uint32_t SO_Y = SO_F32 + 1040;       // the output layer's partial sums (4 quarters x 128 samples x 2 floats)
constexpr uint32_t SO_BAR = SO_Y + 4096;
constexpr uint32_t SO_TMEM = SO_BAR + 8;
constexpr uint32_t SO_END = SO_TMEM + 8;
// over dead operands: accumulator rows on their way to the gradient, in padded rows of floats
constexpr uint32_t GR2 = 68;               // [dW2 | db2] (128 x 65) over H1B, read until phase 2
constexpr uint32_t GR1 = 28;               // [dW1 | db1] (128 x 25) over XA and XB, read until phase 3
static_assert(128 * GR2 * 4 <= SO_D2T - SO_H1B_HI && 128 * GR1 * 4 <= SO_W1, "gradient rows fit the operands they replace");
static_assert(MLP_W1 % 8 == 0 && MLP_W2 % 8 == 0 && MLP_IN % 8 == 0, "weight rows load 16 bytes at a time");
// TMEM columns of the accumulators
constexpr uint32_t TM_Z1 = 0, TM_Z2 = 64, TM_G1 = 128, TM_DW2 = 192, TM_DW1 = 272, TM_COLS = 512;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// shared-memory matrix descriptor: no swizzle, start address, leading byte offset (next 16-byte
// chunk along K), stride byte offset (next 8-row group), descriptor version 1 (bits 46-47)
__device__ __forceinline__ uint64_t mma_sdesc(uint32_t addr, uint32_t sbo) {
   return static_cast<uint64_t>((addr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(128u >> 4) << 16) |
          (static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M = 128
__host__ __device__ constexpr uint32_t mma_idesc(uint32_t n) {
   return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((128u >> 4) << 24);
}
// D[tmem] (+)= A B^T over K = 16 * ksteps: A [128 x K] and B [N x K] K-major with kc chunks along K
__device__ __forceinline__ void mma_k(uint32_t d, uint32_t a, uint32_t b, uint32_t kc, uint32_t ksteps,
                                      uint32_t idesc, bool accumulate) {
   for (uint32_t k = 0; k < ksteps; ++k) {
      const uint64_t ad = mma_sdesc(a + 256 * k, kc * 128), bd = mma_sdesc(b + 256 * k, kc * 128);
      const uint32_t acc = (accumulate || k > 0) ? 1u : 0u;
      asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
                   "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                   : "memory");
   }
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
   asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// operands written by the threads become visible to the tensor cores; then one thread issues
__device__ __forceinline__ void operands_ready() {
   asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   __syncthreads();
   asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// waits (bounded by limit_ns on the global timer) for the MMAs committed as phase `parity`; the whole CTA
// agrees on the outcome
__device__ __forceinline__ bool mma_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns) {
   const uint32_t b = smem_u32(bar);
   uint64_t t0 = 0;
   bool done = false;
   for (uint32_t i = 0; i < (1u << 24) && !done; ++i) {
      uint32_t d;
      asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
                   : "=r"(d)
                   : "r"(b), "r"(parity), "r"(1000u)
                   : "memory");
      done = d != 0;
      if (!done) {
         uint64_t now;
         asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
         if (t0 == 0) t0 = now;
         else if (now - t0 > limit_ns) break;
      }
   }
   done = __syncthreads_and(done) != 0;
   asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
   return done;
}
// 16 consecutive FP32 accumulator columns of this thread's row (its warp's 32 TMEM lanes)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
   uint32_t r[16];
   asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                  "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                : "r"(taddr));
   asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
   for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}
__device__ __forceinline__ void put_bf16(uint8_t* base, uint32_t off, __nv_bfloat16 v) {
   *reinterpret_cast<__nv_bfloat16*>(base + off) = v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
   for (uint32_t o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
   return v;
}
// The warp's sums of 32 values: lane l returns the sum of v[l] (31 shuffles; 160 one value at a time).
__device__ __forceinline__ float warp_sums32(float (&v)[32], uint32_t lane) {
#pragma unroll
   for (uint32_t m = 16; m > 0; m >>= 1) {
      const bool up = lane & m;
#pragma unroll
      for (uint32_t i = 0; i < m; ++i) {
         const float keep = up ? v[i + m] : v[i], send = up ? v[i] : v[i + m];
         v[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, m);
      }
   }
   return v[0];
}
// Eight values as BF16 parts: hi = bf16(v), lo = bf16(v - hi), each 16 bytes.
struct Split8 {
   __align__(16) __nv_bfloat16 hi[8], lo[8];
};
__device__ __forceinline__ Split8 split8(const float* v) {
   Split8 p;
#pragma unroll
   for (uint32_t i = 0; i < 8; ++i) {
      p.hi[i] = __float2bfloat16_rn(v[i]);
      p.lo[i] = __float2bfloat16_rn(v[i] - __bfloat162float(p.hi[i]));
   }
   return p;
}
__device__ __forceinline__ void put8(uint8_t* base, uint32_t off, const __nv_bfloat16 (&v)[8]) {
   *reinterpret_cast<uint4*>(base + off) = *reinterpret_cast<const uint4*>(v);
}

__global__ void __launch_bounds__(TC_T, 1) mlp_grad_kernel(const __nv_bfloat16* __restrict__ w,
                                                           const float* __restrict__ X, const float* __restrict__ T,
                                                           uint32_t n, float inv_total, float* __restrict__ grad,
                                                           float* __restrict__ loss, int* err, bool withhold) {
   extern __shared__ __align__(1024) uint8_t sm[];
   const uint32_t t = threadIdx.x, warp = t >> 5, lane = t & 31;
   const uint32_t r = t & (TC_S - 1), q = t / TC_S, u0 = 16 * q;  // sample row, quarter, its first unit
   const uint32_t s = blockIdx.x * TC_S + r;
   const bool live = s < n;
   uint64_t* bar = reinterpret_cast<uint64_t*>(sm + SO_BAR);
   uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + SO_TMEM);
   float* W3f = reinterpret_cast<float*>(sm + SO_F32);
   float* b1f = W3f + 2 * MLP_H;
   float* b2f = b1f + MLP_H;
   float* b3f = b2f + MLP_H;
   float2* ypart = reinterpret_cast<float2*>(sm + SO_Y);
   if (t == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)));
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
   }
   if (warp == 0) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                   "r"(TM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
   }
   const __nv_bfloat16 zero = __float2bfloat16_rn(0.0f), one = __float2bfloat16_rn(1.0f);
   // weights: W1 [64 x 32] (zeros past the 24 inputs), W2 and W2^T [64 x 64]; the rest as floats
   if (t < MLP_H * 4) {
      const uint32_t j = t / 4, k = 8 * (t % 4);
      uint4 v = make_uint4(0, 0, 0, 0);
      if (k < MLP_IN) v = *reinterpret_cast<const uint4*>(w + MLP_W1 + j * MLP_IN + k);
      *reinterpret_cast<uint4*>(sm + SO_W1 + cm_off(j, k, 4)) = v;
   }
   {
      const uint32_t j = t / 8, k = 8 * (t % 8);
      Split8 v;
      *reinterpret_cast<uint4*>(v.hi) = *reinterpret_cast<const uint4*>(w + MLP_W2 + j * MLP_H + k);
      put8(sm + SO_W2, cm_off(j, k, 8), v.hi);
#pragma unroll
      for (uint32_t i = 0; i < 8; ++i) put_bf16(sm + SO_W2T, cm_off(k + i, j, 8), v.hi[i]);
   }
   if (t < 2 * MLP_H) W3f[t] = __bfloat162float(w[MLP_W3 + t]);
   else if (t < 3 * MLP_H) b1f[t - 2 * MLP_H] = __bfloat162float(w[MLP_B1 + t - 2 * MLP_H]);
   else if (t < 4 * MLP_H) b2f[t - 3 * MLP_H] = __bfloat162float(w[MLP_B2 + t - 3 * MLP_H]);
   else if (t < 4 * MLP_H + MLP_OUT) b3f[t - 4 * MLP_H] = __bfloat162float(w[MLP_B3 + t - 4 * MLP_H]);
   float t0 = 0.0f, t1 = 0.0f;
   if (live) {
      t0 = T[static_cast<size_t>(s) * MLP_OUT];
      t1 = T[static_cast<size_t>(s) * MLP_OUT + 1];
   }
   {  // eight of the sample's features: row r of X (hi, lo) and column r of [X^T; 1; 0]
      const uint32_t k0 = 8 * q;
      float v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (live && k0 < MLP_IN) {
         const float4* src = reinterpret_cast<const float4*>(X + static_cast<size_t>(s) * MLP_IN + k0);
         const float4 a = src[0], b = src[1];
         v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
      }
      const Split8 p = split8(v);
      put8(sm + SO_XA_HI, cm_off(r, k0, 4), p.hi);
      put8(sm + SO_XA_LO, cm_off(r, k0, 4), p.lo);
#pragma unroll
      for (uint32_t i = 0; i < 8; ++i) {
         put_bf16(sm + SO_XB_HI, cm_off(k0 + i, r, 16), k0 + i == MLP_IN ? one : p.hi[i]);
         put_bf16(sm + SO_XB_LO, cm_off(k0 + i, r, 16), p.lo[i]);
      }
   }
   operands_ready();
   const uint32_t tmem = *tmem_slot;
   const uint32_t base = smem_u32(sm);
   const uint32_t lane_addr = tmem + ((32u * (warp & 3)) << 16);
   bool ok = true;
   uint32_t committed = 0;  // MMA phases committed to the barrier (the same in every thread)
   const uint64_t limit = withhold ? 1000000ull : 2000000000ull;
   // ---- phase 0: Z1 = X W1^T
   if (t == 0 && !withhold) {
      mma_k(tmem + TM_Z1, base + SO_XA_HI, base + SO_W1, 4, 2, mma_idesc(64), false);
      mma_k(tmem + TM_Z1, base + SO_XA_LO, base + SO_W1, 4, 2, mma_idesc(64), true);
      mma_commit(bar);
   }
   ++committed;
   ok = mma_wait(bar, 0, limit);
   uint32_t mask1 = 0, mask2 = 0;  // the quarter's units with a positive input
   if (ok) {
      // h1 = relu(z1 + b1): row r of H1 (hi, lo) and column r of [H1^T; 1; 0]
      float z[16];
      tmem_ld16(lane_addr + TM_Z1 + u0, z);
#pragma unroll
      for (uint32_t j = 0; j < 16; ++j) {
         const float a = z[j] + b1f[u0 + j];
         if (a > 0.0f) mask1 |= 1u << j;
         z[j] = fmaxf(a, 0.0f);
      }
#pragma unroll
      for (uint32_t c = 0; c < 16; c += 8) {
         const Split8 p = split8(z + c);
         put8(sm + SO_A_HI, cm_off(r, u0 + c, 8), p.hi);
         put8(sm + SO_A_LO, cm_off(r, u0 + c, 8), p.lo);
#pragma unroll
         for (uint32_t i = 0; i < 8; ++i) {
            put_bf16(sm + SO_H1B_HI, cm_off(u0 + c + i, r, 16), p.hi[i]);
            put_bf16(sm + SO_H1B_LO, cm_off(u0 + c + i, r, 16), p.lo[i]);
         }
      }
#pragma unroll
      for (uint32_t i = 0; i < 4; ++i) {
         const uint32_t u = MLP_H + 4 * q + i;
         put_bf16(sm + SO_H1B_HI, cm_off(u, r, 16), u == MLP_H ? one : zero);
         put_bf16(sm + SO_H1B_LO, cm_off(u, r, 16), zero);
      }
   }
   operands_ready();
   // ---- phase 1: Z2 = H1 W2^T
   if (ok && t == 0) {
      mma_k(tmem + TM_Z2, base + SO_A_HI, base + SO_W2, 8, 4, mma_idesc(64), false);
      mma_k(tmem + TM_Z2, base + SO_A_LO, base + SO_W2, 8, 4, mma_idesc(64), true);
      mma_commit(bar);
   }
   if (ok) {
      ++committed;
      ok = mma_wait(bar, 1, limit);
   }
   float h[16];
   if (ok) {  // the quarter's part of the output layer
      tmem_ld16(lane_addr + TM_Z2 + u0, h);
      float y0 = 0.0f, y1 = 0.0f;
#pragma unroll
      for (uint32_t j = 0; j < 16; ++j) {
         const float a = h[j] + b2f[u0 + j];
         if (a > 0.0f) mask2 |= 1u << j;
         h[j] = fmaxf(a, 0.0f);
         y0 = fmaf(W3f[u0 + j], h[j], y0);
         y1 = fmaf(W3f[MLP_H + u0 + j], h[j], y1);
      }
      ypart[q * TC_S + r] = make_float2(y0, y1);
   }
   __syncthreads();
   if (ok) {
      float y0 = b3f[0], y1 = b3f[1];
#pragma unroll
      for (uint32_t k = 0; k < 4; ++k) {
         const float2 y = ypart[k * TC_S + r];
         y0 += y.x;
         y1 += y.y;
      }
      const float r0 = live ? y0 - t0 : 0.0f, r1 = live ? y1 - t1 : 0.0f;
      const float d30 = 2.0f * r0 * inv_total, d31 = 2.0f * r1 * inv_total;
      if (q == 0) {
         const float e2 = warp_sum(fmaf(r0, r0, r1 * r1));
         const float g30 = warp_sum(d30), g31 = warp_sum(d31);
         if (lane == 0) {
            atomicAdd(loss, e2 * inv_total);
            atomicAdd(grad + MLP_B3, g30);
            atomicAdd(grad + MLP_B3 + 1, g31);
         }
      }
      // delta2 = (W3^T d3) * relu'(z2): row r of D2 (hi, lo), column r of [D2_hi^T; D2_lo^T]
#pragma unroll
      for (uint32_t c = 0; c < 16; c += 8) {
         float d2[8];
#pragma unroll
         for (uint32_t i = 0; i < 8; ++i) {
            const uint32_t u = u0 + c + i;
            d2[i] = (mask2 >> (c + i)) & 1u ? fmaf(W3f[u], d30, W3f[MLP_H + u] * d31) : 0.0f;
         }
         const Split8 p = split8(d2);
         put8(sm + SO_A_HI, cm_off(r, u0 + c, 8), p.hi);
         put8(sm + SO_A_LO, cm_off(r, u0 + c, 8), p.lo);
#pragma unroll
         for (uint32_t i = 0; i < 8; ++i) {
            put_bf16(sm + SO_D2T, cm_off(u0 + c + i, r, 16), p.hi[i]);
            put_bf16(sm + SO_D2T, cm_off(MLP_H + u0 + c + i, r, 16), p.lo[i]);
         }
      }
      // dW3 = sum over the samples of d3 h2^T: the warp's sums, output lane >> 4, unit u0 + (lane & 15)
      float v[32];
#pragma unroll
      for (uint32_t j = 0; j < 16; ++j) {
         v[j] = d30 * h[j];
         v[16 + j] = d31 * h[j];
      }
      const float g = warp_sums32(v, lane);
      atomicAdd(grad + MLP_W3 + (lane >> 4) * MLP_H + u0 + (lane & 15), g);
   }
   operands_ready();
   // ---- phase 2: G1 = D2 W2; [D2_hi^T; D2_lo^T] [H1^T; 1]^T
   if (ok && t == 0) {
      mma_k(tmem + TM_G1, base + SO_A_HI, base + SO_W2T, 8, 4, mma_idesc(64), false);
      mma_k(tmem + TM_G1, base + SO_A_LO, base + SO_W2T, 8, 4, mma_idesc(64), true);
      mma_k(tmem + TM_DW2, base + SO_D2T, base + SO_H1B_HI, 16, 8, mma_idesc(80), false);
      mma_k(tmem + TM_DW2, base + SO_D2T, base + SO_H1B_LO, 16, 8, mma_idesc(80), true);
      mma_commit(bar);
   }
   if (ok) {
      ++committed;
      ok = mma_wait(bar, 0, limit);
   }
   float* g2 = reinterpret_cast<float*>(sm + SO_H1B_HI);
   if (ok) {
      // delta1 = G1 * relu'(z1) into column r of [D1_hi^T; D1_lo^T] (over D2, which phase 2 has read)
      float g[16];
      tmem_ld16(lane_addr + TM_G1 + u0, g);
#pragma unroll
      for (uint32_t j = 0; j < 16; ++j) g[j] = (mask1 >> j) & 1u ? g[j] : 0.0f;
#pragma unroll
      for (uint32_t c = 0; c < 16; c += 8) {
         const Split8 p = split8(g + c);
#pragma unroll
         for (uint32_t i = 0; i < 8; ++i) {
            put_bf16(sm + SO_A_HI, cm_off(u0 + c + i, r, 16), p.hi[i]);
            put_bf16(sm + SO_A_HI, cm_off(MLP_H + u0 + c + i, r, 16), p.lo[i]);
         }
      }
      // dW2 and db2: accumulator row r holds unit r & 63 (hi part for r < 64, lo part above)
      float v[16];
      tmem_ld16(lane_addr + TM_DW2 + u0, v);
#pragma unroll
      for (uint32_t j = 0; j < 16; j += 4)
         *reinterpret_cast<float4*>(g2 + r * GR2 + u0 + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      if (q == 0) {
         tmem_ld16(lane_addr + TM_DW2 + MLP_H, v);
         g2[r * GR2 + MLP_H] = v[0];
      }
   }
   operands_ready();
   // ---- phase 3: [D1_hi^T; D1_lo^T] [X^T; 1]^T
   if (ok && t == 0) {
      mma_k(tmem + TM_DW1, base + SO_A_HI, base + SO_XB_HI, 16, 8, mma_idesc(32), false);
      mma_k(tmem + TM_DW1, base + SO_A_HI, base + SO_XB_LO, 16, 8, mma_idesc(32), true);
      mma_commit(bar);
   }
   // row j of the weights' gradient from accumulator rows j (hi) and 64 + j (lo), four elements a thread
   auto add_rows = [&](const float* rows, uint32_t stride, uint32_t width, float* to, float* bias) {
      for (uint32_t i = t; i < MLP_H * (width / 4); i += TC_T) {
         const uint32_t j = i / (width / 4), k = 4 * (i % (width / 4));
         const float4 a = *reinterpret_cast<const float4*>(rows + j * stride + k);
         const float4 b = *reinterpret_cast<const float4*>(rows + (MLP_H + j) * stride + k);
         atomicAdd(reinterpret_cast<float4*>(to + j * width + k), make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w));
      }
      if (t < MLP_H) atomicAdd(bias + t, rows[t * stride + width] + rows[(MLP_H + t) * stride + width]);
   };
   if (ok) {
      add_rows(g2, GR2, MLP_H, grad + MLP_W2, grad + MLP_B2);
      ++committed;
      ok = mma_wait(bar, 1, limit);
   }
   if (ok) {
      float* g1 = reinterpret_cast<float*>(sm);
      if (q < 2) {
         float v[16];
         tmem_ld16(lane_addr + TM_DW1 + u0, v);
#pragma unroll
         for (uint32_t j = 0; j < 16; j += 4)
            if (u0 + j < GR1)
               *reinterpret_cast<float4*>(g1 + r * GR1 + u0 + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
      }
      __syncthreads();  // ok is the CTA's
      add_rows(g1, GR1, MLP_IN, grad + MLP_W1, grad + MLP_B1);
   } else if (t == 0) {
      atomicExch(err, 1);
   }
   // a wait that gave up leaves MMAs possibly in flight: wait for the phase it gave up on (bounded)
   // before the tensor memory is freed
   if (!ok) mma_wait(bar, (committed - 1) & 1u, limit);
   asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
   __syncthreads();
   if (warp == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TM_COLS) : "memory");
   }
}

__global__ void mlp_adam_kernel(float* __restrict__ master, __nv_bfloat16* __restrict__ w, float* __restrict__ grad,
                                float* __restrict__ m, float* __restrict__ v, float lr, float beta1, float beta2,
                                float eps, float c1, float c2) {
   const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
   if (p >= MLP_NPARAM) return;
   const float g = grad[p];
   const float mm = beta1 * m[p] + (1.0f - beta1) * g;
   const float vv = beta2 * v[p] + (1.0f - beta2) * g * g;
   m[p] = mm;
   v[p] = vv;
   const float x = master[p] - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
   master[p] = x;
   w[p] = __float2bfloat16_rn(x);
   grad[p] = 0.0f;
}

__global__ void mlp_cast_kernel(const float* __restrict__ master, __nv_bfloat16* __restrict__ w) {
   const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
   if (p < MLP_NPARAM) w[p] = __float2bfloat16_rn(master[p]);
}

}  // namespace

cudaError_t mlp_cast(const float* d_master, __nv_bfloat16* d_w, cudaStream_t s) {
   mlp_cast_kernel<<<(MLP_NPARAM + 255) / 256, 256, 0, s>>>(d_master, d_w);
   return cudaGetLastError();
}

cudaError_t mlp_forward(const __nv_bfloat16* d_w, const float* d_X, uint32_t n, float* d_Y, cudaStream_t s) {
   if (n == 0) return cudaSuccess;
   const size_t smem = MLP_NPARAM * sizeof(float);
   mlp_forward_kernel<false><<<(n + FWD_T - 1) / FWD_T, FWD_T, smem, s>>>(d_w, d_X, n, d_Y, MlpScale{}, nullptr, nullptr);
   return cudaGetLastError();
}

cudaError_t mlp_predict(const __nv_bfloat16* d_w, const float* d_X, uint32_t n, const MlpScale& scale, double* d_sel,
                        double* d_cost, cudaStream_t s) {
   if (n == 0) return cudaSuccess;
   const size_t smem = MLP_NPARAM * sizeof(float);
   mlp_forward_kernel<true><<<(n + FWD_T - 1) / FWD_T, FWD_T, smem, s>>>(d_w, d_X, n, nullptr, scale, d_sel, d_cost);
   return cudaGetLastError();
}

cudaError_t mlp_gradient(const __nv_bfloat16* d_w, const float* d_X, const float* d_T, uint32_t n, float* d_grad,
                         float* d_loss, int* d_err, bool withhold, cudaStream_t s) {
   if (n == 0) return cudaSuccess;
   cudaError_t e = cudaFuncSetAttribute(mlp_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SO_END));
   if (e != cudaSuccess) return e;
   mlp_grad_kernel<<<(n + TC_S - 1) / TC_S, TC_T, SO_END, s>>>(d_w, d_X, d_T, n, 1.0f / static_cast<float>(n), d_grad, d_loss,
                                                                   d_err, withhold);
   return cudaGetLastError();
}

cudaError_t mlp_adam(float* d_master, __nv_bfloat16* d_w, float* d_grad, float* d_m, float* d_v, float lr, uint32_t step,
                     cudaStream_t s) {
   const float beta1 = 0.9f, beta2 = 0.999f;
   const float c1 = 1.0f - static_cast<float>(std::pow(beta1, static_cast<double>(step)));
   const float c2 = 1.0f - static_cast<float>(std::pow(beta2, static_cast<double>(step)));
   mlp_adam_kernel<<<(MLP_NPARAM + 255) / 256, 256, 0, s>>>(d_master, d_w, d_grad, d_m, d_v, lr, beta1, beta2, 1e-8f, c1,
                                                            c2);
   return cudaGetLastError();
}

}  // namespace rhygpu
