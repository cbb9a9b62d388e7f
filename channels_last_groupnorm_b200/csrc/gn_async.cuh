// Device helpers of the kernels that stream rows through a ring of shared-memory stages filled by
// asynchronous bulk copies (the wave plan, gn_wave.cu, and the resident plan, gn_resident.cu).
#pragma once
#include "gn_common.cuh"
#include "gn_math.cuh"

namespace gnb200 {

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}
// A consumer warp hands a stage back to the producer only after it has USED the vectors it read from
// the stage.  The shared-memory loads are merely issued when the warp moves on; signalling the stage
// as free right after them let the producer's next TMA copy into the stage (fast when the rows come from
// L2) now and then overtake a load that was still queued, and a warp computed one stage's rows from
// pieces of a later stage.  So the arrival follows the arithmetic in program order - instructions
// issue in order and the arithmetic cannot issue before its operands have arrived - and pin_regs keeps
// the compiler from moving that arithmetic behind the arrival (the output stores of pass B are
// volatile asm statements and stay in front of it by themselves).
template <int N>
__device__ __forceinline__ void pin_regs(float (&a)[N]) {
#pragma unroll
  for (int e = 0; e < N; ++e) asm volatile("" : "+f"(a[e]));
}
__device__ __forceinline__ void release_stage(uint64_t* empty_bar, int lane) {
  __syncwarp();
  if (lane == 0) mbar_arrive(empty_bar);
}
__device__ __forceinline__ float warp_sum_all(float v) {
#pragma unroll
  for (int b = 16; b >= 1; b >>= 1) v += __shfl_xor_sync(0xffffffffu, v, b);
  return v;
}
// streaming 16-byte store: the line is marked evict-first, so results do not push the rows that
// pass B still has to read out of L2
__device__ __forceinline__ void stg128_stream(void* p, const uint4 v) {
  asm volatile("st.global.cs.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
#define kNaN __int_as_float(0x7fc00000)

// ---------------------------------------------------------------------------------------------
// Tensor memory as storage.  No matrix instruction runs here, so an SM's 256 KB of tensor memory are free to hold rows
// between two passes: 512 columns of 128 lanes x 4 bytes.  A warp reaches the 32 lanes of its rank in its warpgroup, so
// the warpgroups of a CTA share the columns out and a thread has kTmemColumns words of its own, i.e. 32 vectors of 16
// bytes that nobody else touches: a store and the load that gets it back need no barrier, only wait::st.
// All these instructions want a whole converged warp, and lane 0 of warp 0 comes back from code of its own (the copies), so
// each begins with a __syncwarp.
// ---------------------------------------------------------------------------------------------
constexpr int kTmemColumns = 128;                  // per warpgroup, hence words per thread
constexpr uint32_t kTmemTotal = 4 * kTmemColumns;  // all of the SM's

// by one whole warp; the base address is valid for the CTA's threads after their next __syncthreads
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot) {
  __syncwarp();
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(smem_slot)), "r"(kTmemTotal)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
// by the same warp, when every thread of the CTA is done with its words: its stores have been waited for too
__device__ __forceinline__ void tmem_free(uint32_t base) {
  __syncwarp();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(kTmemTotal) : "memory");
}
// the calling thread's first word: lane in bits 31..16, column below
__device__ __forceinline__ uint32_t tmem_own(uint32_t base, int warp) {
  return base + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * kTmemColumns;
}
// 16 words from column `col` of the thread's own on
__device__ __forceinline__ void tmem_store16(uint32_t col, const uint4& a, const uint4& b, const uint4& c, const uint4& d) {
  __syncwarp();
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(col),
      "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w), "r"(c.x), "r"(c.y), "r"(c.z), "r"(c.w),
      "r"(d.x), "r"(d.y), "r"(d.z), "r"(d.w)
      : "memory");
}
__device__ __forceinline__ void tmem_store_wait() {
  __syncwarp();
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// the same 16 words back; load and wait are one statement, so that no use of them moves in between
__device__ __forceinline__ void tmem_load16(uint32_t col, uint4& a, uint4& b, uint4& c, uint4& d) {
  __syncwarp();
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(a.x), "=r"(a.y), "=r"(a.z), "=r"(a.w), "=r"(b.x), "=r"(b.y), "=r"(b.z), "=r"(b.w), "=r"(c.x), "=r"(c.y), "=r"(c.z),
        "=r"(c.w), "=r"(d.x), "=r"(d.y), "=r"(d.z), "=r"(d.w)
      : "r"(col)
      : "memory");
}

// mbarrier waits of the streaming kernels.  `gave_up` is the CTA's shared flag: the first wait that runs
// out sets it (and poisons the results, see the callers); from then on no wait of this CTA spends
// its limit again, so a broken run ends after about one limit instead of one limit per stage.
// producer (a single thread):
__device__ __forceinline__ void producer_wait(uint64_t* bar, unsigned parity, volatile int* gave_up, const WaitLimit& lim) {
  if (mbar_try_wait(bar, parity)) return;
  if (*gave_up != 0) return;
  if (!mbar_wait_bounded(bar, parity, lim)) *gave_up = 1;
}
// consumers (whole warps): if the phase is not complete yet, lane 0 alone polls - 256 polling threads
// would take issue slots from the CTAs that share the SM - and afterwards every lane observes the
// completed phase with one more try_wait of its own, which is what makes the TMA's writes visible
// to it.  Returns, alike in all lanes, whether the phase is complete.
__device__ __forceinline__ bool consumer_wait(uint64_t* bar, unsigned parity, volatile int* gave_up, const WaitLimit& lim) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  if ((threadIdx.x & 31) == 0 && *gave_up == 0) {
    if (!mbar_wait_bounded(bar, parity, lim)) *gave_up = 1;
  }
  __syncwarp();
  return __all_sync(0xffffffffu, mbar_try_wait(bar, parity));
}

// untiled bulk copy: both addresses and the size are multiples of 16
__device__ __forceinline__ void bulk_load(uint32_t smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_dst),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// The same for rows that are not read again: their lines are the first that L2 gives up, so the others stay.
__device__ __forceinline__ uint64_t evict_first_policy() {
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  return policy;
}
__device__ __forceinline__ void bulk_load_once(uint32_t smem_dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t policy) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(smem_dst),
               "l"(src), "r"(bytes), "r"(smem_addr(bar)), "l"(policy)
               : "memory");
}

// dx of one 16-byte vector of a 16-bit tensor: dyh = dy * act'(x a + b) with act' in packed half
// precision, dx = ag * dyh + c1 * x + c2.
template <typename T, int ACT, bool PAIRS = kPairs<T>>
__device__ __forceinline__ uint4 bwd_dx_packed(const uint4& xw, const uint4& dw, const float (&a)[8],
                                               const float (&b)[8], const float (&ag)[8], const float (&c1)[8],
                                               const float (&c2)[8]) {
  static_assert(sizeof(T) == 2, "16-bit tensors only");
  float fx[8], fd[8], o[8];
  unpack16<T, 8>(xw, fx);
  unpack16<T, 8>(dw, fd);
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float g0 = 1.f, g1 = 1.f;
    if constexpr (ACT != kActIdentity) {
      float yh0, yh1;
      if constexpr (PAIRS) {
        fma2(yh0, yh1, fx[2 * p], fx[2 * p + 1], a[2 * p], a[2 * p + 1], b[2 * p], b[2 * p + 1]);
      } else {
        yh0 = fmaf(fx[2 * p], a[2 * p], b[2 * p]);
        yh1 = fmaf(fx[2 * p + 1], a[2 * p + 1], b[2 * p + 1]);
      }
      const float2 gf = __half22float2(act_grad_pair<ACT>(yh0, yh1));
      g0 = gf.x;
      g1 = gf.y;
    }
    if constexpr (PAIRS) {
      float t0, t1;
      fma2(t0, t1, c1[2 * p], c1[2 * p + 1], fx[2 * p], fx[2 * p + 1], c2[2 * p], c2[2 * p + 1]);
      fma2(o[2 * p], o[2 * p + 1], ag[2 * p], ag[2 * p + 1], fd[2 * p] * g0, fd[2 * p + 1] * g1, t0, t1);
    } else {
      o[2 * p] = fmaf(ag[2 * p], fd[2 * p] * g0, fmaf(c1[2 * p], fx[2 * p], c2[2 * p]));
      o[2 * p + 1] = fmaf(ag[2 * p + 1], fd[2 * p + 1] * g1, fmaf(c1[2 * p + 1], fx[2 * p + 1], c2[2 * p + 1]));
    }
  }
  return pack16<T, 8>(o);
}

}  // namespace gnb200
