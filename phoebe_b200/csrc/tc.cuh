// sm_100a primitives: tcgen05 (UMMA + TMEM), mbarriers, bulk async copies.
//
// Descriptor bit layouts follow the PTX ISA for tcgen05 (shared-memory
// matrix descriptor, instruction descriptor for .kind::f16/.kind::tf32) as
// also documented in CUTLASS's cute/arch/mma_sm100_desc.hpp.  Every wait on
// an mbarrier is bounded: after kWaitNs of polling it records an error code
// in a global status word and returns false, so a kernel can unwind (free
// TMEM, return) instead of hanging the GPU.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace tc {

constexpr unsigned long long kWaitNs = 2000000000ull;  // give up after 2 s

__device__ __forceinline__ unsigned long long globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ---------------------------------------------------------------------------
// mbarrier
// ---------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}" ::"r"(
                   smem_u32(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: polls for at most kWaitNs (checking a global abort bit every
// 256 polls); on timeout sets *status |= code | abort bit and returns false.
// the bounded poll of mbar_wait, out of line: the waits' call sites stay a
// few instructions each in the hot loops that use them
static __device__ __noinline__ bool mbar_wait_slow(uint64_t* bar, uint32_t parity, int* status, int code) {
  const unsigned long long t0 = globaltimer();
  for (unsigned i = 1;; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 255u) == 0) {
      if (*(volatile int*)status & 0x40000000) return false;  // another CTA gave up
      if (globaltimer() - t0 > kWaitNs) break;
    }
  }
  atomicOr(status, code | 0x40000000);
  return false;
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  return mbar_wait_slow(bar, parity, status, code);
}

// Same bound, with a short sleep between polls: for warps whose waiting must
// not take issue slots from the compute warps sharing their scheduler.
__device__ __forceinline__ bool mbar_wait_sleep(uint64_t* bar, uint32_t parity, int* status, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = globaltimer();
  for (unsigned i = 1;; ++i) {
    __nanosleep(64);
    if (mbar_try_wait(bar, parity)) return true;
    if ((i & 63u) == 0) {
      if (*(volatile int*)status & 0x40000000) return false;
      if (globaltimer() - t0 > kWaitNs) break;
    }
  }
  atomicOr(status, code | 0x40000000);
  return false;
}

// ---------------------------------------------------------------------------
// bulk async copy global -> shared of this CTA (no tensor map)
// ---------------------------------------------------------------------------
__device__ __forceinline__ void bulk_g2s(void* smem_dst, const void* gmem_src, uint32_t bytes,
                                         uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(smem_dst)),
      "l"(gmem_src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// The last copies of a ring have landed: fill k of `issued` (from 0) went to stage k % stages, whose
// barrier completes phase k / stages with it.  Whoever issues copies calls this before the block ends,
// also after a wait that gave up: none is left to write to shared memory that is no longer the block's.
static __device__ __noinline__ void ring_drain(uint64_t* full, unsigned issued, unsigned stages, int* status, int code) {
  for (unsigned k = issued > stages ? issued - stages : 0; k < issued; ++k) {
    const unsigned long long t0 = globaltimer();
    while (!mbar_try_wait(full + k % stages, (k / stages) & 1)) {
      __nanosleep(64);
      if (globaltimer() - t0 > kWaitNs) {
        atomicOr(status, code | 0x40000000);
        return;
      }
    }
  }
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---------------------------------------------------------------------------
// tcgen05: TMEM allocation, MMA, commit, loads, fences
// ---------------------------------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// D[tmem] (+)= A[smem] * B[smem], kind::f16 (bf16 operands, fp32 accumulate)
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                         uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// mbarrier arrives when all previously issued tcgen05.mma of this thread complete
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}

// tcgen05.ld writes its destination registers asynchronously: they may be
// read only after tcgen05.wait::ld.  The compiler sees no dependency between
// the wait and those registers, so the wait also redefines the N loaded
// values through empty asm statements ordered after it: no use of a loaded
// value can then be scheduled above the wait.
template <int N>
__device__ __forceinline__ void tmem_wait_ld(float* v) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < N; ++i) asm volatile("" : "+f"(v[i]));
}

// 32 lanes x 32 bit, 8 consecutive columns per thread
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// 32 lanes x 32 bit, 4 consecutive columns per thread
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, float* v) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}

// ---------------------------------------------------------------------------
// descriptors
// ---------------------------------------------------------------------------
// Shared-memory matrix descriptor, K-major, no swizzle ("interleaved" core
// matrices of 8 rows x 16 bytes stored as 128 contiguous bytes).
//   lbo: byte distance between the two 16-byte K-chunks of one MMA K-step
//   sbo: byte distance between consecutive 8-row groups
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version (sm_100)
  // base offset 0, lbo mode 0, layout type 0 = SWIZZLE_NONE
  return d;
}

// Instruction descriptor, kind::f16 with BF16 A/B, FP32 D, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16_f32(int M, int N) {
  return (1u << 4)                  // D format F32
         | (1u << 7)                // A format BF16
         | (1u << 10)               // B format BF16
         | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Instruction descriptor, kind::f16 with FP16 A/B (format 0), FP32 D, both K-major.
__host__ __device__ constexpr uint32_t idesc_f16_f32(int M, int N) {
  return (1u << 4)                  // D format F32
         | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// Byte offset of element (row, k) in a K-major no-swizzle tile whose rows
// hold Kp elements of esize bytes (core matrix = 8 rows x 16 bytes).
__host__ __device__ __forceinline__ uint32_t core_offset(int row, int k, int Kp, int esize) {
  const int epc = 16 / esize;  // elements per 16-byte chunk
  return (uint32_t)((row >> 3) * (Kp / epc) * 128 + (k / epc) * 128 + (row & 7) * 16 +
                    (k % epc) * esize);
}

}  // namespace tc
