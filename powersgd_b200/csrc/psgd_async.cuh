// Shared-memory barriers with bounded waits, as kernels that fill rings by asynchronous copies and those on the
// tensor cores use them.
#pragma once
#include "psgd_common.cuh"

constexpr uint64_t PSGD_MBAR_LIMIT_NS = 2000000000ull;  // 2 s

__device__ __forceinline__ uint32_t psgd_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void psgd_mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(psgd_smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void psgd_mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(psgd_smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void psgd_mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(psgd_smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool psgd_mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(psgd_smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// False (and the abort flag and the status word set) when the limit expires, or when another wait of the
// CTA has given up already.
__device__ __forceinline__ bool psgd_mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* status) {
  if (psgd_mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = psgd_globaltimer_ns();
  while (!psgd_mbar_try_wait(bar, parity)) {
    if (*abort_flag) return false;
    if (psgd_globaltimer_ns() - t0 > PSGD_MBAR_LIMIT_NS) {
      *abort_flag = 1;
      if (status) {
        // plain store: the word may live in mapped pinned host memory, which the host reads
        *((volatile int*)status) = (int)PSGD_TIMEOUT_MBARRIER;
        __threadfence_system();
      }
      return false;
    }
  }
  return true;
}
// After a wait ran out: time for copies that may still be in flight to land before the CTA's shared memory is
// handed to another one.
__device__ __forceinline__ void psgd_let_copies_land() {
  const uint64_t t0 = psgd_globaltimer_ns();
  while (psgd_globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
}

// Ordinary stores of this thread to shared memory come before asynchronous copies into it that are issued behind a
// later barrier. A barrier alone does not order the two.
__device__ __forceinline__ void psgd_fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// `bytes` (a multiple of 16) of global memory into shared memory, both on 16-byte boundaries.
__device__ __forceinline__ void psgd_bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(psgd_smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(psgd_smem_u32(bar))
               : "memory");
}

// Copies of 4, 8 or 16 bytes of global memory into shared memory that need no registers while they are under way: a loop of them has
// all its copies in flight, where a loop of loads and stores (which the compiler must take for overlapping)
// waits for each. Everybody who reads the copies waits for their own and passes a barrier.
__device__ __forceinline__ void psgd_copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(psgd_smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void psgd_copy8(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(psgd_smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void psgd_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(psgd_smem_u32(dst)), "l"(src) : "memory");
}
// The same by way of L1, for what many CTAs of an SM copy: by way of L2 alone they all meet on its few lines.
__device__ __forceinline__ void psgd_copy16_shared(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(psgd_smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void psgd_copies_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
