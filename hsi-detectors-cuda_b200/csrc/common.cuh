// common.cuh - shared device helpers for the sm_100a kernels.
//
// Hand-written PTX for the pieces the kernels build their pipelines from:
// mbarriers (with bounded waits), 1-D bulk async copies on the TMA engine,
// and a device-side error word that a bounded wait sets instead of hanging.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "hsi_b200.h"

namespace hsi_b200 {

// Largest number of polls a wait makes before it gives up, records
// HSI_E_TIMEOUT and lets the kernel unwind: seconds of wall time, far beyond any
// legitimate wait, short enough that a broken pipeline returns an error.
constexpr uint32_t kWaitLimit = 1u << 26;  // polls of a flag in memory
// Polls of mbar_wait_idle, each of which may suspend the warp for up to kIdleNs.
constexpr uint32_t kIdlePolls = 1u << 22;
constexpr uint32_t kIdleNs = 1000;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count));
}

// Make barrier initialisation visible to the async (TMA) proxy.
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}

// Wait for phase `parity` of `bar` to complete, polling at most kWaitLimit
// times.  Returns false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < kWaitLimit; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
  }
  return false;
}

// The same for kernels that are short of issue slots: a poll without the time
// hint comes back after a few cycles, and the waiting warps take slots from the
// working ones.  RX/ACE on the tensor cores (2048 x 1024 x 113) 375 us with
// mbar_wait, 348 us with this; the screen's logits (2048 x 2048 x 224) 464 and
// 451 us.  Waking costs more: the FP32 scorer, whose consumers wait for every
// stage, is 2 to 4 % slower with it and keeps mbar_wait.
__device__ __forceinline__ bool mbar_wait_idle(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < kIdlePolls; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity), "r"(kIdleNs)
        : "memory");
    if (done) return true;
  }
  return false;
}

// 1-D bulk copy global -> shared on the TMA engine, completing on `bar`.
// dst, src 16-byte aligned; bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// Packed FP32 FMA on sm_100: two lanes per instruction, d = a * b + c, each lane
// rounded as one fmaf.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(r)
      : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
        "l"(*reinterpret_cast<unsigned long long*>(&c)));
  return *reinterpret_cast<float2*>(&r);
}

// Record the first error a kernel hits in the caller's status word (nullable).
__device__ __forceinline__ void record_error(int* status, int code) {
  if (status) atomicCAS(status, 0, code);
}

__device__ __forceinline__ float4 ld_shared_f4(const float* p) {
  return *reinterpret_cast<const float4*>(p);
}

template <typename T>
__host__ __device__ constexpr T div_up(T a, T b) {
  return (a + b - 1) / b;
}

}  // namespace hsi_b200
