// Small helpers of the persistent decode kernel: GPU-scope counters with bounded waits, status-aware mbarrier
// waits, 4-element bf16 loads / stores.
#pragma once
#include <cuda_bf16.h>

#include "../common/ptx.cuh"

namespace agrpo {

namespace {

// Where part i of n begins when `total` is cut into n parts. In 32 bits: a 64-bit division is 2 KB of code, and there were fourteen
// in the persistent kernel. total * n stays far below 2^32 for K blocks, rows and the cache blocks of a sequence.
__device__ __forceinline__ int share(int total, int i, int n) { return (int)((unsigned)total * (unsigned)i / (unsigned)n); }

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void red_release_gpu_add(unsigned int* p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ bool status_set(const int* status) {
  return status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0;
}
// Bounded wait until *ctr >= want. Gives up early when another CTA has already reported a failure. (Relaxed polls and one fence
// at the end instead: 1.51 against 1.47 ms for a step of 16 rows. An acquire empties this SM's L1, so the warps that work
// meanwhile must not depend on it: no spills, page numbers in registers.)
__device__ __forceinline__ bool wait_counter(const unsigned int* ctr, unsigned int want, const int* status) {
  const long long t0 = clock64();
  int it = 0;
  while (ld_acquire_gpu(ctr) < want) {
    if ((++it & 31) == 0) {
      if (status_set(status)) return false;
      if (clock64() - t0 > kWaitBudgetTicks) return false;
    }
  }
  return true;
}
// The counter as one thread of the CTA has seen it, in shared memory: the other warps wait here, so that a counter which every
// CTA increments is polled by one thread per CTA and not by five.
__device__ __forceinline__ void st_release_cta(unsigned int* smem, unsigned int v) {
  asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(smem_u32(smem)), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_cta(const unsigned int* smem) {
  unsigned int v;
  asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(smem_u32(smem)) : "memory");
  return v;
}
__device__ __forceinline__ bool wait_seen(const unsigned int* smem, unsigned int want, const int* status) {
  if (ld_acquire_cta(smem) >= want) return true;
  const long long t0 = clock64();
  int it = 0;
  while (ld_acquire_cta(smem) < want) {
    if ((++it & 255) == 0) {
      if (status_set(status)) return false;
      if (clock64() - t0 > kWaitBudgetTicks) return false;
    }
  }
  return true;
}
// mbarrier wait that also gives up when the status word is set.
__device__ __forceinline__ bool mbar_wait_s(uint64_t* bar, uint32_t parity, const int* status) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  int it = 0;
  while (!mbar_try_wait(bar, parity)) {
    if ((++it & 63) == 0) {
      if (status_set(status)) return false;
      if (clock64() - t0 > kWaitBudgetTicks) return false;
    }
  }
  return true;
}

// Values handed from one CTA to another without a flag: the buffer holds kNotYet (a NaN that no computation produces)
// in every word that has not been written, so the data say themselves that they have arrived and the reader needs one L2
// round trip instead of the three of a fence, a counter and a load. The reader puts kNotYet back; an acquire / release pair
// of the phases in between orders that before the word's next use.
constexpr uint32_t kNotYet = 0xffffffffu;
__device__ __forceinline__ float arrived_value(float v) { return __float_as_uint(v) == kNotYet ? __uint_as_float(0x7fffffffu) : v; }
__device__ __forceinline__ void st_handoff(float* p, float v) {
  asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(arrived_value(v)) : "memory");
}
__device__ __forceinline__ float4 ld_handoff4(const float4* p) {
  float4 v;
  asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ float2 ld_handoff2(const float2* p) {
  float2 v;
  asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ bool has_arrived(float v) { return __float_as_uint(v) != kNotYet; }
__device__ __forceinline__ bool has_arrived(const float4& v) {
  return has_arrived(v.x) && has_arrived(v.y) && has_arrived(v.z) && has_arrived(v.w);
}
__device__ __forceinline__ void clear_handoff4(float4* p) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %1, %1, %1};" ::"l"(p), "r"(kNotYet) : "memory");
}
__device__ __forceinline__ void clear_handoff2(float2* p) {
  asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %1};" ::"l"(p), "r"(kNotYet) : "memory");
}

// Barrier ID of 128 threads that tells all of them alike whether any of them failed.
template <int ID>
__device__ __forceinline__ bool group_bar_or(bool fail) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, %2, 128, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"((uint32_t)fail), "n"(ID)
      : "memory");
  return any != 0;
}

// Loads served by L2: what the persistent kernels read here may have been written by another SM during the same launch,
// and an L1 line of this SM could still hold the value of an earlier layer.
__device__ __forceinline__ sumsq_t ld_sumsq_l2(const sumsq_t* p) { return __ldcg(p); }
__device__ __forceinline__ float4 ld_bf16x4(const __nv_bfloat16* p) {
  const uint2 u = __ldcg(reinterpret_cast<const uint2*>(p));
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void st_bf16x4(__nv_bfloat16* p, float4 v) {
  uint2 u;
  u.x = pack_bf16x2(v.x, v.y);
  u.y = pack_bf16x2(v.z, v.w);
  *reinterpret_cast<uint2*>(p) = u;
}

}  // namespace

}  // namespace agrpo
