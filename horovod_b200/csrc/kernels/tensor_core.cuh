// What the kernels on the 5th-generation tensor cores share: operand
// descriptors, tcgen05 instructions, bounded waits, conversions.
//
// The reference has no counterpart (it takes convolutions from the framework).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

namespace hvd {
namespace kern {

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// Operand without a swizzle: `k_step` bytes between the two core matrices of
// K = 16, `mn_step` bytes between groups of 8 rows (columns).
__device__ __forceinline__ uint64_t operand(uint32_t addr, uint32_t k_step, uint32_t mn_step) {
  return static_cast<uint64_t>((addr >> 4) & 0x3fffu) |
         (static_cast<uint64_t>((k_step >> 4) & 0x3fffu) << 16) |
         (static_cast<uint64_t>((mn_step >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

// Operand in rows of 128 bytes with the 128-byte swizzle. K-major: 8 rows of M
// (or N) are 1024 bytes, `group_step` has no meaning. MN-major: a row is 64
// values of M (or N) at one k, 8 values of k are 1024 bytes and the next 64
// values of M (or N) follow after group_step bytes.
__device__ __forceinline__ uint64_t operand_swizzled(uint32_t addr, uint32_t group_step) {
  return operand(addr, group_step, 1024) | (2ull << 61);
}

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool add) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(add ? 1u : 0u) : "memory");
}

// The barrier completes a phase when the products issued so far are done.
__device__ __forceinline__ void commit(uint32_t bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
      ::"r"(bar) : "memory");
}

// fp32 accumulators, 16-bit operands.
__host__ __device__ constexpr uint32_t instruction(bool bf16, bool a_mn, bool b_mn, int m, int n) {
  return (1u << 4) | ((bf16 ? 1u : 0u) << 7) | ((bf16 ? 1u : 0u) << 10) |
         ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
         (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ bool phase_done(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(bar), "r"(parity), "r"(10000u /* ns */) : "memory");
  return done != 0;
}

__device__ __forceinline__ unsigned long long nanoseconds() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Waits until phase `parity` of the barrier is complete; false when that takes
// longer than `limit` nanoseconds (0: at once).
__device__ __forceinline__ bool wait_bounded(uint32_t bar, uint32_t parity, uint32_t limit) {
  unsigned long long t0 = 0;
  if (limit == 0) return false;
  for (int i = 0;; ++i) {
    if (phase_done(bar, parity)) return true;
    const unsigned long long t = nanoseconds();
    if (i == 0) t0 = t;
    if (t - t0 > limit) return false;
  }
}

template <typename T> __device__ __forceinline__ uint32_t narrow2(float a, float b);
template <> __device__ __forceinline__ uint32_t narrow2<__nv_bfloat16>(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t narrow2<__half>(float a, float b) {
  const __half2 v = __floats2half2_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}
template <typename T> __device__ __forceinline__ float2 widen2(uint32_t v);
template <> __device__ __forceinline__ float2 widen2<__nv_bfloat16>(uint32_t v) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
}
template <> __device__ __forceinline__ float2 widen2<__half>(uint32_t v) {
  return __half22float2(*reinterpret_cast<const __half2*>(&v));
}

}  // namespace kern
}  // namespace hvd
