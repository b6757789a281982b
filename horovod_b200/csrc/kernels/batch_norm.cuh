// What the batch-norm kernels share with the kernels that take one of them in.
//
// The reference has no counterpart (it takes batch normalisation from the framework).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace hvd {
namespace kern {

constexpr int VEC = 8;  // 16-bit elements per 16-byte access

// The next kernel of the stream may be started; it waits for this one's
// results with wait_for_previous().
__device__ __forceinline__ void start_next() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_for_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Bit i of either half word: the sign of channel 2i or 2i + 1.
__device__ __forceinline__ uint32_t spread_signs(uint32_t byte) {
  return (byte & 0xfu) | ((byte & 0xf0u) << 12);
}

// The two sums of channel ch over all copies.
__device__ __forceinline__ double2 total(const double* sums, int C, int copies, int64_t ch) {
  double2 t = make_double2(0.0, 0.0);
#pragma unroll 4
  for (int i = 0; i < copies; ++i) {
    const double* p = sums + static_cast<int64_t>(i) * 2 * C + ch;
    t.x += __ldcg(p);
    t.y += __ldcg(p + C);
  }
  return t;
}

// dx = scale * dz + kx * (x - centre) + kc: the terms of the sums folded per
// channel, in fp64. centre is the mean rounded to the type of x: the difference of the
// two is exact in fp32 (but for values that the other one dwarfs), so channels whose
// mean is many times their spread lose nothing.
struct BackwardTerms {
  float scale, kx, kc, centre;
  double dz, dz_xhat;  // the sums
};
template <typename T>
__device__ __forceinline__ BackwardTerms backward_terms(const double* sums, int C, int copies,
                                                        int64_t ch, double inv_m,
                                                        const float* weight, const float* saved) {
  const double2 sum = total(sums, C, copies, ch);
  BackwardTerms b;
  b.dz = sum.x;
  b.dz_xhat = sum.y;
  const float invstd = saved[C + ch], mean = saved[ch];
  b.scale = (weight ? weight[ch] : 1.f) * invstd;
  b.centre = static_cast<float>(static_cast<T>(mean));
  b.kx = static_cast<float>(-static_cast<double>(b.scale) * invstd * b.dz_xhat * inv_m);
  b.kc = static_cast<float>(-b.scale * b.dz * inv_m -
                            static_cast<double>(b.kx) * (static_cast<double>(mean) - b.centre));
  return b;
}

}  // namespace kern
}  // namespace hvd
