// Conversion of a few arrays between fp32 and a 16-bit type in one launch: the
// weights of a block of layers before its forward, their gradients after its
// backward. Arrays of a block are 0.1 to 10 MB, where a launch takes as long as the
// bytes; one launch per array took 2.5 times as long in all.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "kernels.h"
#include "tensor_core.cuh"

namespace hvd {
namespace kern {

namespace {

constexpr int THREADS = 256, PER_THREAD = 8;
constexpr int CHUNK = THREADS * PER_THREAD;

struct Chunks {
  int first[5];  // of each array, and one past the last
};

template <typename T, bool WIDEN>
__global__ void __launch_bounds__(THREADS)
cast_arrays_kernel(const CastArrays a, const Chunks chunks) {
  int i = 0;
  while (i + 1 < a.n && static_cast<int>(blockIdx.x) >= chunks.first[i + 1]) ++i;
  const int64_t at =
      (static_cast<int64_t>(blockIdx.x) - chunks.first[i]) * CHUNK + threadIdx.x * PER_THREAD;
  const int64_t left = a.counts[i] - at;
  if (left <= 0) return;
  if (WIDEN) {
    const T* from = static_cast<const T*>(a.from[i]) + at;
    float* to = static_cast<float*>(a.to[i]) + at;
    if (left >= PER_THREAD) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(from));
      const float2 p = widen2<T>(v.x), q = widen2<T>(v.y), r = widen2<T>(v.z), s = widen2<T>(v.w);
      reinterpret_cast<float4*>(to)[0] = make_float4(p.x, p.y, q.x, q.y);
      reinterpret_cast<float4*>(to)[1] = make_float4(r.x, r.y, s.x, s.y);
    } else {
      for (int k = 0; k < left; ++k) to[k] = static_cast<float>(from[k]);
    }
  } else {
    const float* from = static_cast<const float*>(a.from[i]) + at;
    T* to = static_cast<T*>(a.to[i]) + at;
    if (left >= PER_THREAD) {
      const float4 p = __ldg(reinterpret_cast<const float4*>(from));
      const float4 q = __ldg(reinterpret_cast<const float4*>(from) + 1);
      *reinterpret_cast<uint4*>(to) = make_uint4(narrow2<T>(p.x, p.y), narrow2<T>(p.z, p.w),
                                                 narrow2<T>(q.x, q.y), narrow2<T>(q.z, q.w));
    } else {
      for (int k = 0; k < left; ++k) to[k] = static_cast<T>(from[k]);
    }
  }
}

}  // namespace

cudaError_t LaunchCastArrays(const CastArrays& a, bool widen, bool bf16, cudaStream_t stream) {
  if (a.n < 1 || a.n > 4) return cudaErrorInvalidValue;
  Chunks chunks;
  int64_t total = 0;
  chunks.first[0] = 0;
  for (int i = 0; i < a.n; ++i) {
    if (reinterpret_cast<uintptr_t>(a.from[i]) % 16 || reinterpret_cast<uintptr_t>(a.to[i]) % 16)
      return cudaErrorInvalidValue;
    total += (a.counts[i] + CHUNK - 1) / CHUNK;
    if (total > INT32_MAX) return cudaErrorInvalidValue;
    chunks.first[i + 1] = static_cast<int>(total);
  }
  if (total == 0) return cudaSuccess;
  CountKernelLaunches(1);
  auto kernel = bf16 ? (widen ? cast_arrays_kernel<__nv_bfloat16, true>
                              : cast_arrays_kernel<__nv_bfloat16, false>)
                     : (widen ? cast_arrays_kernel<__half, true>
                              : cast_arrays_kernel<__half, false>);
  kernel<<<static_cast<unsigned>(total), THREADS, 0, stream>>>(a, chunks);
  return cudaGetLastError();
}

}  // namespace kern
}  // namespace hvd
