// Tiles of channels-last activations ([rows][channels], 16-bit) between global and
// shared memory by TMA: boxes of 64 channels x up to 128 rows with the 128-byte
// swizzle, the layout that operand_swizzled() describes to the tensor cores.
//
// The reference has no counterpart (it takes convolutions from the framework).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "tensor_core.cuh"

namespace hvd {
namespace kern {

constexpr int TILE_M = 128;
constexpr int BOX_BYTES = TILE_M * 128;  // 64 channels of 128 rows

// A matrix [rows][channels] as the TMA sees it: [rows2][rows1][channels], with
// boxes of 64 channels x box1 x box2 rows; pitches in elements. False where the
// driver refuses.
bool MakeMap(CUtensorMap* map, const void* p, bool bf16, int64_t channels, int64_t rows1,
             int64_t rows2, int64_t pitch1, int64_t pitch2, int box1, int box2);
bool TmaAvailable();

// As wait_bounded; also false, soon, when another role of the CTA has set *stop.
__device__ __forceinline__ bool wait_or_stop(uint32_t bar, uint32_t parity, uint32_t limit,
                                             volatile int* stop) {
  unsigned long long t0 = 0;
  if (limit == 0) return false;
  for (int i = 0;; ++i) {
    if (phase_done(bar, parity)) return true;
    if (*stop) return false;
    const unsigned long long t = nanoseconds();
    if (i == 0) t0 = t;
    if (t - t0 > limit) return false;
  }
}

__device__ __forceinline__ void expect_bytes(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
               ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void load_box(uint32_t to, const CUtensorMap* map, int c0, int c1,
                                         int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(to), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(bar) : "memory");
}
__device__ __forceinline__ void store_box(const CUtensorMap* map, int c0, int c1, int c2,
                                          uint32_t from) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];"
               ::"l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(from) : "memory");
}
template <int N> __device__ __forceinline__ void stores_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}

// Where 8 channels (`piece`) of a row lie in a tile of shared memory.
__device__ __forceinline__ uint32_t piece_at(int row, int piece) {
  return piece / 8 * BOX_BYTES + row * 128 + ((piece ^ row) & 7) * 16;
}
__device__ __forceinline__ uint4 load_piece(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}
__device__ __forceinline__ void store_piece(uint32_t at, uint4 v) {
  asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};"
               ::"r"(at), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

__device__ __forceinline__ void load_accumulators(uint32_t at, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
        "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
        "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(at));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace kern
}  // namespace hvd
