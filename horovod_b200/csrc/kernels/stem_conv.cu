// The first convolution of a ResNet, 7x7 / stride 2 / padding 3 on 3 channels,
// forward and gradient of the weights, channels-last 16-bit, as an implicit
// GEMM on the 5th-generation tensor cores. cuDNN has no sm_100 kernel for 3
// channels and pads them to 4 for one of an older architecture.
//
// Input pixels are taken in 2 x 2 blocks of 12 values (16 with padding): the
// convolution is then 4x4 / stride 1 on 16 channels, 16 steps of K = 16, and
// output (i, j) reads the blocks (i .. i + 3, j .. j + 3). A CTA computes 16
// rows of 8 output pixels (M = 128) from a patch of 19 x 11 blocks in shared
// memory, stored without a swizzle as two planes of 16 bytes per block: 8
// neighbouring blocks of a row are then one 8 x 16-byte core matrix, the rows
// of the patch are the stride between core matrices, and the operand of every
// one of the 16 taps is the same descriptor with another start address. No
// im2col is ever stored. The weights stay in shared memory for all tiles of a
// CTA; four CTAs per SM take turns with loading, multiplying and storing, and
// a CTA loads the pixels of its next tile before it waits for the products.
//
// The 4 x 4 blocks of an output are 8 x 8 pixels; the first row and column of
// them lie outside the 7 x 7 window and are multiplied by zero, which would make
// NaN of an infinity or a NaN there. A tile whose patch holds one is therefore
// computed by plain loops over the window (plain_tile).
//
// 256 images of 224 x 224 to 64 channels in bf16 on a B200: forward 168 to 174 us
// (PyTorch's, with cuDNN's padding pass, 1614 us), gradient of the weights 238 to
// 246 us (PyTorch's 926 us). The bytes of either pass take 75 us at the rate of a
// plain copy; the tensor cores' operand reads from shared memory and the turns
// between the phases of a tile take the rest.
//
// Waits are bounded. When one runs out, what the CTA had not finished becomes NaN
// (so that the step is seen to have failed), and a host-visible word per device
// says so (StemConvFailed).
//
// The reference has no counterpart (it takes convolutions from the framework).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>
#include <cstring>
#include <mutex>

#include "kernels.h"
#include "tensor_core.cuh"

namespace hvd {
namespace kern {

namespace {

constexpr int THREADS = 256;
constexpr int TILE_H = 16, TILE_W = 8;                      // output pixels: M = 128
constexpr int PATCH_H = TILE_H + 3, PATCH_W = TILE_W + 3;   // blocks
constexpr int PATCH = PATCH_H * PATCH_W;
constexpr int PLANE_BYTES = PATCH * 16;
constexpr uint16_t NAN16 = 0x7fff;  // a NaN of either 16-bit type
constexpr int TAPS = 16, K_CORES = 2 * TAPS;  // 8 values of K each
static_assert(PATCH <= THREADS, "one block per thread");

// Exponents of two 16-bit values in a word, and the lowest bit of each.
template <typename T> struct Exponent;
template <> struct Exponent<__nv_bfloat16> {
  static constexpr uint32_t ALL = 0x7f807f80u, LOWEST = 0x00800080u;
};
template <> struct Exponent<__half> {
  static constexpr uint32_t ALL = 0x7c007c00u, LOWEST = 0x04000400u;
};

// Whether a value of the block is an infinity or a NaN: only an exponent of
// all ones carries into the sign's place.
template <typename T> __device__ __forceinline__ bool not_finite(const uint32_t (&v)[6]) {
  uint32_t carries = 0u;
#pragma unroll
  for (int i = 0; i < 6; ++i) carries |= (v[i] & Exponent<T>::ALL) + Exponent<T>::LOWEST;
  return (carries & 0x80008000u) != 0u;
}

struct StemShape {
  int n, h, w, ho, wo, channels;  // channels: of the output
  int tiles, tiles_h, tiles_w;
  int64_t ws_o, ws_c, ws_h, ws_w;  // strides of the weights
};

struct TileAt {
  int n, i, j;  // image, first output row and column
};
__device__ __forceinline__ TileAt tile_at(const StemShape& s, int t) {
  const unsigned row = static_cast<unsigned>(t) / s.tiles_w;
  const unsigned n = row / s.tiles_h;
  return {static_cast<int>(n), static_cast<int>(row - n * s.tiles_h) * TILE_H,
          static_cast<int>(t - row * s.tiles_w) * TILE_W};
}

// The 12 values of this thread's block of the patch, two per word (zero
// outside the image). PAIRS: the images are an even number of pixels wide and
// start on a 4-byte boundary, so the six values of a block's row are three
// words, all of them inside the image or none.
template <bool PAIRS>
__device__ __forceinline__ void load_block(const uint16_t* __restrict__ x, const StemShape& s,
                                           const TileAt& t, uint32_t (&v)[6]) {
#pragma unroll
  for (int i = 0; i < 6; ++i) v[i] = 0u;
  const int r = threadIdx.x / PATCH_W, c = threadIdx.x % PATCH_W;
  if (r >= PATCH_H) return;
  const int row = 2 * (t.i + r - 2), col = 2 * (t.j + c - 2);
#pragma unroll
  for (int dr = 0; dr < 2; ++dr) {
    if (row + dr < 0 || row + dr >= s.h) continue;
    const uint16_t* p = x + ((static_cast<int64_t>(t.n) * s.h + row + dr) * s.w + col) * 3;
    if (PAIRS) {
      if (col >= 0 && col < s.w) {
#pragma unroll
        for (int k = 0; k < 3; ++k)
          v[dr * 3 + k] = __ldg(reinterpret_cast<const uint32_t*>(p) + k);
      }
    } else {
      uint32_t e[6] = {0u, 0u, 0u, 0u, 0u, 0u};
#pragma unroll
      for (int k = 0; k < 6; ++k)
        if (col + k / 3 >= 0 && col + k / 3 < s.w) e[k] = __ldg(p + k);
#pragma unroll
      for (int k = 0; k < 3; ++k) v[dr * 3 + k] = e[2 * k] | (e[2 * k + 1] << 16);
    }
  }
}

__device__ __forceinline__ void store_block(unsigned char* patch, const uint32_t (&v)[6]) {
  if (threadIdx.x >= PATCH) return;
  reinterpret_cast<uint4*>(patch)[threadIdx.x] = make_uint4(v[0], v[1], v[2], v[3]);
  reinterpret_cast<uint4*>(patch + PLANE_BYTES)[threadIdx.x] = make_uint4(v[4], v[5], 0u, 0u);
}

// Output pixels [rows][cols] of a tile from the patch and the weights in shared
// memory, by loops over the pixels of each window and no others. y: the
// tile's first pixel.
template <typename T>
__device__ __noinline__ void plain_tile(const unsigned char* patch, const unsigned char* weights,
                                        uint16_t* y, int64_t row_pitch, int rows, int cols,
                                        int C) {
  constexpr int PIXELS = TILE_H * TILE_W;
  const T* p = reinterpret_cast<const T*>(patch);
  const T* w = reinterpret_cast<const T*>(weights);
  const int pixel = threadIdx.x % PIXELS, i = pixel / TILE_W, j = pixel % TILE_W;
  if (i >= rows || j >= cols) return;
  uint16_t* out = y + i * row_pitch + j * C;
  for (int c0 = threadIdx.x / PIXELS * 8; c0 < C; c0 += THREADS / PIXELS * 8) {
    float sum[8] = {};
#pragma unroll 1
    for (int tap = 0; tap < TAPS; ++tap) {
      const int block = (i + tap / 4) * PATCH_W + j + tap % 4;
#pragma unroll 1
      for (int c = 0; c < 12; ++c) {  // (row, column) of the pixel in its block, channel
        if ((tap / 4 == 0 && c / 6 == 0) || (tap % 4 == 0 && c / 3 % 2 == 0)) continue;
        const float value = static_cast<float>(p[(c / 8 * PATCH + block) * 8 + c % 8]);
        const T* wc = w + ((tap * 2 + c / 8) * C + c0) * 8 + c % 8;
#pragma unroll
        for (int o = 0; o < 8; ++o) sum[o] = fmaf(value, static_cast<float>(wc[o * 8]), sum[o]);
      }
    }
    *reinterpret_cast<uint4*>(out + c0) =
        make_uint4(narrow2<T>(sum[0], sum[1]), narrow2<T>(sum[2], sum[3]),
                   narrow2<T>(sum[4], sum[5]), narrow2<T>(sum[6], sum[7]));
  }
}

// Fills the outputs of tiles `tile`, `tile` + grid, ... with NaN.
__device__ __noinline__ void give_up_tiles(uint16_t* y, const StemShape& s, int tile) {
  for (; tile < s.tiles; tile += gridDim.x) {
    const TileAt at = tile_at(s, tile);
    const int rows = min(s.ho - at.i, TILE_H), row_values = min(s.wo - at.j, TILE_W) * s.channels;
    uint16_t* out = y + ((static_cast<int64_t>(at.n) * s.ho + at.i) * s.wo + at.j) * s.channels;
    for (int e = threadIdx.x; e < rows * row_values; e += THREADS)
      out[static_cast<int64_t>(e / row_values) * s.wo * s.channels + e % row_values] = NAN16;
  }
}

template <typename T, bool PAIRS>
__global__ void __launch_bounds__(THREADS, 4)
stem_conv_forward_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ weight,
                         uint16_t* __restrict__ y, const __grid_constant__ StemShape s,
                         const uint32_t idesc, const uint32_t tmem_columns, int* status,
                         const uint32_t wait_ns) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_bar;
  __shared__ uint32_t s_tmem;
  const int C = s.channels;
  unsigned char* patch = smem;                                // [2 planes][PATCH][16 bytes]
  unsigned char* weights = smem + 2 * PLANE_BYTES;            // [K_CORES][C][16 bytes]
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  int tile = blockIdx.x;  // the grid is no larger than the tiles
  TileAt at = tile_at(s, tile);
  uint32_t v[6];
  load_block<PAIRS>(x, s, at, v);
  // A thread fills column k of row o in all 32 core matrices: 16 loads at a
  // time, and all index arithmetic but the last sum outside of them.
  for (int e = threadIdx.x; e < C * 8; e += THREADS) {
    const int o = e / 8, k = e % 8;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int c16 = half * 8 + k;  // (row, column) of the pixel in its block, channel
      const int dr = c16 / 6, dc = c16 / 3 % 2;
      const uint16_t* w = weight + o * s.ws_o + c16 % 3 * s.ws_c + (dr - 1) * s.ws_h +
                          (dc - 1) * s.ws_w;
      uint16_t value[TAPS];
#pragma unroll
      for (int tap = 0; tap < TAPS; ++tap) {
        const bool inside = c16 < 12 && (tap / 4 > 0 || dr > 0) && (tap % 4 > 0 || dc > 0);
        value[tap] = 0;
        if (inside) value[tap] = __ldg(w + tap / 4 * 2 * s.ws_h + tap % 4 * 2 * s.ws_w);
      }
#pragma unroll
      for (int tap = 0; tap < TAPS; ++tap)
        reinterpret_cast<uint16_t*>(weights)[(tap * 2 + half) * C * 8 + e] = value[tap];
    }
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s_bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_addr(&s_tmem)), "r"(tmem_columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;

  uint32_t parity = 0;
  for (; tile < s.tiles; tile += gridDim.x) {
    store_block(patch, v);
    // What the threads wrote is read by the tensor core's proxy.
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    const bool plain = __syncthreads_or(not_finite<T>(v)) != 0;
    if (threadIdx.x == 0 && !plain) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int tap = 0; tap < TAPS; ++tap)
        mma(tmem,
            operand(smem_addr(patch) + (tap / 4 * PATCH_W + tap % 4) * 16, PLANE_BYTES,
                    PATCH_W * 16),
            operand(smem_addr(weights) + tap * 2 * C * 16, C * 16, 128), idesc, tap > 0);
      commit(smem_addr(&s_bar));
    }
    TileAt next = at;
    if (tile + static_cast<int>(gridDim.x) < s.tiles) {
      next = tile_at(s, tile + gridDim.x);
      load_block<PAIRS>(x, s, next, v);
    }
    if (plain) {
      const int64_t row_pitch = static_cast<int64_t>(s.wo) * C;
      plain_tile<T>(patch, weights,
                    y + (static_cast<int64_t>(at.n) * s.ho + at.i) * row_pitch + at.j * C,
                    row_pitch, s.ho - at.i, s.wo - at.j, C);
      __syncthreads();  // the next tile takes the patch's place
      at = next;
      continue;
    }
    const bool ok = wait_bounded(smem_addr(&s_bar), parity, wait_ns);
    parity ^= 1u;
    if (__syncthreads_and(ok) == 0) {
      if (threadIdx.x == 0) *reinterpret_cast<volatile int*>(status) = 1;
      wait_bounded(smem_addr(&s_bar), parity ^ 1u, STEM_WAIT_NS);  // the products in flight
      give_up_tiles(y, s, tile);
      break;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // Warps w and w + 4 read the accumulators of pixels 32 (w % 4) ..., 16
    // channels at a time in turn.
    // A thread's 16 channels are one 32-byte sector of the output.
    const int pixel = warp % 4 * 32 + lane;
    const int i = at.i + pixel / TILE_W, j = at.j + pixel % TILE_W;
    uint16_t* out = y + ((static_cast<int64_t>(at.n) * s.ho + i) * s.wo + j) * C;
    for (int c0 = warp / 4 * 16; c0 < C; c0 += 32) {
      uint32_t r[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
          "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
            "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
            "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
          : "r"(tmem + (static_cast<uint32_t>(warp % 4 * 32) << 16) + c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      uint32_t o[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        o[k] = narrow2<T>(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1]));
      if (i < s.ho && j < s.wo)
        asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                     ::"l"(out + c0), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]),
                     "r"(o[5]), "r"(o[6]), "r"(o[7]) : "memory");
    }
    // The next tile's products wait for these reads (the barrier above).
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    at = next;
  }
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 ::"r"(tmem), "r"(tmem_columns));
}

// ---- gradient of the weights ------------------------------------------------
// D[(tap, channel), o] = sum over output pixels of block value x gradient: the
// same patch is the M operand (M along channels and taps, K along pixels, both
// "MN-major"), the gradients of the tile's pixels are the N operand. M groups
// lie 16 bytes apart, so one M = 128 operand covers 16 consecutive blocks: the
// four taps of a kernel row (groups 0 .. 3) and of the next one (11 .. 14, a
// patch row further on); the other groups multiply values that nobody reads.
// Two pairs of kernel rows x two planes make four accumulators, which stay in
// tensor memory over all tiles of the CTA; each CTA leaves its sums in
// `partial` ([CTA][tap][16 channels][o], fp32) and a second kernel adds them
// up. Two buffers: the next tile is stored while this one is multiplied.
//
// A tile that reaches past the output has gradients of zero there, beside
// pixels that may exist and make NaN of them where they are not finite. A CTA
// whose sums hold an infinity or a NaN, in an image with such tiles, therefore
// computes them again by plain loops over the output pixels that exist
// (plain_sums). (To look at the pixels instead, inside the main loop, costs every
// call 4 to 10%.)

constexpr int DY_PLANE = TILE_H * TILE_W * 16 + 16;  // 16 bytes off: no bank conflicts
constexpr int PATCH_BYTES = (2 * PLANE_BYTES + 127) / 128 * 128;
constexpr int DY_PIECES = 8;  // 16-byte pieces per thread at 128 channels

// The CTA's sums by plain loops. smem: room for a patch and the gradients of a
// tile.
template <typename T, bool PAIRS>
__device__ __noinline__ void plain_sums(const uint16_t* __restrict__ x,
                                        const uint4* __restrict__ dy, float* sums,
                                        const StemShape& s, unsigned char* smem) {
  const int C = s.channels, per_pixel = C / 8;
  const T* p = reinterpret_cast<const T*>(smem);
  uint4* grads = reinterpret_cast<uint4*>(smem + PATCH_BYTES);  // [pixel][C]
  for (int tile = blockIdx.x; tile < s.tiles; tile += gridDim.x) {
    const TileAt at = tile_at(s, tile);
    const int rows = min(s.ho - at.i, TILE_H), cols = min(s.wo - at.j, TILE_W);
    uint32_t v[6];
    load_block<PAIRS>(x, s, at, v);
    __syncthreads();  // the last readers of the buffer
    store_block(smem, v);
    for (int e = threadIdx.x; e < rows * cols * per_pixel; e += THREADS) {
      const int px = e / per_pixel;
      const int64_t i = static_cast<int64_t>(at.n) * s.ho + at.i + px / cols;
      grads[e] = __ldg(dy + (i * s.wo + at.j + px % cols) * per_pixel + e % per_pixel);
    }
    __syncthreads();
    // 8 output channels of a tap and an input channel at a time; a thread has
    // the same ones in every tile.
#pragma unroll 1
    for (int e = threadIdx.x; e < TAPS * 12 * per_pixel; e += THREADS) {
      const int piece = e % per_pixel, c = e / per_pixel % 12, tap = e / per_pixel / 12;
      float* to = sums + (tap * 16 + c) * C + piece * 8;
      float sum[8];
#pragma unroll
      for (int o = 0; o < 8; ++o) sum[o] = tile == static_cast<int>(blockIdx.x) ? 0.f : to[o];
      const uint4* g = grads + piece;
#pragma unroll 1
      for (int i = 0; i < rows; ++i)
#pragma unroll 1
        for (int j = 0; j < cols; ++j, g += per_pixel) {
          const int block = c / 8 * PATCH + (i + tap / 4) * PATCH_W + j + tap % 4;
          const float value = static_cast<float>(p[block * 8 + c % 8]);
          const uint4 raw = *g;
          const T* d = reinterpret_cast<const T*>(&raw);
#pragma unroll
          for (int o = 0; o < 8; ++o) sum[o] = fmaf(value, static_cast<float>(d[o]), sum[o]);
        }
#pragma unroll
      for (int o = 0; o < 8; ++o) to[o] = sum[o];
    }
  }
}

template <typename T, bool PAIRS>
__global__ void __launch_bounds__(THREADS, 2)
stem_conv_wgrad_kernel(const uint16_t* __restrict__ x, const uint4* __restrict__ dy,
                       float* __restrict__ partial, const __grid_constant__ StemShape s,
                       const uint32_t idesc, const uint32_t tmem_columns, int* status,
                       const uint32_t wait_ns) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t s_bar[2];
  __shared__ uint32_t s_tmem;
  const int C = s.channels, per_pixel = C / 8;
  const int buffer_bytes = PATCH_BYTES + (per_pixel * DY_PLANE + 127) / 128 * 128;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  uint32_t v[6];
  uint4 d[DY_PIECES];
  // Where this thread's pieces of the gradients lie: in the tile, relative to
  // the tile's first pixel in dy, and in shared memory.
  int piece_px[DY_PIECES], piece_at[DY_PIECES], piece_to[DY_PIECES];
#pragma unroll
  for (int k = 0; k < DY_PIECES; ++k) {
    const int e = threadIdx.x + k * THREADS, px = e / per_pixel, piece = e - px * per_pixel;
    piece_px[k] = px < TILE_H * TILE_W ? px : -1;
    piece_at[k] = (px / TILE_W * s.wo + px % TILE_W) * per_pixel + piece;
    piece_to[k] = piece * DY_PLANE + px * 16;
  }
  auto load = [&](int tile) {
    const TileAt at = tile_at(s, tile);
    load_block<PAIRS>(x, s, at, v);
    const uint4* p = dy + ((static_cast<int64_t>(at.n) * s.ho + at.i) * s.wo + at.j) * per_pixel;
#pragma unroll
    for (int k = 0; k < DY_PIECES; ++k) {
      d[k] = make_uint4(0u, 0u, 0u, 0u);
      if (piece_px[k] >= 0 && at.i + piece_px[k] / TILE_W < s.ho &&
          at.j + piece_px[k] % TILE_W < s.wo)
        d[k] = __ldg(p + piece_at[k]);
    }
  };
  int tile = blockIdx.x;
  load(tile);  // the grid is no larger than the tiles
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&s_bar[i])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_addr(&s_tmem)), "r"(tmem_columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;

  bool ok = true, finite = true;  // finite: this thread's sums
  uint32_t issued = 0;  // tiles given to the tensor cores
  float* const sums = partial + static_cast<int64_t>(blockIdx.x) * TAPS * 16 * C;
  for (; tile < s.tiles; tile += gridDim.x, ++issued) {
    const uint32_t buffer = issued & 1u, use = issued >> 1;
    unsigned char* patch = smem + buffer * buffer_bytes;
    unsigned char* grads = patch + PATCH_BYTES;
    if (use > 0) ok = wait_bounded(smem_addr(&s_bar[buffer]), (use - 1) & 1u, wait_ns);
    if (__syncthreads_and(ok) == 0) break;
    store_block(patch, v);
#pragma unroll
    for (int k = 0; k < DY_PIECES; ++k)
      if (piece_px[k] >= 0) *reinterpret_cast<uint4*>(grads + piece_to[k]) = d[k];
    if (tile + static_cast<int>(gridDim.x) < s.tiles) load(tile + gridDim.x);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if (threadIdx.x == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int k = 0; k < TILE_H / 2; ++k)  // 16 pixels: two rows of the tile
#pragma unroll
        for (int acc = 0; acc < 4; ++acc)   // kernel rows 2 (acc / 2) and + 1, plane acc % 2
          mma(tmem + acc * C,
              operand(smem_addr(patch) + acc % 2 * PLANE_BYTES +
                          (k * 2 + acc / 2 * 2) * PATCH_W * 16, PATCH_W * 16, 16),
              operand(smem_addr(grads) + k * 256, 128, DY_PLANE), idesc, issued > 0 || k > 0);
      commit(smem_addr(&s_bar[buffer]));
    }
  }
  // The last tile of each buffer.
  for (uint32_t b = 0; b < 2; ++b) {
    const uint32_t uses = (issued + 1 - b) / 2;
    if (uses > 0 && !wait_bounded(smem_addr(&s_bar[b]), (uses - 1) & 1u, wait_ns)) {
      wait_bounded(smem_addr(&s_bar[b]), (uses - 1) & 1u, STEM_WAIT_NS);  // products in flight
      ok = false;
    }
  }
  ok = __syncthreads_and(ok) != 0;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!ok) {
    if (threadIdx.x == 0) *reinterpret_cast<volatile int*>(status) = 1;
    for (int e = threadIdx.x; e < TAPS * 16 * C; e += THREADS) sums[e] = __int_as_float(0x7fffffff);
  } else {
    const int m = warp % 4 * 32 + lane, group = m / 8;
    const bool useful = group < 4 || (group >= 11 && group < 15);
    for (int c0 = warp / 4 * 16; c0 < 4 * C; c0 += 32) {
      uint32_t r[16];
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
          "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
          : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
            "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
            "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
          : "r"(tmem + (static_cast<uint32_t>(warp % 4 * 32) << 16) + c0));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      const int acc = c0 / C, channel = acc % 2 * 8 + m % 8;
      const int tap = (acc / 2 * 2 + group / 11) * 4 + group % 11;
      if (useful && channel < 12) {
        uint4* out = reinterpret_cast<uint4*>(sums + (tap * 16 + channel) * C + c0 % C);
#pragma unroll
        for (int i = 0; i < 4; ++i)
          out[i] = make_uint4(r[4 * i], r[4 * i + 1], r[4 * i + 2], r[4 * i + 3]);
#pragma unroll
        for (int i = 0; i < 16; ++i) finite &= (r[i] & 0x7f800000u) != 0x7f800000u;
      }
    }
  }
  const bool partial_tiles = s.ho % TILE_H != 0 || s.wo % TILE_W != 0;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  const bool plain = __syncthreads_or(!finite && partial_tiles && ok) != 0;
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 ::"r"(tmem), "r"(tmem_columns));
  if (plain) plain_sums<T, PAIRS>(x, dy, sums, s, smem);
}

// dw[o][c][kh][kw] = sum of the CTAs' partial sums, one CTA per (c, kh, kw):
// threads (o, slice of the CTAs), in fp32 within a slice and in fp64 across.
// Bound by the latency of the loads, hence the many slices (16 for 64
// channels; with 4 it took 41 us).
constexpr int SUM_THREADS = 1024;
template <typename T>
__global__ void __launch_bounds__(SUM_THREADS)
stem_conv_wgrad_sum_kernel(const float* __restrict__ partial, uint16_t* __restrict__ dw, int ctas,
                           const StemShape s) {
  __shared__ double sums[SUM_THREADS];
  const int C = s.channels, slices = SUM_THREADS / C;
  const int c = blockIdx.x % 3, kw = blockIdx.x / 3 % 7, kh = blockIdx.x / 21;
  const int tap = (kh + 1) / 2 * 4 + (kw + 1) / 2;
  const int channel = ((kh + 1) % 2 * 2 + (kw + 1) % 2) * 3 + c;
  const int o = threadIdx.x % C, slice = threadIdx.x / C;
  float sum = 0.f;
  if (slice < slices) {
    const float* p = partial + (static_cast<int64_t>(tap) * 16 + channel) * C + o;
#pragma unroll 8
    for (int b = slice; b < ctas; b += slices) sum += __ldg(p + static_cast<int64_t>(b) * 256 * C);
  }
  sums[threadIdx.x] = sum;
  __syncthreads();
  if (threadIdx.x < C) {
    double total = 0.0;
    for (int i = 0; i < slices; ++i) total += sums[i * C + o];
    const uint32_t v = narrow2<T>(static_cast<float>(total), 0.f);
    dw[o * s.ws_o + c * s.ws_c + kh * s.ws_h + kw * s.ws_w] = static_cast<uint16_t>(v);
  }
}

}  // namespace

// Host-visible word per device that a kernel sets when a wait ran out; null
// when there is no memory for them or no such device.
int* TensorCoreStatusWord(int device) {
  constexpr int DEVICES = 64;
  static std::mutex mu;
  static int* words = nullptr;
  std::lock_guard<std::mutex> lock(mu);
  if (words == nullptr) {
    // Also when the first call is being captured into a graph.
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (cudaHostAlloc(reinterpret_cast<void**>(&words), DEVICES * sizeof(int),
                      cudaHostAllocMapped | cudaHostAllocPortable) == cudaSuccess)
      std::memset(words, 0, DEVICES * sizeof(int));
    else
      words = nullptr;
    cudaThreadExchangeStreamCaptureMode(&mode);
  }
  return words != nullptr && device >= 0 && device < DEVICES ? words + device : nullptr;
}

// Offsets inside a tile are 32-bit, 16 rows of the output at 128 channels being the
// longest, as is the number of tiles.
bool StemConvSupported(int64_t n, int64_t h, int64_t w, int64_t channels) {
  constexpr int64_t MOST = 1 << 24;
  return channels >= 16 && channels <= 128 && channels % 16 == 0 && n >= 1 && h >= 1 && w >= 1 &&
         h <= MOST && w <= MOST && n <= (1 << 30) / (((h + 31) / 32) * ((w + 15) / 16));
}

static StemShape MakeShape(int n, int h, int w, int channels, const int64_t* weight_strides) {
  StemShape s;
  s.n = n;
  s.h = h;
  s.w = w;
  s.ho = (h - 1) / 2 + 1;
  s.wo = (w - 1) / 2 + 1;
  s.channels = channels;
  s.tiles_h = (s.ho + TILE_H - 1) / TILE_H;
  s.tiles_w = (s.wo + TILE_W - 1) / TILE_W;
  s.tiles = n * s.tiles_h * s.tiles_w;
  s.ws_o = weight_strides[0];
  s.ws_c = weight_strides[1];
  s.ws_h = weight_strides[2];
  s.ws_w = weight_strides[3];
  return s;
}

// cudaSuccess when the kernels may run; *status is where they report to.
static cudaError_t StemReady(int n, int h, int w, int channels, int** status) {
  if (!StemConvSupported(n, h, w, channels)) return cudaErrorInvalidValue;
  int device = 0;
  const cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  *status = TensorCoreStatusWord(device);
  return *status != nullptr ? cudaSuccess : cudaErrorMemoryAllocation;
}

bool StemConvFailed(int device, bool clear) {
  volatile int* status = TensorCoreStatusWord(device);
  if (status == nullptr) return true;
  const bool failed = *status != 0;
  if (clear) *status = 0;
  return failed;
}

cudaError_t LaunchStemConvForward(const void* x, const void* weight, const int64_t* weight_strides,
                                  void* y, int n, int h, int w, int channels, bool bf16,
                                  cudaStream_t stream, uint32_t wait_ns) {
  int* status = nullptr;
  cudaError_t err = StemReady(n, h, w, channels, &status);
  if (err != cudaSuccess) return err;
  const StemShape s = MakeShape(n, h, w, channels, weight_strides);
  // fp32 accumulators, 16-bit operands, both K-major, M = 128, N = channels.
  const uint32_t idesc = instruction(bf16, false, false, 128, channels);
  uint32_t columns = 32;  // a power of two; four CTAs share the SM's 512
  while (columns < static_cast<uint32_t>(channels)) columns *= 2;
  const int smem = 2 * PLANE_BYTES + K_CORES * channels * 16;
  const bool pairs = w % 2 == 0 && reinterpret_cast<uintptr_t>(x) % 4 == 0;
  auto kernel = bf16 ? (pairs ? stem_conv_forward_kernel<__nv_bfloat16, true>
                              : stem_conv_forward_kernel<__nv_bfloat16, false>)
                     : (pairs ? stem_conv_forward_kernel<__half, true>
                              : stem_conv_forward_kernel<__half, false>);
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) return err;
  const unsigned grid = static_cast<unsigned>(s.tiles < 148 * 4 ? s.tiles : 148 * 4);
  CountKernelLaunches(1);
  kernel<<<grid, THREADS, smem, stream>>>(static_cast<const uint16_t*>(x),
                                          static_cast<const uint16_t*>(weight),
                                          static_cast<uint16_t*>(y), s, idesc, columns, status,
                                          wait_ns);
  return cudaGetLastError();
}

// The four accumulators' columns of tensor memory: a power of two.
static uint32_t WgradColumns(int channels) {
  uint32_t columns = 64;
  while (columns < 4u * static_cast<uint32_t>(channels)) columns *= 2;
  return columns;
}

int StemConvWgradCtas(int n, int h, int w, int channels) {
  const int64_t strides[4] = {0, 0, 0, 0};
  const int tiles = MakeShape(n, h, w, channels, strides).tiles;
  // Two per SM, or one where the accumulators take all of the tensor memory.
  const int most = 148 * (WgradColumns(channels) <= 256 ? 2 : 1);
  return tiles < most ? tiles : most;
}

cudaError_t LaunchStemConvWgrad(const void* x, const void* dy, float* partial, void* dw,
                                const int64_t* weight_strides, int n, int h, int w, int channels,
                                bool bf16, cudaStream_t stream, uint32_t wait_ns) {
  int* status = nullptr;
  cudaError_t err = StemReady(n, h, w, channels, &status);
  if (err != cudaSuccess) return err;
  const StemShape s = MakeShape(n, h, w, channels, weight_strides);
  const int ctas = StemConvWgradCtas(n, h, w, channels);
  // As above, but both operands MN-major.
  const uint32_t idesc = instruction(bf16, true, true, 128, channels);
  const int smem = 2 * (PATCH_BYTES + (channels / 8 * DY_PLANE + 127) / 128 * 128);
  const bool pairs = w % 2 == 0 && reinterpret_cast<uintptr_t>(x) % 4 == 0;
  auto kernel = bf16 ? (pairs ? stem_conv_wgrad_kernel<__nv_bfloat16, true>
                              : stem_conv_wgrad_kernel<__nv_bfloat16, false>)
                     : (pairs ? stem_conv_wgrad_kernel<__half, true>
                              : stem_conv_wgrad_kernel<__half, false>);
  auto sum = bf16 ? stem_conv_wgrad_sum_kernel<__nv_bfloat16> : stem_conv_wgrad_sum_kernel<__half>;
  err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) return err;
  CountKernelLaunches(2);
  kernel<<<ctas, THREADS, smem, stream>>>(static_cast<const uint16_t*>(x),
                                          static_cast<const uint4*>(dy), partial, s, idesc,
                                          WgradColumns(channels), status, wait_ns);
  err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  sum<<<3 * 7 * 7, SUM_THREADS, 0, stream>>>(partial, static_cast<uint16_t*>(dw), ctas, s);
  return cudaGetLastError();
}

}  // namespace kern
}  // namespace hvd
