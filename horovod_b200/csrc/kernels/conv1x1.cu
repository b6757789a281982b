// 1x1 convolutions of a residual network (channels-last, 16-bit) as products on
// the 5th-generation tensor cores, with what surrounds them taken into the
// kernel:
//   forward: the per-channel sums that the batch norm after it needs, so that
//            the output is not read again for its statistics;
//   gradient of the input: the gradient of the skip connection is added before
//            the result is rounded and stored (optionally through the mask of
//            the ReLU that it passes), which replaces a pass of its own over three
//            tensors.
//
// A persistent CTA computes tiles of 128 rows x BN channels of one column of
// tiles: a thread's sums then belong to the same channels in every tile and stay
// in registers. Warp 0 brings 64-deep slices of x into shared memory by TMA, and those
// of w (once for all tiles where they fit, else with every tile), one thread of
// warp 1 issues the products into one of two accumulators in tensor memory, warp 2
// brings the tile that is added, and eight warps take the other accumulator to
// registers, round it, store it to shared memory and from there by TMA. Where k and n
// are small (the first stages of a ResNet) the bytes of x, y and add are the bound, else
// what the SMs move between L2 and shared memory: 308 MB at 8.0 TB/s in the forward of
// 50176 rows from 256 to 1024 channels, whose w is read with every tile.
//
// The kernel alone on a B200, bf16, in us (in brackets: PyTorch's kernel for the product,
// then the pass or passes that are gone; floor: the bytes at a copy's rate):
//   802816 rows, 64 to 256 channels, forward with sums      88 (78, 69)    floor 78
//   802816 rows, 256 to 64                                  79 (77, 22)          78
//   50176 rows, 256 to 1024                                 39 (35, 22)          20
//   802816 rows, gradient of 256 from 64 and the masked sum 147 (79, 140 and 64)  145
//   50176 rows, gradient of 1024 from 256, masked sum       53 (35, 37 and 16)   36
//     with a sum that is not masked                         51 (35, 37)          36
// bench_kernels.py --case conv1x1 measures the calls.
//
// Waits are bounded. When one runs out, what the CTA had not finished becomes
// NaN, its sums too, and TensorCoreStatusWord() of the device is set.
//
// The reference has no counterpart (it takes convolutions from the framework).
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "kernels.h"
#include "tensor_core.cuh"
#include "tma.cuh"

namespace hvd {
namespace kern {

namespace {

constexpr int THREADS = 384;
constexpr int EPILOGUE_WARP = 4, EPILOGUE_THREADS = 256;
constexpr int SLICE_K = 64;
constexpr uint16_t NAN16 = 0x7fff;  // a NaN of either 16-bit type

enum Epilogue : int { STORE_SUMS = 0, ADD = 1, ADD_MASKED = 2 };

// Shared memory: output tiles, w where it stays, and a ring of slices of the
// operands.
constexpr int MOST_SLOTS = 8, MOST_BYTES = 226 * 1024;
template <int BN, int EPI>
struct Layout {
  static constexpr int BUFFER = BN / 64 * BOX_BYTES;
  // Output tiles: one more where a tile is also loaded ahead, one where it is
  // large.
  static constexpr int BUFFERS = BN == 256 ? 1 : EPI >= ADD ? 3 : 2;
  static constexpr int W_SLICE = BN * 128;
};

struct Maps {
  CUtensorMap x, w, add, y;
};

struct Shape {
  int64_t rows;
  int n, slices_k, tiles_m, tiles_n;
  bool w_stays;
  int slots;
  int tile_rows;       // rows of a tile that count: 128, or whole rows of pixels
  int x_step1, x_step2, y_step1, y_step2;  // coordinates of a tile per tile
  int width;           // y's pixels: see pixel_at()
  int64_t pitch_px, pitch_row;  // in elements
  int copies;
};

// Barriers among the epilogue's threads; the second form also says whether
// `ok` holds for all of them.
__device__ __forceinline__ void epilogue_sync() {
  asm volatile("barrier.cta.sync 1, %0;" ::"n"(EPILOGUE_THREADS) : "memory");
}
__device__ __forceinline__ bool epilogue_all(bool ok) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, 2, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all) : "r"(ok ? 1u : 0u), "n"(EPILOGUE_THREADS) : "memory");
  return all != 0;
}

// First element of row `row` of y.
__device__ __forceinline__ int64_t pixel_at(const Shape& s, int64_t row) {
  return row / s.width * s.pitch_row + row % s.width * s.pitch_px;
}

// Fills this CTA's tiles from `tile` on, and its sums, with NaN.
template <int BN>
__device__ __noinline__ void give_up(uint16_t* y, double* sums, const Shape& s, int tile, int step,
                                     int n0) {
  const int t = threadIdx.x - EPILOGUE_WARP * 32;
  for (; tile < s.tiles_m; tile += step)
    for (int e = t; e < s.tile_rows * BN; e += EPILOGUE_THREADS) {
      const int64_t row = static_cast<int64_t>(tile) * s.tile_rows + e / BN;
      if (row < s.rows) y[pixel_at(s, row) + n0 + e % BN] = NAN16;
    }
  if (sums != nullptr && t < BN)
    atomicAdd(sums + n0 + t, __longlong_as_double(0x7ff8000000000000ll));
}

template <typename T, int BN, bool W_MN, int EPI>
__global__ void __launch_bounds__(THREADS, 1)
conv1x1_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Shape s,
               const uint8_t* __restrict__ signs, uint16_t* y, double* sums, int* status,
               const uint32_t wait_ns) {
  using L = Layout<BN, EPI>;
  extern __shared__ unsigned char raw[];
  __shared__ __align__(8) uint64_t s_full[MOST_SLOTS], s_empty[MOST_SLOTS], s_w_full,
      s_acc_full[2],
      s_acc_empty[2], s_add_full[L::BUFFERS], s_add_empty[L::BUFFERS], s_drain;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_stop;
  const uint32_t buffers = (smem_addr(raw) + 1023u) & ~1023u;
  // The slices of w are either before the ring or each behind its slice of x.
  const uint32_t weights = buffers + L::BUFFERS * L::BUFFER;
  const uint32_t slices = weights + (s.w_stays ? s.slices_k * L::W_SLICE : 0);
  const uint32_t slice_bytes = BOX_BYTES + (s.w_stays ? 0 : L::W_SLICE);
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;

  if (threadIdx.x == 0) {
    auto init = [](uint64_t* bar, int count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;"
                   ::"r"(smem_addr(bar)), "r"(count) : "memory");
    };
    for (int i = 0; i < MOST_SLOTS; ++i) init(s_full + i, 1), init(s_empty + i, 1);
    init(&s_w_full, 1);
    for (int i = 0; i < 2; ++i) init(s_acc_full + i, 1), init(s_acc_empty + i, 8);
    for (int i = 0; i < L::BUFFERS; ++i) init(s_add_full + i, 1), init(s_add_empty + i, 1);
    init(&s_drain, 1);
    s_stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_addr(&s_tmem)), "n"(2 * BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;

  // The grid is a multiple of tiles_n.
  const int n0 = blockIdx.x % s.tiles_n * BN;
  const int first = blockIdx.x / s.tiles_n, step = gridDim.x / s.tiles_n;

  if (warp == 0) {
    if (lane == 0) {
      auto load_w = [&](uint32_t to, int k, uint32_t bar) {
        if (W_MN) {
#pragma unroll
          for (int j = 0; j < BN / 64; ++j)
            load_box(to + j * 8192, &maps.w, n0 + j * 64, k * SLICE_K, 0, bar);
        } else {
          load_box(to, &maps.w, k * SLICE_K, n0, 0, bar);
        }
      };
      if (s.w_stays) {
        expect_bytes(smem_addr(&s_w_full), s.slices_k * L::W_SLICE);
        for (int k = 0; k < s.slices_k; ++k)
          load_w(weights + k * L::W_SLICE, k, smem_addr(&s_w_full));
      }
      uint32_t slot = 0, phase = 0, issued = 0;
      bool ok = true;
      for (int tile = first; ok && tile < s.tiles_m; tile += step)
        for (int k = 0; k < s.slices_k; ++k, ++issued) {
          const uint32_t bar = smem_addr(&s_full[slot]), to = slices + slot * slice_bytes;
          ok = wait_or_stop(smem_addr(&s_empty[slot]), phase ^ 1u, wait_ns, &s_stop);
          if (!ok) break;
          expect_bytes(bar, s.tile_rows * 128 + (s.w_stays ? 0 : L::W_SLICE));
          load_box(to, &maps.x, k * SLICE_K, tile * s.x_step1, tile * s.x_step2, bar);
          if (!s.w_stays) load_w(to + BOX_BYTES, k, bar);
          if (++slot == s.slots) slot = 0, phase ^= 1u;
        }
      if (!ok) s_stop = 1;
      // No copy may be in flight when the CTA ends.
      if (s.w_stays) wait_bounded(smem_addr(&s_w_full), 0, STEM_WAIT_NS);
      const uint32_t slots = s.slots;
      for (uint32_t u = issued < slots ? 0 : issued - slots; u < issued; ++u)
        wait_bounded(smem_addr(&s_full[u % slots]), u / slots & 1u, STEM_WAIT_NS);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc =
          instruction(std::is_same<T, __nv_bfloat16>::value, false, W_MN, TILE_M, BN);
      uint32_t slot = 0, phase = 0, i = 0;
      bool ok = !s.w_stays || wait_or_stop(smem_addr(&s_w_full), 0, wait_ns, &s_stop);
      for (int tile = first; ok && tile < s.tiles_m; tile += step, ++i) {
        const uint32_t acc = i & 1u;
        ok = wait_or_stop(smem_addr(&s_acc_empty[acc]), (i >> 1 & 1u) ^ 1u, wait_ns, &s_stop);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int k = 0; k < s.slices_k; ++k) {
          ok = wait_or_stop(smem_addr(&s_full[slot]), phase, wait_ns, &s_stop);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t a = slices + slot * slice_bytes;
          const uint32_t b = s.w_stays ? weights + k * L::W_SLICE : a + BOX_BYTES;
#pragma unroll
          for (int j = 0; j < SLICE_K / 16; ++j)
            mma(tmem + acc * BN, operand_swizzled(a + j * 32, 16),
                W_MN ? operand_swizzled(b + j * 2048, 8192) : operand_swizzled(b + j * 32, 16),
                idesc, k > 0 || j > 0);
          commit(smem_addr(&s_empty[slot]));
          if (++slot == s.slots) slot = 0, phase ^= 1u;
        }
        if (!ok) break;
        commit(smem_addr(&s_acc_full[acc]));
      }
      if (!ok) s_stop = 1;
      commit(smem_addr(&s_drain));  // nor may products be
      wait_bounded(smem_addr(&s_drain), 0, STEM_WAIT_NS);
    }
  } else if (warp == 2) {
    if (EPI >= ADD && lane == 0) {
      uint32_t i = 0;
      bool ok = true;
      for (int tile = first; tile < s.tiles_m; tile += step, ++i) {
        const uint32_t b = i % L::BUFFERS, bar = smem_addr(&s_add_full[b]);
        ok = wait_or_stop(smem_addr(&s_add_empty[b]), (i / L::BUFFERS & 1u) ^ 1u, wait_ns,
                          &s_stop);
        if (!ok) break;
        expect_bytes(bar, s.tile_rows * 128 * (BN / 64));
#pragma unroll
        for (int j = 0; j < BN / 64; ++j)
          load_box(buffers + b * L::BUFFER + j * BOX_BYTES, &maps.add, n0 + j * 64,
                   tile * s.y_step1, tile * s.y_step2, bar);
      }
      if (!ok) s_stop = 1;
      for (uint32_t u = i < L::BUFFERS ? 0 : i - L::BUFFERS; u < i; ++u)
        wait_bounded(smem_addr(&s_add_full[u % L::BUFFERS]), u / L::BUFFERS & 1u, STEM_WAIT_NS);
    }
  } else if (warp >= EPILOGUE_WARP) {
    const int t = threadIdx.x - EPILOGUE_WARP * 32;
    const int row = warp % 4 * 32 + lane, half = (warp - EPILOGUE_WARP) / 4;
    constexpr int COLUMNS = BN / 2;              // of a thread's row
    constexpr int PIECES = BN / 8, ROW_STEP = EPILOGUE_THREADS / PIECES;
    float acc_sum[8], acc_sq[8];  // of channels n0 + t % PIECES * 8 ...
#pragma unroll
    for (int k = 0; k < 8; ++k) acc_sum[k] = acc_sq[k] = 0.f;
    // The signs of a thread's channels, a byte per 8, loaded a tile ahead.
    constexpr int WORDS = COLUMNS / 32;
    uint32_t next_bits[WORDS];
    auto load_bits = [&](int tile) {
      const int64_t r = static_cast<int64_t>(tile) * s.tile_rows + row;
#pragma unroll
      for (int k = 0; k < WORDS; ++k) {
        next_bits[k] = 0u;
        if (row < s.tile_rows && r < s.rows)
          next_bits[k] = __ldg(reinterpret_cast<const uint32_t*>(
              signs + r * (s.n / 8) + (n0 + half * COLUMNS) / 8) + k);
      }
    };
    uint32_t i = 0;
    bool ok = true;
    int tile = first;
    if (EPI == ADD_MASKED && tile < s.tiles_m) load_bits(tile);
    for (; tile < s.tiles_m; tile += step, ++i) {
      const uint32_t acc = i & 1u, b = i % L::BUFFERS, buffer = buffers + b * L::BUFFER;
      const int64_t row0 = static_cast<int64_t>(tile) * s.tile_rows;
      const int valid = static_cast<int>(min(static_cast<int64_t>(s.tile_rows), s.rows - row0));
      uint32_t bits[WORDS];
#pragma unroll
      for (int k = 0; k < WORDS; ++k) bits[k] = next_bits[k];
      if (EPI == ADD_MASKED && tile + step < s.tiles_m) load_bits(tile + step);
      ok = wait_or_stop(smem_addr(&s_acc_full[acc]), i >> 1 & 1u, wait_ns, &s_stop);
      if (EPI >= ADD)
        ok = ok && wait_or_stop(smem_addr(&s_add_full[b]), i / L::BUFFERS & 1u, wait_ns, &s_stop);
      else if (t == 0)
        stores_read<L::BUFFERS - 1>();  // the buffer's last store
      ok = epilogue_all(ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int c = 0; c < COLUMNS; c += 32) {
        uint32_t r[32];
        load_accumulators(tmem + (static_cast<uint32_t>(warp % 4 * 32) << 16) + acc * BN +
                              half * COLUMNS + c, r);
        if (c + 32 == COLUMNS) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          if (lane == 0) arrive(smem_addr(&s_acc_empty[acc]));
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          const uint32_t at = buffer + piece_at(row, (half * COLUMNS + c) / 8 + p);
          float f[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) f[k] = __uint_as_float(r[p * 8 + k]);
          if (EPI >= ADD) {
            const uint4 other = load_piece(at);
            uint32_t w[4] = {other.x, other.y, other.z, other.w};
            if (EPI == ADD_MASKED) {
              // The even channels' bits are the low nibble, the odd ones' the high.
              const uint32_t byte = bits[c / 32] >> (p * 8);
              const uint32_t spread = (byte & 0xfu) | ((byte & 0xf0u) << 12);
#pragma unroll
              for (int k = 0; k < 4; ++k) w[k] &= (spread >> k & 0x00010001u) * 0xffffu;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              const float2 v = widen2<T>(w[k]);
              f[2 * k] += v.x;
              f[2 * k + 1] += v.y;
            }
          }
          store_piece(at, make_uint4(narrow2<T>(f[0], f[1]), narrow2<T>(f[2], f[3]),
                                     narrow2<T>(f[4], f[5]), narrow2<T>(f[6], f[7])));
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      epilogue_sync();
      if (t == 0) {
#pragma unroll
        for (int j = 0; j < BN / 64; ++j)
          store_box(&maps.y, n0 + j * 64, tile * s.y_step1, tile * s.y_step2,
                    buffer + j * BOX_BYTES);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        if (EPI >= ADD && i > 0) {
          stores_read<1>();
          arrive(smem_addr(&s_add_empty[(i - 1) % L::BUFFERS]));
        }
      }
      if (EPI == STORE_SUMS) {
        float tile_sum[8], tile_sq[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) tile_sum[k] = tile_sq[k] = 0.f;
        auto take = [&](int r) {
          const uint4 v = load_piece(buffer + piece_at(r, t % PIECES));
          const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 f = widen2<T>(w[k]);
            tile_sum[2 * k] += f.x;
            tile_sum[2 * k + 1] += f.y;
            tile_sq[2 * k] = fmaf(f.x, f.x, tile_sq[2 * k]);
            tile_sq[2 * k + 1] = fmaf(f.y, f.y, tile_sq[2 * k + 1]);
          }
        };
        if (valid == TILE_M) {
#pragma unroll 4
          for (int r = 0; r < TILE_M; r += ROW_STEP) take(r + t / PIECES);
        } else {
          for (int r = t / PIECES; r < valid; r += ROW_STEP) take(r);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          acc_sum[k] += tile_sum[k];
          acc_sq[k] += tile_sq[k];
        }
      }
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (t == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    if (!ok) {
      if (t == 0) {
        s_stop = 1;
        *reinterpret_cast<volatile int*>(status) = 1;
      }
      give_up<BN>(y, EPI == STORE_SUMS ? sums : nullptr, s, tile, step, n0);
    } else if (EPI == STORE_SUMS) {
      // The slices are no longer in use: every product is done.
      float* red = reinterpret_cast<float*>(raw + (slices - smem_addr(raw)));
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        red[t / PIECES * BN + t % PIECES * 8 + k] = acc_sum[k];
        red[(ROW_STEP + t / PIECES) * BN + t % PIECES * 8 + k] = acc_sq[k];
      }
      epilogue_sync();
      double* mine = sums + static_cast<int64_t>(first % s.copies) * 2 * s.n + n0;
      for (int e = t; e < 2 * BN; e += EPILOGUE_THREADS) {
        const int which = e / BN, channel = e % BN;
        double sum = 0.0;
#pragma unroll 8
        for (int g = 0; g < ROW_STEP; ++g)
          sum += static_cast<double>(red[(which * ROW_STEP + g) * BN + channel]);
        atomicAdd(mine + static_cast<int64_t>(which) * s.n + channel, sum);
      }
    }
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 ::"r"(tmem), "n"(2 * BN));
}

template <typename T, int BN, bool W_MN, int EPI>
cudaError_t LaunchTyped(const Conv1x1& c, Shape s, cudaStream_t stream, int* status,
                        uint32_t wait_ns) {
  using L = Layout<BN, EPI>;
  s.tiles_n = c.n / BN;
  const bool strided = c.strided_x || c.strided_y;
  const int image_rows = strided ? TILE_M / c.width : 0;  // of pixels, in a tile
  s.tile_rows = strided ? image_rows * c.width : TILE_M;
  s.tiles_m = static_cast<int>((c.rows + s.tile_rows - 1) / s.tile_rows);
  Maps maps;
  auto dense = [&](CUtensorMap* map, const void* p, int channels) {
    return MakeMap(map, p, c.bf16, channels, c.rows, 1, channels, c.rows * channels, s.tile_rows,
                   1);
  };
  auto every_other = [&](CUtensorMap* map, const void* p, int channels) {
    return MakeMap(map, p, c.bf16, channels, c.width, c.rows / c.width, 2 * channels,
                   4ll * c.width * channels, c.width, image_rows);
  };
  s.x_step1 = c.strided_x ? 0 : s.tile_rows;
  s.x_step2 = c.strided_x ? image_rows : 0;
  s.y_step1 = c.strided_y ? 0 : s.tile_rows;
  s.y_step2 = c.strided_y ? image_rows : 0;
  s.width = c.strided_y ? c.width : 1;
  s.pitch_px = 2 * c.n;
  s.pitch_row = c.strided_y ? 4ll * c.width * c.n : c.n;
  bool ok = c.strided_x ? every_other(&maps.x, c.x, c.k) : dense(&maps.x, c.x, c.k);
  ok = ok && (c.strided_y ? every_other(&maps.y, c.y, c.n) : dense(&maps.y, c.y, c.n));
  if (EPI >= ADD)
    ok = ok && (c.strided_y ? every_other(&maps.add, c.add, c.n) : dense(&maps.add, c.add, c.n));
  else
    maps.add = maps.y;
  const int w_rows = W_MN ? c.k : c.n, w_cols = W_MN ? c.n : c.k;
  ok = ok && MakeMap(&maps.w, c.w, c.bf16, w_cols, w_rows, 1, w_cols,
                     static_cast<int64_t>(w_rows) * w_cols, W_MN ? SLICE_K : BN, 1);
  if (!ok) return cudaErrorInvalidValue;
  auto kernel = conv1x1_kernel<T, BN, W_MN, EPI>;
  // w stays in shared memory for all tiles of a CTA where three slices of x still fit
  // beside it: gradient of 1024 channels from 256 with the masked sum, 50176 rows, 53 us,
  // 62 with w read for every tile; of 256 from 64, 802816 rows, 147 to 152, 174 without.
  const int fixed = 1024 + L::BUFFERS * L::BUFFER, all_of_w = s.slices_k * L::W_SLICE;
  s.w_stays = fixed + all_of_w + 3 * BOX_BYTES <= MOST_BYTES;
  const int slice = BOX_BYTES + (s.w_stays ? 0 : L::W_SLICE);
  const int before = fixed + (s.w_stays ? all_of_w : 0);
  s.slots = (MOST_BYTES - before) / slice;
  if (s.slots > MOST_SLOTS) s.slots = MOST_SLOTS;
  const int bytes = before + s.slots * slice;
  const cudaError_t err =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (err != cudaSuccess) return err;
  int per_column = 148 / s.tiles_n;  // CTAs of a column of tiles
  if (per_column < 1) per_column = 1;
  if (per_column > s.tiles_m) per_column = s.tiles_m;
  CountKernelLaunches(1);
  kernel<<<per_column * s.tiles_n, THREADS, bytes, stream>>>(
      maps, s, c.signs, static_cast<uint16_t*>(c.y), c.sums, status, wait_ns);
  return cudaGetLastError();
}

template <typename T, int BN>
cudaError_t LaunchWidth(const Conv1x1& c, const Shape& s, cudaStream_t stream, int* status,
                        uint32_t wait_ns) {
  if (!c.w_transposed) return LaunchTyped<T, BN, false, STORE_SUMS>(c, s, stream, status, wait_ns);
  if constexpr (BN <= 128) {
    if (c.signs == nullptr) return LaunchTyped<T, BN, true, ADD>(c, s, stream, status, wait_ns);
    return LaunchTyped<T, BN, true, ADD_MASKED>(c, s, stream, status, wait_ns);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

bool Conv1x1Supported(int64_t rows, int k, int n) {
  return rows >= 1 && rows <= INT32_MAX - 256 && k >= 64 && n >= 64 && k % 64 == 0 &&
         n % 64 == 0 && k <= 65536 && n <= 65536;
}

bool Conv1x1StrideSupported(int64_t rows, int width) {
  return width >= 1 && width <= TILE_M && rows % width == 0;
}

cudaError_t LaunchConv1x1(const Conv1x1& c, cudaStream_t stream, uint32_t wait_ns) {
  if (!Conv1x1Supported(c.rows, c.k, c.n)) return cudaErrorInvalidValue;
  if ((c.strided_x || c.strided_y) && !Conv1x1StrideSupported(c.rows, c.width))
    return cudaErrorInvalidValue;
  // The forward has a batch norm behind it, the gradient something to add: PyTorch's
  // kernels cost less where they do not.
  if (c.w_transposed ? c.add == nullptr || c.sums != nullptr
                     : c.add != nullptr || c.signs != nullptr || c.sums == nullptr || c.copies < 1)
    return cudaErrorInvalidValue;
  if ((c.strided_x && c.strided_y) || (c.signs != nullptr && c.strided_y) || !TmaAvailable())
    return cudaErrorInvalidValue;
  // (The maps refuse what else is off its boundary.)
  if (reinterpret_cast<uintptr_t>(c.signs) % 4 != 0) return cudaErrorInvalidValue;
  int device = 0;
  const cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  int* status = TensorCoreStatusWord(device);
  if (status == nullptr) return cudaErrorMemoryAllocation;
  Shape s = {};
  s.rows = c.rows;
  s.n = c.n;
  s.slices_k = c.k / SLICE_K;
  s.copies = c.copies;
  const int64_t tiles_m = (c.rows + TILE_M - 1) / TILE_M;
  // Wider tiles read x less often, which is what the loop over k waits for: 50176 rows,
  // 256 to 1024 channels: 70, 43 and 39 us with 64, 128 and 256; 6272 rows, 1024 to 256:
  // 18, 14 and 16. Tiles of 256 want two for every SM (6272 rows, 256 to 1024: 12 us with
  // 128, 14 with 256). With a tile to add, 128 leaves room for three of them ahead.
  int width = 64;
  if (c.n % 128 == 0) width = 128;
  if (c.n % 256 == 0 && c.add == nullptr && tiles_m * (c.n / 256) >= 2 * 148) width = 256;
  if (c.bf16)
    return width == 256   ? LaunchWidth<__nv_bfloat16, 256>(c, s, stream, status, wait_ns)
           : width == 128 ? LaunchWidth<__nv_bfloat16, 128>(c, s, stream, status, wait_ns)
                          : LaunchWidth<__nv_bfloat16, 64>(c, s, stream, status, wait_ns);
  return width == 256   ? LaunchWidth<__half, 256>(c, s, stream, status, wait_ns)
         : width == 128 ? LaunchWidth<__half, 128>(c, s, stream, status, wait_ns)
                        : LaunchWidth<__half, 64>(c, s, stream, status, wait_ns);
}

}  // namespace kern
}  // namespace hvd
