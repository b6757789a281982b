// Backward of a wide batch norm and of the narrow-to-wide 1x1 convolution before it
// (the end of a residual block) in one kernel, channels-last, 16-bit: with
//   dz = dy where the block's output was above zero,
//   dx = scale * dz + kx * (x - centre) + kc     (batch norm; x: the convolution's output)
//   da = dx * W,   dW = dx^T * a                 (convolution; a: its input)
// dx, the widest tensor of the block, exists in shared memory only. Apart, its store
// and its two reads are 1.2 of the 2.3 GB that move per block of 802816 rows, 256
// and 64 channels.
//
// A persistent CTA takes tiles of 128 rows. Warp 0 copies dy, x and the signs into
// a ring of slots of a few rows, and tiles of a, by TMA; 16 warps form dx from a slot
// and store it to the tile; the same tile is the K-major operand of da (K: channels)
// and the MN-major one of dW (K: rows). dW stays in tensor memory over all tiles of the
// CTA and goes to `partial` ([CTA][cout][cin], fp32) at the end, where a second kernel
// adds it up in fp64. One thread of warp 1 issues the products, 4 warps round and store
// da. All channels of dx in one CTA, and all of dW in its tensor memory, are what
// limits the kernel to 256 wide and 64 narrow channels.
//
// Bound by the bytes of dy, x, a and da. 802816 rows, 256 and 64 channels, bf16, with
// the batch norm's sums: 359 to 361 us (290 for the bytes), of which this kernel takes 215;
// the kernels apart 345 and 167 to 180 (bench_kernels.py --case norm_conv). 2304
// rows: 24 us, apart 28. The copies alone take 320 us, with the forming of dx, but no
// products, 333. A tile of dx of its own for the products to work on while the
// next is formed leaves no room for the ring: with loads into registers instead, which
// wait for one another, it took 468 us.
//
// Waits are bounded. When one runs out, what the CTA had not finished becomes NaN,
// dW too, and TensorCoreStatusWord() of the device is set.
//
// The reference has no counterpart (it takes both layers from the framework).
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "batch_norm.cuh"
#include "kernels.h"
#include "tma.cuh"

namespace hvd {
namespace kern {

namespace {

constexpr int CIN = 64;
constexpr int EPILOGUE_WARP = 2, EPILOGUE_THREADS = 128;
constexpr int FORM_WARP = 6, FORM_THREADS = 512;
constexpr int THREADS = FORM_WARP * 32 + FORM_THREADS;
constexpr int SLOTS = 5;
constexpr uint16_t NAN16 = 0x7fff;

struct Maps {
  CUtensorMap w, a;
};

struct Args {
  const uint16_t* dy;
  const uint8_t* signs;
  const uint16_t* x;
  uint16_t* da;  // null: not wanted
  const double* sums;
  const float *gamma, *saved;
  float *dgamma, *dbeta, *partial;
  int64_t rows;
  int tiles, copies;
  int* status;
  uint32_t wait_ns;
};

template <int COUT> struct Layout {
  static constexpr int WIDE = COUT / 64 * BOX_BYTES;  // a tile of dx
  static constexpr int W = COUT * 128;
  // A thread forms 8 channels of one row of a slot: dy, x and signs of the rows.
  static constexpr int SLOT_ROWS = FORM_THREADS / (COUT / VEC);
  static constexpr int SLOT_X = SLOT_ROWS * COUT * 2, SLOT_SIGNS = 2 * SLOT_X;
  static constexpr int SLOT = 2 * SLOT_X + SLOT_ROWS * COUT / 8;
  static constexpr int BYTES = 1024 + WIDE + 2 * BOX_BYTES + W + SLOTS * SLOT;
};

// `bytes` (a multiple of 16) of contiguous memory.
__device__ __forceinline__ void load_bytes(uint32_t to, const void* from, uint32_t bytes,
                                           uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      ::"r"(to), "l"(from), "r"(bytes), "r"(bar) : "memory");
}
template <int ID> __device__ __forceinline__ bool all_of(bool ok, int threads) {
  uint32_t all;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.and.pred q, %3, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
      : "=r"(all) : "r"(ok ? 1u : 0u), "r"(threads), "n"(ID) : "memory");
  return all != 0;
}

template <typename T, int COUT>
__global__ void __launch_bounds__(THREADS, 1)
norm_conv_backward_kernel(const __grid_constant__ Maps maps, const __grid_constant__ Args p) {
  using L = Layout<COUT>;
  constexpr bool BF16 = std::is_same<T, __nv_bfloat16>::value;
  constexpr int GROUPS = COUT / VEC;                       // threads per row
  constexpr int BLOCKS_M = COUT / 128;                     // of dW
  constexpr uint32_t COLUMNS = 2 * CIN + BLOCKS_M * CIN > 128 ? 256 : 128;
  extern __shared__ unsigned char raw[];
  __shared__ __align__(16) float s_scale[COUT], s_kx[COUT], s_kc[COUT], s_centre[COUT];
  __shared__ __align__(8) uint64_t s_w_full, s_dx_full[2], s_dx_empty, s_a_full[2], s_a_empty[2],
      s_acc_full[2], s_acc_empty[2], s_slot_full[SLOTS], s_slot_empty[SLOTS], s_done;
  __shared__ uint32_t s_tmem;
  __shared__ volatile int s_stop;
  const uint32_t wide = (smem_addr(raw) + 1023u) & ~1023u;
  const uint32_t narrow = wide + L::WIDE, weights = narrow + 2 * BOX_BYTES,
                 slots = weights + L::W;
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  // From the last rows to the first: the kernel before this one read the last ones
  // last, and they are still in L2.
  const int tiles = (p.tiles - static_cast<int>(blockIdx.x) + gridDim.x - 1) / gridDim.x;
  auto tile_of = [&](int i) {
    return p.tiles - 1 - static_cast<int>(blockIdx.x) - i * static_cast<int>(gridDim.x);
  };

  if (threadIdx.x == 0) {
    auto init = [](uint64_t* bar, int count) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;"
                   ::"r"(smem_addr(bar)), "r"(count) : "memory");
    };
    for (int i = 0; i < 2; ++i) {
      init(s_a_full + i, 1);
      init(s_a_empty + i, 1);
      init(s_acc_full + i, 1);
      init(s_acc_empty + i, EPILOGUE_THREADS / 32);
    }
    for (int i = 0; i < SLOTS; ++i) init(s_slot_full + i, 1), init(s_slot_empty + i, FORM_THREADS / 32);
    for (int i = 0; i < 2; ++i) init(s_dx_full + i, FORM_THREADS / 32);  // halves of the rows
    init(&s_dx_empty, 1);
    init(&s_w_full, 1);
    init(&s_done, 1);
    s_stop = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_addr(&s_tmem)), "n"(COLUMNS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  wait_for_previous();
  for (int ch = threadIdx.x; ch < COUT; ch += THREADS) {
    const BackwardTerms b = backward_terms<T>(p.sums, COUT, p.copies, ch,
                                              1.0 / static_cast<double>(p.rows), p.gamma, p.saved);
    s_scale[ch] = b.scale;
    s_kx[ch] = b.kx;
    s_kc[ch] = b.kc;
    s_centre[ch] = b.centre;
    if (blockIdx.x == 0) {
      p.dgamma[ch] = static_cast<float>(b.dz_xhat);
      p.dbeta[ch] = static_cast<float>(b.dz);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem, tmem_dw = tmem + 2 * CIN;

  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      expect_bytes(smem_addr(&s_w_full), L::W);
      // Boxes of 128 rows of W; one after the other, they are rows of 128 bytes.
#pragma unroll
      for (int j = 0; j < COUT / 128; ++j)
        load_box(weights + j * BOX_BYTES, &maps.w, 0, j * 128, 0, smem_addr(&s_w_full));
      int a_tiles = 0;
      uint32_t n = 0;  // slots
      for (int i = 0; ok && i < tiles; ++i) {
        const int64_t first = static_cast<int64_t>(tile_of(i)) * TILE_M;
        ok = wait_or_stop(smem_addr(&s_a_empty[i & 1]), (i >> 1 & 1) ^ 1, p.wait_ns, &s_stop);
        if (!ok) break;
        expect_bytes(smem_addr(&s_a_full[i & 1]), BOX_BYTES);
        load_box(narrow + (i & 1) * BOX_BYTES, &maps.a, 0, tile_of(i) * TILE_M, 0,
                 smem_addr(&s_a_full[i & 1]));
        ++a_tiles;
        for (int r = 0; r < TILE_M; r += L::SLOT_ROWS, ++n) {
          const uint32_t slot = n % SLOTS, to = slots + slot * L::SLOT,
                         bar = smem_addr(&s_slot_full[slot]);
          ok = wait_or_stop(smem_addr(&s_slot_empty[slot]), (n / SLOTS & 1) ^ 1, p.wait_ns,
                            &s_stop);
          if (!ok) break;
          // (Rows past the end are no copies: of a slot of those, the barrier alone.)
          const int64_t left = p.rows - first - r;
          const uint32_t rows = left < 0 ? 0u : left < L::SLOT_ROWS ? left : L::SLOT_ROWS;
          expect_bytes(bar, rows * (2 * COUT * 2 + COUT / 8));
          if (rows > 0) {
            const int64_t at = (first + r) * COUT;
            load_bytes(to, p.dy + at, rows * COUT * 2, bar);
            load_bytes(to + L::SLOT_X, p.x + at, rows * COUT * 2, bar);
            load_bytes(to + L::SLOT_SIGNS, p.signs + at / 8, rows * COUT / 8, bar);
          }
        }
      }
      if (!ok) s_stop = 1;
      // No copy may be in flight when the CTA ends.
      wait_bounded(smem_addr(&s_w_full), 0, STEM_WAIT_NS);
      for (uint32_t u = n < SLOTS ? 0 : n - SLOTS; u < n; ++u)
        wait_bounded(smem_addr(&s_slot_full[u % SLOTS]), u / SLOTS & 1, STEM_WAIT_NS);
      for (int u = a_tiles < 2 ? 0 : a_tiles - 2; u < a_tiles; ++u)
        wait_bounded(smem_addr(&s_a_full[u & 1]), u >> 1 & 1, STEM_WAIT_NS);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t to_da = instruction(BF16, false, true, TILE_M, CIN);
      constexpr uint32_t to_dw = instruction(BF16, true, true, 128, CIN);
      ok = wait_or_stop(smem_addr(&s_w_full), 0, p.wait_ns, &s_stop);
      for (int i = 0; ok && i < tiles; ++i) {
        const uint32_t b = i & 1, phase = i >> 1 & 1, dx = wide, a = narrow + b * BOX_BYTES;
        auto add_dw = [&](int half) {
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int m = 0; m < BLOCKS_M; ++m)
#pragma unroll
            for (int j = 0; j < TILE_M / 32; ++j) {
              const int k = half * (TILE_M / 32) + j;  // 16 rows
              mma(tmem_dw + m * CIN,
                  operand_swizzled(dx + m * 2 * BOX_BYTES + k * 2048, BOX_BYTES),
                  operand_swizzled(a + k * 2048, 0), to_dw, i > 0 || k > 0);
            }
        };
        // The first half of the rows goes into dW while the second one is formed.
        ok = wait_or_stop(smem_addr(&s_a_full[b]), phase, p.wait_ns, &s_stop) &&
             wait_or_stop(smem_addr(&s_dx_full[0]), i & 1, p.wait_ns, &s_stop);
        if (!ok) break;
        add_dw(0);
        ok = wait_or_stop(smem_addr(&s_dx_full[1]), i & 1, p.wait_ns, &s_stop) &&
             (p.da == nullptr ||
              wait_or_stop(smem_addr(&s_acc_empty[b]), phase ^ 1, p.wait_ns, &s_stop));
        if (!ok) break;
        add_dw(1);
        if (p.da != nullptr) {
#pragma unroll
          for (int k = 0; k < COUT / 16; ++k)
            mma(tmem + b * CIN, operand_swizzled(dx + k / 4 * BOX_BYTES + k % 4 * 32, 16),
                operand_swizzled(weights + k * 2048, 0), to_da, k > 0);
          commit(smem_addr(&s_acc_full[b]));
        }
        commit(smem_addr(&s_a_empty[b]));
        commit(smem_addr(&s_dx_empty));
      }
      if (!ok) s_stop = 1;
      commit(smem_addr(&s_done));
      wait_bounded(smem_addr(&s_done), 0, STEM_WAIT_NS);
    }
  } else if (warp >= FORM_WARP) {
    const int t = threadIdx.x - FORM_WARP * 32, group = t % GROUPS, row0 = t / GROUPS;
    float scale[VEC], kx[VEC], kc[VEC], centre[VEC];
#pragma unroll
    for (int k = 0; k < VEC; ++k) {
      scale[k] = s_scale[group * VEC + k];
      kx[k] = s_kx[group * VEC + k];
      kc[k] = s_kc[group * VEC + k];
      centre[k] = s_centre[group * VEC + k];
    }
    const uint32_t to = wide + piece_at(row0, group);
    uint32_t n = 0;
    for (int i = 0; ok && i < tiles; ++i) {
      const int64_t left = p.rows - static_cast<int64_t>(tile_of(i)) * TILE_M - row0;
      for (int r0 = 0; r0 < TILE_M; r0 += L::SLOT_ROWS, ++n) {
        const uint32_t slot = n % SLOTS, from = slots + slot * L::SLOT;
        ok = wait_or_stop(smem_addr(&s_slot_full[slot]), n / SLOTS & 1, p.wait_ns, &s_stop);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint4 d = load_piece(from + t * 16), x = load_piece(from + L::SLOT_X + t * 16);
        uint32_t byte;
        asm volatile("ld.shared.u8 %0, [%1];"
                     : "=r"(byte) : "r"(from + L::SLOT_SIGNS + t) : "memory");
        __syncwarp();
        if (lane == 0) arrive(smem_addr(&s_slot_empty[slot]));
        const uint32_t signs = spread_signs(byte);
        const uint32_t dw[4] = {d.x, d.y, d.z, d.w}, xw[4] = {x.x, x.y, x.z, x.w};
        uint32_t o[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float2 z = widen2<T>(dw[k] & ((signs >> k & 0x00010001u) * 0xffffu));
          const float2 f = widen2<T>(xw[k]);
          const int c = 2 * k;
          o[k] = narrow2<T>(
              fmaf(scale[c], z.x, fmaf(kx[c], f.x - centre[c], kc[c])),
              fmaf(scale[c + 1], z.y, fmaf(kx[c + 1], f.y - centre[c + 1], kc[c + 1])));
        }
        uint4 v = make_uint4(o[0], o[1], o[2], o[3]);
        // Rows past the end (whatever the slot holds there) are zeros.
        if (left <= r0) v = make_uint4(0u, 0u, 0u, 0u);
        if (r0 == 0) {  // the products of the tile before
          ok = wait_or_stop(smem_addr(&s_dx_empty), (i & 1) ^ 1, p.wait_ns, &s_stop);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
        store_piece(to + r0 * 128, v);
        const int done = r0 + L::SLOT_ROWS;
        if (done == TILE_M / 2 || done == TILE_M) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) arrive(smem_addr(&s_dx_full[done / TILE_M]));
        }
      }
    }
    if (!ok) s_stop = 1;
    // (The MMA thread is told by s_stop.)
  } else if (warp >= EPILOGUE_WARP) {
    const int row = warp % 4 * 32 + lane;
    int i = 0;
    for (; p.da != nullptr && i < tiles; ++i) {
      const uint32_t b = i & 1;
      ok = wait_or_stop(smem_addr(&s_acc_full[b]), i >> 1 & 1, p.wait_ns, &s_stop);
      ok = all_of<2>(ok, EPILOGUE_THREADS);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // A thread's row is 128 contiguous bytes of da, four sectors.
      const int64_t at = static_cast<int64_t>(tile_of(i)) * TILE_M + row;
      uint16_t* out = p.da + at * CIN;
#pragma unroll
      for (int c = 0; c < CIN; c += 32) {
        uint32_t r[32];
        load_accumulators(tmem + (static_cast<uint32_t>(warp % 4 * 32) << 16) + b * CIN + c, r);
        if (c + 32 == CIN) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          if (lane == 0) arrive(smem_addr(&s_acc_empty[b]));
        }
        if (at >= p.rows) continue;
#pragma unroll
        for (int k = 0; k < 32; k += 16) {
          uint32_t o[8];
#pragma unroll
          for (int j = 0; j < 8; ++j)
            o[j] = narrow2<T>(__uint_as_float(r[k + 2 * j]), __uint_as_float(r[k + 2 * j + 1]));
          asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                       ::"l"(out + c + k), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]),
                       "r"(o[5]), "r"(o[6]), "r"(o[7]) : "memory");
        }
      }
    }
    if (!ok) {
      s_stop = 1;
      for (; i < tiles; ++i)
        for (int e = threadIdx.x - EPILOGUE_WARP * 32; e < TILE_M * CIN; e += EPILOGUE_THREADS) {
          const int64_t r = static_cast<int64_t>(tile_of(i)) * TILE_M + e / CIN;
          if (r < p.rows) p.da[r * CIN + e % CIN] = NAN16;
        }
    }
  }
  __syncwarp();
  // Every product is done: the MMA thread waited for them.
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  const bool all_ok = __syncthreads_and(ok && s_stop == 0) != 0;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!all_ok && threadIdx.x == 0) *reinterpret_cast<volatile int*>(p.status) = 1;
  // dW: the epilogue's warps, a block of 128 rows after the other.
  if (warp >= EPILOGUE_WARP && warp < FORM_WARP) {
#pragma unroll
    for (int m = 0; m < BLOCKS_M; ++m) {
      float* out = p.partial + (static_cast<int64_t>(blockIdx.x) * COUT + m * 128 +
                                warp % 4 * 32 + lane) * CIN;
#pragma unroll
      for (int c = 0; c < CIN; c += 32) {
        uint32_t r[32];
        load_accumulators(tmem_dw + (static_cast<uint32_t>(warp % 4 * 32) << 16) + m * CIN + c, r);
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
          const uint4 v = make_uint4(r[k], r[k + 1], r[k + 2], r[k + 3]);
          *reinterpret_cast<uint4*>(out + c + k) =
              all_ok ? v : make_uint4(0x7fffffffu, 0x7fffffffu, 0x7fffffffu, 0x7fffffffu);
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 ::"r"(tmem), "n"(COLUMNS));
}

// dW = sum of the CTAs' parts, in fp64. Bound by the latency of the loads: 8 threads
// to a value, and the loads of each independent.
constexpr int SUM_THREADS = 256, SUM_SLICES = 8;
template <typename T>
__global__ void __launch_bounds__(SUM_THREADS)
sum_partials_kernel(const float* __restrict__ partial, T* __restrict__ dw, int parts, int values,
                    int cin, int64_t stride_o, int64_t stride_i) {
  __shared__ double sums[SUM_SLICES][SUM_THREADS / SUM_SLICES];
  const int at = threadIdx.x % (SUM_THREADS / SUM_SLICES), slice = threadIdx.x / (SUM_THREADS / SUM_SLICES);
  const int e = blockIdx.x * (SUM_THREADS / SUM_SLICES) + at;
  double sum = 0.0;
#pragma unroll 8
  for (int i = slice; i < parts; i += SUM_SLICES)
    sum += static_cast<double>(__ldg(partial + static_cast<int64_t>(i) * values + e));
  sums[slice][at] = sum;
  __syncthreads();
  if (slice == 0) {
    for (int i = 1; i < SUM_SLICES; ++i) sum += sums[i][at];
    dw[e / cin * stride_o + e % cin * stride_i] = static_cast<T>(static_cast<float>(sum));
  }
}

template <typename T, int COUT>
cudaError_t LaunchTyped(const NormConvBackward& n, cudaStream_t stream, int* status,
                        uint32_t wait_ns) {
  using L = Layout<COUT>;
  Args p;
  p.dy = static_cast<const uint16_t*>(n.dy);
  p.signs = n.signs;
  p.x = static_cast<const uint16_t*>(n.x);
  p.da = static_cast<uint16_t*>(n.da);
  p.sums = n.sums;
  p.copies = BatchNormCopies(COUT);
  p.gamma = n.gamma;
  p.saved = n.saved;
  p.dgamma = n.dgamma;
  p.dbeta = n.dbeta;
  p.partial = n.partial;
  p.rows = n.rows;
  p.tiles = static_cast<int>((n.rows + TILE_M - 1) / TILE_M);
  p.status = status;
  p.wait_ns = wait_ns;
  Maps maps;
  const bool ok = MakeMap(&maps.w, n.w, n.bf16, CIN, COUT, 1, CIN, COUT * CIN, 128, 1) &&
            MakeMap(&maps.a, n.a, n.bf16, CIN, n.rows, 1, CIN, n.rows * CIN, TILE_M, 1);
  if (!ok) return cudaErrorInvalidValue;
  auto kernel = norm_conv_backward_kernel<T, COUT>;
  cudaError_t err =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::BYTES);
  if (err != cudaSuccess) return err;
  const int parts = NormConvBackwardParts(n.rows);
  CountKernelLaunches(2);
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(static_cast<unsigned>(parts));
  config.blockDim = dim3(THREADS);
  config.dynamicSmemBytes = L::BYTES;
  config.stream = stream;
  config.attrs = &attr;
  config.numAttrs = 1;
  err = cudaLaunchKernelEx(&config, kernel, static_cast<const Maps>(maps),
                           static_cast<const Args>(p));
  if (err != cudaSuccess) return err;
  constexpr int VALUES = COUT * CIN, PER_CTA = SUM_THREADS / SUM_SLICES;
  if (n.dw_fp32)
    sum_partials_kernel<float><<<VALUES / PER_CTA, SUM_THREADS, 0, stream>>>(
        n.partial, static_cast<float*>(n.dw), parts, VALUES, CIN, n.dw_stride_o, n.dw_stride_i);
  else
    sum_partials_kernel<T><<<VALUES / PER_CTA, SUM_THREADS, 0, stream>>>(
        n.partial, static_cast<T*>(n.dw), parts, VALUES, CIN, n.dw_stride_o, n.dw_stride_i);
  return cudaGetLastError();
}

}  // namespace

bool NormConvBackwardSupported(int64_t rows, int cout, int cin) {
  return rows >= 1 && rows <= INT32_MAX - 256 && cin == CIN && (cout == 128 || cout == 256);
}

int NormConvBackwardParts(int64_t rows) {
  const int64_t tiles = (rows + TILE_M - 1) / TILE_M;
  return tiles < 148 ? static_cast<int>(tiles) : 148;
}

cudaError_t LaunchNormConvBackward(const NormConvBackward& n, cudaStream_t stream,
                                   uint32_t wait_ns) {
  if (!NormConvBackwardSupported(n.rows, n.cout, n.cin)) return cudaErrorInvalidValue;
  // What is copied, loaded and stored in 16 (da: 32) bytes at a time.
  for (const void* p : {n.dy, n.x, n.a, n.w, static_cast<const void*>(n.signs),
                        static_cast<const void*>(n.saved), static_cast<const void*>(n.partial)})
    if (reinterpret_cast<uintptr_t>(p) % 16 != 0) return cudaErrorInvalidValue;
  if (reinterpret_cast<uintptr_t>(n.da) % 32 != 0) return cudaErrorInvalidValue;
  int device = 0;
  cudaError_t err = cudaGetDevice(&device);
  if (err != cudaSuccess) return err;
  int* status = TensorCoreStatusWord(device);
  if (status == nullptr) return cudaErrorMemoryAllocation;
  if (!n.summed)
    err = LaunchBatchNormBackwardSums(n.dy, n.signs, n.x, n.rows, n.cout, n.bf16, n.sums, n.gamma,
                                      n.saved, stream);
  if (err != cudaSuccess) return err;
  if (n.bf16)
    return n.cout == 256 ? LaunchTyped<__nv_bfloat16, 256>(n, stream, status, wait_ns)
                         : LaunchTyped<__nv_bfloat16, 128>(n, stream, status, wait_ns);
  return n.cout == 256 ? LaunchTyped<__half, 256>(n, stream, status, wait_ns)
                       : LaunchTyped<__half, 128>(n, stream, status, wait_ns);
}

}  // namespace kern
}  // namespace hvd
