// Training-mode batch normalisation for channels-last (NHWC) 16-bit
// activations, fused with what surrounds it in a residual network:
//   forward : statistics -> y = relu(x * scale + shift [+ residual])
//   backward: dz = dy * (y > 0); per-channel sum(dz), sum(dz * xhat);
//             dx = scale * (dz - sum(dz)/M - xhat * sum(dz*xhat)/M); dres = dz
// The tensor is treated as a row-major [M = N*H*W, C] matrix. A thread owns 8
// consecutive channels (one 16-byte access per row), a warp covers 256
// consecutive channels of one row (or several rows when C is smaller), so every
// access is a fully coalesced 512-byte line. Each pass is bound by HBM traffic:
// the forward reads x twice and writes y once (the PyTorch eager sequence
// batch_norm + add + relu makes eight passes), the backward reads dy and x
// twice and writes dx (and dres). The backward never reads y: without a
// residual, y > 0 follows from x and the saved scale and shift by the
// forward's own arithmetic; with one, the forward leaves one bit per element.
//
// Of 256 x 256 x 56 x 56 with a residual in bf16 (411 MB a tensor) the four
// kernels take 70, 204, 138 and 270 us on a B200, 0.92-0.94 of the rate of a
// plain copy of the bytes they move; with the output read back 78, 204, 194 and
// 336 us.
//
// The second kernel of a pair walks the rows from the last to the first, so
// what the first kernel read last is still in L2 when the second one starts,
// and is launched while the first one still runs (programmatic dependent
// launch), which hides its launch latency.
//
// Per-channel sums are accumulated in fp32 per thread (a few dozen groups of
// rows), in fp64 across the warps of a CTA and across CTAs (atomicAdd on
// doubles), then mean/variance are formed in fp64. Additions to one address
// follow each other at about 18 ns, so the CTAs share several copies of the
// accumulators (bn_copies) and the second kernel adds those up.
//
// The reference has no counterpart: it takes batch normalisation from the
// framework (horovod/torch/sync_batch_norm.py:98-199 calls
// torch.batch_norm_stats / batch_norm_elemt / batch_norm_backward_reduce).
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "batch_norm.cuh"
#include "kernels.h"

namespace hvd {
namespace kern {

namespace {

constexpr int BN_THREADS = 256;
// Resident CTAs per SM the compiler must leave room for (register budget):
// these are streaming kernels whose throughput is set by the bytes in flight
// per SM, i.e. by occupancy.
constexpr int BN_MIN_BLOCKS = 3;        // <= 85 registers per thread
constexpr int BN_MIN_BLOCKS_STATS = 4;  // <= 64 registers per thread
constexpr int UNROLL = 4;  // rows in flight per thread

// Two channels per 32-bit word.
template <typename T> struct Pair;
template <> struct Pair<__nv_bfloat16> {
  using type = __nv_bfloat162;
  static __device__ __forceinline__ float2 widen(type v) { return __bfloat1622float2(v); }
  static __device__ __forceinline__ type narrow(float a, float b) {
    return __floats2bfloat162_rn(a, b);
  }
};
template <> struct Pair<__half> {
  using type = __half2;
  static __device__ __forceinline__ float2 widen(type v) { return __half22float2(v); }
  static __device__ __forceinline__ type narrow(float a, float b) {
    return __floats2half2_rn(a, b);
  }
};

// 8 channels of one row.
template <typename T> struct Vec8 {
  using P = typename Pair<T>::type;
  uint32_t w[VEC / 2];
  __device__ __forceinline__ P pair(int i) const { return *reinterpret_cast<const P*>(&w[i]); }
  __device__ __forceinline__ void set(int i, P v) { w[i] = *reinterpret_cast<uint32_t*>(&v); }
};

template <typename T> __device__ __forceinline__ Vec8<T> ldg16(const T* p) {
  Vec8<T> v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]) : "l"(p));
  return v;
}
template <typename T> __device__ __forceinline__ void stg16(T* p, const Vec8<T>& v) {
  asm volatile("st.global.v4.u32 [%0], {%1,%2,%3,%4};" ::"l"(p), "r"(v.w[0]), "r"(v.w[1]),
               "r"(v.w[2]), "r"(v.w[3]) : "memory");
}
// The signs of 8 outputs in one byte: the even channels in the low nibble, the
// odd ones in the high nibble. `positive` holds an all-ones half word for each
// channel whose output is above zero.
__device__ __forceinline__ uint32_t pack_signs(const uint32_t (&positive)[VEC / 2]) {
  const uint32_t t = (positive[0] & 0x00010001u) | (positive[1] & 0x00020002u) |
                     (positive[2] & 0x00040004u) | (positive[3] & 0x00080008u);
  return (t | (t >> 12)) & 0xffu;
}
// Thread geometry shared by all four kernels.
struct Tile {
  int txg;        // channel groups (of 8 channels) per CTA along x: min(C/8, 32)
  int ty;         // rows handled in parallel by a CTA: BN_THREADS / txg
  int tx, row;    // this thread's position
  int64_t group;  // global channel group of this thread
  __device__ __forceinline__ Tile(int C) {
    const int cg = C / VEC;
    txg = cg < 32 ? cg : 32;
    ty = BN_THREADS / txg;
    tx = threadIdx.x % txg;
    row = threadIdx.x / txg;
    group = static_cast<int64_t>(blockIdx.x) * txg + tx;
  }
};

// Rows [r0, r1) of CTA `by`.
__device__ __forceinline__ void cta_rows(int64_t M, int by, int64_t* r0, int64_t* r1) {
  const int64_t per = (M + gridDim.y - 1) / gridDim.y;
  *r0 = min(by * per, M);
  *r1 = min(*r0 + per, M);
}

// Calls rows(U or 1, at): at is the element of the thread's first row, the
// others lie t.ty rows further on (for_rows) or back (for_rows_back) each.
template <int U, typename F>
__device__ __forceinline__ void for_rows(const Tile& t, int64_t r0, int64_t r1, int C, F rows) {
  const int64_t stride = static_cast<int64_t>(t.ty) * C;
  int64_t at = (r0 + t.row) * C + t.group * VEC;
  int64_t left = r1 - r0 - t.row;
  for (; left > (U - 1) * t.ty; left -= U * t.ty, at += U * stride)
    rows(std::integral_constant<int, U>(), at);
  for (; left > 0; left -= t.ty, at += stride) rows(std::integral_constant<int, 1>(), at);
}
template <int U, typename F>
__device__ __forceinline__ void for_rows_back(const Tile& t, int64_t r0, int64_t r1, int C,
                                              F rows) {
  const int64_t stride = static_cast<int64_t>(t.ty) * C;
  int64_t at = (r1 - 1 - t.row) * C + t.group * VEC;
  int64_t left = r1 - r0 - t.row;
  for (; left > (U - 1) * t.ty; left -= U * t.ty, at -= U * stride)
    rows(std::integral_constant<int, U>(), at);
  for (; left > 0; left -= t.ty, at -= stride) rows(std::integral_constant<int, 1>(), at);
}

// Sums `acc` (N values per channel of the thread) over the threads of the
// CTA that own the same channel group and adds the totals to the fp64
// accumulators: pairwise by shuffles inside a warp, in fp64 across warps.
// sums: [copies][2][C]; CTA y adds to copy y % copies. Of three values, the first and
// the third go to `more`.
template <int N>
__device__ __forceinline__ void reduce_to_global(const Tile& t, float (&acc)[N][VEC], int C,
                                                 int copies, double* sums,
                                                 double* more = nullptr) {
  constexpr int WARPS = BN_THREADS / 32;
  // Rows of 36 words: the threads of a warp, which read 8 rows of 4 words
  // below, hit 32 different banks.
  __shared__ float red[WARPS][N * VEC][36];
  for (int lanes = 16; lanes >= t.txg; lanes >>= 1) {
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < VEC; ++i) acc[k][i] += __shfl_xor_sync(0xffffffffu, acc[k][i], lanes);
  }
  const int warp = threadIdx.x / 32;
  if (static_cast<int>(threadIdx.x % 32) < t.txg) {
#pragma unroll
    for (int k = 0; k < N; ++k)
#pragma unroll
      for (int i = 0; i < VEC; ++i) red[warp][k * VEC + i][t.tx] = acc[k][i];
  }
  __syncthreads();
  const int64_t mine = static_cast<int64_t>(blockIdx.y % copies) * 2 * C +
                       static_cast<int64_t>(blockIdx.x) * t.txg * VEC;
  // N * VEC * txg <= 256 N totals, N rounds of 256 threads at most.
  for (int idx = threadIdx.x; idx < t.txg * N * VEC; idx += BN_THREADS) {
    const int i = idx % VEC, tx = idx / VEC % t.txg, k = idx / VEC / t.txg;
    double sum = 0.0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) sum += static_cast<double>(red[w][k * VEC + i][tx]);
    const int64_t at = mine + tx * VEC + i;
    if (k < 2) atomicAdd(sums + at + static_cast<int64_t>(k) * C, sum);
    if (N == 3 && k != 1) atomicAdd(more + at + (k == 2 ? C : 0), sum);
  }
}

template <typename T>
__global__ void __launch_bounds__(BN_THREADS, BN_MIN_BLOCKS_STATS)
bn_stats_kernel(const T* __restrict__ x, int64_t M, int C, int copies,
                double* __restrict__ sums) {
  const Tile t(C);
  int64_t r0, r1;
  cta_rows(M, blockIdx.y, &r0, &r1);
  float acc[2][VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) acc[0][i] = acc[1][i] = 0.f;
  const int64_t stride = static_cast<int64_t>(t.ty) * C;
  for_rows<UNROLL>(t, r0, r1, C, [&](auto count, int64_t at) {
    constexpr int U = decltype(count)::value;
    Vec8<T> v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = ldg16(x + at + u * stride);
    // The rows of one round are summed among themselves first: a quarter of
    // the additions into the long-running sums.
#pragma unroll
    for (int i = 0; i < VEC / 2; ++i) {
      float2 s = make_float2(0.f, 0.f), q = make_float2(0.f, 0.f);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float2 f = Pair<T>::widen(v[u].pair(i));
        s.x += f.x;
        s.y += f.y;
        q.x = fmaf(f.x, f.x, q.x);
        q.y = fmaf(f.y, f.y, q.y);
      }
      acc[0][2 * i] += s.x;
      acc[0][2 * i + 1] += s.y;
      acc[1][2 * i] += q.x;
      acc[1][2 * i + 1] += q.y;
    }
  });
  start_next();
  reduce_to_global(t, acc, C, copies, sums);
}

// Most channels of a CTA. Their per-channel values are formed by one thread
// each: in every thread, the fp64 arithmetic would take longer than the rows of
// a small tensor.
constexpr int BN_CTA_CHANNELS = 32 * VEC;

// relu(x * scale + shift [+ residual]) of 8 channels.
template <typename T, bool RELU, bool RES>
__device__ __forceinline__ Vec8<T> normalise(const Vec8<T>& x, const Vec8<T>& res,
                                             const float (&scale)[VEC], const float (&shift)[VEC]) {
  Vec8<T> o;
#pragma unroll
  for (int i = 0; i < VEC / 2; ++i) {
    const float2 a = Pair<T>::widen(x.pair(i));
    float2 f = make_float2(fmaf(a.x, scale[2 * i], shift[2 * i]),
                           fmaf(a.y, scale[2 * i + 1], shift[2 * i + 1]));
    if (RES) {
      const float2 b = Pair<T>::widen(res.pair(i));
      f.x += b.x;
      f.y += b.y;
    }
    typename Pair<T>::type v = Pair<T>::narrow(f.x, f.y);
    if (RELU) v = __hmax2(v, Pair<T>::narrow(0.f, 0.f));
    o.set(i, v);
  }
  return o;
}

__device__ __forceinline__ void load8(const float* p, float (&v)[VEC]) {
  const float4 a = *reinterpret_cast<const float4*>(p);
  const float4 b = *reinterpret_cast<const float4*>(p + 4);
  v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
  v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

// What a channel of x is multiplied with, and what is added. The first CTA of a
// column also writes `saved` (rows mean, invstd and shift of [3, C]) and the running
// statistics.
struct ForwardTerms {
  float scale, shift;
};
__device__ __forceinline__ ForwardTerms forward_terms(const BatchNormForward& n, int64_t M, int C,
                                                      double inv_m, int copies, int64_t ch,
                                                      bool first) {
  const double2 sum = total(n.sums, C, copies, ch);
  const double m = sum.x * inv_m;
  double var = sum.y * inv_m - m * m;
  if (var < 0.0) var = 0.0;
  const float mean = static_cast<float>(m);
  const float invstd = static_cast<float>(rsqrt(var + static_cast<double>(n.eps)));
  const float scale = (n.weight ? n.weight[ch] : 1.f) * invstd;
  const float shift = (n.bias ? n.bias[ch] : 0.f) - mean * scale;
  if (first) {
    n.saved[ch] = mean;
    n.saved[C + ch] = invstd;
    n.saved[2 * static_cast<int64_t>(C) + ch] = shift;
    if (n.running_mean != nullptr) {
      const double unbiased =
          M > 1 ? var * static_cast<double>(M) / static_cast<double>(M - 1) : var;
      n.running_mean[ch] = (1.f - n.momentum) * n.running_mean[ch] + n.momentum * mean;
      n.running_var[ch] =
          (1.f - n.momentum) * n.running_var[ch] + n.momentum * static_cast<float>(unbiased);
    }
  }
  return {scale, shift};
}

template <typename T, bool RELU, bool RES>
__global__ void __launch_bounds__(BN_THREADS, BN_MIN_BLOCKS)
bn_apply_kernel(const T* __restrict__ x, const T* __restrict__ res, T* __restrict__ y,
                uint8_t* __restrict__ signs, int64_t M, int C, double inv_m, int copies,
                const BatchNormForward n) {
  const Tile t(C);
  const int by = gridDim.y - 1 - blockIdx.y;
  int64_t r0, r1;
  cta_rows(M, by, &r0, &r1);
  __shared__ __align__(16) float s_scale[BN_CTA_CHANNELS];
  __shared__ __align__(16) float s_shift[BN_CTA_CHANNELS];
  wait_for_previous();
  if (n.batches != nullptr && by == 0 && blockIdx.x == 0 && threadIdx.x == 0) *n.batches += 1;
  if (static_cast<int>(threadIdx.x) < t.txg * VEC) {
    const int64_t ch = static_cast<int64_t>(blockIdx.x) * t.txg * VEC + threadIdx.x;
    const ForwardTerms f = forward_terms(n, M, C, inv_m, copies, ch, by == 0);
    s_scale[threadIdx.x] = f.scale;
    s_shift[threadIdx.x] = f.shift;
  }
  __syncthreads();
  float scale[VEC], shift[VEC];
  load8(s_scale + t.tx * VEC, scale);
  load8(s_shift + t.tx * VEC, shift);
  const int64_t stride = static_cast<int64_t>(t.ty) * C;
  for_rows_back<UNROLL>(t, r0, r1, C, [&](auto count, int64_t at0) {
    constexpr int U = decltype(count)::value;
    Vec8<T> a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = ldg16(x + at0 - u * stride);
      if (RES) b[u] = ldg16(res + at0 - u * stride);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t at = at0 - u * stride;
      const Vec8<T> o = normalise<T, RELU, RES>(a[u], b[u], scale, shift);
      stg16(y + at, o);
      if (RELU && RES) {
        uint32_t positive[VEC / 2];
#pragma unroll
        for (int i = 0; i < VEC / 2; ++i)
          positive[i] = __hgt2_mask(o.pair(i), Pair<T>::narrow(0.f, 0.f));
        signs[at / VEC] = static_cast<uint8_t>(pack_signs(positive));
      }
    }
  });
}

// relu(batch norm of x + batch norm of r) and its signs: the end of a residual block
// whose skip connection has a convolution and a batch norm of its own, which is then
// neither stored nor read. The four of a ResNet-50 step at batch 256 take 416 us, 676
// with a pass for the skip connection's batch norm. Bound by HBM.
template <typename T>
__global__ void __launch_bounds__(BN_THREADS, BN_MIN_BLOCKS)
bn_apply_pair_kernel(const T* __restrict__ x, const T* __restrict__ r, T* __restrict__ y,
                     uint8_t* __restrict__ signs, int64_t M, int C, double inv_m, int copies,
                     const BatchNormForward nx, const BatchNormForward nr) {
  const Tile t(C);
  const int by = gridDim.y - 1 - blockIdx.y;
  int64_t r0, r1;
  cta_rows(M, by, &r0, &r1);
  __shared__ __align__(16) float s_x[BN_CTA_CHANNELS], s_r[BN_CTA_CHANNELS],
      s_shift[BN_CTA_CHANNELS];
  wait_for_previous();
  if (by == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
    if (nx.batches != nullptr) *nx.batches += 1;
    if (nr.batches != nullptr) *nr.batches += 1;
  }
  if (static_cast<int>(threadIdx.x) < t.txg * VEC) {
    const int64_t ch = static_cast<int64_t>(blockIdx.x) * t.txg * VEC + threadIdx.x;
    const ForwardTerms fx = forward_terms(nx, M, C, inv_m, copies, ch, by == 0);
    const ForwardTerms fr = forward_terms(nr, M, C, inv_m, copies, ch, by == 0);
    s_x[threadIdx.x] = fx.scale;
    s_r[threadIdx.x] = fr.scale;
    s_shift[threadIdx.x] = fx.shift + fr.shift;
  }
  __syncthreads();
  float sx[VEC], sr[VEC], shift[VEC];
  load8(s_x + t.tx * VEC, sx);
  load8(s_r + t.tx * VEC, sr);
  load8(s_shift + t.tx * VEC, shift);
  const int64_t stride = static_cast<int64_t>(t.ty) * C;
  for_rows_back<UNROLL>(t, r0, r1, C, [&](auto count, int64_t at0) {
    constexpr int U = decltype(count)::value;
    Vec8<T> a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      a[u] = ldg16(x + at0 - u * stride);
      b[u] = ldg16(r + at0 - u * stride);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t at = at0 - u * stride;
      Vec8<T> o;
      uint32_t positive[VEC / 2];
#pragma unroll
      for (int i = 0; i < VEC / 2; ++i) {
        const float2 f = Pair<T>::widen(a[u].pair(i)), g = Pair<T>::widen(b[u].pair(i));
        const int j = 2 * i, k = 2 * i + 1;
        const typename Pair<T>::type zero = Pair<T>::narrow(0.f, 0.f);
        const typename Pair<T>::type v =
            __hmax2(Pair<T>::narrow(fmaf(f.x, sx[j], fmaf(g.x, sr[j], shift[j])),
                                    fmaf(f.y, sx[k], fmaf(g.y, sr[k], shift[k]))), zero);
        positive[i] = __hgt2_mask(v, zero);
        o.set(i, v);
      }
      stg16(y + at, o);
      signs[at / VEC] = static_cast<uint8_t>(pack_signs(positive));
    }
  });
}

// Where the backward gets relu's mask from.
enum Mask : int {
  MASK_NONE = 0,   // no relu
  MASK_X = 1,      // x, scale and shift: relu without a residual
  MASK_SIGNS = 2,  // the forward's bits: relu of a sum with a residual
};

// dz of channels 2i and 2i + 1: dy where the output was above zero. x: the
// two inputs; signs: spread_signs() of the forward's byte. MASK_X repeats the
// forward's arithmetic, rounding included.
template <typename T, int MASK>
__device__ __forceinline__ uint32_t masked(int i, uint32_t dy, float2 x, uint32_t signs,
                                           const float (&scale)[VEC], const float (&shift)[VEC]) {
  if (MASK == MASK_X)
    return dy & __hgt2_mask(Pair<T>::narrow(fmaf(x.x, scale[2 * i], shift[2 * i]),
                                            fmaf(x.y, scale[2 * i + 1], shift[2 * i + 1])),
                            Pair<T>::narrow(0.f, 0.f));
  if (MASK == MASK_SIGNS) return dy & (((signs >> i) & 0x00010001u) * 0xffffu);
  return dy;
}

// sum(dz) and sum(dz * xhat) per channel.
template <typename T, int MASK>
__global__ void __launch_bounds__(BN_THREADS, BN_MIN_BLOCKS)
bn_backward_reduce_kernel(const T* __restrict__ dy, const uint8_t* __restrict__ signs,
                          const T* __restrict__ x, int64_t M, int C,
                          const float* __restrict__ weight, const float* __restrict__ saved,
                          int copies, double* __restrict__ sums) {
  const Tile t(C);
  int64_t r0, r1;
  cta_rows(M, blockIdx.y, &r0, &r1);
  const int64_t off = t.group * VEC;
  float mean[VEC], scale[VEC], shift[VEC];
  load8(saved + off, mean);
  if (MASK == MASK_X) {
    load8(saved + C + off, scale);
    load8(saved + 2 * static_cast<int64_t>(C) + off, shift);
#pragma unroll
    for (int i = 0; i < VEC; ++i) scale[i] *= weight ? weight[off + i] : 1.f;
  }
  float acc[2][VEC];
#pragma unroll
  for (int i = 0; i < VEC; ++i) acc[0][i] = acc[1][i] = 0.f;
  const int64_t stride = static_cast<int64_t>(t.ty) * C;
  // MASK_X keeps 16 more values per thread: four rows would spill.
  for_rows<MASK == MASK_X ? 3 : UNROLL>(t, r0, r1, C, [&](auto count, int64_t at0) {
    constexpr int U = decltype(count)::value;
    Vec8<T> d[U], a[U];
    uint32_t m[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t at = at0 + u * stride;
      d[u] = ldg16(dy + at);
      a[u] = ldg16(x + at);
      m[u] = MASK == MASK_SIGNS ? spread_signs(__ldg(signs + at / VEC)) : 0u;
    }
#pragma unroll
    for (int i = 0; i < VEC / 2; ++i) {
      float2 s = make_float2(0.f, 0.f), p = make_float2(0.f, 0.f);
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float2 f = Pair<T>::widen(a[u].pair(i));
        d[u].w[i] = masked<T, MASK>(i, d[u].w[i], f, m[u], scale, shift);
        const float2 dz = Pair<T>::widen(d[u].pair(i));
        s.x += dz.x;
        s.y += dz.y;
        p.x = fmaf(dz.x, f.x - mean[2 * i], p.x);
        p.y = fmaf(dz.y, f.y - mean[2 * i + 1], p.y);
      }
      acc[0][2 * i] += s.x;
      acc[0][2 * i + 1] += s.y;
      acc[1][2 * i] += p.x;
      acc[1][2 * i + 1] += p.y;
    }
  });
  start_next();
  float invstd[VEC];
  load8(saved + C + off, invstd);
#pragma unroll
  for (int i = 0; i < VEC; ++i) acc[1][i] *= invstd[i];
  reduce_to_global(t, acc, C, copies, sums);
}

// The same for two batch norms whose sum went through the ReLU: dz is one for both.
// The four of a ResNet-50 step at batch 256 take 389 us, 533 one after the other.
template <typename T>
__global__ void __launch_bounds__(BN_THREADS, BN_MIN_BLOCKS)
bn_backward_reduce_pair_kernel(const T* __restrict__ dy, const uint8_t* __restrict__ signs,
                               const T* __restrict__ x, const T* __restrict__ r, int64_t M, int C,
                               const float* __restrict__ saved_x,
                               const float* __restrict__ saved_r, int copies,
                               double* __restrict__ sums_x, double* __restrict__ sums_r) {
  const Tile t(C);
  int64_t r0, r1;
  cta_rows(M, blockIdx.y, &r0, &r1);
  const int64_t off = t.group * VEC;
  float mean_x[VEC], mean_r[VEC], acc[3][VEC];
  load8(saved_x + off, mean_x);
  load8(saved_r + off, mean_r);
#pragma unroll
  for (int i = 0; i < VEC; ++i) acc[0][i] = acc[1][i] = acc[2][i] = 0.f;
  const int64_t stride = static_cast<int64_t>(t.ty) * C;
  // (Three rows would spill.)
  for_rows<2>(t, r0, r1, C, [&](auto count, int64_t at0) {
    constexpr int U = decltype(count)::value;
    Vec8<T> d[U], a[U], b[U];
    uint32_t m[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t at = at0 + u * stride;
      d[u] = ldg16(dy + at);
      a[u] = ldg16(x + at);
      b[u] = ldg16(r + at);
      m[u] = spread_signs(__ldg(signs + at / VEC));
    }
#pragma unroll
    for (int i = 0; i < VEC / 2; ++i) {
      const int j = 2 * i, k = 2 * i + 1;
      float2 s = make_float2(0.f, 0.f), p = s, q = s;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const float2 f = Pair<T>::widen(a[u].pair(i)), g = Pair<T>::widen(b[u].pair(i));
        d[u].w[i] &= ((m[u] >> i) & 0x00010001u) * 0xffffu;
        const float2 dz = Pair<T>::widen(d[u].pair(i));
        s.x += dz.x;
        s.y += dz.y;
        p.x = fmaf(dz.x, f.x - mean_x[j], p.x);
        p.y = fmaf(dz.y, f.y - mean_x[k], p.y);
        q.x = fmaf(dz.x, g.x - mean_r[j], q.x);
        q.y = fmaf(dz.y, g.y - mean_r[k], q.y);
      }
      acc[0][j] += s.x;
      acc[0][k] += s.y;
      acc[1][j] += p.x;
      acc[1][k] += p.y;
      acc[2][j] += q.x;
      acc[2][k] += q.y;
    }
  });
  start_next();
  float invstd_x[VEC], invstd_r[VEC];
  load8(saved_x + C + off, invstd_x);
  load8(saved_r + C + off, invstd_r);
#pragma unroll
  for (int i = 0; i < VEC; ++i) {
    acc[1][i] *= invstd_x[i];
    acc[2][i] *= invstd_r[i];
  }
  reduce_to_global(t, acc, C, copies, sums_x, sums_r);
}

template <typename T, int MASK, bool DRES>
__global__ void __launch_bounds__(BN_THREADS, BN_MIN_BLOCKS)
bn_backward_apply_kernel(const T* __restrict__ dy, const uint8_t* __restrict__ signs,
                         const T* __restrict__ x, T* __restrict__ dx, T* __restrict__ dres,
                         int64_t M, int C, double inv_m, const float* __restrict__ weight,
                         const float* __restrict__ saved, int copies,
                         const double* __restrict__ sums, float* __restrict__ dweight,
                         float* __restrict__ dbias) {
  const Tile t(C);
  const int by = gridDim.y - 1 - blockIdx.y;
  int64_t r0, r1;
  cta_rows(M, by, &r0, &r1);
  // The centre costs 2 us of 359 (256 x 64 x 112 x 112, both kernels); two of them to a
  // register, 23.
  __shared__ __align__(16) float s_scale[BN_CTA_CHANNELS], s_shift[BN_CTA_CHANNELS],
      s_kx[BN_CTA_CHANNELS], s_kc[BN_CTA_CHANNELS], s_centre[BN_CTA_CHANNELS];
  wait_for_previous();
  if (static_cast<int>(threadIdx.x) < t.txg * VEC) {
    const int64_t ch = static_cast<int64_t>(blockIdx.x) * t.txg * VEC + threadIdx.x;
    const BackwardTerms b = backward_terms<T>(sums, C, copies, ch, inv_m, weight, saved);
    s_scale[threadIdx.x] = b.scale;
    s_shift[threadIdx.x] = saved[2 * static_cast<int64_t>(C) + ch];
    s_centre[threadIdx.x] = b.centre;
    s_kx[threadIdx.x] = b.kx;
    s_kc[threadIdx.x] = b.kc;
    if (by == 0) {
      if (dweight) dweight[ch] = static_cast<float>(b.dz_xhat);
      if (dbias) dbias[ch] = static_cast<float>(b.dz);
    }
  }
  __syncthreads();
  float scale[VEC], shift[VEC], kx[VEC], kc[VEC], centre[VEC];
  load8(s_scale + t.tx * VEC, scale);
  load8(s_kx + t.tx * VEC, kx);
  load8(s_kc + t.tx * VEC, kc);
  load8(s_centre + t.tx * VEC, centre);
  if (MASK == MASK_X) load8(s_shift + t.tx * VEC, shift);
  const int64_t stride = static_cast<int64_t>(t.ty) * C;
  for_rows_back<UNROLL>(t, r0, r1, C, [&](auto count, int64_t at0) {
    constexpr int U = decltype(count)::value;
    Vec8<T> d[U], a[U];
    uint32_t m[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t at = at0 - u * stride;
      d[u] = ldg16(dy + at);
      a[u] = ldg16(x + at);
      m[u] = MASK == MASK_SIGNS ? spread_signs(__ldg(signs + at / VEC)) : 0u;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t at = at0 - u * stride;
      Vec8<T> g;
#pragma unroll
      for (int i = 0; i < VEC / 2; ++i) {
        const float2 f = Pair<T>::widen(a[u].pair(i));
        d[u].w[i] = masked<T, MASK>(i, d[u].w[i], f, m[u], scale, shift);
        const float2 z = Pair<T>::widen(d[u].pair(i));
        const int j = 2 * i, k = 2 * i + 1;
        g.set(i, Pair<T>::narrow(fmaf(scale[j], z.x, fmaf(kx[j], f.x - centre[j], kc[j])),
                                 fmaf(scale[k], z.y, fmaf(kx[k], f.y - centre[k], kc[k]))));
      }
      stg16(dx + at, g);
      if (DRES) stg16(dres + at, d[u]);
    }
  });
}

// The gradients of both inputs of such a pair. 64 values per channel group stay in
// registers, hence two CTAs per SM. The three of a ResNet-50 step at batch 256 that take
// this path: 319 us, 341 one after the other.
template <typename T>
__global__ void __launch_bounds__(BN_THREADS, 2)
bn_backward_apply_pair_kernel(const T* __restrict__ dy, const uint8_t* __restrict__ signs,
                              const T* __restrict__ x, const T* __restrict__ r,
                              T* __restrict__ dx, T* __restrict__ dr, int64_t M, int C,
                              double inv_m, int copies, const BatchNormBackward nx,
                              const BatchNormBackward nr) {
  const Tile t(C);
  const int by = gridDim.y - 1 - blockIdx.y;
  int64_t r0, r1;
  cta_rows(M, by, &r0, &r1);
  __shared__ __align__(16) float s_terms[2][4][BN_CTA_CHANNELS];
  wait_for_previous();
  if (static_cast<int>(threadIdx.x) < t.txg * VEC) {
    const int64_t ch = static_cast<int64_t>(blockIdx.x) * t.txg * VEC + threadIdx.x;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const BatchNormBackward& n = k == 0 ? nx : nr;
      const BackwardTerms b = backward_terms<T>(n.sums, C, copies, ch, inv_m, n.weight, n.saved);
      s_terms[k][0][threadIdx.x] = b.scale;
      s_terms[k][1][threadIdx.x] = b.kx;
      s_terms[k][2][threadIdx.x] = b.kc;
      s_terms[k][3][threadIdx.x] = b.centre;
      if (by == 0) {
        n.dweight[ch] = static_cast<float>(b.dz_xhat);
        n.dbias[ch] = static_cast<float>(b.dz);
      }
    }
  }
  __syncthreads();
  float scale[2][VEC], kx[2][VEC], kc[2][VEC], centre[2][VEC];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    load8(s_terms[k][0] + t.tx * VEC, scale[k]);
    load8(s_terms[k][1] + t.tx * VEC, kx[k]);
    load8(s_terms[k][2] + t.tx * VEC, kc[k]);
    load8(s_terms[k][3] + t.tx * VEC, centre[k]);
  }
  const int64_t stride = static_cast<int64_t>(t.ty) * C;
  for_rows_back<3>(t, r0, r1, C, [&](auto count, int64_t at0) {
    constexpr int U = decltype(count)::value;
    Vec8<T> d[U], in[2][U];
    uint32_t m[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t at = at0 - u * stride;
      d[u] = ldg16(dy + at);
      in[0][u] = ldg16(x + at);
      in[1][u] = ldg16(r + at);
      m[u] = spread_signs(__ldg(signs + at / VEC));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t at = at0 - u * stride;
      Vec8<T> g[2];
#pragma unroll
      for (int i = 0; i < VEC / 2; ++i) {
        d[u].w[i] &= ((m[u] >> i) & 0x00010001u) * 0xffffu;
        const float2 z = Pair<T>::widen(d[u].pair(i));
        const int j = 2 * i, l = 2 * i + 1;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const float2 f = Pair<T>::widen(in[k][u].pair(i));
          g[k].set(i, Pair<T>::narrow(
              fmaf(scale[k][j], z.x, fmaf(kx[k][j], f.x - centre[k][j], kc[k][j])),
              fmaf(scale[k][l], z.y, fmaf(kx[k][l], f.y - centre[k][l], kc[k][l]))));
        }
      }
      stg16(dx + at, g[0]);
      stg16(dr + at, g[1]);
    }
  });
}

// Copies of the per-channel accumulators: 8 up to 256 channels, fewer beyond
// (more channels are spread over more CTAs, so fewer of them meet at one
// address). One copy and 1184 CTAs took 23 us for the statistics of 256 x 256 x
// 14 x 14, 8 copies and 592 CTAs take 7.3; 16 and more cost the second kernel
// more than they save the first.
int bn_copies(int C) { return C <= 256 ? 8 : C < 2048 ? 2048 / C : 1; }

// The kernels that sum run as one wave of resident CTAs: each CTA ends with its
// additions to the accumulators.
constexpr int BN_CTAS_STATS = 148 * BN_MIN_BLOCKS_STATS;
constexpr int BN_CTAS_REDUCE = 148 * BN_MIN_BLOCKS;
// The kernels that write start with reading the sums, which one wave of CTAs does
// least often: small tensors get one. In large ones more and shorter CTAs even
// out the SMs. The line lies where the two meet, which differs: with 64 to 1024
// channels in bf16 both kernels together take, with one wave, against 1184 CTAs,
//   16 Mi elements  forward 0.89-0.95 of the time  backward 0.92-0.96
//   32 Mi                   0.96-1.00                       0.94-0.98
//   64 Mi                   0.99-1.03                       0.96-1.01
//   96 Mi                   1.02-1.04                       0.98-1.03
//   192 Mi                  1.03-1.05                       0.98-1.03
// (the higher figures with a residual).
int bn_apply_ctas(int64_t M, int C) { return M * C <= (64 << 20) ? 148 * BN_MIN_BLOCKS : 148 * 8; }

dim3 bn_grid(int64_t M, int C, int ctas) {
  const int cg = C / VEC;
  const int txg = cg < 32 ? cg : 32;
  const int ty = BN_THREADS / txg;
  const int ctiles = cg / txg;
  // At most `ctas` in total (a few more would be a second wave), at least 4 *
  // ty rows each.
  int64_t by = ctas / ctiles;
  const int64_t max_by = (M + 4 * ty - 1) / (4 * ty);
  if (by > max_by) by = max_by;
  if (by < 1) by = 1;
  if (by > 65535) by = 65535;
  return dim3(static_cast<unsigned>(ctiles), static_cast<unsigned>(by), 1);
}

bool bn_shape_ok(int64_t M, int C) {
  if (M < 1 || C < VEC || C % VEC != 0) return false;
  const int cg = C / VEC;
  // Channel groups must tile into CTAs of min(cg, 32) groups, and that width
  // must divide the CTA size.
  const int txg = cg < 32 ? cg : 32;
  return cg % txg == 0 && BN_THREADS % txg == 0;
}

}  // namespace

bool BatchNormSupported(int64_t rows, int channels) { return bn_shape_ok(rows, channels); }

int BatchNormCopies(int channels) { return bn_copies(channels); }

int64_t BatchNormScratchDoubles(int channels) {
  return static_cast<int64_t>(2) * bn_copies(channels) * channels;
}

// Launches the second kernel of a pair so that it may start while the first
// one is still running (it waits for the results itself).
template <typename... P, typename... A>
static cudaError_t LaunchDependent(void (*kernel)(P...), dim3 grid, cudaStream_t stream,
                                   A... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = grid;
  config.blockDim = dim3(BN_THREADS);
  config.stream = stream;
  config.attrs = &attr;
  config.numAttrs = 1;
  return cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
}

template <typename T>
static cudaError_t SumsTyped(const void* x, int64_t M, int C, const BatchNormForward& n,
                             cudaStream_t stream) {
  if (n.summed) return cudaSuccess;
  CountKernelLaunches(1);
  bn_stats_kernel<T><<<bn_grid(M, C, BN_CTAS_STATS), BN_THREADS, 0, stream>>>(
      static_cast<const T*>(x), M, C, bn_copies(C), n.sums);
  return cudaGetLastError();
}

template <typename T>
static cudaError_t ForwardTyped(const void* x, const void* res, void* y, uint8_t* signs, int64_t M,
                                int C, const BatchNormForward& n, bool relu,
                                cudaStream_t stream) {
  const cudaError_t err = SumsTyped<T>(x, M, C, n, stream);
  if (err != cudaSuccess) return err;
  auto kernel = relu && res ? bn_apply_kernel<T, true, true>
                : relu      ? bn_apply_kernel<T, true, false>
                : res       ? bn_apply_kernel<T, false, true>
                            : bn_apply_kernel<T, false, false>;
  return LaunchDependent(kernel, bn_grid(M, C, bn_apply_ctas(M, C)), stream,
                         static_cast<const T*>(x), static_cast<const T*>(res),
                         static_cast<T*>(y), signs, M, C, 1.0 / static_cast<double>(M),
                         bn_copies(C), n);
}

template <typename T>
static cudaError_t PairForwardTyped(const void* x, const void* r, void* y, uint8_t* signs,
                                    int64_t M, int C, const BatchNormForward& nx,
                                    const BatchNormForward& nr, cudaStream_t stream) {
  cudaError_t err = SumsTyped<T>(r, M, C, nr, stream);
  if (err == cudaSuccess) err = SumsTyped<T>(x, M, C, nx, stream);
  if (err != cudaSuccess) return err;
  return LaunchDependent(bn_apply_pair_kernel<T>, bn_grid(M, C, bn_apply_ctas(M, C)), stream,
                         static_cast<const T*>(x), static_cast<const T*>(r), static_cast<T*>(y),
                         signs, M, C, 1.0 / static_cast<double>(M), bn_copies(C), nx, nr);
}

template <typename T>
static cudaError_t PairSumsTyped(const void* dy, const uint8_t* signs, const void* x,
                                 const void* r, int64_t M, int C, const BatchNormBackward& nx,
                                 const BatchNormBackward& nr, cudaStream_t stream) {
  CountKernelLaunches(1);
  bn_backward_reduce_pair_kernel<T><<<bn_grid(M, C, BN_CTAS_REDUCE), BN_THREADS, 0, stream>>>(
      static_cast<const T*>(dy), signs, static_cast<const T*>(x), static_cast<const T*>(r), M, C,
      nx.saved, nr.saved, bn_copies(C), nx.sums, nr.sums);
  return cudaGetLastError();
}

template <typename T>
static cudaError_t PairBackwardTyped(const void* dy, const uint8_t* signs, const void* x,
                                     const void* r, void* dx, void* dr, int64_t M, int C,
                                     const BatchNormBackward& nx, const BatchNormBackward& nr,
                                     cudaStream_t stream) {
  const cudaError_t err = PairSumsTyped<T>(dy, signs, x, r, M, C, nx, nr, stream);
  if (err != cudaSuccess) return err;
  CountKernelLaunches(1);
  return LaunchDependent(bn_backward_apply_pair_kernel<T>, bn_grid(M, C, 148 * 2), stream,
                         static_cast<const T*>(dy), signs, static_cast<const T*>(x),
                         static_cast<const T*>(r), static_cast<T*>(dx), static_cast<T*>(dr), M, C,
                         1.0 / static_cast<double>(M), bn_copies(C), nx, nr);
}

template <typename T>
static cudaError_t BackwardTyped(const void* dy, const uint8_t* signs, const void* x, void* dx,
                                 void* dres, int64_t M, int C, double* sums, const float* weight,
                                 const float* saved, float* dweight, float* dbias, bool relu,
                                 cudaStream_t stream) {
  const int copies = bn_copies(C);
  const T* dyt = static_cast<const T*>(dy);
  const T* xt = static_cast<const T*>(x);
  const int mask = !relu ? MASK_NONE : signs == nullptr ? MASK_X : MASK_SIGNS;
  // A gradient of the residual never comes with MASK_X: that is a layer
  // without one.
  if (mask == MASK_X && dres != nullptr) return cudaErrorInvalidValue;
  auto reduce = mask == MASK_NONE ? bn_backward_reduce_kernel<T, MASK_NONE>
                : mask == MASK_X  ? bn_backward_reduce_kernel<T, MASK_X>
                                  : bn_backward_reduce_kernel<T, MASK_SIGNS>;
  reduce<<<bn_grid(M, C, BN_CTAS_REDUCE), BN_THREADS, 0, stream>>>(dyt, signs, xt, M, C, weight,
                                                                   saved, copies, sums);
  cudaError_t err = cudaGetLastError();
  if (err != cudaSuccess) return err;
  auto apply = mask == MASK_NONE ? (dres ? bn_backward_apply_kernel<T, MASK_NONE, true>
                                         : bn_backward_apply_kernel<T, MASK_NONE, false>)
               : mask == MASK_X  ? bn_backward_apply_kernel<T, MASK_X, false>
                                 : (dres ? bn_backward_apply_kernel<T, MASK_SIGNS, true>
                                         : bn_backward_apply_kernel<T, MASK_SIGNS, false>);
  return LaunchDependent(apply, bn_grid(M, C, bn_apply_ctas(M, C)), stream, dyt, signs, xt,
                         static_cast<T*>(dx), static_cast<T*>(dres), M, C,
                         1.0 / static_cast<double>(M), weight, saved, copies, sums, dweight,
                         dbias);
}

cudaError_t LaunchBatchNormForward(const void* x, const void* residual, void* y, uint8_t* signs,
                                   int64_t rows, int channels, bool bf16,
                                   const BatchNormForward& n, bool relu, cudaStream_t stream) {
  if (!bn_shape_ok(rows, channels)) return cudaErrorInvalidValue;
  if (relu && residual != nullptr && signs == nullptr) return cudaErrorInvalidValue;
  CountKernelLaunches(1);
  return bf16 ? ForwardTyped<__nv_bfloat16>(x, residual, y, signs, rows, channels, n, relu, stream)
              : ForwardTyped<__half>(x, residual, y, signs, rows, channels, n, relu, stream);
}

cudaError_t LaunchBatchNormPairForward(const void* x, const void* r, void* y, uint8_t* signs,
                                       int64_t rows, int channels, bool bf16,
                                       const BatchNormForward& nx, const BatchNormForward& nr,
                                       cudaStream_t stream) {
  if (!bn_shape_ok(rows, channels)) return cudaErrorInvalidValue;
  CountKernelLaunches(1);
  return bf16 ? PairForwardTyped<__nv_bfloat16>(x, r, y, signs, rows, channels, nx, nr, stream)
              : PairForwardTyped<__half>(x, r, y, signs, rows, channels, nx, nr, stream);
}

cudaError_t LaunchBatchNormPairSums(const void* dy, const uint8_t* signs, const void* x,
                                    const void* r, int64_t rows, int channels, bool bf16,
                                    const BatchNormBackward& nx, const BatchNormBackward& nr,
                                    cudaStream_t stream) {
  if (!bn_shape_ok(rows, channels)) return cudaErrorInvalidValue;
  return bf16 ? PairSumsTyped<__nv_bfloat16>(dy, signs, x, r, rows, channels, nx, nr, stream)
              : PairSumsTyped<__half>(dy, signs, x, r, rows, channels, nx, nr, stream);
}

cudaError_t LaunchBatchNormPairBackward(const void* dy, const uint8_t* signs, const void* x,
                                        const void* r, void* dx, void* dr, int64_t rows,
                                        int channels, bool bf16, const BatchNormBackward& nx,
                                        const BatchNormBackward& nr, cudaStream_t stream) {
  if (!bn_shape_ok(rows, channels)) return cudaErrorInvalidValue;
  return bf16 ? PairBackwardTyped<__nv_bfloat16>(dy, signs, x, r, dx, dr, rows, channels, nx, nr,
                                                 stream)
              : PairBackwardTyped<__half>(dy, signs, x, r, dx, dr, rows, channels, nx, nr,
                                          stream);
}

cudaError_t LaunchBatchNormBackwardSums(const void* dy, const uint8_t* signs, const void* x,
                                        int64_t rows, int channels, bool bf16,
                                        double* sums_zeroed, const float* weight,
                                        const float* saved, cudaStream_t stream) {
  if (!bn_shape_ok(rows, channels) || signs == nullptr) return cudaErrorInvalidValue;
  CountKernelLaunches(1);
  const dim3 grid = bn_grid(rows, channels, BN_CTAS_REDUCE);
  const int copies = bn_copies(channels);
  if (bf16)
    bn_backward_reduce_kernel<__nv_bfloat16, MASK_SIGNS><<<grid, BN_THREADS, 0, stream>>>(
        static_cast<const __nv_bfloat16*>(dy), signs, static_cast<const __nv_bfloat16*>(x), rows,
        channels, weight, saved, copies, sums_zeroed);
  else
    bn_backward_reduce_kernel<__half, MASK_SIGNS><<<grid, BN_THREADS, 0, stream>>>(
        static_cast<const __half*>(dy), signs, static_cast<const __half*>(x), rows, channels,
        weight, saved, copies, sums_zeroed);
  return cudaGetLastError();
}

cudaError_t LaunchBatchNormBackward(const void* dy, const uint8_t* signs, const void* x, void* dx,
                                    void* dresidual, int64_t rows, int channels, bool bf16,
                                    double* sums_zeroed, const float* weight, const float* saved,
                                    float* dweight, float* dbias, bool relu,
                                    cudaStream_t stream) {
  if (!bn_shape_ok(rows, channels)) return cudaErrorInvalidValue;
  CountKernelLaunches(2);
  return bf16 ? BackwardTyped<__nv_bfloat16>(dy, signs, x, dx, dresidual, rows, channels,
                                             sums_zeroed, weight, saved, dweight, dbias, relu,
                                             stream)
              : BackwardTyped<__half>(dy, signs, x, dx, dresidual, rows, channels, sums_zeroed,
                                      weight, saved, dweight, dbias, relu, stream);
}

}  // namespace kern
}  // namespace hvd
