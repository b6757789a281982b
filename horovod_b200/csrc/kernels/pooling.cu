// 3x3 / stride 2 / padding 1 max pooling on channels-last 16-bit activations
// (the ResNet stem), forward and backward. Both passes are bound by HBM: the
// forward reads x and writes y and half a byte per output element that says
// which of the nine window positions won; the backward reads dy and those
// nibbles and writes dx, a gather without atomics.
//
// Forward: one thread owns 8 channels (16 bytes) of one output column and
// walks down several output rows. It reduces each input row to the maximum of
// its three columns and keeps the row that two windows share in registers, so
// an output pixel costs 6 loads and 6 comparisons instead of 9 and 9;
// comparisons and selections work on two 16-bit channels at a time.
// Backward: one thread owns 8 channels of a 2 x 2 block of input pixels and
// walks down block rows. Such a block is covered by four windows, two of which
// the next block down needs again: 2 loads of dy per 4 pixels instead of 9.
// The ResNet-50 stem at batch 256 (256 x 64 x 112 x 112, bf16) takes 204 us
// forward and backward on a B200; one output or input pixel per thread, with a
// byte per index, took 521 us. The bytes that have to move (x, y, dy, dx) take
// 159 us at the rate of a plain copy.
//
// Ties go to the first maximum in scan order (rows, then columns) and NaN
// wins over everything, which is the rule of PyTorch's max_pool2d, so the
// gradients agree with it element for element.
//
// The reference has no counterpart (it takes pooling from the framework).
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>

#include "kernels.h"

namespace hvd {
namespace kern {

namespace {

constexpr int POOL_THREADS = 256;

template <typename T> struct Pair;
template <> struct Pair<__half> { using type = __half2; };
template <> struct Pair<__nv_bfloat16> { using type = __nv_bfloat162; };

// 8 channels of one pixel.
template <typename T> union Vec8 {
  uint4 raw;
  uint32_t w[4];
  typename Pair<T>::type p[4];
  T e[8];
};

// The best value so far and where it came from, two channels per word.
struct Best {
  uint32_t v[4];
  uint32_t at[4];
};

// Takes over the channels of (f, at) that beat b: greater, or NaN. A NaN stays
// (every comparison with it is false) until a later NaN replaces it, and of
// equal values the first stays, as in PyTorch.
template <typename T>
__device__ __forceinline__ void take_better(Best& b, const Vec8<T>& f, const uint32_t (&at)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    Vec8<T> old;
    old.w[i] = b.v[i];
    const uint32_t m = __hgt2_mask(f.p[i], old.p[i]) | __hneu2_mask(f.p[i], f.p[i]);
    b.v[i] = (f.w[i] & m) | (b.v[i] & ~m);
    b.at[i] = (at[i] & m) | (b.at[i] & ~m);
  }
}

// Maximum over columns w0 .. w0 + 2 of an input row; `at` holds the position
// inside the window's first row (0, 1, 2). Column w0 + 1 always exists.
template <typename T, typename I>
__device__ __forceinline__ Best row_best(const uint4* __restrict__ row, int w0, int W, int C8) {
  const bool left = w0 >= 0, right = w0 + 2 < W;
  Vec8<T> a, m, c;
  a.raw = m.raw = __ldg(row + static_cast<I>(w0 + 1) * C8);
  c.raw = make_uint4(0, 0, 0, 0);
  if (left) a.raw = __ldg(row + static_cast<I>(w0) * C8);
  if (right) c.raw = __ldg(row + static_cast<I>(w0 + 2) * C8);
  const uint32_t one[4] = {0x00010001u, 0x00010001u, 0x00010001u, 0x00010001u};
  const uint32_t two[4] = {0x00020002u, 0x00020002u, 0x00020002u, 0x00020002u};
  Best b;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    b.v[i] = a.w[i];
    b.at[i] = left ? 0u : 0x00010001u;
  }
  if (left) take_better<T>(b, m, one);
  if (right) take_better<T>(b, c, two);
  return b;
}

// Bit position of channel i's nibble in the index word of 8 channels: the even
// channels lie in the low half, the odd ones in the high half, as in the words
// of two channels above.
__host__ __device__ constexpr int nibble_shift(int i) { return (i >> 1) * 4 + (i & 1) * 16; }

// Five CTAs per SM (48 registers): forward 109 us, 117 with four of 57.
// I: type of the flat vector index. Tensors of fewer than 2^31 vectors (every
// practical activation) use 32-bit index arithmetic: the divisions cost several
// times the pooling itself when done in 64 bits.
template <typename T, typename I>
__global__ void __launch_bounds__(POOL_THREADS, 5)
maxpool3s2_forward_kernel(const uint4* __restrict__ x, uint4* __restrict__ y,
                          uint32_t* __restrict__ idx, I total, int H, int W, int C8, int Ho,
                          int Wo, int rows) {
  I t = blockIdx.x * static_cast<I>(POOL_THREADS) + threadIdx.x;
  if (t >= total) return;
  const int c8 = static_cast<int>(t % C8);
  t /= C8;
  const int ow = static_cast<int>(t % Wo);
  t /= Wo;
  const int strips = (Ho + rows - 1) / rows;
  const int oh0 = static_cast<int>(t % strips) * rows;
  const I n = t / strips;
  const int oh1 = min(oh0 + rows, Ho);
  const int w0 = ow * 2 - 1;
  const I pitch = static_cast<I>(W) * C8;
  const uint4* in = x + (n * H + oh0 * 2) * pitch + c8;  // middle row of the first window
  const I step = static_cast<I>(Wo) * C8;
  I o = ((n * Ho + oh0) * Wo + ow) * C8 + c8;
  Best above;  // the row above the window's middle row
  bool have_above = oh0 > 0;
  if (have_above) above = row_best<T, I>(in - pitch, w0, W, C8);
  for (int oh = oh0; oh < oh1; ++oh) {
    Best best = row_best<T, I>(in, w0, W, C8);
    const bool have_below = oh * 2 + 1 < H;
    Best below;
    if (have_below) below = row_best<T, I>(in + pitch, w0, W, C8);
    Vec8<T> f;
    uint32_t at[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      f.w[i] = best.v[i];
      at[i] = best.at[i] + 0x00030003u;
    }
    if (have_above) {
      best = above;
      take_better<T>(best, f, at);
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i) best.at[i] = at[i];
    }
    if (have_below) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        f.w[i] = below.v[i];
        at[i] = below.at[i] + 0x00060006u;
      }
      take_better<T>(best, f, at);
      above = below;
    }
    have_above = have_below;
    y[o] = make_uint4(best.v[0], best.v[1], best.v[2], best.v[3]);
    idx[o] = best.at[0] | (best.at[1] << 4) | (best.at[2] << 8) | (best.at[3] << 12);
    in += 2 * pitch;
    o += step;
  }
}

// The gradient of one window and which of its positions gets it.
struct Window {
  uint4 dy;
  uint32_t idx;
};

template <typename T, typename I>
__global__ void __launch_bounds__(POOL_THREADS)
maxpool3s2_backward_kernel(const uint4* __restrict__ dy, const uint32_t* __restrict__ idx,
                           uint4* __restrict__ dx, I total, int H, int W, int C8, int Ho, int Wo,
                           int rows) {
  I t = blockIdx.x * static_cast<I>(POOL_THREADS) + threadIdx.x;
  if (t >= total) return;
  const int c8 = static_cast<int>(t % C8);
  t /= C8;
  // Block (a, b) holds input rows 2a, 2a + 1 and columns 2b, 2b + 1; there are
  // as many blocks as output pixels.
  const int b = static_cast<int>(t % Wo);
  t /= Wo;
  const int strips = (Ho + rows - 1) / rows;
  const int a0 = static_cast<int>(t % strips) * rows;
  const I n = t / strips;
  const int a1 = min(a0 + rows, Ho);
  const bool right = b + 1 < Wo;       // window (., b + 1) exists
  const bool odd_col = b * 2 + 1 < W;  // column 2b + 1 exists
  const I step = static_cast<I>(Wo) * C8;
  I o = ((n * Ho + a0) * Wo + b) * C8 + c8;
  const I pitch = static_cast<I>(W) * C8;
  uint4* out = dx + (n * H + a0 * 2) * pitch + static_cast<I>(b) * 2 * C8 + c8;
  auto load = [&](I at, bool exists) {
    Window w;
    w.dy = make_uint4(0, 0, 0, 0);
    w.idx = 0xffffffffu;  // no position
    if (exists) {
      w.dy = __ldg(dy + at);
      w.idx = __ldg(idx + at);
    }
    return w;
  };
  auto add = [](float (&acc)[8], const Window& w, uint32_t pos) {
    Vec8<T> g;
    g.raw = w.dy;
    const uint32_t differs = w.idx ^ (pos * 0x11111111u);
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if ((differs & (0xfu << nibble_shift(i))) == 0) acc[i] += static_cast<float>(g.e[i]);
  };
  auto put = [](uint4* p, const float (&acc)[8]) {
    Vec8<T> r;
#pragma unroll
    for (int i = 0; i < 8; ++i) r.e[i] = static_cast<T>(acc[i]);
    *p = r.raw;
  };
  Window w00 = load(o, true), w01 = load(o + C8, right);
  for (int a = a0; a < a1; ++a) {
    const bool below = a + 1 < Ho;
    const Window w10 = load(o + step, below), w11 = load(o + step + C8, below && right);
    {
      float acc[8] = {};
      add(acc, w00, 4);
      put(out, acc);
    }
    if (odd_col) {
      float acc[8] = {};
      add(acc, w00, 5);
      add(acc, w01, 3);
      put(out + C8, acc);
    }
    if (a * 2 + 1 < H) {
      {
        float acc[8] = {};
        add(acc, w00, 7);
        add(acc, w10, 1);
        put(out + pitch, acc);
      }
      if (odd_col) {
        float acc[8] = {};
        add(acc, w00, 8);
        add(acc, w01, 6);
        add(acc, w10, 2);
        add(acc, w11, 0);
        put(out + pitch + C8, acc);
      }
    }
    w00 = w10;
    w01 = w11;
    o += step;
    out += 2 * pitch;
  }
}

// Output rows per thread: as many as leave the GPU two full sets of resident
// threads, at most 8 (the row or pair of windows that a strip's first step
// loads again is then an eighth of its traffic, and comes from L2).
int StripRows(long long columns, int ho) {
  int rows = 8;
  while (rows > 1 && columns * ((ho + rows - 1) / rows) < 2LL * 148 * 2048) rows /= 2;
  return rows;
}

// Whether every vector index of the larger tensor, plus one block, fits a
// 32-bit int.
bool Fits32(long long input_vectors) { return input_vectors + POOL_THREADS < (1LL << 31); }

}  // namespace

bool MaxPool3s2Supported(int channels) { return channels > 0 && channels % 8 == 0; }

cudaError_t LaunchMaxPool3s2Forward(const void* x, void* y, uint32_t* idx, int n, int h, int w,
                                    int channels, bool bf16, cudaStream_t stream) {
  if (!MaxPool3s2Supported(channels)) return cudaErrorInvalidValue;
  const int ho = (h + 2 - 3) / 2 + 1, wo = (w + 2 - 3) / 2 + 1;
  const long long columns = static_cast<long long>(n) * wo * (channels / 8);
  if (columns * ho == 0) return cudaSuccess;
  const int rows = StripRows(columns, ho);
  const long long total = columns * ((ho + rows - 1) / rows);
  const unsigned blocks = static_cast<unsigned>((total + POOL_THREADS - 1) / POOL_THREADS);
  CountKernelLaunches(1);
  const bool small = Fits32(static_cast<long long>(n) * h * w * (channels / 8));
#define HVD_POOL_FWD(T, I)                                                                   \
  maxpool3s2_forward_kernel<T, I><<<blocks, POOL_THREADS, 0, stream>>>(                      \
      static_cast<const uint4*>(x), static_cast<uint4*>(y), idx, static_cast<I>(total), h, w, \
      channels / 8, ho, wo, rows)
  if (bf16) {
    if (small) HVD_POOL_FWD(__nv_bfloat16, int); else HVD_POOL_FWD(__nv_bfloat16, long long);
  } else {
    if (small) HVD_POOL_FWD(__half, int); else HVD_POOL_FWD(__half, long long);
  }
#undef HVD_POOL_FWD
  return cudaGetLastError();
}

cudaError_t LaunchMaxPool3s2Backward(const void* dy, const uint32_t* idx, void* dx, int n, int h,
                                     int w, int channels, bool bf16, cudaStream_t stream) {
  if (!MaxPool3s2Supported(channels)) return cudaErrorInvalidValue;
  const int ho = (h + 2 - 3) / 2 + 1, wo = (w + 2 - 3) / 2 + 1;
  const long long columns = static_cast<long long>(n) * wo * (channels / 8);
  if (columns * ho == 0) return cudaSuccess;
  const int rows = StripRows(columns, ho);
  const long long total = columns * ((ho + rows - 1) / rows);
  const unsigned blocks = static_cast<unsigned>((total + POOL_THREADS - 1) / POOL_THREADS);
  CountKernelLaunches(1);
  const bool small = Fits32(static_cast<long long>(n) * h * w * (channels / 8));
#define HVD_POOL_BWD(T, I)                                                                   \
  maxpool3s2_backward_kernel<T, I><<<blocks, POOL_THREADS, 0, stream>>>(                     \
      static_cast<const uint4*>(dy), idx, static_cast<uint4*>(dx), static_cast<I>(total), h, w, \
      channels / 8, ho, wo, rows)
  if (bf16) {
    if (small) HVD_POOL_BWD(__nv_bfloat16, int); else HVD_POOL_BWD(__nv_bfloat16, long long);
  } else {
    if (small) HVD_POOL_BWD(__half, int); else HVD_POOL_BWD(__half, long long);
  }
#undef HVD_POOL_BWD
  return cudaGetLastError();
}

}  // namespace kern
}  // namespace hvd
