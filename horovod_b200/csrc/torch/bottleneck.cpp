// A ResNet bottleneck block (1x1, 3x3, 1x1 convolutions with batch norms, ReLUs
// and the skip connection) in training as one autograd node. What it saves over
// the sequence of its layers, per block:
//   - the statistics of a 1x1 convolution's output come from the convolution;
//   - the gradient of the skip connection is never stored: the first
//     convolution's gradient kernel adds dy where the block's output was above
//     zero, in place of a store and a pass over three tensors;
//   - the backward of the last batch norm and convolution (of the first stage's
//     sizes) is one kernel, which stores no gradient of the batch norm's input;
//   - the batch norm of the skip connection is formed where it is added, and the two
//     batch norms' backwards read dy once;
//   - the weights are cast in one launch, and so are their gradients.
// The 3x3 convolution, the gradients of the weights and some 1x1 convolutions are
// PyTorch's.
#include <ATen/autocast_mode.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <array>
#include <cstdint>
#include <vector>

#include "../kernels/kernels.h"
#include "model_ops.h"

namespace hvd {

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

constexpr auto CL = at::MemoryFormat::ChannelsLast;

// Layers of a block: the three convolutions in order, then the one of the
// skip connection (its weights are undefined tensors where there is none).
constexpr int LAYERS = 4, DOWN = 3;

// Names of what a node keeps beside its saved tensors. (Compiled autograd finds tensors
// there, but not lists of them.)
constexpr const char* WEIGHT[LAYERS] = {"w0", "w1", "w2", "w3"};
constexpr const char* BETA[LAYERS] = {"b0", "b1", "b2", "b3"};

struct Norm {
  Tensor mean, var, batches;
  double momentum = 0.0, eps = 0.0;
};

struct Block {
  std::array<Norm, LAYERS> norms;
  int64_t stride = 1;
  at::ScalarType type = at::kBFloat16;
};

cudaStream_t Stream() { return at::cuda::getCurrentCUDAStream(); }

void Check(cudaError_t err, const char* what) {
  TORCH_CHECK(err == cudaSuccess, what, ": ", cudaGetErrorString(err));
}

// t in a memory format and on a 16-byte boundary, which is how the kernels read it.
Tensor Dense(const Tensor& t, at::MemoryFormat format) {
  const Tensor c = t.contiguous(format);
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 16 == 0 ? c : c.clone(format);
}

int64_t Rows(const Tensor& t) { return t.numel() / t.size(1); }
int Channels(const Tensor& t) { return static_cast<int>(t.size(1)); }

Tensor NewActivations(const Tensor& like, int64_t channels, int64_t h, int64_t w) {
  return at::empty({like.size(0), channels, h, w}, like.options(), CL);
}

// Casts of up to LAYERS tensors in one launch; undefined ones are passed over.
// The results have the strides of `layouts`, or of `from` where that is dense.
std::array<Tensor, LAYERS> Cast(const std::array<Tensor, LAYERS>& from, at::ScalarType to,
                                const std::array<Tensor, LAYERS>* layouts = nullptr) {
  std::array<Tensor, LAYERS> out;
  kern::CastArrays a;
  bool bf16 = true;
  for (int i = 0; i < LAYERS; ++i) {
    const Tensor& f = from[i];
    if (!f.defined()) continue;
    if (f.scalar_type() == to) {
      out[i] = f;
      continue;
    }
    const Tensor& layout = layouts ? (*layouts)[i] : f;
    if (layout.is_non_overlapping_and_dense()) {
      out[i] = at::empty_strided(layout.sizes(), layout.strides(), f.options().dtype(to));
      // The order of the elements in memory: strides of dimensions of size 1 do
      // not matter.
      bool same = true;
      for (int64_t d = 0; d < f.dim(); ++d)
        same = same && (f.size(d) == 1 || f.stride(d) == out[i].stride(d));
      if (same && reinterpret_cast<uintptr_t>(f.data_ptr()) % 16 == 0) {
        a.from[a.n] = f.data_ptr();
        a.to[a.n] = out[i].data_ptr();
        a.counts[a.n++] = f.numel();
        bf16 = (to == at::kFloat ? f.scalar_type() : to) == at::kBFloat16;
        continue;
      }
      out[i].copy_(f);
    } else {
      out[i] = f.to(to);
    }
  }
  if (a.n > 0) Check(kern::LaunchCastArrays(a, to == at::kFloat, bf16, Stream()), "casts");
  if (layouts == nullptr)
    for (Tensor& t : out)  // the kernels' operands: rows of input channels, aligned
      if (t.defined() && t.size(2) == 1 &&
          (!t.is_contiguous() || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0))
        t = t.clone(at::MemoryFormat::Contiguous);
  return out;
}

// Sums of a batch norm's input: scratch, and whether they are in it already. Has to
// live until the kernels that read them are launched.
struct Sums {
  double* p = nullptr;
  Tensor own;
  bool ready = false;
  Sums() = default;
  Sums(const Tensor& like, int channels) {
    p = ZeroedDoubles(kern::BatchNormScratchDoubles(channels), like, Stream(), &own);
  }
};

// Whether the forward of a 1x1 convolution is this library's. Up to 512 input
// channels it costs less than PyTorch's and the pass for the statistics; beyond,
// PyTorch's kernels move the operands between L2 and the SMs less often (1024 to 256
// channels, 50176 rows: 36 us against 25 and 7 for the statistics).
bool OwnForward(int64_t rows, int64_t k, int64_t n) {
  return k <= 512 && kern::Conv1x1Supported(rows, static_cast<int>(k), static_cast<int>(n));
}

// Whether y of a 1x1 convolution with a stride of 2 lies on every other pixel of x.
bool EveryOther(const Tensor& x) {
  return x.size(2) % 2 == 0 && x.size(3) % 2 == 0 &&
         kern::Conv1x1StrideSupported(Rows(x) / 4, static_cast<int>(x.size(3) / 2));
}

Tensor ConvForward(const Tensor& x, const Tensor& w, int64_t stride, Sums* sums) {
  const int64_t kernel = w.size(2), n = w.size(0);
  const int64_t ho = (x.size(2) - 1) / stride + 1, wo = (x.size(3) - 1) / stride + 1;
  if (kernel == 1 && OwnForward(x.size(0) * ho * wo, x.size(1), n) &&
      (stride == 1 || (stride == 2 && EveryOther(x)))) {
    kern::Conv1x1 c;
    Tensor y = NewActivations(x, n, ho, wo);
    c.x = x.data_ptr();
    c.w = w.data_ptr();
    c.y = y.data_ptr();
    c.rows = Rows(y);
    c.k = Channels(x);
    c.n = static_cast<int>(n);
    c.sums = sums->p;
    c.copies = kern::BatchNormCopies(c.n);
    c.strided_x = stride == 2;
    c.width = static_cast<int>(wo);
    c.bf16 = x.scalar_type() == at::kBFloat16;
    Check(kern::LaunchConv1x1(c, Stream()), "1x1 convolution");
    sums->ready = true;
    return y;
  }
  const int64_t pad = kernel / 2;
  return at::convolution(x, w, {}, {stride, stride}, {pad, pad}, {1, 1}, false, {0, 0}, 1)
      .contiguous(CL);
}

// The batch norm's arguments; *saved: what the backward needs of the statistics.
kern::BatchNormForward Describe(const Tensor& weight, const Tensor& bias, const Norm& norm,
                                const Sums& sums, Tensor* saved) {
  const int64_t C = weight.numel();
  *saved = at::empty({3, C}, weight.options());
  kern::BatchNormForward n;
  n.sums = sums.p;
  n.summed = sums.ready;
  n.weight = FloatPtrOrNull(weight, C, "weight");
  n.bias = FloatPtrOrNull(bias, C, "bias");
  n.eps = static_cast<float>(norm.eps);
  n.momentum = static_cast<float>(norm.momentum);
  n.saved = saved->data_ptr<float>();
  n.running_mean = norm.mean.data_ptr<float>();
  n.running_var = norm.var.data_ptr<float>();
  n.batches = norm.batches.defined() ? norm.batches.data_ptr<int64_t>() : nullptr;
  return n;
}

// relu(batch norm of x [+ residual, or batch norm of it]); signs are for the latter two.
Tensor NormForward(const Tensor& x, const kern::BatchNormForward& n, const Tensor& residual,
                   const kern::BatchNormForward* of_residual, Tensor* signs) {
  const int C = Channels(x);
  const bool bf16 = x.scalar_type() == at::kBFloat16;
  Tensor y = at::empty_like(x, x.options(), CL);
  if (residual.defined()) *signs = at::empty({Rows(x), C / 8}, x.options().dtype(at::kByte));
  uint8_t* bits = residual.defined() ? signs->data_ptr<uint8_t>() : nullptr;
  const void* r = residual.defined() ? residual.data_ptr() : nullptr;
  Check(of_residual ? kern::LaunchBatchNormPairForward(x.data_ptr(), r, y.data_ptr(), bits, Rows(x),
                                                       C, bf16, n, *of_residual, Stream())
                    : kern::LaunchBatchNormForward(x.data_ptr(), r, y.data_ptr(), bits, Rows(x), C,
                                                   bf16, n, true, Stream()),
        "batch norm forward");
  return y;
}

struct NormGradients {
  Tensor x, residual, weight, bias;
};

// Of the two batch norms whose sum is the block's output: their sums alone, or the
// gradients too.
kern::BatchNormBackward Describe(const Tensor& weight, const Tensor& saved, const Sums& sums,
                                 NormGradients* g) {
  kern::BatchNormBackward n;
  n.sums = sums.p;
  n.weight = FloatPtrOrNull(weight, weight.numel(), "weight");
  n.saved = saved.data_ptr<float>();
  if (g != nullptr) {
    g->weight = at::empty_like(weight);
    g->bias = at::empty_like(weight);
    n.dweight = g->weight.data_ptr<float>();
    n.dbias = g->bias.data_ptr<float>();
  }
  return n;
}

// signs (where defined): dy counts where the block's output was above zero;
// otherwise relu says whether this layer had a ReLU of its own.
NormGradients NormBackward(const Tensor& dy, const Tensor& x, const Tensor& weight,
                           const Tensor& saved, const Tensor& signs, bool relu,
                           bool want_residual) {
  const int C = Channels(x);
  NormGradients g;
  g.x = at::empty_like(x, x.options(), CL);
  if (want_residual) g.residual = at::empty_like(x, x.options(), CL);
  g.weight = at::empty({C}, x.options().dtype(at::kFloat));
  g.bias = at::empty({C}, x.options().dtype(at::kFloat));
  Sums sums(x, C);
  Check(kern::LaunchBatchNormBackward(
            dy.data_ptr(), signs.defined() ? signs.data_ptr<uint8_t>() : nullptr, x.data_ptr(),
            g.x.data_ptr(), want_residual ? g.residual.data_ptr() : nullptr, Rows(x), C,
            x.scalar_type() == at::kBFloat16, sums.p, FloatPtrOrNull(weight, C, "weight"),
            saved.data_ptr<float>(), g.weight.data_ptr<float>(), g.bias.data_ptr<float>(), relu,
            Stream()),
        "batch norm backward");
  return g;
}

// Gradients of a batch norm behind a 1x1 convolution and of that convolution, together.
struct TailGradients {
  Tensor a, w, weight, bias;  // of the convolution's input and weight, of the batch norm
};

bool OwnTail(const Tensor& out, const Tensor& w, int64_t stride) {
  return stride == 1 && w.size(2) == 1 &&
         kern::NormConvBackwardSupported(Rows(out), Channels(out), static_cast<int>(w.size(1)));
}

// a: the convolution's input; leaf: its weight as the user has it.
TailGradients TailBackward(const Tensor& dy, const Tensor& signs, const Tensor& x, const Tensor& a,
                           const Tensor& w, const Tensor& weight, const Tensor& saved,
                           const Tensor& leaf, const Sums& sums, bool want_a) {
  kern::NormConvBackward n;
  const auto fp32 = x.options().dtype(at::kFloat);
  TailGradients g;
  n.rows = Rows(x);
  n.cout = Channels(x);
  n.cin = Channels(a);
  n.bf16 = x.scalar_type() == at::kBFloat16;
  if (want_a) g.a = at::empty_like(a, a.options(), CL);
  g.w = leaf.is_non_overlapping_and_dense()
            ? at::empty_strided(leaf.sizes(), leaf.strides(), leaf.options())
            : at::empty(leaf.sizes(), leaf.options());
  g.weight = at::empty({n.cout}, fp32);
  g.bias = at::empty({n.cout}, fp32);
  const Tensor partial =
      at::empty({kern::NormConvBackwardParts(n.rows), n.cout, n.cin}, fp32,
                at::MemoryFormat::Contiguous);
  n.dy = dy.data_ptr();
  n.x = x.data_ptr();
  n.a = a.data_ptr();
  n.w = w.data_ptr();
  n.signs = signs.data_ptr<uint8_t>();
  n.da = want_a ? g.a.data_ptr() : nullptr;
  n.dw = g.w.data_ptr();
  n.dw_fp32 = g.w.scalar_type() == at::kFloat;
  n.dw_stride_o = g.w.stride(0);
  n.dw_stride_i = g.w.stride(1);
  n.sums = sums.p;
  n.summed = sums.ready;
  n.gamma = FloatPtrOrNull(weight, n.cout, "weight");
  n.saved = saved.data_ptr<float>();
  n.dgamma = g.weight.data_ptr<float>();
  n.dbeta = g.bias.data_ptr<float>();
  n.partial = partial.data_ptr<float>();
  Check(kern::LaunchNormConvBackward(n, Stream()), "batch norm and convolution backward");
  return g;
}

// PyTorch's gradients of a convolution: of the input (where wanted) and the weight.
std::pair<Tensor, Tensor> ConvBackward(const Tensor& dy, const Tensor& x, const Tensor& w,
                                       int64_t stride, bool want_x, bool want_w) {
  if (!want_x && !want_w) return {};
  const int64_t pad = w.size(2) / 2;
  auto g = at::convolution_backward(dy, x, w, c10::nullopt, {stride, stride}, {pad, pad}, {1, 1},
                                    false, {0, 0}, 1, {want_x, want_w, false});
  return {want_x ? std::get<0>(g).contiguous(CL) : Tensor(), std::get<1>(g)};
}

// Gradient of a 1x1 convolution's input, plus `add` (where `signs`, if defined, say
// so). every_other: the result is `add` itself, changed at every other pixel.
Tensor ConvInputGradient(const Tensor& dy, const Tensor& w, const Tensor& add, const Tensor& signs,
                         bool every_other) {
  kern::Conv1x1 c;
  Tensor dx = every_other ? add : at::empty_like(add, add.options(), CL);
  c.x = dy.data_ptr();
  c.w = w.data_ptr();
  c.y = dx.data_ptr();
  c.add = add.data_ptr();
  if (signs.defined()) c.signs = signs.data_ptr<uint8_t>();
  c.rows = Rows(dy);
  c.k = Channels(dy);
  c.n = Channels(dx);
  c.w_transposed = true;
  c.strided_y = every_other;
  c.width = static_cast<int>(dy.size(3));
  c.bf16 = dy.scalar_type() == at::kBFloat16;
  Check(kern::LaunchConv1x1(c, Stream()), "gradient of a 1x1 convolution");
  return dx;
}

// A weight with the value that a forward worked on, for gradients of gradients: the
// leaf may have changed since, and its gradients are those of the cast.
class AsOfForward : public torch::autograd::Function<AsOfForward> {
 public:
  static Variable forward(AutogradContext* ctx, const Variable& leaf, const Variable& value) {
    ctx->saved_data["type"] = static_cast<int64_t>(leaf.scalar_type());
    return value.clone();
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    if (!grads[0].defined()) return {Tensor(), Tensor()};
    const auto type = static_cast<at::ScalarType>(ctx->saved_data["type"].toInt());
    return {grads[0].to(type), Tensor()};
  }
};

// The block by PyTorch's operations, for gradients of its gradients. w: in the type of x.
Tensor Composition(const Tensor& x, const std::array<Tensor, LAYERS>& w,
                   const std::array<Tensor, LAYERS>& g, const std::array<Tensor, LAYERS>& b,
                   const std::vector<double>& eps, int64_t stride) {
  auto layer = [&](int i, const Tensor& in, int64_t s) {
    const int64_t pad = w[i].size(2) / 2;
    const Tensor out =
        at::convolution(in, w[i], {}, {s, s}, {pad, pad}, {1, 1}, false, {0, 0}, 1);
    return at::batch_norm(out, g[i], b[i], {}, {}, true, 0.0, eps[i], true);
  };
  const Tensor a1 = at::relu(layer(0, x, 1)), a2 = at::relu(layer(1, a1, stride));
  const Tensor skip = w[DOWN].defined() ? layer(DOWN, x, stride) : x;
  return at::relu(layer(2, a2, 1) + skip);
}

// What a backward has saved, by layer.
struct Kept {
  Tensor x, a1, a2, signs;
  std::array<Tensor, LAYERS> w, gammas, out, saved;
};

// Saved tensors went through the user's hooks, if there are any. Their values and
// shapes are the forward's; the kernels read them by pointer, so that is looked at.
void CheckKept(const Kept& k, int layers, const Tensor& dy, int64_t stride) {
  bool ok = k.x.defined() && k.x.dim() == 4;
  auto is = [&](const Tensor& t, at::ScalarType type, at::IntArrayRef sizes) {
    ok = ok && t.defined() && t.layout() == at::kStrided && t.device() == dy.device() &&
         t.scalar_type() == type && t.sizes() == sizes;
  };
  std::array<int64_t, LAYERS> c;
  for (int i = 0; i < layers; ++i) c[i] = k.gammas[i].defined() ? k.gammas[i].numel() : 0;
  if (ok) {
    const at::ScalarType type = k.x.scalar_type();
    const int64_t n = dy.size(0), h = k.x.size(2), w = k.x.size(3), ho = dy.size(2),
                  wo = dy.size(3), cx = k.x.size(1);
    ok = (type == at::kBFloat16 || type == at::kHalf) && (h - 1) / stride + 1 == ho &&
         (w - 1) / stride + 1 == wo && c[2] == dy.size(1);
    is(k.x, type, {n, cx, h, w});
    is(k.a1, type, {n, c[0], h, w});
    is(k.a2, type, {n, c[1], ho, wo});
    is(k.signs, at::kByte, {n * ho * wo, c[2] / 8});
    is(k.w[0], type, {c[0], cx, 1, 1});
    is(k.w[1], type, {c[1], c[0], 3, 3});
    is(k.w[2], type, {c[2], c[1], 1, 1});
    if (layers > DOWN) is(k.w[DOWN], type, {c[2], cx, 1, 1});
    is(k.out[0], type, {n, c[0], h, w});
    is(k.out[1], type, {n, c[1], ho, wo});
    for (int i = 2; i < layers; ++i) is(k.out[i], type, {n, c[2], ho, wo});
    for (int i = 0; i < layers; ++i) {
      is(k.gammas[i], at::kFloat, k.gammas[i].sizes());
      is(k.saved[i], at::kFloat, {3, c[i]});
    }
  }
  TORCH_CHECK(ok, "bottleneck: a saved tensor has come back with another shape, type or device");
}

class Bottleneck : public torch::autograd::Function<Bottleneck> {
 public:
  static Variable forward(AutogradContext* ctx, const Variable& x, const Variable& w0,
                          const Variable& g0, const Variable& b0, const Variable& w1,
                          const Variable& g1, const Variable& b1, const Variable& w2,
                          const Variable& g2, const Variable& b2,
                          const c10::optional<Tensor>& w3o, const c10::optional<Tensor>& g3o,
                          const c10::optional<Tensor>& b3o, const Block& block) {
    const bool down = w3o.has_value();
    const Tensor w3 = down ? *w3o : Tensor(), g3 = down ? *g3o : Tensor(),
                 b3 = down ? *b3o : Tensor();
    c10::impl::ExcludeDispatchKeyGuard no_autocast(c10::DispatchKey::AutocastCUDA);
    const std::array<Tensor, LAYERS> weights = {w0, w1, w2, w3}, gammas = {g0, g1, g2, g3},
                                     betas = {b0, b1, b2, b3};
    c10::cuda::CUDAGuard guard(x.device());
    const auto w = Cast(weights, block.type);
    std::array<Tensor, LAYERS> out, saved;  // of the convolutions; of the batch norms
    Tensor signs;
    std::array<kern::BatchNormForward, LAYERS> norms;
    std::vector<Sums> sums;  // kept until the kernels are launched
    sums.reserve(LAYERS);
    auto convolve = [&](int i, const Tensor& in, int64_t stride) {
      sums.emplace_back(x, static_cast<int>(w[i].size(0)));
      out[i] = ConvForward(in, w[i], stride, &sums.back());
      norms[i] = Describe(gammas[i], betas[i], block.norms[i], sums.back(), &saved[i]);
    };
    convolve(0, x, 1);
    const Tensor a1 = NormForward(out[0], norms[0], {}, nullptr, nullptr);
    convolve(1, a1, block.stride);
    const Tensor a2 = NormForward(out[1], norms[1], {}, nullptr, nullptr);
    if (down) convolve(DOWN, x, block.stride);
    convolve(2, a2, 1);
    const Tensor y = NormForward(out[2], norms[2], down ? out[DOWN] : x,
                                 down ? &norms[DOWN] : nullptr, &signs);
    // Like relu's own backward, this one refuses to run when somebody has
    // changed y in place, although it does not read it.
    variable_list keep = {x, y, a1, a2, signs};
    for (int i = 0; i < (down ? LAYERS : DOWN); ++i)
      for (const Tensor& t : {w[i], gammas[i], out[i], saved[i]}) keep.push_back(t);
    ctx->save_for_backward(keep);
    std::vector<double> eps;
    for (const Norm& norm : block.norms) eps.push_back(norm.eps);
    ctx->saved_data.reserve(3 + 2 * LAYERS);
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["stride"] = block.stride;
    // For the edges of gradients of gradients. Every backward works on the casts: the
    // weights may have changed since.
    const int layers = down ? LAYERS : DOWN;
    for (int i = 0; i < layers; ++i) ctx->saved_data[WEIGHT[i]] = weights[i];
    // A gradient needs no betas, a gradient of a gradient does: changes are noticed
    // there alone.
    std::vector<int64_t> versions;
    for (int i = 0; i < layers; ++i) {
      ctx->saved_data[BETA[i]] = betas[i];
      versions.push_back(betas[i].is_inference() ? 0 : betas[i]._version());
    }
    ctx->saved_data["versions"] = versions;
    return y;
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    // Inputs: x, then weight, gamma and beta of each layer.
    variable_list result(1 + 3 * LAYERS + 1);
    if (!grads[0].defined()) return result;
    const variable_list keep = ctx->get_saved_variables();
    const bool down = keep.size() > 5 + 4 * DOWN;
    const int layers = down ? LAYERS : DOWN;
    const int64_t stride = ctx->saved_data["stride"].toInt();
    Kept k;
    Tensor &x = k.x, &a1 = k.a1, &a2 = k.a2, &signs = k.signs;
    auto &w = k.w, &gammas = k.gammas, &out = k.out, &saved = k.saved;
    std::array<Tensor, LAYERS> weights;
    x = keep[0], a1 = keep[2], a2 = keep[3], signs = keep[4];
    for (int i = 0; i < layers; ++i) {
      const size_t at = 5 + 4 * static_cast<size_t>(i);
      w[i] = keep[at], gammas[i] = keep[at + 1], out[i] = keep[at + 2], saved[i] = keep[at + 3];
      weights[i] = ctx->saved_data[WEIGHT[i]].toTensor();
    }
    CheckKept(k, layers, grads[0], stride);
    auto wanted = [&](int input) { return ctx->needs_input_grad(input); };
    if (at::GradMode::is_enabled()) {
      const auto versions = ctx->saved_data["versions"].toIntVector();
      std::array<Tensor, LAYERS> betas;
      for (int i = 0; i < layers; ++i) {
        betas[i] = ctx->saved_data[BETA[i]].toTensor();
        TORCH_CHECK(betas[i].is_inference() || betas[i]._version() == versions[i],
                    "one of the variables needed for gradient computation has been modified by an "
                    "inplace operation: the bias of a block's batch norm");
      }
      variable_list inputs;
      std::vector<size_t> to;
      auto add = [&](size_t i, const Tensor& t) {
        if (t.defined() && wanted(static_cast<int>(i))) inputs.push_back(t), to.push_back(i);
      };
      add(0, x);
      for (int i = 0; i < LAYERS; ++i)
        add(1 + 3 * i, weights[i]), add(2 + 3 * i, gammas[i]), add(3 + 3 * i, betas[i]);
      std::array<Tensor, LAYERS> then;
      for (int i = 0; i < layers; ++i) then[i] = AsOfForward::apply(weights[i], w[i].detach());
      const Tensor y =
          Composition(x, then, gammas, betas, ctx->saved_data["eps"].toDoubleVector(), stride);
      const variable_list g = torch::autograd::grad({y}, inputs, {grads[0]}, true, true, true);
      for (size_t i = 0; i < to.size(); ++i) result[to[i]] = g[i];
      return result;
    }
    c10::cuda::CUDAGuard guard(x.device());
    x = Dense(x, CL), a1 = Dense(a1, CL), a2 = Dense(a2, CL);
    signs = Dense(signs, at::MemoryFormat::Contiguous);
    for (int i = 0; i < layers; ++i) {
      out[i] = Dense(out[i], CL);
      if (i != 1) w[i] = Dense(w[i], at::MemoryFormat::Contiguous);  // (the 3x3 is PyTorch's)
      gammas[i] = Dense(gammas[i], at::MemoryFormat::Contiguous);
      saved[i] = Dense(saved[i], at::MemoryFormat::Contiguous);
    }
    Tensor dy = grads[0];
    if (dy.scalar_type() != x.scalar_type()) dy = dy.to(x.scalar_type());
    dy = Activations(dy.contiguous(CL), "dy");
    std::array<Tensor, LAYERS> dw;
    auto norm = [&](int i, const Tensor& d, const Tensor& mask, bool want_residual) {
      NormGradients g = NormBackward(d, out[i], gammas[i], saved[i], mask, true, want_residual);
      if (wanted(2 + 3 * i)) result[2 + 3 * i] = g.weight;
      if (wanted(3 + 3 * i)) result[3 + 3 * i] = g.bias;
      return g;
    };
    const bool want_x = wanted(0);
    // Whether anything before the first (the second) ReLU wants a gradient: the input and
    // the first layers of a network are often frozen.
    const bool need_a1 = want_x || wanted(1) || wanted(2) || wanted(3);
    const bool need_a2 = need_a1 || wanted(4) || wanted(5) || wanted(6);
    // The gradients of x through the first convolution and through the skip
    // connection meet in a kernel of this library where it takes the shapes.
    const bool fused = kern::Conv1x1Supported(Rows(x), Channels(out[0]), Channels(x));
    Tensor da2, da1, dx, skip, mask;
    if (!down && fused) skip = dy, mask = signs;
    auto keep_norm = [&](int i, const NormGradients& g) {
      if (wanted(2 + 3 * i)) result[2 + 3 * i] = g.weight;
      if (wanted(3 + 3 * i)) result[3 + 3 * i] = g.bias;
    };
    // The batch norms of the end of the block and of its skip connection have dy in
    // common. Their convolutions' gradients come from the kernel that forms theirs
    // (OwnTail) or from what is formed here. The kernel stores no gradient of the skip
    // connection: where x itself is that, another kernel (`fused`) has to add it.
    const bool tails = OwnTail(out[2], w[2], 1) &&
                       (down ? OwnTail(out[DOWN], w[DOWN], stride) : fused || !want_x);
    Sums sums2, sums3;
    if (down || tails) sums2 = Sums(x, Channels(out[2]));
    if (down) sums3 = Sums(x, Channels(out[2]));
    NormGradients g2, g3;
    if (down) {
      const bool bf16 = x.scalar_type() == at::kBFloat16;
      const kern::BatchNormBackward n2 = Describe(gammas[2], saved[2], sums2, &g2),
                                    n3 = Describe(gammas[DOWN], saved[DOWN], sums3, &g3);
      const int C = Channels(dy);
      if (tails) {
        Check(kern::LaunchBatchNormPairSums(dy.data_ptr(), signs.data_ptr<uint8_t>(),
                                            out[2].data_ptr(), out[DOWN].data_ptr(), Rows(dy), C,
                                            bf16, n2, n3, Stream()),
              "batch norm backward");
        sums2.ready = sums3.ready = true;
      } else {
        g2.x = at::empty_like(out[2], out[2].options(), CL);
        g3.x = at::empty_like(out[2], out[2].options(), CL);
        Check(kern::LaunchBatchNormPairBackward(
                  dy.data_ptr(), signs.data_ptr<uint8_t>(), out[2].data_ptr(),
                  out[DOWN].data_ptr(), g2.x.data_ptr(), g3.x.data_ptr(), Rows(dy), C, bf16, n2,
                  n3, Stream()),
              "batch norm backward");
        keep_norm(2, g2);
        keep_norm(DOWN, g3);
      }
    } else if (!tails) {
      g2 = norm(2, dy, signs, want_x && !fused);
      if (want_x && !fused) skip = g2.residual;
    }
    // The gradient of the convolution's input `in`, where wanted.
    auto tail = [&](int i, const Tensor& in, int64_t s, Tensor d_out, const Sums& sums,
                    bool want_in) {
      Tensor d_in;
      if (!want_in && !wanted(1 + 3 * i) && !wanted(2 + 3 * i) && !wanted(3 + 3 * i)) return d_in;
      if (tails) {
        const TailGradients g = TailBackward(dy, signs, out[i], in, w[i], gammas[i], saved[i],
                                             weights[i], sums, want_in);
        if (wanted(2 + 3 * i)) result[2 + 3 * i] = g.weight;
        if (wanted(3 + 3 * i)) result[3 + 3 * i] = g.bias;
        if (wanted(1 + 3 * i)) result[1 + 3 * i] = g.w;
        return g.a;
      }
      std::tie(d_in, dw[i]) = ConvBackward(d_out, in, w[i], s, want_in, wanted(1 + 3 * i));
      return d_in;
    };
    da2 = tail(2, a2, 1, g2.x, sums2, need_a2);
    g2.x.reset();
    Tensor d2, d1;
    if (need_a2) d2 = norm(1, da2, {}, false).x;
    da2.reset();
    std::tie(da1, dw[1]) = ConvBackward(d2, a1, w[1], stride, need_a1, wanted(4));
    if (need_a1) d1 = norm(0, da1, {}, false).x;
    da1.reset();
    if (down) {
      const bool scatter = stride == 2 && EveryOther(x) &&
                           kern::Conv1x1Supported(Rows(dy), Channels(dy), Channels(x));
      if (want_x && scatter) {
        // Its gradient of x is zero but for every fourth pixel: added in place.
        std::tie(dx, dw[0]) = ConvBackward(d1, x, w[0], 1, true, wanted(1));
        ConvInputGradient(g3.x, w[DOWN], dx, {}, true);
        dw[DOWN] = ConvBackward(g3.x, x, w[DOWN], stride, false, wanted(10)).second;
      } else {
        skip = tail(DOWN, x, stride, g3.x, sums3, want_x);
      }
    }
    if (!dx.defined()) {
      std::tie(dx, dw[0]) = ConvBackward(d1, x, w[0], 1, want_x && !fused, wanted(1));
      if (want_x) dx = fused ? ConvInputGradient(d1, w[0], skip, mask, false) : dx.add_(skip);
    }
    if (want_x) result[0] = dx;
    // (Weights whose gradients are there already have no dw.)
    for (int i = 0; i < LAYERS; ++i)
      if (dw[i].defined() && weights[i].scalar_type() != at::kFloat) {
        result[1 + 3 * i] = dw[i];
        dw[i].reset();
      }
    const auto wide = Cast(dw, at::kFloat, &weights);
    for (int i = 0; i < LAYERS; ++i)
      if (wide[i].defined()) result[1 + 3 * i] = wide[i];
    return result;
  }
};

}  // namespace

void BindBottleneck(py::module_& m) {
  // (x, [weight, gamma, beta, running mean, running variance, count of batches or
  //  None] per layer, [(momentum, eps)] per layer, stride)
  // Wrapped, so that what a saved-tensor hook raises arrives as what it is (a
  // checkpointed region ends its second forward that way), and so do PyTorch's errors.
  m.def("bottleneck", torch::wrap_pybind_function([](
                          const Tensor& x,
                          const std::vector<std::vector<c10::optional<Tensor>>>& layers,
                          const std::vector<std::pair<double, double>>& rates, int64_t stride) {
    TORCH_CHECK(layers.size() >= DOWN && layers.size() <= LAYERS && rates.size() == layers.size(),
                "bottleneck: three or four layers");
    CheckActivations(x, "x");
    TORCH_CHECK(x.numel() > 0 && reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0,
                "bottleneck: x must have elements and start on a 16-byte boundary");
    TORCH_CHECK(stride == 1 || stride == 2, "bottleneck: a stride of 1 or 2");
    Block block;
    block.stride = stride;
    block.type = x.scalar_type();
    std::array<Tensor, 3 * LAYERS> p;
    for (size_t i = 0; i < layers.size(); ++i) {
      TORCH_CHECK(layers[i].size() == 6, "bottleneck: six tensors per layer");
      for (int k = 0; k < 5; ++k)
        TORCH_CHECK(layers[i][k].has_value() && layers[i][k]->device() == x.device(),
                    "bottleneck: tensors of a layer must be on the device of x");
      for (int k = 0; k < 3; ++k) p[3 * i + k] = *layers[i][k];
      TORCH_CHECK(p[3 * i].dim() == 4, "bottleneck: weights of convolutions are 4-D");
      TORCH_CHECK(p[3 * i].scalar_type() == at::kFloat || p[3 * i].scalar_type() == block.type,
                  "bottleneck: weights of convolutions are float32 or of the type of x");
      const int64_t C = p[3 * i].size(0);
      for (int k = 1; k < 5; ++k) FloatPtrOrNull(layers[i][k], C, "a batch norm's tensor");
      Norm& n = block.norms[i];
      n.mean = *layers[i][3];
      n.var = *layers[i][4];
      if (layers[i][5].has_value()) n.batches = *layers[i][5];
      TORCH_CHECK(!n.batches.defined() || (n.batches.is_cuda() && n.batches.numel() == 1 &&
                                           n.batches.scalar_type() == at::kLong),
                  "num_batches_tracked must be one int64 on the GPU");
      n.momentum = rates[i].first;
      n.eps = rates[i].second;
      TORCH_CHECK(kern::BatchNormSupported(1, static_cast<int>(C)), "bottleneck does not support ",
                  C, " channels");
    }
    // The kernels take the sizes of a weight from its neighbours.
    const bool down = layers.size() > DOWN;
    const int64_t c0 = p[0].size(0), c1 = p[3].size(0), c2 = p[6].size(0), cx = x.size(1);
    const auto is = [&](int k, at::IntArrayRef sizes) { return p[k].sizes() == sizes; };
    TORCH_CHECK(is(0, {c0, cx, 1, 1}) && is(3, {c1, c0, 3, 3}) && is(6, {c2, c1, 1, 1}) &&
                    (down ? is(9, {c2, cx, 1, 1}) : c2 == cx && stride == 1),
                "bottleneck: the weights' shapes do not match x and one another");
    py::gil_scoped_release unlocked;
    auto skip = [&](int k) {
      return p[k].defined() ? c10::optional<Tensor>(p[k]) : c10::nullopt;
    };
    return Bottleneck::apply(x, p[0], p[1], p[2], p[3], p[4], p[5], p[6], p[7], p[8], skip(9),
                             skip(10), skip(11), block);
  }));
}

}  // namespace hvd
