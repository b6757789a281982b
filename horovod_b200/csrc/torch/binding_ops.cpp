// Python entry points of the model-side kernels but those of the residual block.
// They run on the caller's current CUDA stream like any torch op.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <atomic>
#include <cstdint>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "../kernels/kernels.h"
#include "model_ops.h"

namespace hvd {

void CheckActivations(const at::Tensor& t, const char* what) {
  TORCH_CHECK(t.is_cuda(), what, " must be a CUDA tensor");
  TORCH_CHECK(t.dim() == 4, what, " must be 4-D (N, C, H, W)");
  TORCH_CHECK(t.scalar_type() == at::kBFloat16 || t.scalar_type() == at::kHalf, what,
              " must be bfloat16 or float16");
  TORCH_CHECK(t.is_contiguous(at::MemoryFormat::ChannelsLast), what,
              " must be contiguous in channels_last memory format");
}

// t, checked, for kernels that access it 16 bytes at a time: a view that starts
// between two such boundaries (a slice of a flat buffer) is copied.
at::Tensor Activations(const at::Tensor& t, const char* what) {
  CheckActivations(t, what);
  if (reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0) return t;
  return t.clone(at::MemoryFormat::ChannelsLast);
}

const float* FloatPtrOrNull(const c10::optional<at::Tensor>& t, int64_t channels,
                            const char* what) {
  if (!t.has_value() || !t->defined()) return nullptr;
  TORCH_CHECK(t->is_cuda() && t->scalar_type() == at::kFloat && t->is_contiguous() &&
                  t->numel() == channels,
              what, " must be a contiguous float32 CUDA vector with one entry per channel");
  return t->data_ptr<float>();
}

// Zero-filled scratch for the batch-norm reductions without a fill launch per
// call: slices are handed out from a per-stream pool that is cleared with one
// memset whenever it has been used up. The memset is queued behind the consumers of
// all slices whose `own` is gone, so a slice is zero when the first kernel that was
// given it runs. Where a slice is still held, by the caller itself (a block of layers
// keeps the sums of one layer while it asks for the next one's) or by another thread
// that launches to the same stream, a memset could erase sums that nobody has read or
// come before kernels that still add to theirs: such a pool is left to its holders and
// a new one takes its place. A stream that is being captured gets memory of its own,
// filled inside the graph: every replay has to start from zeros, and slices of the
// pool would be cleared by none.
double* ZeroedDoubles(int64_t count, const at::Tensor& like, cudaStream_t stream,
                      at::Tensor* own) {
  // (The default stream cannot be captured. Asking takes 0.2 to 0.4 us on the host,
  // of 9.4 for a small forward.)
  if (stream != nullptr &&
      c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) {
    *own = at::zeros({count}, like.options().dtype(at::kDouble));
    return own->data_ptr<double>();
  }
  struct Pool {
    at::Tensor buf;
    int64_t used = 0;
  };
  constexpr int64_t POOL_DOUBLES = 1 << 20;  // 8 MB
  static std::mutex mu;
  static std::map<std::pair<int, cudaStream_t>, Pool> pools;
  TORCH_CHECK(count <= POOL_DOUBLES, "batch norm scratch request too large");
  const int64_t need = (count + 31) / 32 * 32;  // 256-byte slices
  // Memory is allocated and given back outside the lock: the allocator may ask for the
  // interpreter's lock (to note a stack), which a thread that waits for this one can hold.
  at::Tensor fresh, old;
  for (;;) {
    {
      std::lock_guard<std::mutex> lock(mu);
      Pool& p = pools[{like.get_device(), stream}];
      bool room = p.buf.defined() && p.used + need <= POOL_DOUBLES;
      if (!room && p.buf.defined() && p.buf.use_count() == 1) {
        // Another thread's launches came before it let go of its slice.
        std::atomic_thread_fence(std::memory_order_acquire);
        const cudaError_t err =
            cudaMemsetAsync(p.buf.data_ptr(), 0, POOL_DOUBLES * sizeof(double), stream);
        TORCH_CHECK(err == cudaSuccess, "batch norm scratch: ", cudaGetErrorString(err));
        p.used = 0;
        room = true;
      }
      if (!room && fresh.defined()) {
        old = std::move(p.buf);
        p.buf = std::move(fresh);
        p.used = 0;
        room = true;
      }
      if (room) {
        *own = p.buf;
        double* out = p.buf.data_ptr<double>() + p.used;
        p.used += need;
        return out;
      }
    }
    fresh = at::zeros({POOL_DOUBLES}, like.options().dtype(at::kDouble));
  }
}

namespace {

// Whether t holds fp32 values next to p's, element for element.
bool SgdLike(const at::Tensor& p, const at::Tensor& t) {
  return t.defined() && t.layout() == at::kStrided && t.scalar_type() == at::kFloat &&
         t.device() == p.device() && t.sizes() == p.sizes() && t.strides() == p.strides();
}

// What the multi-tensor SGD kernel takes: fp32 on a GPU, a gradient of the
// same memory layout, and no gaps in it.
bool SgdReady(const at::Tensor& p, const at::Tensor& g) {
  return p.is_cuda() && p.layout() == at::kStrided && p.scalar_type() == at::kFloat &&
         SgdLike(p, g) && p.is_non_overlapping_and_dense();
}


struct NormOutputs {
  at::Tensor y, saved, signs;
};

NormOutputs NormForward(at::Tensor x, c10::optional<at::Tensor> residual,
                        const c10::optional<at::Tensor>& weight,
                        const c10::optional<at::Tensor>& bias,
                        const c10::optional<at::Tensor>& running_mean,
                        const c10::optional<at::Tensor>& running_var, double momentum, double eps,
                        bool relu, const c10::optional<at::Tensor>& batches) {
  x = Activations(x, "x");
  const int64_t C = x.size(1), M = x.numel() / C;
  TORCH_CHECK(kern::BatchNormSupported(M, static_cast<int>(C)),
              "fused batch norm does not support ", C, " channels");
  const void* res = nullptr;
  if (residual.has_value() && residual->defined()) {
    residual = Activations(*residual, "residual");
    TORCH_CHECK(residual->sizes() == x.sizes() && residual->scalar_type() == x.scalar_type(),
                "residual must match x");
    res = residual->data_ptr();
  }
  c10::cuda::CUDAGuard guard(x.device());
  cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  at::Tensor y = at::empty_like(x, x.options(), at::MemoryFormat::ChannelsLast);
  at::Tensor saved = at::empty({3, C}, x.options().dtype(at::kFloat));
  at::Tensor signs;
  if (relu && res != nullptr) signs = at::empty({M, C / 8}, x.options().dtype(at::kByte));
  at::Tensor own;
  double* sums =
      ZeroedDoubles(kern::BatchNormScratchDoubles(static_cast<int>(C)), x, stream, &own);
  float* rm = nullptr;
  float* rv = nullptr;
  if (running_mean.has_value() && running_mean->defined()) {
    rm = const_cast<float*>(FloatPtrOrNull(running_mean, C, "running_mean"));
    rv = const_cast<float*>(FloatPtrOrNull(running_var, C, "running_var"));
    TORCH_CHECK(rv != nullptr, "running_var must accompany running_mean");
  }
  int64_t* count = nullptr;
  if (batches.has_value() && batches->defined()) {
    TORCH_CHECK(batches->device() == x.device() && batches->scalar_type() == at::kLong &&
                    batches->numel() == 1,
                "num_batches_tracked must be one int64 on the device of x");
    count = batches->data_ptr<int64_t>();
  }
  kern::BatchNormForward n;
  n.sums = sums;
  n.weight = FloatPtrOrNull(weight, C, "weight");
  n.bias = FloatPtrOrNull(bias, C, "bias");
  n.eps = static_cast<float>(eps);
  n.momentum = static_cast<float>(momentum);
  n.saved = saved.data_ptr<float>();
  n.running_mean = rm;
  n.running_var = rv;
  n.batches = count;
  const cudaError_t err = kern::LaunchBatchNormForward(
      x.data_ptr(), res, y.data_ptr(), signs.defined() ? signs.data_ptr<uint8_t>() : nullptr, M,
      static_cast<int>(C), x.scalar_type() == at::kBFloat16, n, relu, stream);
  TORCH_CHECK(err == cudaSuccess, "fused batch norm forward: ", cudaGetErrorString(err));
  return {y, saved, signs};
}

struct NormGradients {
  at::Tensor x, residual, weight, bias;
};

NormGradients NormBackward(at::Tensor dy, at::Tensor x, const c10::optional<at::Tensor>& weight,
                           at::Tensor saved, const c10::optional<at::Tensor>& signs,
                           bool relu, bool want_dresidual) {
  x = Activations(x, "x");
  dy = Activations(dy, "dy");
  TORCH_CHECK(dy.sizes() == x.sizes() && dy.scalar_type() == x.scalar_type(), "dy must match x");
  const int64_t C = x.size(1), M = x.numel() / C;
  TORCH_CHECK(saved.is_cuda() && saved.scalar_type() == at::kFloat && saved.is_contiguous() &&
                  saved.numel() == 3 * C,
              "saved must be the tensor returned by bn_forward");
  // (A saved-tensor hook may have moved it.)
  if (reinterpret_cast<uintptr_t>(saved.data_ptr()) % 16 != 0) saved = saved.clone();
  const uint8_t* sign_bits = nullptr;
  if (signs.has_value() && signs->defined()) {
    TORCH_CHECK(signs->is_cuda() && signs->scalar_type() == at::kByte &&
                    signs->is_contiguous() && signs->numel() * 8 == x.numel(),
                "signs must be the tensor returned by bn_forward");
    sign_bits = signs->data_ptr<uint8_t>();
  }
  c10::cuda::CUDAGuard guard(x.device());
  cudaStream_t stream = at::cuda::getCurrentCUDAStream();
  at::Tensor dx = at::empty_like(x, x.options(), at::MemoryFormat::ChannelsLast);
  at::Tensor dres;
  if (want_dresidual) dres = at::empty_like(x, x.options(), at::MemoryFormat::ChannelsLast);
  auto fopt = x.options().dtype(at::kFloat);
  at::Tensor dweight = at::empty({C}, fopt), dbias = at::empty({C}, fopt);
  at::Tensor own;
  double* sums =
      ZeroedDoubles(kern::BatchNormScratchDoubles(static_cast<int>(C)), x, stream, &own);
  cudaError_t err = kern::LaunchBatchNormBackward(
      dy.data_ptr(), sign_bits, x.data_ptr(), dx.data_ptr(),
      want_dresidual ? dres.data_ptr() : nullptr, M, static_cast<int>(C),
      x.scalar_type() == at::kBFloat16, sums,
      FloatPtrOrNull(weight, C, "weight"), saved.data_ptr<float>(), dweight.data_ptr<float>(),
      dbias.data_ptr<float>(), relu, stream);
  TORCH_CHECK(err == cudaSuccess, "fused batch norm backward: ", cudaGetErrorString(err));
  return {dx, dres, dweight, dbias};
}

c10::optional<at::Tensor> OrNone(const at::Tensor& t) {
  return t.defined() ? c10::optional<at::Tensor>(t) : c10::nullopt;
}

// The layer as an autograd node. In Python (horovod_b200/ops/batch_norm.py keeps
// such a node for what this one cannot take part in), the node's own work took
// 45 us of a forward and backward of 110 on the host.
class NormNode : public torch::autograd::Function<NormNode> {
 public:
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& x,
                            c10::optional<at::Tensor> residual,
                            const c10::optional<at::Tensor>& weight,
                            const c10::optional<at::Tensor>& bias,
                            const c10::optional<at::Tensor>& running_mean,
                            const c10::optional<at::Tensor>& running_var, double momentum,
                            double eps, bool relu, c10::optional<at::Tensor> batches) {
    if (residual.has_value()) residual = residual->contiguous(at::MemoryFormat::ChannelsLast);
    if (batches.has_value() &&
        (batches->device() != x.device() || batches->scalar_type() != at::kLong)) {
      batches->add_(1);
      batches = c10::nullopt;
    }
    const NormOutputs o = NormForward(x, residual, weight, bias, running_mean, running_var,
                                      momentum, eps, relu, batches);
    // The kernels do without y; like relu's own backward, this one still
    // refuses to run when somebody has changed it in place.
    ctx->save_for_backward({x, relu ? o.y : at::Tensor(), weight.value_or(at::Tensor()), o.saved,
                            o.signs});
    ctx->saved_data["flags"] = static_cast<int64_t>((relu ? 1 : 0) | (residual.has_value() ? 2 : 0) |
                                                    (weight.has_value() ? 4 : 0) |
                                                    (bias.has_value() ? 8 : 0));
    return o.y;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx,
                                                 torch::autograd::variable_list grads) {
    torch::autograd::variable_list result(10);
    if (!grads[0].defined()) return result;
    const auto keep = ctx->get_saved_variables();
    const at::Tensor &x = keep[0], &weight = keep[2], &saved = keep[3], &signs = keep[4];
    const int64_t flags = ctx->saved_data["flags"].toInt();
    at::Tensor dy = grads[0];
    if (dy.scalar_type() != x.scalar_type()) dy = dy.to(x.scalar_type());
    dy = dy.contiguous(at::MemoryFormat::ChannelsLast);
    // The edges of the node are those of the tensors that were given.
    const NormGradients g = NormBackward(dy, x, OrNone(weight), saved, OrNone(signs), flags & 1,
                                         (flags & 2) != 0 && ctx->needs_input_grad(1));
    result[0] = g.x;
    result[1] = g.residual;
    if (flags & 4) result[2] = g.weight;
    if (flags & 8) result[3] = g.bias;
    return result;
  }
};

}  // namespace

void BindModelOps(py::module_& m) {
  m.def("bn_supported", [](int64_t rows, int64_t channels) {
    return kern::BatchNormSupported(rows, static_cast<int>(channels));
  });
  // (x, residual?, weight?, bias?, running_mean?, running_var?, momentum, eps, relu,
  //  num_batches_tracked?)
  //   -> (y, saved, signs or None): saved holds what the backward needs of the
  //      statistics, signs (with a residual and a ReLU) which outputs are above zero
  m.def("bn_forward", [](const at::Tensor& x, const c10::optional<at::Tensor>& residual,
                         const c10::optional<at::Tensor>& weight,
                         const c10::optional<at::Tensor>& bias,
                         const c10::optional<at::Tensor>& running_mean,
                         const c10::optional<at::Tensor>& running_var, double momentum, double eps,
                         bool relu, const c10::optional<at::Tensor>& batches) {
    const NormOutputs o = NormForward(x, residual, weight, bias, running_mean, running_var,
                                      momentum, eps, relu, batches);
    return std::make_tuple(o.y, o.saved, OrNone(o.signs));
  });
  // (dy, x, weight?, saved, signs?, relu, want_dresidual)
  //   -> (dx, dresidual or None, dweight, dbias)
  m.def("bn_backward", [](const at::Tensor& dy, const at::Tensor& x,
                          const c10::optional<at::Tensor>& weight, const at::Tensor& saved,
                          const c10::optional<at::Tensor>& signs, bool relu,
                          bool want_dresidual) {
    const NormGradients g = NormBackward(dy, x, weight, saved, signs, relu, want_dresidual);
    return std::make_tuple(g.x, OrNone(g.residual), g.weight, g.bias);
  });
  // The whole layer, differentiable: y, or None where the kernels cannot take the
  // call (the caller then composes PyTorch's operations). Wrapped, so that what a
  // saved-tensor hook raises arrives as what it is: a checkpointed region ends its second
  // forward that way.
  m.def("bn_act", torch::wrap_pybind_function([](
                      const at::Tensor& x, const c10::optional<at::Tensor>& residual,
                      const c10::optional<at::Tensor>& weight,
                      const c10::optional<at::Tensor>& bias,
                      const c10::optional<at::Tensor>& running_mean,
                      const c10::optional<at::Tensor>& running_var, double momentum, double eps,
                      bool relu,
                      const c10::optional<at::Tensor>& batches) -> c10::optional<at::Tensor> {
    if (!x.is_cuda() || x.dim() != 4 ||
        (x.scalar_type() != at::kBFloat16 && x.scalar_type() != at::kHalf) ||
        !x.is_contiguous(at::MemoryFormat::ChannelsLast) || x.numel() == 0 ||
        !kern::BatchNormSupported(x.numel() / x.size(1), static_cast<int>(x.size(1))))
      return c10::nullopt;
    if (residual.has_value() &&
        (residual->sizes() != x.sizes() || residual->scalar_type() != x.scalar_type()))
      return c10::nullopt;
    return NormNode::apply(x, residual, weight, bias, running_mean, running_var, momentum, eps,
                           relu, batches);
  }));

  // ---- max pooling 3x3 / stride 2 / padding 1 (channels-last, 16-bit) -------
  m.def("maxpool3s2_supported", [](int64_t channels) {
    return kern::MaxPool3s2Supported(static_cast<int>(channels));
  });
  // x -> (y, idx): idx holds one word per 8 output channels (a nibble for the
  // winning window position of each).
  m.def("maxpool3s2_forward", [](at::Tensor x) {
    x = Activations(x, "x");
    const int64_t N = x.size(0), C = x.size(1), H = x.size(2), W = x.size(3);
    TORCH_CHECK(kern::MaxPool3s2Supported(static_cast<int>(C)),
                "fused max pooling needs a channel count that is a multiple of 8");
    const int64_t Ho = (H + 2 - 3) / 2 + 1, Wo = (W + 2 - 3) / 2 + 1;
    c10::cuda::CUDAGuard guard(x.device());
    cudaStream_t stream = at::cuda::getCurrentCUDAStream();
    at::Tensor y = at::empty({N, C, Ho, Wo}, x.options(), at::MemoryFormat::ChannelsLast);
    at::Tensor idx = at::empty({N, Ho, Wo, C / 8}, x.options().dtype(at::kInt));
    cudaError_t err = kern::LaunchMaxPool3s2Forward(
        x.data_ptr(), y.data_ptr(), reinterpret_cast<uint32_t*>(idx.data_ptr<int32_t>()),
        static_cast<int>(N), static_cast<int>(H), static_cast<int>(W), static_cast<int>(C),
        x.scalar_type() == at::kBFloat16, stream);
    TORCH_CHECK(err == cudaSuccess, "fused max pooling forward: ", cudaGetErrorString(err));
    return std::make_tuple(y, idx);
  });
  // (dy, idx, H, W) -> dx
  m.def("maxpool3s2_backward", [](at::Tensor dy, const at::Tensor& idx, int64_t H, int64_t W) {
    dy = Activations(dy, "dy");
    const int64_t N = dy.size(0), C = dy.size(1);
    TORCH_CHECK(idx.is_cuda() && idx.scalar_type() == at::kInt && idx.is_contiguous() &&
                    idx.numel() * 8 == dy.numel(),
                "idx must be the tensor returned by maxpool3s2_forward");
    TORCH_CHECK(dy.size(2) == (H + 2 - 3) / 2 + 1 && dy.size(3) == (W + 2 - 3) / 2 + 1,
                "dy does not match the pooled size of an input of ", H, " x ", W);
    c10::cuda::CUDAGuard guard(dy.device());
    cudaStream_t stream = at::cuda::getCurrentCUDAStream();
    at::Tensor dx = at::empty({N, C, H, W}, dy.options(), at::MemoryFormat::ChannelsLast);
    cudaError_t err = kern::LaunchMaxPool3s2Backward(
        dy.data_ptr(), reinterpret_cast<const uint32_t*>(idx.data_ptr<int32_t>()), dx.data_ptr(),
        static_cast<int>(N), static_cast<int>(H), static_cast<int>(W), static_cast<int>(C),
        dy.scalar_type() == at::kBFloat16, stream);
    TORCH_CHECK(err == cudaSuccess, "fused max pooling backward: ", cudaGetErrorString(err));
    return dx;
  });

  // ---- 7x7 / stride 2 convolution of 3 channels (channels-last, 16-bit) ------
  m.def("stem_conv_supported", &kern::StemConvSupported);  // (n, h, w, channels)
  // Whether a kernel's wait has run out on this device.
  m.def("stem_conv_failed", &kern::StemConvFailed, py::arg("device"), py::arg("clear") = false);
  m.def("stem_conv_forward", [](const at::Tensor& x, const at::Tensor& weight, uint32_t wait_ns) {
    CheckActivations(x, "x");
    const int64_t N = x.size(0), H = x.size(2), W = x.size(3), C = weight.size(0);
    TORCH_CHECK(weight.is_cuda() && weight.device() == x.device() &&
                    weight.scalar_type() == x.scalar_type() && weight.dim() == 4 &&
                    weight.size(1) == 3 && weight.size(2) == 7 && weight.size(3) == 7 &&
                    x.size(1) == 3,
                "stem_conv_forward: x must have 3 channels and weight the shape [C, 3, 7, 7]");
    TORCH_CHECK(kern::StemConvSupported(N, H, W, C), "stem_conv_forward does not support ", N,
                " images of ", H, " x ", W, " to ", C, " channels");
    c10::cuda::CUDAGuard guard(x.device());
    at::Tensor y = at::empty({N, C, (H - 1) / 2 + 1, (W - 1) / 2 + 1}, x.options(),
                             at::MemoryFormat::ChannelsLast);
    cudaError_t err = kern::LaunchStemConvForward(
        x.data_ptr(), weight.data_ptr(), weight.strides().data(), y.data_ptr(),
        static_cast<int>(N), static_cast<int>(H), static_cast<int>(W), static_cast<int>(C),
        x.scalar_type() == at::kBFloat16, at::cuda::getCurrentCUDAStream(), wait_ns);
    TORCH_CHECK(err == cudaSuccess, "stem convolution: ", cudaGetErrorString(err));
    return y;
  }, py::arg("x"), py::arg("weight"), py::arg("wait_ns") = kern::STEM_WAIT_NS);

  // (x, dy, weight) -> gradient of the weight
  m.def("stem_conv_wgrad", [](const at::Tensor& x, at::Tensor dy, const at::Tensor& weight,
                              uint32_t wait_ns) {
    CheckActivations(x, "x");
    dy = Activations(dy, "dy");
    const int64_t N = x.size(0), H = x.size(2), W = x.size(3), C = weight.size(0);
    TORCH_CHECK(weight.scalar_type() == x.scalar_type() && weight.device() == x.device() &&
                    weight.dim() == 4 && weight.size(1) == 3 && weight.size(2) == 7 &&
                    weight.size(3) == 7 && x.size(1) == 3,
                "stem_conv_wgrad: x must have 3 channels and weight the shape [C, 3, 7, 7]");
    TORCH_CHECK(dy.scalar_type() == x.scalar_type() && dy.device() == x.device() &&
                    dy.size(0) == N && dy.size(1) == C && dy.size(2) == (H - 1) / 2 + 1 &&
                    dy.size(3) == (W - 1) / 2 + 1,
                "stem_conv_wgrad: dy does not match x and weight");
    TORCH_CHECK(kern::StemConvSupported(N, H, W, C), "stem_conv_wgrad does not support ", N,
                " images of ", H, " x ", W, " to ", C, " channels");
    c10::cuda::CUDAGuard guard(x.device());
    const int64_t ctas = kern::StemConvWgradCtas(static_cast<int>(N), static_cast<int>(H),
                                                 static_cast<int>(W), static_cast<int>(C));
    at::Tensor partial = at::empty({ctas * 256 * C}, x.options().dtype(at::kFloat),
                                   at::MemoryFormat::Contiguous);
    at::Tensor dw = at::empty_like(weight);
    cudaError_t err = kern::LaunchStemConvWgrad(
        x.data_ptr(), dy.data_ptr(), partial.data_ptr<float>(), dw.data_ptr(),
        dw.strides().data(), static_cast<int>(N), static_cast<int>(H), static_cast<int>(W),
        static_cast<int>(C), x.scalar_type() == at::kBFloat16, at::cuda::getCurrentCUDAStream(),
        wait_ns);
    TORCH_CHECK(err == cudaSuccess, "stem convolution gradient: ", cudaGetErrorString(err));
    return dw;
  }, py::arg("x"), py::arg("dy"), py::arg("weight"), py::arg("wait_ns") = kern::STEM_WAIT_NS);

  // ---- multi-tensor SGD ------------------------------------------------------
  // One step over a parameter list, in one launch per 256 tensors. bufs holds
  // a momentum buffer (or None) per parameter; it is empty when momentum is 0.
  // Parameters without a gradient are passed over. Returns whether it launched
  // and the positions of those that the kernel cannot take (see SgdReady) or that
  // have no buffer yet, untouched. Where one has a buffer that does not match
  // it, nothing is launched: a step that fails leaves every parameter as it was.
  m.def("sgd_step", [](const std::vector<at::Tensor>& params,
                       const std::vector<c10::optional<at::Tensor>>& bufs, double lr,
                       double momentum, double dampening, double weight_decay, bool nesterov,
                       bool first_step, bool maximize) {
    const bool with_bufs = momentum != 0.0;
    TORCH_CHECK(bufs.size() == (with_bufs ? params.size() : 0), "sgd_step: list lengths differ");
    std::vector<int64_t> rest;
    std::vector<size_t> ready;
    bool launch = true;
    for (size_t i = 0; i < params.size(); ++i) {
      const at::Tensor& g = params[i].grad();
      if (!g.defined()) continue;
      bool taken = SgdReady(params[i], g);
      if (taken && with_bufs) {
        const bool exists = bufs[i].has_value() && bufs[i]->defined();
        taken = exists && SgdLike(params[i], *bufs[i]);
        if (exists && !taken) launch = false;
      }
      if (taken)
        ready.push_back(i);
      else
        rest.push_back(static_cast<int64_t>(i));
    }
    if (!launch) return std::make_pair(false, rest);
    kern::SgdTensors t;
    size_t next = 0;
    while (next < ready.size()) {
      // The run of tensors from here on that share a device, as many as fit.
      const at::Device device = params[ready[next]].device();
      t.n = 0;
      int64_t chunks = 0;
      t.first_chunk[0] = 0;
      for (; next < ready.size() && t.n < kern::SGD_MAX_TENSORS; ++next) {
        const at::Tensor& p = params[ready[next]];
        if (p.device() != device) break;
        const int64_t more =
            (p.numel() + kern::SGD_CHUNK_ELEMS - 1) / kern::SGD_CHUNK_ELEMS;
        if (chunks + more > INT32_MAX) break;
        chunks += more;
        t.params[t.n] = p.data_ptr<float>();
        t.grads[t.n] = p.grad().const_data_ptr<float>();
        t.bufs[t.n] = with_bufs ? bufs[ready[next]]->data_ptr<float>() : nullptr;
        t.counts[t.n] = p.numel();
        t.first_chunk[++t.n] = static_cast<int32_t>(chunks);
      }
      TORCH_CHECK(t.n > 0, "sgd_step: a parameter is too large");
      c10::cuda::CUDAGuard guard(device);
      cudaError_t err = kern::LaunchFusedSgd(
          t, static_cast<float>(lr), static_cast<float>(momentum), static_cast<float>(dampening),
          static_cast<float>(weight_decay), nesterov, first_step, maximize,
          at::cuda::getCurrentCUDAStream());
      TORCH_CHECK(err == cudaSuccess, "fused SGD: ", cudaGetErrorString(err));
    }
    return std::make_pair(true, rest);
  });
}

}  // namespace hvd
