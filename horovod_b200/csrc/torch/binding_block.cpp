// Python entry points of the ResNet block's kernels. They run on the caller's
// current CUDA stream like any torch op.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <cstdint>
#include <tuple>

#include "../kernels/kernels.h"
#include "model_ops.h"

namespace hvd {

void BindBlockOps(py::module_& m) {
  m.def("conv1x1_supported", &kern::Conv1x1Supported);  // (rows, k, n)
  // The kernel alone. x: channels-last activations; w: [n, k], or [k, n] with
  // w_transposed; add (zeros where there is none), signs: see kernels.h. With scatter, y
  // is written to (and add read from) every other pixel of `y`; with gather, x is read
  // that way.
  //   -> (y, sums of [2, n] in fp64 or None)
  m.def("conv1x1", [](const at::Tensor& x, const at::Tensor& w, bool w_transposed,
                      const c10::optional<at::Tensor>& add,
                      const c10::optional<at::Tensor>& signs, bool want_sums, bool gather,
                      bool scatter, uint32_t wait_ns) {
    TORCH_CHECK(x.is_cuda() && x.dim() == 4 && x.is_contiguous(at::MemoryFormat::ChannelsLast) &&
                    (x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kHalf),
                "conv1x1: x must be 16-bit channels-last CUDA activations");
    TORCH_CHECK(w.is_cuda() && w.dim() == 2 && w.is_contiguous() && w.device() == x.device() &&
                    w.scalar_type() == x.scalar_type() && w.size(w_transposed ? 0 : 1) == x.size(1),
                "conv1x1: w does not match x");
    const int64_t n = w.size(w_transposed ? 1 : 0), factor = gather ? 2 : 1;
    TORCH_CHECK(x.size(2) % factor == 0 && x.size(3) % factor == 0, "conv1x1: odd size");
    const int64_t ho = x.size(2) / factor, wo = x.size(3) / factor;
    kern::Conv1x1 c;
    c.rows = x.size(0) * ho * wo;
    c.k = static_cast<int>(x.size(1));
    c.n = static_cast<int>(n);
    TORCH_CHECK(kern::Conv1x1Supported(c.rows, c.k, c.n), "conv1x1 does not support ", c.rows,
                " rows of ", c.k, " to ", c.n, " channels");
    c10::cuda::CUDAGuard guard(x.device());
    at::Tensor y;
    if (scatter) {
      TORCH_CHECK(add.has_value() && add->size(2) == 2 * ho && add->size(3) == 2 * wo,
                  "conv1x1: scatter needs add of twice the size");
      y = add->clone(at::MemoryFormat::ChannelsLast);
    } else {
      y = at::empty({x.size(0), n, ho, wo}, x.options(), at::MemoryFormat::ChannelsLast);
    }
    if (add.has_value()) {
      TORCH_CHECK(add->sizes() == y.sizes() && add->scalar_type() == x.scalar_type() &&
                      add->device() == x.device() &&
                      add->is_contiguous(at::MemoryFormat::ChannelsLast),
                  "conv1x1: add does not match");
      c.add = scatter ? y.data_ptr() : add->data_ptr();
    }
    at::Tensor zeros;
    if (w_transposed && !add.has_value()) {
      zeros = at::zeros_like(y);
      c.add = zeros.data_ptr();
    }
    if (signs.has_value()) {
      TORCH_CHECK(signs->is_cuda() && signs->scalar_type() == at::kByte &&
                      signs->is_contiguous() && signs->numel() * 8 == y.numel(),
                  "conv1x1: signs do not match");
      c.signs = signs->data_ptr<uint8_t>();
    }
    at::Tensor sums;
    if (!w_transposed || want_sums) {
      c.copies = kern::BatchNormCopies(c.n);
      sums = at::zeros({c.copies, 2, n}, x.options().dtype(at::kDouble));
      c.sums = sums.data_ptr<double>();
    }
    c.x = x.data_ptr();
    c.w = w.data_ptr();
    c.y = y.data_ptr();
    c.w_transposed = w_transposed;
    c.strided_x = gather;
    c.strided_y = scatter;
    c.width = static_cast<int>(wo);
    c.bf16 = x.scalar_type() == at::kBFloat16;
    const cudaError_t err = kern::LaunchConv1x1(c, at::cuda::getCurrentCUDAStream(), wait_ns);
    TORCH_CHECK(err == cudaSuccess, "1x1 convolution: ", cudaGetErrorString(err));
    return std::make_tuple(y, want_sums ? c10::optional<at::Tensor>(sums.sum(0)) : c10::nullopt);
  }, py::arg("x"), py::arg("w"), py::arg("w_transposed") = false, py::arg("add") = c10::nullopt,
     py::arg("signs") = c10::nullopt, py::arg("want_sums") = false, py::arg("gather") = false,
     py::arg("scatter") = false, py::arg("wait_ns") = kern::STEM_WAIT_NS);

  m.def("norm_conv_backward_supported", &kern::NormConvBackwardSupported);  // (rows, cout, cin)
  // (dy, signs, x, a, w, gamma, saved) -> (da, dw, dgamma, dbeta): see kernels.h.
  m.def("norm_conv_backward", [](const at::Tensor& dy, const at::Tensor& signs,
                                 const at::Tensor& x, const at::Tensor& a, const at::Tensor& w,
                                 const at::Tensor& gamma, const at::Tensor& saved,
                                 uint32_t wait_ns) {
    CheckActivations(dy, "dy");
    CheckActivations(x, "x");
    CheckActivations(a, "a");
    const int64_t cout = x.size(1), cin = a.size(1), rows = x.numel() / cout;
    TORCH_CHECK(kern::NormConvBackwardSupported(rows, static_cast<int>(cout),
                                                static_cast<int>(cin)),
                "norm_conv_backward does not support ", rows, " rows of ", cin, " to ", cout,
                " channels");
    TORCH_CHECK(dy.sizes() == x.sizes() && a.numel() / cin == rows && w.is_contiguous() &&
                    w.is_cuda() && w.size(0) == cout && w.numel() == cout * cin &&
                    dy.scalar_type() == x.scalar_type() && a.scalar_type() == x.scalar_type() &&
                    w.scalar_type() == x.scalar_type() && signs.is_contiguous() &&
                    signs.is_cuda() && signs.scalar_type() == at::kByte &&
                    signs.numel() * 8 == x.numel() && saved.is_contiguous() && saved.is_cuda() &&
                    saved.scalar_type() == at::kFloat && saved.numel() == 3 * cout,
                "norm_conv_backward: tensors do not match");
    c10::cuda::CUDAGuard guard(x.device());
    const auto fp32 = x.options().dtype(at::kFloat);
    at::Tensor da = at::empty_like(a, a.options(), at::MemoryFormat::ChannelsLast);
    at::Tensor dw = at::empty({cout, cin}, fp32, at::MemoryFormat::Contiguous);
    at::Tensor dgamma = at::empty({cout}, fp32), dbeta = at::empty({cout}, fp32), own;
    at::Tensor partial = at::empty({kern::NormConvBackwardParts(rows) * cout * cin}, fp32,
                                   at::MemoryFormat::Contiguous);
    kern::NormConvBackward n;
    n.dy = dy.data_ptr();
    n.x = x.data_ptr();
    n.a = a.data_ptr();
    n.w = w.data_ptr();
    n.signs = signs.data_ptr<uint8_t>();
    n.da = da.data_ptr();
    n.dw = dw.data_ptr();
    n.dw_fp32 = true;
    n.dw_stride_o = cin;
    n.dw_stride_i = 1;
    cudaStream_t stream = at::cuda::getCurrentCUDAStream();
    n.sums = ZeroedDoubles(kern::BatchNormScratchDoubles(static_cast<int>(cout)), x, stream, &own);
    n.summed = false;
    n.gamma = FloatPtrOrNull(gamma, cout, "gamma");
    n.saved = saved.data_ptr<float>();
    n.dgamma = dgamma.data_ptr<float>();
    n.dbeta = dbeta.data_ptr<float>();
    n.partial = partial.data_ptr<float>();
    n.rows = rows;
    n.cout = static_cast<int>(cout);
    n.cin = static_cast<int>(cin);
    n.bf16 = x.scalar_type() == at::kBFloat16;
    const cudaError_t err = kern::LaunchNormConvBackward(n, stream, wait_ns);
    TORCH_CHECK(err == cudaSuccess, "batch norm and convolution backward: ",
                cudaGetErrorString(err));
    return std::make_tuple(da, dw, dgamma, dbeta);
  }, py::arg("dy"), py::arg("signs"), py::arg("x"), py::arg("a"), py::arg("w"), py::arg("gamma"),
     py::arg("saved"), py::arg("wait_ns") = kern::STEM_WAIT_NS);
}

}  // namespace hvd
