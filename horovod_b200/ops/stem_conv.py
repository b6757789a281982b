"""The first convolution of a ResNet (7x7, stride 2, padding 3, 3 channels) for
channels-last bf16/fp16 inputs on this library's tensor-core kernel
(csrc/kernels/stem_conv.cu), with PyTorch's convolution everywhere else and
for the gradient of the input.

``HOROVOD_B200_FUSED_STEM=0`` leaves everything to PyTorch, and so does a wait
that has run out inside the kernel: the results of that call are NaN, later ones
on the device are PyTorch's.

``StemConv2d`` is an ``nn.Conv2d`` (same parameters and state_dict keys). The
reference has no counterpart (it takes convolutions from the framework).
"""
import os
import warnings

import torch
import torch.nn as nn

from horovod_b200.ops._native import PLAIN, plain_autograd


def _extension():
    from horovod_b200 import _C
    return _C


def tensor_core_kernels_enabled(device):
    """False from when a wait inside one of them has run out on the device."""
    if _extension().stem_conv_failed(device.index):
        warnings.warn("a wait inside a convolution's kernel ran out on %s; the results of that "
                      "call are NaN, and PyTorch's convolution runs from now on" % device)
        return False
    return True


def _enabled(device):
    return os.environ.get("HOROVOD_B200_FUSED_STEM", "1") == "1" and \
        tensor_core_kernels_enabled(device)


class _StemConv(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, weight):
        ctx.save_for_backward(x, weight)
        return _extension().stem_conv_forward(x, weight)

    @staticmethod
    def backward(ctx, dy):
        x, weight = ctx.saved_tensors
        need_x, need_w = ctx.needs_input_grad
        # A gradient of this gradient is PyTorch's.
        native = need_w and not torch.is_grad_enabled() and weight.dtype == dy.dtype and \
            _enabled(x.device)
        dx = dw = None
        if need_x or (need_w and not native):
            dx, dw, _ = torch.ops.aten.convolution_backward(
                dy, x, weight, None, [2, 2], [3, 3], [1, 1], False, [0, 0], 1,
                [need_x, need_w and not native, False])
        if native:
            dw = _extension().stem_conv_wgrad(
                x, dy.contiguous(memory_format=torch.channels_last), weight)
        return dx, dw


class StemConv2d(nn.Conv2d):
    """``nn.Conv2d`` that runs the kernel where it can."""

    def _kernel_dtype(self, x):
        """The 16-bit type the convolution runs in, or None for PyTorch's own:
        another geometry, memory format or type, and what a custom autograd
        function cannot take part in: tracing, transforms, tensors and modes
        with an __torch_dispatch__ of their own."""
        if not (type(x) in PLAIN and type(self.weight) in PLAIN
                and x.is_cuda and x.dim() == 4 and x.size(1) == 3 and x.numel() > 0
                and self.kernel_size == (7, 7) and self.stride == (2, 2)
                and self.padding == (3, 3) and self.dilation == (1, 1) and self.groups == 1
                and self.bias is None and self.padding_mode == "zeros"
                and self.weight.device == x.device
                and x.is_contiguous(memory_format=torch.channels_last)):
            return None
        if torch.is_autocast_enabled("cuda"):
            dtype = torch.get_autocast_dtype("cuda")
        elif x.dtype == self.weight.dtype:
            dtype = x.dtype
        else:
            return None
        if dtype not in (torch.bfloat16, torch.float16) or \
                x.dtype not in (torch.float32, torch.bfloat16, torch.float16) or \
                self.weight.dtype not in (torch.float32, torch.bfloat16, torch.float16):
            return None
        if not plain_autograd():
            return None
        n, _, h, w = x.shape
        if not _extension().stem_conv_supported(n, h, w, self.out_channels) or \
                not _enabled(x.device):
            return None
        return dtype

    def forward(self, x):
        dtype = self._kernel_dtype(x)
        if dtype is None:
            return super().forward(x)
        return _StemConv.apply(x.to(dtype), self.weight.to(dtype))
