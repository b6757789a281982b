"""Fused training-mode batch normalisation (+ residual add + ReLU) for
channels-last bf16/fp16 activations, backed by this library's CUDA kernels
(csrc/kernels/batch_norm.cu), with a plain PyTorch fallback everywhere else
(CPU, fp32, NCHW, eval mode, channel counts the kernels do not tile).

``BatchNormAct2d`` is a drop-in ``nn.BatchNorm2d`` (same parameters, buffers
and state_dict keys) whose forward takes an optional residual:

    y = relu(batch_norm(x) + residual)

The eager PyTorch sequence batch_norm -> add -> relu makes eight passes over
the activation in forward and nine in backward; the fused kernels make three
or four and five or six. The reference has no counterpart (it takes batch normalisation
from the framework; horovod/torch/sync_batch_norm.py:98-199 composes
torch.batch_norm_stats / batch_norm_elemt / batch_norm_backward_reduce).
"""
import os

import torch
import torch.nn as nn
import torch.nn.functional as F

from horovod_b200.ops._native import PLAIN, plain_autograd


def _extension():
    from horovod_b200 import _C
    return _C


def fused_batch_norm_available(x, momentum):
    """True when the CUDA kernels can take this input."""
    if os.environ.get("HOROVOD_B200_FUSED_BN", "1") != "1":
        return False
    if not (x.is_cuda and x.dim() == 4 and x.dtype in (torch.bfloat16, torch.float16)):
        return False
    if momentum is None or not x.is_contiguous(memory_format=torch.channels_last):
        return False
    channels = x.size(1)
    return _extension().bn_supported(x.numel() // channels, channels)


def _native(*tensors):
    """Whether the layer may run as its native autograd node."""
    return plain_autograd() and all(t is None or type(t) in PLAIN for t in tensors)


class _FusedBatchNormAct(torch.autograd.Function):
    """The layer where its native node (bn_act) cannot be used."""

    @staticmethod
    def forward(ctx, x, residual, weight, bias, running_mean, running_var, momentum, eps, relu,
                batches):
        y, saved, signs = _extension().bn_forward(x, residual, weight, bias, running_mean,
                                                  running_var, momentum, eps, relu, batches)
        # The kernels do without y; like relu's own backward, this one still
        # refuses to run when somebody has changed it in place.
        ctx.save_for_backward(x, y if relu else None, weight, saved, signs)
        ctx.relu = relu
        ctx.has_residual = residual is not None
        return y

    @staticmethod
    def backward(ctx, dy):
        x, _, weight, saved, signs = ctx.saved_tensors
        if dy.dtype != x.dtype:
            dy = dy.to(x.dtype)
        dy = dy.contiguous(memory_format=torch.channels_last)
        want_dres = ctx.has_residual and ctx.needs_input_grad[1]
        dx, dres, dweight, dbias = _extension().bn_backward(
            dy, x, weight, saved, signs, ctx.relu, want_dres)
        if weight is None:
            dweight = None
        return dx, dres, dweight, dbias if ctx.needs_input_grad[3] else None, None, None, None, \
            None, None, None


def batch_norm_act(x, weight, bias, running_mean, running_var, residual=None, training=True,
                   momentum=0.1, eps=1e-5, relu=True, num_batches_tracked=None):
    """relu(batch_norm(x) + residual), fused on the GPU when possible.
    ``num_batches_tracked`` (optional, an int64 tensor) is incremented."""
    if training and momentum is not None and x.is_cuda and \
            os.environ.get("HOROVOD_B200_FUSED_BN", "1") == "1" and \
            _native(x, residual, weight, bias, running_mean, running_var):
        y = _extension().bn_act(x, residual, weight, bias, running_mean, running_var, momentum,
                                eps, relu, num_batches_tracked)
        if y is not None:
            return y
    elif training and fused_batch_norm_available(x, momentum) and \
            (residual is None or (residual.shape == x.shape and residual.dtype == x.dtype)):
        if residual is not None:
            residual = residual.contiguous(memory_format=torch.channels_last)
        if num_batches_tracked is not None and (num_batches_tracked.device != x.device or
                                                num_batches_tracked.dtype != torch.int64):
            num_batches_tracked.add_(1)
            num_batches_tracked = None
        return _FusedBatchNormAct.apply(x, residual, weight, bias, running_mean, running_var,
                                        float(momentum), float(eps), bool(relu),
                                        num_batches_tracked)
    if num_batches_tracked is not None:
        num_batches_tracked.add_(1)
    out = F.batch_norm(x, running_mean, running_var, weight, bias, training,
                       0.0 if momentum is None else momentum, eps)
    if residual is not None:
        out = out + residual
    return F.relu(out) if relu else out


class BatchNormAct2d(nn.BatchNorm2d):
    """``nn.BatchNorm2d`` followed by an optional residual add and ReLU."""

    def __init__(self, num_features, relu=True, **kwargs):
        super().__init__(num_features, **kwargs)
        self.relu = relu

    def forward(self, x, residual=None):
        self._check_input_dim(x)
        batches = self.num_batches_tracked if self.training and self.track_running_stats else None
        training = self.training or (self.running_mean is None and self.running_var is None)
        momentum = self.momentum
        if momentum is None and self.training and self.track_running_stats:
            if batches is not None:  # counted here: the average needs the count first
                batches.add_(1)
                batches = None
            momentum = 1.0 / float(self.num_batches_tracked)
        return batch_norm_act(
            x, self.weight, self.bias,
            self.running_mean if not self.training or self.track_running_stats else None,
            self.running_var if not self.training or self.track_running_stats else None,
            residual=residual, training=training, momentum=momentum, eps=self.eps,
            relu=self.relu, num_batches_tracked=batches)
