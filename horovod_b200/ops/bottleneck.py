"""A ResNet bottleneck block in training as one autograd node
(csrc/torch/bottleneck.cpp): the statistics of the batch norms behind its 1x1
convolutions come out of the convolutions' kernel (csrc/kernels/conv1x1.cu), and
the gradient of the skip connection is added inside one.

``fused_bottleneck_available`` says whether a block and its input can take it. What
it cannot represent is left to the sequence of layers: evaluation mode, other
memory formats and types, layers of other classes, hooks on a layer, tracing,
transforms, modes that watch functions. ``HOROVOD_B200_FUSED_BLOCK=0`` leaves every
block to its layers.

The reference has no counterpart (it takes convolutions and batch normalisation from
the framework).
"""
import os

import torch
import torch.nn as nn
from torch.nn.modules.module import _has_any_global_hook

from horovod_b200.ops._native import PLAIN, functions_watched, plain_autograd
from horovod_b200.ops.batch_norm import BatchNormAct2d
from horovod_b200.ops.stem_conv import tensor_core_kernels_enabled


def _extension():
    from horovod_b200 import _C
    return _C


def _observed(module):
    """Whether somebody would miss a call of this module."""
    return bool(module._forward_hooks or module._forward_pre_hooks or module._backward_hooks
                or module._backward_pre_hooks or "forward" in module.__dict__)


def _plain_conv(conv, kernel, stride, dtypes, device):
    weight = conv._parameters.get("weight")
    return (type(conv) is nn.Conv2d and conv.kernel_size == (kernel, kernel)
            and conv.stride == (stride, stride)
            and conv.padding == (kernel // 2, kernel // 2) and conv.dilation == (1, 1)
            and conv.groups == 1 and conv.bias is None and conv.padding_mode == "zeros"
            and type(weight) in PLAIN and weight.dtype in dtypes and weight.device == device
            # (A weight may have been replaced without the layer's attributes.)
            and weight.shape == (conv.out_channels, conv.in_channels, kernel, kernel)
            and not _observed(conv))


def _plain_norm(norm, relu, conv, device):
    if not (type(norm) is BatchNormAct2d and norm.relu is relu and norm.training
            and norm.track_running_stats and norm.momentum is not None and norm.affine
            and norm.num_features == conv.out_channels and not _observed(norm)):
        return False
    # (Some of them may be attributes of another kind.)
    weight, bias = norm._parameters.get("weight"), norm._parameters.get("bias")
    mean, var = norm._buffers.get("running_mean"), norm._buffers.get("running_var")
    batches = norm._buffers.get("num_batches_tracked")
    for t in (weight, bias, mean, var):
        if not (type(t) in PLAIN and t.dtype == torch.float32 and t.device == device
                and t.is_contiguous()):
            return False
    return type(batches) in PLAIN and batches.dtype == torch.int64 and batches.device == device


def _layers(block):
    """(convolution, batch norm, kernel size, stride, has a ReLU) of every layer, or
    None when one of them is something else."""
    for conv in (block.conv1, block.conv2, block.conv3):
        if type(conv) is not nn.Conv2d:
            return None
    stride = block.conv2.stride[0]
    layers = [(block.conv1, block.bn1, 1, 1, True), (block.conv2, block.bn2, 3, stride, True),
              (block.conv3, block.bn3, 1, 1, True)]
    down = block.downsample
    if down is not None:
        if type(down) is not nn.Sequential or len(down) != 2 or _observed(down) or \
                type(down[0]) is not nn.Conv2d:
            return None
        layers.append((down[0], down[1], 1, stride, False))
    return layers


def fused_bottleneck_available(block, x):
    """The layers of the block for ``fused_bottleneck``, or None."""
    if not (type(x) in PLAIN and x.is_cuda and x.dim() == 4 and x.numel() > 0
            and x.dtype in (torch.bfloat16, torch.float16)):
        return None
    if os.environ.get("HOROVOD_B200_FUSED_BLOCK", "1") != "1" or \
            os.environ.get("HOROVOD_B200_FUSED_BN", "1") != "1" or _has_any_global_hook() or \
            not plain_autograd() or functions_watched():
        return None
    if not x.is_contiguous(memory_format=torch.channels_last) or x.data_ptr() % 16 != 0:
        return None
    if torch.is_autocast_enabled("cuda"):
        if torch.get_autocast_dtype("cuda") != x.dtype:
            return None
        dtypes = (torch.float32, x.dtype)
    else:
        dtypes = (x.dtype,)
    layers = _layers(block)
    if layers is None:
        return None
    device, channels = x.device, x.size(1)
    into = (channels, block.conv1.out_channels, block.conv2.out_channels, channels)
    norm_supported = _extension().bn_supported
    for (conv, norm, kernel, stride, relu), inputs in zip(layers, into):
        if stride not in (1, 2) or conv.in_channels != inputs or \
                not _plain_conv(conv, kernel, stride, dtypes, device) or \
                not _plain_norm(norm, relu, conv, device) or \
                not norm_supported(1, conv.out_channels):
            return None
    if len(layers) == 3 and (layers[1][3] != 1 or block.conv3.out_channels != channels):
        return None
    if len(layers) == 4 and layers[3][0].out_channels != block.conv3.out_channels:
        return None
    if not norm_supported(1, channels) or not tensor_core_kernels_enabled(device):
        return None
    return layers


def fused_bottleneck(x, layers):
    """relu(layer 2(layer 1(layer 0(x))) + skip), every layer a convolution, a
    batch norm and (but for the skip connection's) a ReLU."""
    tensors, rates = [], []
    for conv, norm, _, _, _ in layers:
        p, b = norm._parameters, norm._buffers
        tensors.append((conv._parameters["weight"], p["weight"], p["bias"], b["running_mean"],
                        b["running_var"], b["num_batches_tracked"]))
        rates.append((norm.momentum, norm.eps))
    return _extension().bottleneck(x, tensors, rates, layers[1][3])
