"""When a call may go straight to a native autograd node."""
import torch
import torch.nn as nn
from torch.autograd import forward_ad
from torch.overrides import _get_current_function_mode_stack
from torch.utils._device import DeviceContext
from torch.utils._python_dispatch import is_in_torch_dispatch_mode

#: Tensors without a __torch_dispatch__ or __torch_function__ of their own.
PLAIN = (torch.Tensor, nn.Parameter)


def plain_autograd():
    """False under what a native autograd node cannot take part in: tracing,
    compilation, forward mode, functorch's transforms, dispatch modes."""
    return not (torch.jit.is_tracing() or torch.compiler.is_compiling()
                or forward_ad._current_level >= 0
                or torch._C._are_functorch_transforms_active() or is_in_torch_dispatch_mode())


def functions_watched():
    """Whether a mode is to see the calls of torch's functions, those that a native node
    has no calls of among them. A device as a context is a mode too, one that changes
    where tensors are made and nothing else."""
    return torch._C._len_torch_function_stack() > 0 and \
        any(type(mode) is not DeviceContext for mode in _get_current_function_mode_stack())
