"""Which layers a residual block hands to its native node, as far as that is decided
by the layers alone."""
import torch
import torch.nn as nn

from horovod_b200.ops import bottleneck

CPU = torch.device("cpu")


def _plain_conv(weight=None, cin=64, cout=32, kernel=1):
    conv = nn.Conv2d(cin, cout, kernel, padding=kernel // 2, bias=False)
    if weight is not None:
        conv.weight = nn.Parameter(torch.randn(weight))
    return bottleneck._plain_conv(conv, kernel, 1, (torch.float32,), CPU)


def test_weights_that_do_not_fit_their_layer():
    """Replaced without the layer's attributes: PyTorch's convolution says what is wrong."""
    assert _plain_conv() and _plain_conv((32, 64, 1, 1)) and _plain_conv(kernel=3)
    assert not _plain_conv((32, 48, 1, 1))       # fewer inputs
    assert not _plain_conv((24, 64, 1, 1))       # fewer outputs
    assert not _plain_conv((32, 64, 3, 3))       # another size
    assert not _plain_conv((32, 64, 1, 1), kernel=3)
    assert not _plain_conv((32, 64, 1))          # not even four dimensions


def test_modes_that_watch_functions():
    from torch.overrides import TorchFunctionMode

    from horovod_b200.ops._native import functions_watched

    class Watch(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    assert not functions_watched()
    with torch.device("cpu"):
        assert not functions_watched()
        with Watch():
            assert functions_watched()
            with torch.device("cpu"):  # the one below it still watches
                assert functions_watched()
    assert not functions_watched()


def test_batch_norms_whose_tensors_are_plain_attributes():
    """As after some functional rewrites: left to the layer, which reads attributes."""
    from horovod_b200.ops.batch_norm import BatchNormAct2d

    def plain(name=None):
        norm, conv = BatchNormAct2d(32), nn.Conv2d(64, 32, 1, bias=False)
        if name is not None:
            value = getattr(norm, name).detach()
            delattr(norm, name)
            norm.__dict__[name] = value
        return bottleneck._plain_norm(norm, True, conv, CPU)

    assert plain()
    for name in ("weight", "bias", "running_mean", "running_var", "num_batches_tracked"):
        assert not plain(name)
