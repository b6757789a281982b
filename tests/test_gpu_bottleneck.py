"""The ResNet block as one node: the 1x1 convolution kernels at the edges of
their tiles, the block against its layers and against 64 bits, and what is left to
the layers."""
import copy

import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu
CL = torch.channels_last


def _dev():
    return torch.device("cuda", 0)


def _act(g, n, c, h, w, dtype):
    return torch.randn(n, h, w, c, device=_dev(), generator=g).to(dtype).permute(0, 3, 1, 2)


def _signs(mask):
    """A byte per 8 channels: even channels in the low nibble, odd ones above."""
    m = mask.permute(0, 2, 3, 1).reshape(-1, mask.size(1) // 8, 8).int()
    bits = sum(m[..., c] << i for i, c in enumerate([0, 2, 4, 6, 1, 3, 5, 7]))
    return bits.to(torch.uint8).contiguous()


def _close(got, want, dtype):
    """One rounding of every value to 16 bits (half a unit in the last place), and
    the order of the fp32 sums, which is far below it."""
    half_ulp = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    err = (got.double() - want).abs()
    lim = half_ulp * want.abs() + 1e-4 * want.abs().max()
    assert bool((err <= lim).all()), (err - lim).max().item()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,k,co,h,w", [
    (1, 64, 64, 1, 1),        # one row
    (1, 64, 128, 8, 16),      # exactly one tile
    (3, 128, 64, 11, 13),     # a ragged second and third one
    (2, 192, 320, 9, 7),      # channels that are multiples of 64 only
    (4, 512, 2048, 7, 7),     # a few rows, many columns of tiles
    (16, 256, 128, 35, 35),   # tiles of 128 columns
    (32, 64, 256, 29, 28),    # tiles of 256 columns, several per CTA, a ragged last one
    (1, 64, 64, 128, 2),      # (with a stride) rows of one pixel, of 128
    (1, 64, 64, 2, 128),
])
def test_conv1x1_kernels(dtype, n, k, co, h, w):
    from horovod_b200 import _C
    g = torch.Generator(device=_dev()).manual_seed(1)
    weight = (torch.randn(co, k, device=_dev(), generator=g) / k ** 0.5).to(dtype)
    x, dy, add = _act(g, n, k, h, w, dtype), _act(g, n, co, h, w, dtype), _act(g, n, k, h, w, dtype)
    y, sums = _C.conv1x1(x, weight, want_sums=True)
    _close(y, torch.einsum("nkhw,ok->nohw", x.double(), weight.double()), dtype)
    rows = y.double().permute(0, 2, 3, 1).reshape(-1, co)
    # fp32 sums of what was stored: 2^-24 of the terms' magnitudes per addition,
    # a few hundred additions in a row at most
    for got, terms in ((sums[0], rows), (sums[1], rows * rows)):
        assert bool(((got - terms.sum(0)).abs() <= 2e-5 * terms.abs().sum(0) + 1e-12).all())
    assert torch.equal(_C.conv1x1(x, weight)[0], y)
    ref = torch.einsum("nohw,ok->nkhw", dy.double(), weight.double())
    _close(_C.conv1x1(dy, weight, w_transposed=True)[0], ref, dtype)
    _close(_C.conv1x1(dy, weight, w_transposed=True, add=add)[0], ref + add.double(), dtype)
    mask = torch.rand(n, k, h, w, device=_dev(), generator=g) > 0.5
    _close(_C.conv1x1(dy, weight, w_transposed=True, add=add, signs=_signs(mask))[0],
           ref + add.double() * mask, dtype)
    # every other pixel of twice the size
    big = _act(g, n, k, 2 * h, 2 * w, dtype)
    wide = big.double()
    wide[:, :, ::2, ::2] += ref
    _close(_C.conv1x1(dy, weight, w_transposed=True, add=big, scatter=True)[0], wide, dtype)
    y2, sums2 = _C.conv1x1(big, weight, gather=True, want_sums=True)
    y3, sums3 = _C.conv1x1(big[:, :, ::2, ::2].contiguous(memory_format=CL), weight,
                           want_sums=True)
    assert torch.equal(y2, y3)
    torch.testing.assert_close(sums2, sums3, rtol=1e-5, atol=1e-3)


def test_conv1x1_values_that_are_not_finite():
    """Infinities and NaN reach the rows that hold them and no others."""
    from horovod_b200 import _C
    g = torch.Generator(device=_dev()).manual_seed(2)
    x = _act(g, 2, 64, 9, 9, torch.bfloat16)
    weight = torch.randn(64, 64, device=_dev(), generator=g).bfloat16()
    clean = _C.conv1x1(x, weight)[0]
    x[0, 3, 2, 1], x[1, 5, 8, 8] = float("inf"), float("nan")
    y, sums = _C.conv1x1(x, weight, want_sums=True)
    touched = torch.zeros(2, 1, 9, 9, dtype=torch.bool, device=_dev())
    touched[0, 0, 2, 1] = touched[1, 0, 8, 8] = True
    assert torch.equal(torch.where(touched, 0, y), torch.where(touched, 0, clean))
    assert not bool(y[0, :, 2, 1].isfinite().any()) and bool(y[1, :, 8, 8].isnan().all())
    assert bool(sums.isnan().all())


def test_conv1x1_wait_that_runs_out():
    """The results are NaN, the device is marked, and nothing is left behind."""
    from horovod_b200 import _C
    g = torch.Generator(device=_dev()).manual_seed(3)
    x, add = _act(g, 8, 64, 30, 30, torch.bfloat16), _act(g, 8, 64, 30, 30, torch.bfloat16)
    big = _act(g, 8, 64, 60, 60, torch.bfloat16)
    weight = torch.randn(64, 64, device=_dev(), generator=g).bfloat16()
    calls = [dict(want_sums=True), dict(w_transposed=True), dict(w_transposed=True, add=add),
             dict(w_transposed=True, add=big, scatter=True)]
    try:
        for kw in calls:
            before = _C.conv1x1(x, weight, **kw)
            assert not _C.stem_conv_failed(0)
            y, sums = _C.conv1x1(x, weight, wait_ns=0, **kw)
            torch.cuda.synchronize()
            assert _C.stem_conv_failed(0, clear=True)
            if "scatter" in kw:
                assert bool(y[:, :, ::2, ::2].isnan().all())
                assert torch.equal(y[:, :, 1::2], big[:, :, 1::2])
            else:
                assert bool(y.isnan().all())
            assert sums is None or bool(sums[0].isnan().all())
            again = _C.conv1x1(x, weight, **kw)
            assert torch.equal(again[0], before[0])
        block, x = _block(64, 16, 1, False), _act(g, 2, 64, 8, 8, torch.bfloat16)
        assert _available(block, x)
        _C.conv1x1(x, weight, wait_ns=0)
        torch.cuda.synchronize()
        with pytest.warns(UserWarning, match="ran out"):
            assert not _available(block, x)
    finally:
        torch.cuda.synchronize()
        _C.stem_conv_failed(0, clear=True)


def _tail(g, n, cout, h, w, dtype):
    """What the backward of a batch norm behind a 1x1 convolution of 64 channels gets:
    dy, signs, x, a, weight, gamma, saved."""
    from horovod_b200 import _C
    x, res, dy = (_act(g, n, cout, h, w, dtype) for _ in range(3))
    a = _act(g, n, 64, h, w, dtype).relu_()
    weight = (torch.randn(cout, 64, device=_dev(), generator=g) / 8).to(dtype)
    gamma = torch.rand(cout, device=_dev(), generator=g) + 0.5
    _, saved, signs = _C.bn_forward(x, res, gamma, torch.zeros_like(gamma), None, None, 0.1, 1e-5,
                                    True, None)
    return dy, signs, x, a, weight, gamma, saved


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("n,cout,h,w", [
    (1, 256, 1, 2), (1, 128, 1, 17),                   # a few rows: one slot of the ring
    (1, 256, 8, 16), (1, 128, 8, 16),                  # exactly one tile
    (3, 256, 9, 11), (2, 128, 13, 10),                 # a ragged last one
    (64, 256, 29, 23), (64, 128, 29, 23),              # several per CTA
])
def test_norm_conv_backward(dtype, n, cout, h, w):
    """dx is formed as by the batch norm's own kernel, bit for bit; da is its product
    with the weight, rounded once; dW sums in fp32 (and fp64 across CTAs)."""
    from horovod_b200 import _C
    g = torch.Generator(device=_dev()).manual_seed(11)
    dy, signs, x, a, weight, gamma, saved = _tail(g, n, cout, h, w, dtype)
    da, dw, dgamma, dbeta = _C.norm_conv_backward(dy, signs, x, a, weight, gamma, saved)
    dx, _, dgamma_ref, dbeta_ref = _C.bn_backward(dy, x, gamma, saved, signs, True, False)
    _close(da, torch.einsum("nohw,ok->nkhw", dx.double(), weight.double()), dtype)
    want = torch.einsum("nohw,nkhw->ok", dx.double(), a.double())
    terms = torch.einsum("nohw,nkhw->ok", dx.double().abs(), a.double().abs())
    assert bool(((dw - want).abs() <= 1e-5 * terms + 1e-12).all())
    # the sums' atomics come in any order
    torch.testing.assert_close(dgamma, dgamma_ref, rtol=1e-6, atol=1e-6)
    torch.testing.assert_close(dbeta, dbeta_ref, rtol=1e-6, atol=1e-6)


def test_norm_conv_backward_values_that_are_not_finite():
    """A NaN in an activation reaches its column of dW and nothing else; one in the
    batch norm's input reaches all of its channel."""
    from horovod_b200 import _C
    g = torch.Generator(device=_dev()).manual_seed(12)
    dy, signs, x, a, weight, gamma, saved = _tail(g, 3, 256, 9, 11, torch.bfloat16)
    da, dw, _, _ = _C.norm_conv_backward(dy, signs, x, a, weight, gamma, saved)
    a[2, 7, 8, 10] = float("nan")  # of the last, ragged tile
    da2, dw2, _, _ = _C.norm_conv_backward(dy, signs, x, a, weight, gamma, saved)
    assert torch.equal(da, da2) and bool(dw2[:, 7].isnan().all())
    assert torch.equal(dw2[:, :7], dw[:, :7]) and torch.equal(dw2[:, 8:], dw[:, 8:])
    x[1, 200, 3, 3] = float("inf")
    da3, dw3, dgamma, _ = _C.norm_conv_backward(dy, signs, x, a, weight, gamma, saved)
    assert bool(da3.isnan().all()) and bool(dgamma[200].isfinite().logical_not())
    assert bool(dw3[200].isfinite().logical_not().all())
    assert torch.equal(dw3[:200, :7], dw[:200, :7])


def test_norm_conv_backward_wait_that_runs_out():
    from horovod_b200 import _C
    g = torch.Generator(device=_dev()).manual_seed(13)
    args = _tail(g, 40, 256, 28, 28, torch.bfloat16)
    before = _C.norm_conv_backward(*args)
    try:
        da, dw, _, _ = _C.norm_conv_backward(*args, wait_ns=0)
        torch.cuda.synchronize()
        assert _C.stem_conv_failed(0, clear=True)
        assert bool(da.isnan().all()) and bool(dw.isnan().all())
    finally:
        torch.cuda.synchronize()
        _C.stem_conv_failed(0, clear=True)
    again = _C.norm_conv_backward(*args)
    assert all(_rel(p, q) <= 1e-6 for p, q in zip(again, before))


def _block(inplanes, planes, stride, down, seed=0):
    from horovod_b200.models.resnet import Bottleneck
    from horovod_b200.ops.batch_norm import BatchNormAct2d
    torch.manual_seed(seed)
    downsample = nn.Sequential(nn.Conv2d(inplanes, planes * 4, 1, stride=stride, bias=False),
                               BatchNormAct2d(planes * 4, relu=False)) if down else None
    block = Bottleneck(inplanes, planes, stride, downsample)
    for m in block.modules():
        if isinstance(m, nn.BatchNorm2d):
            nn.init.uniform_(m.weight, 0.5, 1.5)
            nn.init.normal_(m.bias, std=0.1)
    return block.to(_dev()).to(memory_format=CL)


def _available(block, x):
    from horovod_b200.ops.bottleneck import fused_bottleneck_available
    with torch.autocast("cuda", dtype=x.dtype):
        return fused_bottleneck_available(block, x) is not None


def _step(block, x, dy, autocast=True):
    """y, the gradients of x and of every parameter, and the buffers."""
    block.zero_grad()
    x = x.detach().clone(memory_format=CL).requires_grad_(True)
    with torch.autocast("cuda", dtype=torch.bfloat16 if x.dtype == torch.float64 else x.dtype,
                        enabled=autocast and x.dtype != torch.float64):
        y = block(x)
    y.backward(dy.to(y.dtype))
    out = {"y": y.detach(), "dx": x.grad}
    out.update({n: p.grad for n, p in block.named_parameters()})
    out.update({n: b.clone() for n, b in block.named_buffers()})
    return out


def _rel(a, b):
    return ((a.double() - b.double()).norm() / (b.double().norm() + 1e-30)).item()


SHAPES = [
    (256, 64, 1, False, 4, 12, 10, torch.bfloat16), (64, 64, 1, True, 4, 12, 10, torch.bfloat16),
    (256, 128, 2, True, 4, 12, 10, torch.float16),
    (64, 64, 1, True, 16, 28, 27, torch.float16), (256, 64, 2, True, 3, 10, 10, torch.bfloat16),
    (256, 128, 2, True, 4, 11, 9, torch.bfloat16),    # odd sizes: PyTorch's strided layers
    (64, 64, 2, True, 1, 2, 260, torch.bfloat16),     # and rows of more than 128 pixels
    (1024, 256, 1, False, 9, 7, 7, torch.float16),    # the first convolution is PyTorch's
    (32, 8, 1, False, 4, 9, 9, torch.bfloat16),       # too few channels for the kernels
    (32, 16, 2, True, 4, 8, 8, torch.bfloat16),
]


@pytest.mark.parametrize("shape", SHAPES)
def test_block_is_as_close_to_64_bits_as_its_layers(shape, monkeypatch):
    inplanes, planes, stride, down, n, h, w, dtype = shape
    block = _block(inplanes, planes, stride, down)
    g = torch.Generator(device=_dev()).manual_seed(4)
    x = _act(g, n, inplanes, h, w, dtype).relu_()
    dy = _act(g, n, planes * 4, (h - 1) // stride + 1, (w - 1) // stride + 1, dtype)
    assert _available(block, x)
    fused = _step(copy.deepcopy(block), x, dy)
    monkeypatch.setenv("HOROVOD_B200_FUSED_BLOCK", "0")
    assert not _available(block, x)
    layers = _step(copy.deepcopy(block), x, dy)
    exact = _step(copy.deepcopy(block).double(), x.double(), dy.double())
    for name, want in exact.items():
        if not want.is_floating_point():
            assert torch.equal(fused[name], want), name
            continue
        # Values that pass a ReLU or not by their last bit make most of either
        # error; which ones do is chance.
        assert _rel(fused[name], want) <= 1.15 * _rel(layers[name], want) + 2e-3, name
    for name, p in block.named_parameters():
        assert fused[name].stride() == p.stride() and fused[name].dtype == p.dtype


@pytest.mark.parametrize("change", ["contiguous", "transposed", "flat", "16 bit", "frozen",
                                    "expanded dy", "strided dy"])
def test_block_with_other_layouts(change, monkeypatch):
    """Weights and gradients in layouts other than the usual one: as the layers."""
    block = _block(256, 64, 2, True)
    g = torch.Generator(device=_dev()).manual_seed(5)
    x = _act(g, 4, 256, 12, 10, torch.bfloat16).relu_()
    dy = _act(g, 4, 256, 6, 5, torch.bfloat16)
    params = dict(block.named_parameters())
    if change == "contiguous":
        block = block.to(memory_format=torch.contiguous_format)
    elif change == "transposed":
        for name in ("conv1.weight", "conv3.weight", "downsample.0.weight"):
            p = params[name]
            p.data = p.data[:, :, 0, 0].t().contiguous().t()[:, :, None, None]
    elif change == "flat":  # off a 16-byte boundary
        for p in params.values():
            if p.dim() == 4:
                flat = torch.empty(p.numel() + 1, device=_dev())
                p.data = torch.as_strided(flat, p.shape, p.stride(), 1).copy_(p.data)
    elif change == "16 bit":
        for p in params.values():
            if p.dim() == 4:
                p.data = p.data.bfloat16()
    elif change == "frozen":
        for name in ("conv1.weight", "bn2.weight", "bn3.bias", "downsample.0.weight"):
            params[name].requires_grad_(False)
    elif change == "expanded dy":
        dy = torch.full((1, 1, 1, 1), 0.5, device=_dev()).bfloat16().expand(4, 256, 6, 5)
    elif change == "strided dy":
        dy = dy.contiguous()

    def step(block):
        xx = x.detach().clone(memory_format=CL).requires_grad_(True)
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=change != "16 bit"):
            y = block(xx)
        y.backward(dy)
        return [y.detach(), xx.grad] + [p.grad for p in block.parameters()]

    from horovod_b200.ops.bottleneck import fused_bottleneck_available
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=change != "16 bit"):
        assert fused_bottleneck_available(block, x) is not None
    fused = step(copy.deepcopy(block))
    monkeypatch.setenv("HOROVOD_B200_FUSED_BLOCK", "0")
    layers = step(copy.deepcopy(block))
    for a, b in zip(fused, layers):
        assert (a is None) == (b is None)
        # the two round the same values in the same places but for a few
        assert a is None or (_rel(a, b) <= 4e-2 and a.dtype == b.dtype)


class _Add(nn.Module):
    def __init__(self, norm):
        super().__init__()
        self.norm = norm

    def forward(self, x, residual):
        return self.norm(x) + residual


@pytest.mark.parametrize("inplanes,planes,stride,down", [
    (256, 64, 1, False), (64, 64, 1, True), (256, 128, 2, True), (512, 128, 1, False)])
def test_block_whose_input_wants_no_gradient(inplanes, planes, stride, down):
    """The parameters' gradients are those of a block whose input does."""
    block = _block(inplanes, planes, stride, down)
    g = torch.Generator(device=_dev()).manual_seed(14)
    x = _act(g, 4, inplanes, 12, 10, torch.bfloat16).relu_()
    assert _available(block, x)
    params = list(block.parameters())

    def grads(x):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = block(x)
        return torch.autograd.grad(y, params, torch.ones_like(y))

    for a, b in zip(grads(x), grads(x.detach().requires_grad_(True))):
        assert _rel(a, b) <= 2e-2  # sums in another order


def test_block_leaves_the_rest_to_its_layers():
    from horovod_b200.ops.bottleneck import fused_bottleneck_available
    g = torch.Generator(device=_dev()).manual_seed(6)
    x = _act(g, 2, 256, 8, 8, torch.bfloat16)

    def plain(block, x=x, autocast=torch.bfloat16):
        with torch.autocast("cuda", dtype=autocast or torch.bfloat16, enabled=autocast is not None):
            assert fused_bottleneck_available(block, x) is None
            return block(x)

    def changed(f):
        block = _block(256, 64, 1, False)
        f(block)
        return block

    assert _available(_block(256, 64, 1, False), x)
    plain(_block(256, 64, 1, False), x.contiguous())
    plain(_block(256, 64, 1, False), autocast=torch.float16)
    plain(_block(256, 64, 1, False), x.float())
    flat = torch.empty(x.numel() + 1, device=_dev(), dtype=x.dtype)
    plain(_block(256, 64, 1, False), torch.as_strided(flat, x.shape, x.stride(), 1).copy_(x))
    plain(changed(lambda b: b.eval()))
    plain(changed(lambda b: b.bn2.eval()))
    plain(changed(lambda b: setattr(b.bn1, "momentum", None)))
    plain(changed(lambda b: setattr(b.bn1, "relu", False)))
    plain(changed(lambda b: setattr(b, "bn1", nn.BatchNorm2d(64).to(_dev()))))
    plain(changed(lambda b: setattr(b.conv2, "dilation", (2, 2))
                  or setattr(b.conv2, "padding", (2, 2))))
    plain(changed(lambda b: nn.utils.parametrizations.weight_norm(b.conv1)))
    # layers without a stride, channels or statistics of their own
    plain(changed(lambda b: setattr(b, "conv1", nn.Sequential(b.conv1))))
    plain(changed(lambda b: setattr(b, "conv2", nn.Sequential(b.conv2))))
    plain(changed(lambda b: setattr(b, "bn3", _Add(b.bn3))))
    plain(changed(lambda b: setattr(b, "downsample", nn.Sequential(nn.Identity(), nn.Identity()))))
    plain(changed(lambda b: setattr(b, "downsample", nn.Identity())))
    calls = []
    plain(changed(lambda b: b.conv2.register_forward_hook(lambda *a: calls.append(1))))
    plain(changed(lambda b: b.bn3.register_full_backward_hook(lambda *a: None)))
    assert calls == [1]
    handle = nn.modules.module.register_module_forward_hook(lambda *a: calls.append(2))
    try:
        plain(_block(256, 64, 1, False))
    finally:
        handle.remove()
    assert calls.count(2) > 3
    from torch.autograd import forward_ad
    with forward_ad.dual_level():
        plain(_block(256, 64, 1, False))
    block, seen = _block(256, 64, 1, False), []
    torch.func.vmap(lambda t: seen.append(fused_bottleneck_available(block, t)) or t)(x[None])
    assert seen == [None]


def test_block_under_autograds_other_uses():
    """Gradients of gradients, a second backward, saved-tensor hooks, weights that
    change between forward and backward, an output that does."""
    block = _block(256, 64, 1, False)
    g = torch.Generator(device=_dev()).manual_seed(7)
    x = _act(g, 2, 256, 8, 8, torch.bfloat16).requires_grad_(True)
    inputs = [x] + list(block.parameters())

    def forward():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return block(x)

    y = forward()
    dy = torch.ones_like(y)
    first = torch.autograd.grad(y, inputs, dy, retain_graph=True)
    again = torch.autograd.grad(y, inputs, dy, retain_graph=True)
    for a, b in zip(first, again):
        assert _rel(a, b) <= 1e-3  # sums of the batch norms in another order
    graph = torch.autograd.grad(y, inputs, dy, create_graph=True)
    for a, b in zip(graph, first):
        assert _rel(a, b) <= 0.15  # PyTorch's composition, which rounds elsewhere
    second = torch.autograd.grad(sum(t.float().square().sum() for t in graph), inputs)
    assert all(bool(t.isfinite().all()) for t in second)
    assert second[1].norm().item() > 0

    saved = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: saved.append(1) or t.cpu(),
                                                  lambda t: t.to(_dev())):
        y = forward()
    for a, b in zip(torch.autograd.grad(y, inputs, dy), first):
        assert _rel(a, b) <= 1e-3
    assert saved

    y = forward()
    before = block.conv1.weight.detach().clone()
    with torch.no_grad():
        block.conv1.weight.zero_()
    for a, b in zip(torch.autograd.grad(y, inputs, dy), first):
        assert _rel(a, b) <= 1e-3
    with torch.no_grad():
        block.conv1.weight.copy_(before)
    y = forward()
    y.detach().add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(y, inputs, dy)


def test_block_in_a_graph():
    """A captured step replays with new inputs as the same step does eagerly."""
    block = _block(256, 128, 2, True)
    g = torch.Generator(device=_dev()).manual_seed(8)
    x = _act(g, 4, 256, 8, 8, torch.bfloat16).requires_grad_(True)
    dy = _act(g, 4, 512, 4, 4, torch.bfloat16)
    inputs = [x] + list(block.parameters())

    def step():
        with torch.autocast("cuda", dtype=torch.bfloat16, cache_enabled=False):
            y = block(x)
        return [y] + list(torch.autograd.grad(y, inputs, dy))

    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        for _ in range(2):
            step()
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        captured = step()
    for _ in range(2):
        with torch.no_grad():
            x.copy_(_act(g, 4, 256, 8, 8, torch.bfloat16))
        graph.replay()
        torch.cuda.synchronize()
        replayed = [t.clone() for t in captured]
        for a, b in zip(replayed, step()):
            assert _rel(a, b) <= 2e-2  # sums in another order


def test_block_on_two_streams():
    """Two streams at once: each has the results of one alone."""
    g = torch.Generator(device=_dev()).manual_seed(9)
    blocks = [_block(256, 64, 1, False, seed) for seed in (1, 2)]
    xs = [_act(g, 16, 256, 28, 28, torch.bfloat16) for _ in blocks]
    dy = _act(g, 16, 256, 28, 28, torch.bfloat16)
    alone = [_step(copy.deepcopy(b), x, dy) for b, x in zip(blocks, xs)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in blocks]
    together = []
    for b, x, s in zip(blocks, xs, streams):
        with torch.cuda.stream(s):
            together.append(_step(b, x, dy))
    torch.cuda.synchronize()
    for a, b in zip(alone, together):
        assert max(_rel(b[k], a[k]) for k in a if a[k].is_floating_point()) <= 2e-2


@pytest.mark.parametrize("inplanes,planes,stride", [(64, 64, 1), (256, 128, 2), (1024, 256, 2)])
def test_block_holds_its_sums_while_others_ask_for_scratch(inplanes, planes, stride):
    """The zeroed scratch of the batch norms is cleared whenever it has been handed out
    once. Wherever in a step of a block that happens, and for whatever was written
    before, every step has the results of the first."""
    from horovod_b200 import _C
    import random
    block = _block(inplanes, planes, stride, True)
    for m in block.modules():
        if isinstance(m, nn.BatchNorm2d):
            m.momentum = 1.0  # the running statistics are those of the step
    g = torch.Generator(device=_dev()).manual_seed(21)
    x = _act(g, 2, inplanes, 8, 6, torch.bfloat16).relu_()
    dy = _act(g, 2, planes * 4, 8 // stride, 6 // stride, torch.bfloat16)
    assert _available(block, x)
    other = _act(g, 1, 64, 2, 2, torch.bfloat16)
    rng = random.Random(22)  # where in a step the scratch is used up: all over it
    want, worst = None, None
    for _ in range(1200):
        for _ in range(rng.randrange(8)):
            _C.bn_forward(other, None, None, None, None, None, 0.1, 1e-5, False, None)
        got = [t.double() for t in _step(block, x, dy).values() if t.is_floating_point()]
        if want is None:
            want, worst = got, torch.zeros(len(got), device=_dev(), dtype=torch.float64)
        worst = torch.maximum(worst, torch.stack(
            [(a - b).norm() / (b.norm() + 1e-30) for a, b in zip(got, want)]))
    # Sums in another order: a value in a few thousand rounds the other way or passes
    # a ReLU (2^-8 and 1 of its size). Sums that are lost change all values of a layer.
    assert bool((worst <= 5e-2).all()), worst.tolist()


def test_blocks_of_two_threads_on_one_stream():
    """Each thread has the results of one alone."""
    import threading
    g = torch.Generator(device=_dev()).manual_seed(23)
    blocks = [_block(64, 64, 1, True, seed) for seed in (1, 2)]
    x = _act(g, 2, 64, 8, 6, torch.bfloat16)
    dy = _act(g, 2, 256, 8, 6, torch.bfloat16)
    worst = {}

    def work(i):
        params = list(blocks[i].parameters())

        def step():
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = blocks[i](x)
            return [y.detach()] + list(torch.autograd.grad(y, params, dy))
        want = first[i]
        worst[i] = torch.zeros(len(want), device=_dev(), dtype=torch.float64)
        for _ in range(300):
            worst[i] = torch.maximum(worst[i], torch.stack(
                [(a.double() - b.double()).norm() / (b.double().norm() + 1e-30)
                 for a, b in zip(step(), want)]))

    first = []
    for b in blocks:
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = b(x)
        first.append([y.detach()] + list(torch.autograd.grad(y, list(b.parameters()), dy)))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i in range(2):
        assert bool((worst[i] <= 5e-2).all()), worst[i].tolist()


@pytest.mark.parametrize("inplanes,planes,stride,down", [
    (256, 64, 1, False), (64, 64, 1, True), (256, 128, 2, True), (32, 16, 2, True)])
def test_block_whose_saved_tensors_come_back_in_another_layout(inplanes, planes, stride, down):
    """save_on_cpu(pin_memory=True) packs into contiguous memory: what comes back is NCHW."""
    block = _block(inplanes, planes, stride, down)
    g = torch.Generator(device=_dev()).manual_seed(24)
    x = _act(g, 4, inplanes, 12, 10, torch.bfloat16).relu_().requires_grad_(True)
    inputs = [x] + list(block.parameters())
    assert _available(block, x)

    def grads():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = block(x)
        return y

    y = grads()
    want = torch.autograd.grad(y, inputs, torch.ones_like(y))
    with torch.autograd.graph.save_on_cpu(pin_memory=True):
        y = grads()
    for a, b in zip(torch.autograd.grad(y, inputs, torch.ones_like(y)), want):
        assert _rel(a, b) <= 2e-2  # sums in another order


def test_block_whose_saved_tensors_come_back_off_a_boundary():
    """And with what does not fit the forward's, the backward raises."""
    block = _block(64, 64, 1, True)
    g = torch.Generator(device=_dev()).manual_seed(25)
    x = _act(g, 4, 64, 12, 10, torch.bfloat16).relu_().requires_grad_(True)
    inputs = [x] + list(block.parameters())

    def off(t):
        flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
        return torch.as_strided(flat, t.shape, t.stride(), 1).copy_(t)

    def run(unpack):
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = block(x)
        return torch.autograd.grad(y, inputs, torch.ones_like(y))

    for a, b in zip(run(off), run(lambda t: t)):
        assert _rel(a, b) <= 2e-2  # sums in another order
    for spoil in (lambda t: t[:1], lambda t: t.cpu(),
                  lambda t: t.float() if t.dtype == torch.bfloat16 else t):
        with pytest.raises(RuntimeError, match="saved"):
            run(spoil)


@pytest.mark.parametrize("name,shape", [
    ("conv1", (64, 128, 1, 1)), ("conv2", (64, 32, 3, 3)), ("conv2", (64, 64, 1, 1)),
    ("conv3", (256, 32, 1, 1)), ("downsample", (256, 128, 1, 1))])
def test_block_with_a_weight_of_another_shape(name, shape):
    """One that was replaced without the layer's attributes raises, as in the layers."""
    from horovod_b200.ops.bottleneck import fused_bottleneck, fused_bottleneck_available
    block = _block(256, 64, 2, True)
    g = torch.Generator(device=_dev()).manual_seed(32)
    x = _act(g, 2, 256, 8, 8, torch.bfloat16)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        layers = fused_bottleneck_available(block, x)
        assert layers is not None
        conv = block.downsample[0] if name == "downsample" else getattr(block, name)
        conv.weight = nn.Parameter(torch.randn(shape, device=_dev()))
        assert fused_bottleneck_available(block, x) is None
        with pytest.raises(RuntimeError, match="shapes do not match"):
            fused_bottleneck(x, layers)
        with pytest.raises(RuntimeError):
            block(x)
    with pytest.raises(RuntimeError, match="16-byte"):
        flat = torch.empty(x.numel() + 1, device=_dev(), dtype=x.dtype)
        fused_bottleneck(torch.as_strided(flat, x.shape, x.stride(), 1), layers)


def _block_of(widths):
    """A block without a convolution in its skip connection whose convolutions have
    widths of their own, as after the pruning of channels."""
    block = _block(widths[0], 64, 1, False)
    convs, norms = ("conv1", "conv2", "conv3"), ("bn1", "bn2", "bn3")
    from horovod_b200.ops.batch_norm import BatchNormAct2d
    for i, (conv, norm) in enumerate(zip(convs, norms)):
        kernel = 3 if i == 1 else 1
        setattr(block, conv, nn.Conv2d(widths[i], widths[i + 1], kernel, padding=kernel // 2,
                                       bias=False))
        setattr(block, norm, BatchNormAct2d(widths[i + 1], relu=True))
    return block.to(_dev()).to(memory_format=CL)


@pytest.mark.parametrize("widths", [
    (256, 32, 64, 256),   # the end of the block is this library's, its first convolution is not
    (128, 32, 64, 128), (128, 64, 64, 128),
    (256, 64, 32, 256),   # the other way round
    (256, 32, 32, 256), (512, 128, 64, 512)])
@pytest.mark.parametrize("want_x", [True, False])
def test_block_with_widths_of_its_own(widths, want_x, monkeypatch):
    block = _block_of(widths)
    g = torch.Generator(device=_dev()).manual_seed(26)
    x = _act(g, 4, widths[0], 12, 10, torch.bfloat16).relu_()
    dy = _act(g, 4, widths[0], 12, 10, torch.bfloat16)
    assert _available(block, x)

    def step(block):
        xx = x.detach().clone(memory_format=CL).requires_grad_(want_x)
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = block(xx)
        y.backward(dy)
        return [y.detach()] + ([xx.grad] if want_x else []) + [p.grad for p in block.parameters()]

    fused = step(copy.deepcopy(block))
    monkeypatch.setenv("HOROVOD_B200_FUSED_BLOCK", "0")
    layers = step(copy.deepcopy(block))
    for a, b in zip(fused, layers):
        # the two round the same values in the same places but for a few
        assert _rel(a, b) <= 4e-2


def _composed(block, x):
    """The block by PyTorch's operations under bf16 autocast."""
    import torch.nn.functional as F

    def layer(conv, norm, x):
        out = F.conv2d(x, conv.weight.to(x.dtype), None, conv.stride, conv.padding)
        return F.batch_norm(out, None, None, norm.weight, norm.bias, True, 0.0, norm.eps)

    out = F.relu(layer(block.conv2, block.bn2, F.relu(layer(block.conv1, block.bn1, x))))
    skip = layer(*block.downsample, x) if block.downsample is not None else x
    return F.relu(layer(block.conv3, block.bn3, out) + skip)


@pytest.mark.parametrize("inplanes,planes,stride,down", [(256, 64, 1, False), (64, 64, 1, True),
                                                         (256, 128, 2, True)])
def test_block_gradients_of_gradients(inplanes, planes, stride, down):
    """Those of PyTorch's operations, also of weights as they were in the forward."""
    block = _block(inplanes, planes, stride, down)
    g = torch.Generator(device=_dev()).manual_seed(27)
    x = _act(g, 4, inplanes, 12, 10, torch.bfloat16).relu_().requires_grad_(True)
    dy = _act(g, 4, planes * 4, 12 // stride, 10 // stride, torch.bfloat16)
    inputs = [x] + list(block.parameters())
    assert _available(block, x)

    def second(first):
        return torch.autograd.grad(sum(t.float().square().sum() for t in first), inputs)

    first = torch.autograd.grad(_composed(block, x), inputs, dy, create_graph=True)
    want = [t.detach() for t in first] + list(second(first))
    for change in (False, True):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = block(x)
        weights = [m.weight for m in block.modules() if isinstance(m, nn.Conv2d)]
        before = [w.detach().clone() for w in weights]
        if change:
            with torch.no_grad():
                for w in weights:
                    w.mul_(-2.0)
        first = torch.autograd.grad(y, inputs, dy, create_graph=True)
        got = [t.detach() for t in first] + list(second(first))
        with torch.no_grad():
            for w, b in zip(weights, before):
                w.copy_(b)
        for i, (a, b) in enumerate(zip(got, want)):
            # the same operations, whose convolutions' sums may have another order
            assert _rel(a, b) <= 2e-2, (change, i)


def test_block_whose_batch_norms_change_after_the_forward():
    """A bias is not needed for the backward, a weight is; both for a gradient's."""
    block = _block(256, 64, 1, False)
    g = torch.Generator(device=_dev()).manual_seed(28)
    x = _act(g, 4, 256, 8, 8, torch.bfloat16).relu_().requires_grad_(True)
    inputs = [x] + list(block.parameters())

    def forward():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            return block(x)

    y = forward()
    want = torch.autograd.grad(y, inputs, torch.ones_like(y))
    y = forward()
    with torch.no_grad():
        block.bn2.bias.add_(0.0)
    got = torch.autograd.grad(y, inputs, torch.ones_like(y), retain_graph=True)
    for a, b in zip(got, want):
        assert _rel(a, b) <= 2e-2  # sums in another order
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(y, inputs, torch.ones_like(y), create_graph=True)
    y = forward()
    with torch.no_grad():
        block.bn2.weight.add_(0.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(y, inputs, torch.ones_like(y))


@pytest.mark.parametrize("what", ["block", "norm"])
def test_recomputed_activations(what):
    """A checkpointed region ends its second forward with an exception out of a
    saved-tensor hook, which has to arrive as what it is."""
    from torch.utils.checkpoint import checkpoint
    block = _block(256, 64, 1, False)
    layer = block if what == "block" else block.bn3
    g = torch.Generator(device=_dev()).manual_seed(30)
    x = _act(g, 2, 256, 8, 8, torch.bfloat16).requires_grad_(True)
    inputs = [x] + list(layer.parameters())

    def grads(f):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = f(x)
        return torch.autograd.grad(y, inputs, torch.ones_like(y))

    for a, b in zip(grads(lambda x: checkpoint(layer, x, use_reentrant=False)), grads(layer)):
        assert _rel(a, b) <= 2e-2  # sums in another order

    class Stop(Exception):
        pass

    def stop(t):
        raise Stop()

    with torch.autograd.graph.saved_tensors_hooks(stop, lambda t: t), pytest.raises(Stop):
        grads(layer)


def test_block_under_function_modes():
    """A mode that watches functions sees the layers' convolutions; a default device
    is no such mode."""
    from torch.overrides import TorchFunctionMode

    class Watch(TorchFunctionMode):
        seen = 0

        def __torch_function__(self, func, types, args=(), kwargs=None):
            Watch.seen += func in (torch.conv2d, nn.functional.conv2d)
            return func(*args, **(kwargs or {}))

    block = _block(256, 64, 1, False)
    g = torch.Generator(device=_dev()).manual_seed(29)
    x = _act(g, 2, 256, 8, 8, torch.bfloat16)
    with torch.device("cuda"):
        assert _available(block, x)
        with Watch(), torch.autocast("cuda", dtype=torch.bfloat16):
            block(x)
    assert Watch.seen == 3


@pytest.mark.parametrize("down", [False, True])
def test_block_does_not_compute_gradients_that_nobody_wants(down):
    """With the first layers frozen and an input without a gradient, the backward ends
    at the layers that are trained: fewer launches, the same gradients."""
    from horovod_b200 import _C
    block = _block(64 if down else 256, 64, 1, down)
    g = torch.Generator(device=_dev()).manual_seed(31)
    x = _act(g, 2, 64 if down else 256, 8, 8, torch.bfloat16)
    dy = _act(g, 2, 256, 8, 8, torch.bfloat16)

    def step():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = block(x)
        before = _C.kernel_launch_count()
        y.backward(dy)
        torch.cuda.synchronize()
        grads = {n: p.grad for n, p in block.named_parameters() if p.requires_grad}
        block.zero_grad()
        return _C.kernel_launch_count() - before, grads

    every, want = step()
    last = every
    for frozen in ("conv1", "bn1", "conv2", "bn2") + (("downsample",) if down else ()):
        for p in getattr(block, frozen).parameters():
            p.requires_grad_(False)
        launches, got = step()
        for n, t in got.items():
            assert _rel(t, want[n]) <= 2e-2, n  # sums in another order
        if not frozen.startswith("conv"):
            assert launches < last  # the batch norm's two kernels and more
            last = launches


def test_kernels_refuse_what_starts_off_a_boundary():
    from horovod_b200 import _C
    g = torch.Generator(device=_dev()).manual_seed(33)

    def off(t):
        flat = torch.empty(t.numel() + 1, device=t.device, dtype=t.dtype)
        return torch.as_strided(flat, t.shape, t.stride(), 1).copy_(t)

    args = _tail(g, 3, 256, 9, 11, torch.bfloat16)
    for i in (0, 1, 2, 3, 4, 6):  # gamma is read value by value
        with pytest.raises(RuntimeError, match="invalid argument"):
            _C.norm_conv_backward(*[off(t) if i == k else t for k, t in enumerate(args)])
    da, dw, _, _ = _C.norm_conv_backward(*args)
    args = tuple(off(t) if k == 5 else t for k, t in enumerate(args))
    assert torch.equal(_C.norm_conv_backward(*args)[0], da)
    x, add = _act(g, 2, 64, 9, 9, torch.bfloat16), _act(g, 2, 64, 9, 9, torch.bfloat16)
    weight = torch.randn(64, 64, device=_dev(), generator=g).bfloat16()
    signs = _signs(add > 0)
    for kw in (dict(x=off(x)), dict(w=off(weight)), dict(add=off(add)), dict(signs=off(signs))):
        with pytest.raises(RuntimeError, match="invalid argument"):
            _C.conv1x1(**{**dict(x=x, w=weight, w_transposed=True, add=add, signs=signs), **kw})


@pytest.mark.parametrize("down", [False, True])
def test_block_under_compiled_autograd(down):
    """A backward that is traced runs the node as it is."""
    from torch._dynamo import compiled_autograd
    block = _block(64 if down else 256, 64, 1, down)
    g = torch.Generator(device=_dev()).manual_seed(34)
    x = _act(g, 2, 64 if down else 256, 8, 8, torch.bfloat16).requires_grad_(True)
    inputs = [x] + list(block.parameters())
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = block(x)
    want = torch.autograd.grad(y, inputs, torch.ones_like(y), retain_graph=True)
    with compiled_autograd._enable(lambda graph: graph):
        y.backward(torch.ones_like(y))
    for t, b in zip(inputs, want):
        assert _rel(t.grad, b) <= 2e-2  # sums in another order


_RECORDED = """
import threading, torch
from horovod_b200.models.resnet import Bottleneck
from horovod_b200.ops.batch_norm import BatchNormAct2d
torch.cuda.memory._record_memory_history(enabled="all", stacks="python")
down = torch.nn.Sequential(torch.nn.Conv2d(64, 256, 1, bias=False), BatchNormAct2d(256, relu=False))
block = Bottleneck(64, 64, 1, down).cuda().to(memory_format=torch.channels_last)
norm = BatchNormAct2d(256).cuda()

def blocks():
    x = torch.randn(2, 8, 6, 64, device="cuda").bfloat16().permute(0, 3, 1, 2)
    for _ in range(400):
        with torch.autocast("cuda", dtype=torch.bfloat16):
            block(x).sum().backward()

def norms():
    x = torch.randn(2, 8, 6, 256, device="cuda").bfloat16().permute(0, 3, 1, 2)
    for _ in range(4000):
        norm(x)

threads = [threading.Thread(target=f) for f in (blocks, norms)]
[t.start() for t in threads]
[t.join() for t in threads]
torch.cuda.synchronize()
print("done")
"""


def test_two_threads_while_allocations_are_recorded():
    """The allocator then takes the interpreter's lock, which one thread holds while it
    waits for the scratch that the other one is given: nobody waits for both."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    run = subprocess.run([sys.executable, "-c", _RECORDED], cwd=root, capture_output=True,
                         text=True, timeout=200)
    assert run.returncode == 0 and "done" in run.stdout, run.stderr[-2000:]
