"""The model-side and single-rank kernels at the sizes where they can go wrong:
remainders of their tiles and strips, both sides of each dispatch rule (but for
pooling's 64-bit indices, which take tensors of 34 GB), and values that are not
finite."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _dev():
    return torch.device("cuda", 0)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape", [
    (1, 8, 2, 3), (1, 8, 3, 2), (2, 24, 17, 18),  # one output row per thread
    (64, 64, 67, 66),                             # strips of 1 and 2 rows
    (64, 256, 67, 67), (64, 512, 67, 67),         # strips of 4 and 8 rows, ragged
])
def test_max_pool_strips(dtype, shape):
    """Values are few, so ties are the rule; gradients are small whole numbers,
    whose sums are exact in any order."""
    from horovod_b200.ops.pooling import fused_max_pool_available, max_pool_3x3_s2
    g = torch.Generator(device=_dev()).manual_seed(1)
    x = torch.randint(-3, 4, shape, device=_dev(), generator=g).to(dtype)
    flat = x.view(-1)
    flat[::101] = float("-inf")
    flat[::1009] = float("nan")
    x = x.contiguous(memory_format=torch.channels_last).requires_grad_(True)
    ref_x = x.detach().float().requires_grad_(True)
    assert fused_max_pool_available(x)
    y = max_pool_3x3_s2(x)
    ref = F.max_pool2d(ref_x, 3, stride=2, padding=1)
    assert torch.equal(torch.nan_to_num(y.float(), nan=99.0), torch.nan_to_num(ref, nan=99.0))
    go = torch.randint(-8, 9, ref.shape, device=_dev(), generator=g).to(dtype)
    y.backward(go.contiguous(memory_format=torch.channels_last))
    ref.backward(go.float())
    assert torch.equal(x.grad.float(), ref_x.grad)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("with_res", [False, True])
@pytest.mark.parametrize("shape", [
    (1, 8, 1, 3), (3, 8, 31, 33),            # 1 channel group: 256 rows per step of a CTA
    (2, 64, 9, 7), (1, 256, 5, 5), (5, 512, 7, 7),  # fewer rows than a round, and remainders
    (37, 32, 53, 51), (8, 2048, 13, 11),     # several rounds per CTA
])
def test_batch_norm_mask_without_the_output(shape, with_res, dtype):
    """The backward finds relu's mask without reading the output. Whole-number
    gradients have exact sums, so the gradient of the bias must equal the sum
    over the outputs above zero to the last bit, and the residual's gradient
    the masked one; tiny scales put outputs where fp16 rounds them to zero."""
    from horovod_b200.ops.batch_norm import batch_norm_act, fused_batch_norm_available
    dev, c = _dev(), shape[1]
    g = torch.Generator(device=dev).manual_seed(3)

    def act():
        return torch.randn(shape, device=dev, generator=g).to(dtype).contiguous(
            memory_format=torch.channels_last)

    x = act().requires_grad_(True)
    res = act().requires_grad_(True) if with_res else None
    weight = torch.rand(c, device=dev, generator=g) - 0.3
    weight[::3] *= 1e-7
    bias = 0.3 * torch.randn(c, device=dev, generator=g)
    bias[::3] = 0.0
    weight.requires_grad_(True)
    bias.requires_grad_(True)
    assert fused_batch_norm_available(x, 0.1)
    y = batch_norm_act(x, weight, bias, None, None, residual=res)
    dy = torch.randint(-4, 5, shape, device=dev, generator=g).to(dtype).contiguous(
        memory_format=torch.channels_last)
    y.backward(dy)
    dz = dy.double() * (y > 0)
    assert torch.equal(bias.grad.double(), dz.sum((0, 2, 3)))
    if with_res:
        assert torch.equal(res.grad.double(), dz)
    # dx against 64 bits with the same mask: the 16-bit rounding of the result
    # and of the inputs of a sum of three terms
    xd = x.detach().double()
    var, mean = torch.var_mean(xd, (0, 2, 3), unbiased=False, keepdim=True)
    invstd = torch.rsqrt(var + 1e-5)
    xhat = (xd - mean) * invstd
    dx = weight.detach().double().view(1, c, 1, 1) * invstd * (
        dz - dz.mean((0, 2, 3), keepdim=True) - xhat * (dz * xhat).mean((0, 2, 3), keepdim=True))
    eps = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    # 1e-5 of the largest: 32-bit terms that cancel; 6e-8: fp16's smallest step
    bound = eps * dx.abs() + 1e-5 * dx.abs().amax() + 6e-8
    assert bool(((x.grad.double() - dx).abs() <= bound).all())


@pytest.mark.parametrize("with_res", [False, True])
def test_batch_norm_beyond_64_mi_elements(with_res):
    """The writing kernels' other grid."""
    test_batch_norm_mask_without_the_output((21, 64, 224, 224), with_res, torch.bfloat16)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("ratio", [1, 50, 300, 1000])
def test_batch_norm_gradient_of_channels_far_from_zero(ratio, dtype):
    """Means of up to `ratio` times the spread, and a gradient that follows x, so
    that the terms of dx nearly cancel. Against the same formula in 64 bits with
    the kernel's own statistics: left are the fp32 terms' roundings (2^-24 each, of
    the terms' sizes; 2^-19 with those of the sums behind them) and that of the
    result."""
    from horovod_b200 import _C
    dev, shape = _dev(), (4, 64, 31, 33)
    g = torch.Generator(device=dev).manual_seed(14)

    def column(v):
        return v.double().view(1, -1, 1, 1)

    mean = ratio * (0.5 + 0.5 * torch.rand(64, device=dev, generator=g))
    mean[::2] *= -1
    x = (torch.randn(shape, device=dev, generator=g) + mean.view(1, -1, 1, 1)).to(dtype)
    x = x.contiguous(memory_format=torch.channels_last)
    weight = 0.5 + torch.rand(64, device=dev, generator=g)
    _, saved, _ = _C.bn_forward(x, None, weight, None, None, None, 0.1, 1e-5, False, None)
    xc = x.double() - column(saved[0])
    xhat = xc * column(saved[1])
    # whole numbers: their sums are exact
    dy = (30 * xhat + torch.randn(shape, device=dev, generator=g)).clamp(-200, 200).round()
    dy = dy.to(dtype).contiguous(memory_format=torch.channels_last)
    dx = _C.bn_backward(dy, x, weight, saved, None, False, False)[0].double()
    dz, dims = dy.double(), (0, 2, 3)
    scale = column(weight) * column(saved[1])
    terms = [scale * dz, -scale * dz.mean(dims, keepdim=True),
             -scale * xhat * (dz * xhat).mean(dims, keepdim=True)]
    want = sum(terms)
    eps = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    bound = eps * want.abs() + 2.0 ** -19 * sum(t.abs() for t in terms) + 6e-8
    assert bool(((dx - want).abs() <= bound).all())


def test_batch_norm_residual_without_a_gradient():
    from horovod_b200.ops.batch_norm import batch_norm_act
    g = torch.Generator(device=_dev()).manual_seed(4)
    x, res, dy = (torch.randn(3, 16, 5, 5, device=_dev(), generator=g).bfloat16().contiguous(
        memory_format=torch.channels_last) for _ in range(3))
    grads = []
    for wanted in (True, False):
        xi = x.clone(memory_format=torch.preserve_format).requires_grad_(True)
        y = batch_norm_act(xi, None, None, None, None,
                           residual=res.clone(memory_format=torch.preserve_format)
                           .requires_grad_(wanted))
        y.backward(dy)
        grads.append(xi.grad)
    assert torch.equal(*grads)


@pytest.fixture(scope="module")
def hvd():
    import horovod_b200.torch as hvd
    hvd.init()
    torch.cuda.set_device(0)
    yield hvd
    hvd.shutdown()


SIZES = [1, 3, 4, 5, 2047, 2048, 8191, 8192 + 7, (1 << 20) + 1, (3 << 20) + 5]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float64, torch.int64,
                                   torch.uint8])
def test_one_rank_collectives_move_every_element(hvd, dtype):
    """Sizes around a vector, a round of a CTA and a whole grid, and inputs
    that do not start on a 16-byte boundary. The results of scaled ones are
    prescale, round, postscale, round, as with several ranks."""
    g = torch.Generator(device=_dev()).manual_seed(5)
    holder = torch.randint(0, 100, (max(SIZES) + 3,), device=_dev(), generator=g).to(dtype)
    tensors = [holder[:n] for n in SIZES] + [holder[1:1 + n] for n in SIZES]
    for x, y in zip(tensors, hvd.grouped_allreduce(tensors, op=hvd.Sum, name="edge.%s" % dtype)):
        assert torch.equal(x, y)
    for i, x in enumerate(tensors):
        name = "edge.%s.%d" % (dtype, i)
        assert torch.equal(hvd.reducescatter(x, op=hvd.Sum, name=name + ".rs"), x)
        assert torch.equal(hvd.allgather(x, name=name + ".ag"), x)
        assert torch.equal(hvd.alltoall(x, name=name + ".a2a"), x)
        if dtype.is_floating_point:
            wide = torch.float64 if dtype == torch.float64 else torch.float32
            want = ((x.to(wide) * 0.3).to(dtype).to(wide) * 1.7).to(dtype)
            for got in (hvd.reducescatter(x, op=hvd.Sum, prescale_factor=0.3, postscale_factor=1.7,
                                          name=name + ".rss"),
                        hvd.allreduce(x, op=hvd.Sum, prescale_factor=0.3, postscale_factor=1.7,
                                      name=name + ".ars")):
                assert torch.equal(got, want)


@pytest.mark.parametrize("dtype", [torch.float16, torch.int32, torch.int8])
def test_one_rank_collectives_of_the_other_types(hvd, dtype):
    test_one_rank_collectives_move_every_element(hvd, dtype)


@pytest.mark.parametrize("wire", [torch.float16, torch.bfloat16])
def test_one_rank_wire_cast_sizes(hvd, wire):
    g = torch.Generator(device=_dev()).manual_seed(6)
    holder = torch.randn(max(SIZES) + 3, device=_dev(), generator=g)
    for i, x in enumerate([holder[:n] for n in SIZES] + [holder[1:1 + n] for n in SIZES]):
        y = x.clone()
        hvd.synchronize(hvd.allreduce_async_(y, op=hvd.Sum, wire_dtype=wire,
                                             name="edge.wire.%s.%d" % (wire, i)))
        assert torch.equal(y, x.to(wire).float())


@pytest.mark.parametrize("momentum", [0.0, 0.9])
def test_fused_sgd_many_tensors(momentum):
    """More tensors than one launch takes, sizes around a chunk, tensors that
    are not 16-byte aligned and parameters without a gradient."""
    from horovod_b200 import _C
    from horovod_b200.torch.fused_sgd import FusedSGD
    g = torch.Generator(device=_dev()).manual_seed(7)
    sizes = [1, 3, 4, 4095, 4096, 4097, 8193, 0] * 40 + [(1 << 20) + 3]
    holders = [torch.randn(n + 1, device=_dev(), generator=g) for n in sizes]
    ps = [h[i % 2:i % 2 + n].detach().requires_grad_(True)
          for i, (h, n) in enumerate(zip(holders, sizes))]
    qs = [p.detach().clone().requires_grad_(True) for p in ps]
    kwargs = dict(lr=0.1, momentum=momentum, weight_decay=1e-3)
    opt, ref = FusedSGD(ps, **kwargs), torch.optim.SGD(qs, foreach=False, **kwargs)
    for step in range(3):
        for i, (p, q) in enumerate(zip(ps, qs)):
            if i % 11 == step:
                p.grad = q.grad = None
                continue
            p.grad = torch.randn(p.shape, device=_dev(), generator=g)
            q.grad = p.grad.clone()
        before = _C.kernel_launch_count()
        opt.step()
        assert _C.kernel_launch_count() - before >= 2, "321 tensors take two launches"
        ref.step()
    for p, q in zip(ps, qs):
        torch.testing.assert_close(p, q, rtol=1e-5, atol=1e-6)
    assert len(opt.state) == len(ref.state) or momentum == 0


def test_fused_sgd_updates_all_or_nothing():
    """A momentum buffer that the kernel cannot take leaves every parameter as
    it was; one of another memory layout is put into the right one."""
    from horovod_b200 import _C
    from horovod_b200.torch.fused_sgd import FusedSGD
    g = torch.Generator(device=_dev()).manual_seed(15)
    shapes = [(5,), (8, 4, 3, 3), (7, 3), (2, 2)]
    ps = [torch.randn(s, device=_dev(), generator=g) for s in shapes]
    ps.append(torch.randn(3, device=_dev(), generator=g).double())  # left to PyTorch
    qs = [p.clone().requires_grad_(True) for p in ps]
    ps = [p.requires_grad_(True) for p in ps]
    kwargs = dict(lr=0.1, momentum=0.9, weight_decay=1e-3)
    opt, ref = FusedSGD(ps, **kwargs), torch.optim.SGD(qs, foreach=False, **kwargs)

    def gradients():
        for p, q in zip(ps, qs):
            p.grad = torch.randn(p.shape, device=_dev(), generator=g).to(p.dtype)
            q.grad = p.grad.clone()

    def compare():
        for p, q in zip(ps, qs):
            torch.testing.assert_close(p, q, rtol=1e-5, atol=1e-6)

    gradients()
    opt.step()
    ref.step()
    compare()
    good = opt.state[ps[2]]["momentum_buffer"]
    opt.state[ps[1]]["momentum_buffer"] = opt.state[ps[1]]["momentum_buffer"].contiguous(
        memory_format=torch.channels_last)
    gradients()
    for bad in (good.double(), good.cpu(), torch.zeros(6, 3, device=_dev())):
        opt.state[ps[2]]["momentum_buffer"] = bad
        before, launches = [p.detach().clone() for p in ps], _C.kernel_launch_count()
        with pytest.raises(RuntimeError, match="momentum buffer"):
            opt.step()
        assert _C.kernel_launch_count() == launches
        assert all(torch.equal(p, b) for p, b in zip(ps, before))
    opt.state[ps[2]]["momentum_buffer"] = good
    opt.step()
    ref.step()
    compare()
    assert opt.state[ps[1]]["momentum_buffer"].stride() == ps[1].stride()


@pytest.mark.parametrize("name", ["fp16", "bf16"])
def test_compression_inside_the_kernel(hvd, name):
    """allreduce and grouped_allreduce of fp32 tensors with this library's
    compressors: values, layouts, dtypes and gradients of the casts around it."""
    compression = getattr(hvd.Compression, name)
    g = torch.Generator(device=_dev()).manual_seed(8)
    base = torch.randn(6, 8, 5, 7, device=_dev(), generator=g)
    xs = [base, base.contiguous(memory_format=torch.channels_last), base[:, ::2], base[..., 1:],
          torch.randn((), device=_dev(), generator=g), base.flatten()[1:1 + 4099],
          torch.empty(0, device=_dev())]
    leaves = [x.detach().requires_grad_(True) for x in xs]
    ys = hvd.grouped_allreduce(leaves, name="cmp.%s" % name, compression=compression)
    for i, (x, y) in enumerate(zip(xs, ys)):
        want = x.to(compression.wire_dtype).float()
        assert y.dtype == torch.float32 and y.stride() == want.stride() and torch.equal(y, want)
        z = hvd.allreduce(x, name="cmp.%s.%d" % (name, i), compression=compression)
        assert z.stride() == want.stride() and torch.equal(z, want)
    dys = [torch.randn(y.shape, device=_dev(), generator=g) for y in ys]
    for dx, dy in zip(torch.autograd.grad(ys, leaves, dys), dys):
        assert torch.equal(dx, dy.to(compression.wire_dtype).float())
    # other types keep the casts outside
    for dtype in (torch.float64, torch.bfloat16, torch.int32):
        v = torch.arange(9, device=_dev()).to(dtype)
        out = hvd.allreduce(v, name="cmp.%s.%s" % (name, dtype), compression=compression,
                            op=hvd.Sum)
        assert out.dtype == dtype and torch.equal(out, v)


def test_fused_sgd_leaves_the_buffers_of_other_types():
    """A buffer that is put into another layout leaves those of parameters that
    are PyTorch's as they are: fp32 sums of a 16-bit parameter stay fp32."""
    from horovod_b200.torch.fused_sgd import FusedSGD
    ps = [torch.zeros(4, 6, device=_dev(), dtype=d).requires_grad_(True)
          for d in (torch.float32, torch.float16)]
    opt = FusedSGD(ps, lr=0.5, momentum=0.5)
    for p in ps:
        p.grad = torch.ones_like(p)
        opt.state[p]["momentum_buffer"] = torch.full((6, 4), 2.0 ** -13, device=_dev()).t()
    opt.step()
    # 1 + 2^-14 is a number of 24 bits, not of 11
    assert opt.state[ps[0]]["momentum_buffer"].stride() == ps[0].stride()
    for p in ps:
        buf = opt.state[p]["momentum_buffer"]
        assert buf.dtype == torch.float32 and bool((buf == 1 + 2.0 ** -14).all())


def test_compression_refuses_what_is_refused_without(hvd):
    """Permuted tensors: with the casts inside the kernel as with those outside."""
    x = torch.randn(4, 6, device=_dev())
    for compression in (hvd.Compression.none, hvd.Compression.fp16, hvd.Compression.bf16):
        for t in (x.t(), x.double().t(), x.cpu().t()):
            with pytest.raises(ValueError, match="contiguous"):
                hvd.allreduce(t, name="permuted", compression=compression)
            with pytest.raises(ValueError, match="contiguous"):
                hvd.grouped_allreduce([x, t], name="permuted.g", compression=compression)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("shape,channels", [
    ((1, 3, 1, 1), 16), ((2, 3, 33, 17), 64), ((3, 3, 32, 16), 48),  # one past a tile, a tile
    ((2, 3, 31, 50), 128), ((5, 3, 97, 131), 64), ((40, 3, 224, 224), 64),  # several per CTA
])
def test_stem_convolution(shape, channels, dtype):
    """Against the same convolution in 64 bits: fp32 accumulators, so what is
    left is the rounding of the result."""
    from horovod_b200.ops.stem_conv import StemConv2d
    g = torch.Generator(device=_dev()).manual_seed(9)
    conv = StemConv2d(3, channels, 7, stride=2, padding=3, bias=False).to(_dev())
    conv = conv.to(memory_format=torch.channels_last)
    x = torch.randn(shape, device=_dev(), generator=g).contiguous(
        memory_format=torch.channels_last)
    with torch.autocast("cuda", dtype=dtype):
        assert conv._kernel_dtype(x) == dtype
        y = conv(x)
    assert y.dtype == dtype and y.is_contiguous(memory_format=torch.channels_last)
    xd, wd = x.to(dtype).double(), conv.weight.detach().to(dtype).double()
    want = F.conv2d(xd, wd, stride=2, padding=3)
    # 147 products of at most |x| |w| each in fp32, then one rounding
    size = F.conv2d(xd.abs(), wd.abs(), stride=2, padding=3)
    eps = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert bool(((y.double() - want).abs() <= eps * want.abs() + 2e-5 * size + 6e-8).all())
    dy = torch.randn(y.shape, device=_dev(), generator=g).to(dtype)
    y.backward(dy)
    dw = torch.nn.grad.conv2d_weight(xd, wd.shape, dy.double(), stride=2, padding=3)
    assert (conv.weight.grad.double() - dw).norm() <= 1e-2 * dw.norm()
    # fp32 without autocast is PyTorch's
    assert conv._kernel_dtype(x) is None


@pytest.mark.parametrize("shape,channels", [
    ((8, 3, 224, 224), 80), ((8, 3, 225, 223), 128), ((40, 3, 97, 131), 64),
])
def test_stem_convolution_many_tiles_per_cta(shape, channels):
    """Accumulators and buffers used again, at widths with one and with two
    gradient CTAs per SM; every element against 64 bits, weights in PyTorch's own
    memory format."""
    from horovod_b200 import _C
    g = torch.Generator(device=_dev()).manual_seed(17)
    x = torch.randn(shape, device=_dev(), generator=g).bfloat16().contiguous(
        memory_format=torch.channels_last)
    w = torch.randn(channels, 3, 7, 7, device=_dev(), generator=g).bfloat16()
    y = _C.stem_conv_forward(x, w)
    dy = torch.randn(y.shape, device=_dev(), generator=g).bfloat16().contiguous(
        memory_format=torch.channels_last)
    dw = _C.stem_conv_wgrad(x, dy, w)
    xd, wd, dyd = x.double(), w.double(), dy.double()

    def wgrad(a, b):
        return torch.nn.grad.conv2d_weight(a, w.shape, b, stride=2, padding=3)

    for got, want, size in (
            (y, F.conv2d(xd, wd, stride=2, padding=3),
             F.conv2d(xd.abs(), wd.abs(), stride=2, padding=3)),
            (dw, wgrad(xd, dyd), wgrad(xd.abs(), dyd.abs()))):
        # one rounding to bf16, and the products' fp32 sums
        bound = 2.0 ** -8 * want.abs() + 2e-5 * size
        assert bool(((got.double() - want).abs() <= bound).all())
    assert dw.stride() == w.stride()


@pytest.mark.parametrize("width", [20, 21])
def test_stem_convolution_in_a_16_bit_model(width):
    """Without autocast, with an input that needs a gradient, and with gradients
    of gradients, which are PyTorch's: next to an nn.Conv2d in 64 bits."""
    from horovod_b200.ops.stem_conv import StemConv2d
    g = torch.Generator(device=_dev()).manual_seed(18)
    conv = StemConv2d(3, 32, 7, stride=2, padding=3, bias=False).to(_dev()).half()
    ref = torch.nn.Conv2d(3, 32, 7, stride=2, padding=3, bias=False).to(_dev()).double()
    ref.load_state_dict(conv.state_dict())
    x = torch.randn(3, 3, 18, width, device=_dev(), generator=g).half().contiguous(
        memory_format=torch.channels_last)
    results = []
    for module, dtype in ((conv, torch.float16), (ref, torch.float64)):
        xi = x.to(dtype).requires_grad_(True)
        y = module(xi)
        gi = torch.Generator(device=_dev()).manual_seed(19)
        dy = torch.randn(y.shape, device=_dev(), generator=gi).half().to(dtype)
        dy.requires_grad_(True)
        plain = torch.autograd.grad(y, [xi, module.weight], dy, retain_graph=True)
        first = torch.autograd.grad(y, [xi, module.weight], dy, create_graph=True)
        second = torch.autograd.grad(sum((t * t).sum() for t in first) * 1e-3,
                                     [xi, module.weight, dy])
        results.append([y, *plain, *first, *second])
    assert conv._kernel_dtype(x) == torch.float16
    for got, want in zip(*results):
        # a few roundings to fp16 on the way: 2^-11 each
        assert (got.double() - want).norm() <= 2e-3 * want.norm()


def _kinds(t):
    """0 for finite values, 1 for NaN, 2 and 3 for the infinities."""
    return t.isnan() * 1 + t.isposinf() * 2 + t.isneginf() * 3


#: (row, column, channel) of what is not finite in a 67 x 45 image: even and odd
#: rows and columns, corners, both sides of a tile's edge (rows 31 / 32, columns
#: 15 / 16) and the last, partial tiles (from row 64 and column 32)
_SPECIAL_PIXELS = [(8, 8, 0), (9, 8, 1), (8, 9, 2), (9, 9, 0), (0, 0, 1), (66, 44, 2), (31, 15, 0),
                   (32, 16, 1), (31, 16, 2), (32, 15, 0), (65, 40, 1), (20, 43, 2), (64, 32, 0)]


def _special_images(dtype, value):
    """An image per special pixel, one with all of them and a finite one."""
    g = torch.Generator().manual_seed(10)
    x = torch.randn(len(_SPECIAL_PIXELS) + 2, 3, 67, 45, generator=g).to(dtype)
    for n, (r, c, ch) in enumerate(_SPECIAL_PIXELS):
        x[n, ch, r, c] = value
        x[-2, ch, r, c] = value
    return x.contiguous(memory_format=torch.channels_last)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("channels", [16, 64])
def test_stem_convolution_of_special_values(channels, value, dtype):
    """Infinities and NaN reach the outputs whose 7 x 7 window holds them, and
    no others."""
    from horovod_b200 import _C
    x = _special_images(dtype, value)
    w = torch.randn(channels, 3, 7, 7, generator=torch.Generator().manual_seed(11)).to(dtype)
    # five times over: more tiles than CTAs, so that both kinds follow each other
    many = torch.cat([x] * 5).contiguous(memory_format=torch.channels_last)
    y = _C.stem_conv_forward(many.to(_dev()), w.to(_dev())).cpu()
    assert all(torch.equal(y[:len(x)].view(torch.int16), part.view(torch.int16))
               for part in y.split(len(x)))
    y = y[:len(x)]
    want = F.conv2d(x.double(), w.double(), stride=2, padding=3)
    assert torch.equal(_kinds(y), _kinds(want)) and bool(want[:-1].isfinite().logical_not().any())
    finite = want.isfinite()
    # as above: 147 products in fp32, then one rounding
    size = F.conv2d(torch.nan_to_num(x.double().abs(), 0.0, 0.0, 0.0), w.double().abs(), stride=2,
                    padding=3)
    eps = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    bound = eps * want.abs() + 2e-5 * size + 6e-8
    assert bool(((y.double() - want).abs() <= bound)[finite].all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("channels", [16, 64])
def test_stem_gradient_of_special_values(channels, value, dtype):
    """Infinities and NaN reach the taps that some output pixel multiplies
    with them, also where a tile reaches past the output."""
    from horovod_b200 import _C
    images = _special_images(dtype, value)
    w = torch.zeros(channels, 3, 7, 7, dtype=dtype)
    g = torch.Generator().manual_seed(12)
    dy = torch.randn(len(images), channels, 34, 23, generator=g).to(dtype)
    # each image by itself, and many at once (more tiles than CTAs), of which
    # only one is not finite
    many = images[-1:].repeat(90, 1, 1, 1)
    many[-1] = images[5]
    more = torch.randn(len(many), channels, 34, 23, generator=g).to(dtype)
    for x, d in [(images[n:n + 1], dy[n:n + 1]) for n in range(len(images))] + [(many, more)]:
        x, d = (t.contiguous(memory_format=torch.channels_last) for t in (x, d))
        dw = _C.stem_conv_wgrad(x.to(_dev()), d.to(_dev()), w.to(_dev())).cpu()
        want = torch.nn.grad.conv2d_weight(x.double(), w.shape, d.double(), stride=2, padding=3)
        assert torch.equal(_kinds(dw), _kinds(want))
        # the sum of the products' sizes in fp32, then one rounding
        size = torch.nn.grad.conv2d_weight(torch.nan_to_num(x.double().abs(), 0.0, 0.0, 0.0),
                                           w.shape, d.double().abs(), stride=2, padding=3)
        eps = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
        bound = eps * want.abs() + 2e-5 * size + 6e-8
        assert bool(((dw.double() - want).abs() <= bound)[want.isfinite()].all())


def _fallback_conv(use):
    """Runs `use` under conditions in which a StemConv2d is PyTorch's."""
    from horovod_b200 import _C
    from horovod_b200.ops.stem_conv import StemConv2d
    conv = StemConv2d(3, 16, 7, stride=2, padding=3, bias=False).to(_dev()).bfloat16()
    x = torch.randn(2, 3, 20, 20, device=_dev()).bfloat16().contiguous(
        memory_format=torch.channels_last)
    assert conv._kernel_dtype(x) == torch.bfloat16
    with use():
        assert conv._kernel_dtype(x) is None
        before = _C.kernel_launch_count()
        y = conv(x)
        y.sum().backward()
        assert _C.kernel_launch_count() == before
        assert torch.equal(y, F.conv2d(x, conv.weight, stride=2, padding=3))
    assert conv._kernel_dtype(x) == torch.bfloat16


def test_stem_convolution_left_to_pytorch():
    """Dispatch modes and tensor subclasses see PyTorch's convolution, as with an
    nn.Conv2d; a weight with gaps is taken by the kernels."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from torch.utils.flop_counter import FlopCounterMode
    from horovod_b200.ops.stem_conv import StemConv2d
    _fallback_conv(lambda: FlopCounterMode(display=False))

    class Quiet(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))
    _fallback_conv(Quiet)

    class Subclass(torch.Tensor):
        pass
    conv = StemConv2d(3, 16, 7, stride=2, padding=3, bias=False).to(_dev()).bfloat16()
    x = torch.randn(2, 3, 20, 20, device=_dev()).bfloat16().contiguous(
        memory_format=torch.channels_last)
    assert conv._kernel_dtype(x.as_subclass(Subclass)) is None
    assert isinstance(conv(x.as_subclass(Subclass)), Subclass)

    wide = torch.randn(16, 3, 7, 14, device=_dev()).bfloat16()
    gaps = wide[..., ::2].detach().requires_grad_(True)
    dense = gaps.detach().clone(memory_format=torch.contiguous_format).requires_grad_(True)
    grads = []
    for w in (gaps, dense):
        conv.weight = torch.nn.Parameter(w.detach())
        assert conv._kernel_dtype(x) == torch.bfloat16
        y = conv(x)
        y.backward(torch.ones_like(y))
        grads.append((y, conv.weight.grad))
    assert not gaps.is_contiguous()
    assert torch.equal(grads[0][0], grads[1][0]) and torch.equal(grads[0][1], grads[1][1])


def test_stem_convolution_switch(monkeypatch):
    import contextlib

    @contextlib.contextmanager
    def off():
        with monkeypatch.context() as m:
            m.setenv("HOROVOD_B200_FUSED_STEM", "0")
            yield
    _fallback_conv(off)


@pytest.mark.parametrize("channels", [16, 128])
def test_stem_convolution_whose_waits_run_out(channels):
    """A limit of 0 makes every wait run out (the kernels then wait for their
    products in flight all the same): results are NaN, the device is marked, and
    the module goes on with PyTorch's convolution."""
    import contextlib
    from horovod_b200 import _C
    x = torch.randn(90, 3, 67, 45, device=_dev()).bfloat16().contiguous(
        memory_format=torch.channels_last)
    w = torch.randn(channels, 3, 7, 7, device=_dev()).bfloat16()
    dy = torch.randn(90, channels, 34, 23, device=_dev()).bfloat16().contiguous(
        memory_format=torch.channels_last)
    y, dw = _C.stem_conv_forward(x, w), _C.stem_conv_wgrad(x, dy, w)
    assert not _C.stem_conv_failed(0)
    try:
        assert bool(_C.stem_conv_forward(x, w, wait_ns=0).isnan().all())
        assert _C.stem_conv_failed(0) and _C.stem_conv_failed(0, clear=True)
        assert not _C.stem_conv_failed(0)
        assert bool(_C.stem_conv_wgrad(x, dy, w, wait_ns=0).isnan().all())
        assert _C.stem_conv_failed(0, clear=True)

        @contextlib.contextmanager
        def failed():
            _C.stem_conv_forward(x, w, wait_ns=0)
            torch.cuda.synchronize()
            with pytest.warns(UserWarning, match="ran out"):
                yield
            _C.stem_conv_failed(0, clear=True)
        _fallback_conv(failed)
    finally:
        torch.cuda.synchronize()
        _C.stem_conv_failed(0, clear=True)
    # nothing is left behind
    assert torch.equal(_C.stem_conv_forward(x, w), y)
    assert torch.equal(_C.stem_conv_wgrad(x, dy, w), dw)


@pytest.mark.parametrize("offset", [1, 2, 4, 7])
def test_activations_off_a_16_byte_boundary(offset):
    """Slices of flat buffers as inputs and as gradients: the same results as
    from tensors of their own."""
    from horovod_b200.ops.batch_norm import batch_norm_act
    from horovod_b200.ops.pooling import max_pool_3x3_s2
    from horovod_b200.ops.stem_conv import StemConv2d
    g = torch.Generator(device=_dev()).manual_seed(13)

    def pair(n, c, h, w):
        """The same values at an offset and on a boundary."""
        flat = torch.randn(n * c * h * w + offset, device=_dev(), generator=g).bfloat16()
        view = flat[offset:].view(n, h, w, c).permute(0, 3, 1, 2)
        assert view.data_ptr() % 16 == 2 * offset
        return view, view.clone(memory_format=torch.channels_last)

    conv = StemConv2d(3, 16, 7, stride=2, padding=3, bias=False).to(_dev()).bfloat16()
    cases = [
        (lambda x: batch_norm_act(x, None, None, None, None), [pair(3, 16, 9, 7)]),
        (lambda x, r: batch_norm_act(x, None, None, None, None, residual=r),
         [pair(3, 16, 9, 7), pair(3, 16, 9, 7)]),
        (max_pool_3x3_s2, [pair(3, 16, 9, 7)]),
        (conv, [pair(3, 3, 18, 20)]), (conv, [pair(3, 3, 17, 19)]),
    ]
    for fn, inputs in cases:
        dy, results = None, []
        for which in (0, 1):
            leaves = [p[which].detach().requires_grad_(fn is not conv) for p in inputs]
            conv.weight.grad = None
            y = fn(*leaves)
            dy = dy or pair(*y.shape)
            y.backward(dy[which])
            results.append([y] + ([conv.weight.grad] if fn is conv else [t.grad for t in leaves]))
        for a, b in zip(*results):
            assert torch.equal(a, b)


def test_model_kernels_in_a_replayed_graph():
    """Stem convolution, batch norm, pooling and a batch norm with a residual,
    forward and backward, captured twice (on one stream, as graphs are) and
    replayed on new inputs, with other calls in between: as without a graph."""
    import copy
    from horovod_b200.ops import BatchNormAct2d
    from horovod_b200.ops.pooling import MaxPool3x3s2
    from horovod_b200.ops.stem_conv import StemConv2d
    torch.manual_seed(16)

    class Net(torch.nn.Module):
        def __init__(self):
            super().__init__()
            self.conv = StemConv2d(3, 16, 7, stride=2, padding=3, bias=False)
            self.bn1, self.bn2 = BatchNormAct2d(16, relu=True), BatchNormAct2d(16, relu=True)
            self.pool = MaxPool3x3s2()

        def forward(self, x):
            with torch.autocast("cuda", dtype=torch.bfloat16):
                y = self.pool(self.bn1(self.conv(x)))
                return self.bn2(y, y)

    def step(net, x, dy):
        for p in net.parameters():
            p.grad = None
        y = net(x)
        y.backward(dy)
        return [y.detach()] + [p.grad for p in net.parameters()]

    net = Net().to(_dev()).to(memory_format=torch.channels_last)
    twin = copy.deepcopy(net)
    x = torch.randn(9, 3, 61, 47, device=_dev()).contiguous(memory_format=torch.channels_last)
    dy = torch.randn(9, 16, 16, 12, device=_dev()).bfloat16().contiguous(
        memory_format=torch.channels_last)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(net, x, dy)
        step(twin, x, dy)
    torch.cuda.current_stream().wait_stream(side)
    graphs = [torch.cuda.CUDAGraph(), torch.cuda.CUDAGraph()]
    results = []
    for graph in graphs:
        with torch.cuda.graph(graph):
            results.append(step(net, x, dy))
    for which in (0, 1, 1, 0, 1):
        x.copy_(torch.randn_like(x))
        graphs[which].replay()
        captured = results[which]
        for got, want in zip(captured, step(twin, x, dy)):
            # the sums over CTAs come in any order: 16-bit values may round elsewhere
            assert (got.double() - want.double()).norm() <= 1e-3 * want.double().norm()
        for got, want in zip(net.buffers(), twin.buffers()):
            torch.testing.assert_close(got, want)


@pytest.mark.parametrize("momentum", [0.1, None])
def test_batch_norm_counts_batches_once(momentum):
    from horovod_b200.ops.batch_norm import BatchNormAct2d
    bn = BatchNormAct2d(16, momentum=momentum).to(_dev())
    x = torch.randn(2, 16, 5, 5, device=_dev()).contiguous(memory_format=torch.channels_last)
    for i, t in enumerate((x.bfloat16(), x, x.half())):  # the kernel, PyTorch, the kernel
        bn(t)
        assert int(bn.num_batches_tracked) == i + 1
    bn.eval()
    bn(x.bfloat16())
    assert int(bn.num_batches_tracked) == 3
