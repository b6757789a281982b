"""The work whose speed this repository keeps track of on one GPU: what a user's
program has the library do, through its public entry points.

``listed()`` names the cases of record, ``draw()`` gives more of the same
ranges. A case is a dict of plain values whose ``kind`` says which path it is:

  train          a whole training step of a ResNet (forward, backward,
                 hvd.DistributedOptimizer over hvd.FusedSGD) under bf16 autocast
  bn             hvd's BatchNormAct2d in training mode, forward and backward
  pool           the 3x3 / stride 2 max pooling of the ResNet stem, forward and
                 backward
  sgd            the optimizer step alone, over the tensors of a ResNet
  allreduce      one blocking hvd.allreduce of a small tensor
  grouped        hvd.grouped_allreduce of the gradients of transformer blocks,
                 with or without 16-bit compression
  reducescatter, allgather, alltoall
                 one blocking call on one large tensor

Everything runs in one process, which is a job of one rank.
"""
import math

import torch
import torch.nn.functional as F

import horovod_b200.torch as hvd
from horovod_b200.models.resnet import ResNet
from horovod_b200.models.transformer import Block
from horovod_b200.ops.batch_norm import BatchNormAct2d
from horovod_b200.ops.pooling import MaxPool3x3s2
from horovod_b200.torch.fused_sgd import FusedSGD

DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16,
          "int64": torch.int64}
COMPRESSION = {"none": hvd.Compression.none, "fp16": hvd.Compression.fp16,
               "bf16": hvd.Compression.bf16}
#: Depths of the ResNet family by number of bottleneck blocks per stage.
DEPTHS = {14: (1, 1, 1, 1), 26: (2, 2, 2, 2), 50: (3, 4, 6, 3), 101: (3, 4, 23, 3)}
MOST_BN_ELEMENTS = 256 * 256 * 56 * 56


def listed():
    return [
        # The synthetic benchmark: ResNet-50, 256 images of 224 x 224 per GPU.
        {"name": "train_b256", "kind": "train", "batch": 256, "image": 224},
        # The same script at its default batch of 32 images: the GPU's work per
        # step is short and the host's matters.
        {"name": "train_b32", "kind": "train", "batch": 32, "image": 224},
        # Last batch norm of a first-stage block at batch 256: the largest
        # activation of ResNet-50, with the skip connection and the ReLU.
        {"name": "bn_residual_stage1", "kind": "bn", "batch": 256, "channels": 256, "h": 56,
         "w": 56, "dtype": "bf16", "residual": True, "relu": True},
        # The batch norm that occurs most often: inside a third-stage block.
        {"name": "bn_relu_stage3", "kind": "bn", "batch": 256, "channels": 256, "h": 14,
         "w": 14, "dtype": "bf16", "residual": False, "relu": True},
        # A last-stage batch norm at a small batch, in fp16.
        {"name": "bn_residual_small", "kind": "bn", "batch": 13, "channels": 512, "h": 7, "w": 7,
         "dtype": "fp16", "residual": True, "relu": True},
        # The stem's pooling at batch 256.
        {"name": "pool_stem", "kind": "pool", "batch": 256, "channels": 64, "h": 112, "w": 112,
         "dtype": "bf16"},
        # The optimizer step of ResNet-50: 161 tensors, 25.6 M parameters.
        {"name": "sgd_resnet50", "kind": "sgd", "depth": 50, "width": 64, "nesterov": False,
         "weight_decay": 1e-4},
        # Averaging a metric over the ranks: one number.
        {"name": "allreduce_metric", "kind": "allreduce", "count": 1, "dtype": "fp32"},
        # The gradients of four BERT-large blocks sent as fp16.
        {"name": "grouped_fp16_4_blocks", "kind": "grouped", "blocks": 4, "d_model": 1024,
         "d_ff": 4096, "compression": "fp16"},
        # Sharding one flat gradient of ResNet-50's size.
        {"name": "reducescatter_flat", "kind": "reducescatter", "rows": 25557032, "width": 1,
         "dtype": "fp32"},
        # Collecting the outputs of an evaluation whose last batch is ragged.
        {"name": "allgather_outputs", "kind": "allgather", "rows": 16377, "width": 1024,
         "dtype": "bf16"},
        # Sending embedding rows to the ranks that own them.
        {"name": "alltoall_embeddings", "kind": "alltoall", "rows": 65536, "width": 128,
         "dtype": "fp32"},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["train", "bn", "bn", "pool", "sgd", "allreduce", "grouped",
                       "reducescatter", "allgather", "alltoall"])
    if kind == "train":
        image = rng.randint(96, 256)
        most = min(256, 256 * 224 * 224 // (image * image))
        return {"kind": kind, "batch": _log(rng, 4, most), "image": image}
    if kind == "bn":
        channels = 2 ** rng.randint(4, 11)
        h = _log(rng, 4, 112)
        w = max(4, min(112, h + rng.randint(-3, 3)))
        most = max(1, min(256, MOST_BN_ELEMENTS // (channels * h * w)))
        residual = rng.random() < 0.4
        return {"kind": kind, "batch": _log(rng, 1, most), "channels": channels, "h": h, "w": w,
                "dtype": rng.choice(["bf16", "bf16", "fp16"]), "residual": residual,
                "relu": residual or rng.random() < 0.8}
    if kind == "pool":
        h = _log(rng, 16, 128)
        return {"kind": kind, "batch": _log(rng, 1, 200), "channels": 8 * rng.randint(4, 12),
                "h": h, "w": max(16, h + rng.randint(-5, 5)),
                "dtype": rng.choice(["bf16", "bf16", "fp16"])}
    if kind == "sgd":
        return {"kind": kind, "depth": rng.choice(sorted(DEPTHS)), "width": rng.randint(8, 96),
                "nesterov": rng.random() < 0.3, "weight_decay": rng.choice([0.0, 1e-4, 5e-5])}
    if kind == "allreduce":
        return {"kind": kind, "count": _log(rng, 1, 1 << 20),
                "dtype": rng.choice(["fp32", "fp32", "bf16", "fp16", "int64"])}
    if kind == "grouped":
        d_model = 64 * rng.randint(2, 16)
        return {"kind": kind, "blocks": rng.randint(1, 4), "d_model": d_model,
                "d_ff": 4 * d_model + rng.choice([0, 0, 2, 7]),
                "compression": rng.choice(["none", "fp16", "fp16", "bf16"])}
    width = rng.choice([1, 3, 64, 127, 128, 768, 1000, 1024])
    return {"kind": kind, "rows": max(1, _log(rng, 1 << 10, 1 << 25) // width), "width": width,
            "dtype": rng.choice(["fp32", "fp32", "bf16", "fp16"])}


# ---- inputs -------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _flat_views(shapes, device="cuda"):
    """One flat fp32 buffer and a tensor for every (shape, stride), each on a
    512-byte boundary as the caching allocator would place it."""
    offsets, total = [], 0
    for shape, _ in shapes:
        offsets.append(total)
        total += (math.prod(shape) + 127) // 128 * 128
    flat = torch.zeros(total, device=device)
    return flat, [torch.as_strided(flat, shape, stride, off)
                  for (shape, stride), off in zip(shapes, offsets)]


def _resnet(depth, width, device):
    with torch.device(device):
        return ResNet(DEPTHS[depth], width=width)


def _lay_out(params):
    """Puts the parameters into one flat buffer so that a step can hand back all
    of them as one tensor."""
    flat, views = _flat_views([(tuple(p.shape), p.stride()) for p in params])
    for p, v in zip(params, views):
        v.copy_(p.data)
        p.data = v
    return flat


def _momentum(optimizer, params):
    """Momentum buffers as a program that resumes from a checkpoint has them."""
    flat, views = _flat_views([(tuple(p.shape), p.stride()) for p in params])
    for p, v in zip(params, views):
        optimizer.state[p]["momentum_buffer"] = v
    return flat


def _prepare_train(case, seed):
    torch.manual_seed(seed)
    model = _resnet(50, 64, "cuda").to(memory_format=torch.channels_last)
    params = list(model.parameters())
    weights = _lay_out(params)
    optimizer = hvd.DistributedOptimizer(
        FusedSGD(params, lr=0.01, momentum=0.9, weight_decay=1e-4),
        named_parameters=model.named_parameters())
    _momentum(optimizer, params)
    hvd.broadcast_parameters(model.state_dict(), root_rank=0)
    g = _generator(seed)
    x = torch.randn(case["batch"], 3, case["image"], case["image"], device="cuda", generator=g)
    y = torch.randint(0, 1000, (case["batch"],), device="cuda", generator=g)
    return {"model": model, "optimizer": optimizer, "weights": weights,
            "x": x.contiguous(memory_format=torch.channels_last), "y": y}


def _run_train(s):
    s["optimizer"].zero_grad()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = F.cross_entropy(s["model"](s["x"]), s["y"])
    loss.backward()
    s["optimizer"].step()
    return s["weights"]


def _activation(case, g):
    return torch.randn(case["batch"], case["h"], case["w"], case["channels"], device="cuda",
                       dtype=DTYPES[case["dtype"]], generator=g).permute(0, 3, 1, 2)


def _prepare_bn(case, seed):
    g = _generator(seed)
    c = case["channels"]
    bn = BatchNormAct2d(c, relu=case["relu"]).cuda()
    with torch.no_grad():  # a layer in the middle of training
        bn.weight.copy_(0.5 + torch.rand(c, device="cuda", generator=g))
        bn.bias.copy_(0.1 * torch.randn(c, device="cuda", generator=g))
    x = _activation(case, g)
    # Channels with means and spreads of their own, as a convolution gives them.
    spread = (0.25 + torch.rand(c, device="cuda", generator=g)).to(x.dtype)
    mean = (0.5 * torch.randn(c, device="cuda", generator=g)).to(x.dtype)
    x.mul_(spread.view(1, c, 1, 1)).add_(mean.view(1, c, 1, 1))
    x.requires_grad_(True)
    residual = _activation(case, g).relu_().requires_grad_(True) if case["residual"] else None
    return {"bn": bn, "x": x, "residual": residual, "dy": _activation(case, g).mul_(0.01)}


def _run_bn(s):
    bn, x, residual = s["bn"], s["x"], s["residual"]
    y = bn(x, residual)
    wanted = [x, bn.weight, bn.bias] + ([residual] if residual is not None else [])
    grads = torch.autograd.grad(y, wanted, s["dy"])
    return [y.detach(), bn.running_mean, bn.running_var, *grads]


def _prepare_pool(case, seed):
    g = _generator(seed)
    x = _activation(case, g).relu_().requires_grad_(True)
    h, w = (case["h"] + 1) // 2, (case["w"] + 1) // 2
    return {"pool": MaxPool3x3s2(), "x": x, "dy": _activation({**case, "h": h, "w": w}, g)}


def _run_pool(s):
    y = s["pool"](s["x"])
    return y.detach(), torch.autograd.grad(y, s["x"], s["dy"])[0]


def _prepare_sgd(case, seed):
    g = _generator(seed)
    model = _resnet(case["depth"], case["width"], "meta").to(memory_format=torch.channels_last)
    shapes = [(tuple(p.shape), p.stride()) for p in model.parameters()]
    weights, views = _flat_views(shapes)
    weights.normal_(std=0.05, generator=g)
    params = [torch.nn.Parameter(v) for v in views]
    flat, grads = _flat_views(shapes)
    flat.normal_(std=0.01, generator=g)
    for p, v in zip(params, grads):
        p.grad = v
    optimizer = hvd.DistributedOptimizer(
        FusedSGD(params, lr=0.01, momentum=0.9, weight_decay=case["weight_decay"],
                 nesterov=case["nesterov"]))
    momentum = _momentum(optimizer, params)
    momentum.normal_(std=0.05, generator=g)
    return {"optimizer": optimizer, "weights": weights, "momentum": momentum}


def _run_sgd(s):
    s["optimizer"].step()
    return s["weights"], s["momentum"]


def _values(shape, dtype, g):
    if dtype == torch.int64:
        return torch.randint(-1000, 1000, shape, device="cuda", generator=g)
    return torch.randn(shape, device="cuda", dtype=dtype, generator=g)


def _prepare_one_tensor(case, seed):
    shape = (case["count"],) if case["kind"] == "allreduce" else \
        (case["rows"],) if case["width"] == 1 else (case["rows"], case["width"])
    return {"x": _values(shape, DTYPES[case["dtype"]], _generator(seed))}


def _run_allreduce(s):
    # Means of floating-point metrics, sums of counts.
    op = hvd.Average if s["x"].is_floating_point() else hvd.Sum
    return hvd.allreduce(s["x"], name="metric", op=op)


def _prepare_grouped(case, seed):
    g = _generator(seed)
    with torch.device("meta"):
        block = Block(case["d_model"], 1, case["d_ff"], causal=False, pre_norm=False)
    shapes = [tuple(p.shape) for p in block.parameters()] * case["blocks"]
    return {"x": [_values(shape, torch.float32, g) for shape in shapes],
            "compression": COMPRESSION[case["compression"]]}


def _run_grouped(s):
    return hvd.grouped_allreduce(s["x"], name="gradients", compression=s["compression"])


def _run_reducescatter(s):
    return hvd.reducescatter(s["x"], name="shard")


def _run_allgather(s):
    return hvd.allgather(s["x"], name="outputs")


def _run_alltoall(s):
    return hvd.alltoall(s["x"], splits=[s["x"].size(0)], name="rows")


PREPARE = {"train": _prepare_train, "bn": _prepare_bn, "pool": _prepare_pool, "sgd": _prepare_sgd,
           "grouped": _prepare_grouped}
RUN = {"train": _run_train, "bn": _run_bn, "pool": _run_pool, "sgd": _run_sgd,
       "allreduce": _run_allreduce, "grouped": _run_grouped, "reducescatter": _run_reducescatter,
       "allgather": _run_allgather, "alltoall": _run_alltoall}


def prepare(case, seed):
    if not hvd.is_initialized():
        hvd.init()
        torch.cuda.set_device(hvd.local_rank())
    return {"kind": case["kind"],
            **PREPARE.get(case["kind"], _prepare_one_tensor)(case, seed)}


def run(state):
    return RUN[state["kind"]](state)


# ---- what a pass cannot do without ---------------------------------------------

def _parameters(depth, width):
    return sum(p.numel() for p in _resnet(depth, width, "meta").parameters())


def work(case):
    """Bytes: each input read once, each output written once."""
    kind = case["kind"]
    if kind == "train":
        # 4.09 G multiply-adds per 224 x 224 image in forward, twice that in
        # backward; images, weights, gradients and momentum.
        flops = 3 * 2 * 4.09e9 * case["batch"] * (case["image"] / 224.0) ** 2
        return {"bytes": case["batch"] * case["image"] ** 2 * 12.0 + 5 * 4 * _parameters(50, 64),
                "flops": flops}
    if kind == "bn":
        n = case["batch"] * case["channels"] * case["h"] * case["w"]
        # x, dy (and the residual) in; y, dx (and the residual's gradient) out
        return {"bytes": n * 2.0 * (6 if case["residual"] else 4), "flops": 20.0 * n}
    if kind == "pool":
        n = case["batch"] * case["channels"]
        small = ((case["h"] + 1) // 2) * ((case["w"] + 1) // 2)
        return {"bytes": n * 2.0 * (2 * case["h"] * case["w"] + 2 * small), "flops": 9.0 * n * small}
    if kind == "sgd":
        n = _parameters(case["depth"], case["width"])
        return {"bytes": 5 * 4.0 * n, "flops": 6.0 * n}
    if kind == "grouped":
        d, f = case["d_model"], case["d_ff"]
        n = case["blocks"] * (4 * d * d + 2 * d * f + 9 * d + f)
        return {"bytes": 2 * 4.0 * n, "flops": 0}
    n = case["count"] if kind == "allreduce" else case["rows"] * case["width"]
    return {"bytes": 2.0 * n * torch.empty((), dtype=DTYPES[case["dtype"]]).element_size(),
            "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "train":
        # Of the weights. Against a step whose batch norms round elsewhere (the
        # PyTorch composition) they differ by 6e-5 / sqrt(batch) after two
        # steps, at most by 1.4e-2 / sqrt(batch) of their root mean square; one
        # step moves them by 8e-4 / sqrt(batch).
        root = math.sqrt(case["batch"])
        return {"rel": 2.5e-4 / root, "max": 6e-2 / root}
    if kind == "bn":
        # Rounding of the results; the sums behind them are wider. A value that
        # is zero but for its rounding may pass the ReLU or not, and takes its
        # gradient with it: 0.94 of the root mean square was the largest
        # difference from a computation in 64 bits.
        return {"rel": 7e-3 if case["dtype"] == "bf16" else 9e-4, "max": 0.99}
    if kind == "sgd":
        return {"rel": 3e-7}
    return "exact"  # one rank: data movement and casts


# ---- what a pass returns, in 64 bits ---------------------------------------------

def _exact_bn(s):
    bn, x, residual = s["bn"], s["x"], s["residual"]
    n = x.numel() // x.size(1)

    def column(v):
        return v.view(1, -1, 1, 1)

    with torch.no_grad():
        xhat = x.double()
        var, mean = torch.var_mean(xhat, (0, 2, 3), unbiased=False)
        xhat.sub_(column(mean)).mul_(column(torch.rsqrt(var + bn.eps)))
        weight, bias = bn.weight.double(), bn.bias.double()
        y = (xhat * column(weight)).add_(column(bias))
        if residual is not None:
            y.add_(residual)
        dz = s["dy"].double()
        if bn.relu:
            y.relu_()
            dz.mul_(y > 0)
        db, dw = dz.sum((0, 2, 3)), (dz * xhat).sum((0, 2, 3))
        dx = xhat.mul_(column(-dw / n)).add_(dz).sub_(column(db / n))
        dx.mul_(column(weight * torch.rsqrt(var + bn.eps)))
        keep = 1.0 - bn.momentum
        unbiased = var * (n / max(n - 1, 1))
        running = [bn.running_mean.double() * keep + mean * bn.momentum,
                   bn.running_var.double() * keep + unbiased * bn.momentum]
        return [y, *running, dx, dw, db] + ([dz] if residual is not None else [])


def _exact_pool(s):
    x = s["x"].detach().double().requires_grad_(True)
    y = F.max_pool2d(x, 3, stride=2, padding=1)
    return y.detach(), torch.autograd.grad(y, x, s["dy"].double())[0]


def _exact_sgd(case, s):
    optimizer = s["optimizer"]
    weights, momentum = s["weights"].double(), s["momentum"].double()
    for p in optimizer.param_groups[0]["params"]:
        m = optimizer.state[p]["momentum_buffer"]
        w64 = torch.as_strided(weights, p.shape, p.stride(), p.storage_offset())
        m64 = torch.as_strided(momentum, m.shape, m.stride(), m.storage_offset())
        g = p.grad.double() + case["weight_decay"] * w64
        m64.mul_(0.9).add_(g)
        w64.sub_(0.01 * (g + 0.9 * m64 if case["nesterov"] else m64))
    return weights.detach(), momentum


def exact(case, seed):
    """What ``run`` returns for these inputs, computed by PyTorch in 64 bits. A
    training step of the whole model has no such value here."""
    kind = case["kind"]
    if kind == "train":
        return None
    s = prepare(case, seed)
    if kind == "bn":
        return _exact_bn(s)
    if kind == "pool":
        return _exact_pool(s)
    if kind == "sgd":
        with torch.no_grad():
            return _exact_sgd(case, s)
    if kind == "grouped":  # the cast is part of what was asked for
        sent = {"none": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}
        return [x.to(sent[case["compression"]]).float() for x in s["x"]]
    return s["x"].clone()  # one rank
