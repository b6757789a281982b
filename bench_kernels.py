"""Single-GPU micro-benchmark of the library's local kernels, reported against
the measured HBM copy bandwidth (MEASURED_PEAKS.json: hbm_gbs).

    python bench_kernels.py                 # all cases
    python bench_kernels.py --case fused_local --mb 512 --iters 3   # small ncu target

Cases
  fused_local   the fused multi-tensor allreduce kernel on one rank (LOCAL
                variant): reads 161 ResNet-50-shaped gradient tensors, scales
                and writes them back in one launch (read + write = 2x bytes).
  fused_fp16    same with float16 tensors.
  reducescatter reduce-scatter of one rank: one pass of the fused allreduce
                kernel's LOCAL variant (read + write = 2x bytes).
  exchange      allgather of one rank through the exchange kernel: with nobody
                to send to it is one copy into the output (2x bytes).
  batch_norm    fused batch norm + residual + ReLU on a channels-last bf16
                activation of 256 x 256 x 56 x 56 (411 MB): forward (statistics
                pass + apply pass: read x twice, read the residual, write y and
                a bit per element = 4.0625x bytes) and backward (reduce pass
                reads dy, x and the bits; apply pass reads them again and writes
                dx and dres = 6.125x bytes), timed with CUDA events on the current
                stream, next to the PyTorch eager composition batch_norm -> add ->
                relu on the same tensors, which moves other bytes.
  stem_conv     7x7 / stride 2 / padding 3 convolution of 256 images of 224 x 224
                x 3 to 64 channels in bf16: forward reads x and writes y (488 MB),
                the weights' gradient reads x and dy. Next to PyTorch's.
  conv1x1       1x1 convolutions of ResNet-50's first and third stage (256 images of
                56 x 56 and 14 x 14) in bf16: forward, which reads x and writes y
                and the sums of a batch norm (the call clears them too), and the
                gradient of the input, which reads dy, the skip connection's
                gradient and a bit per element of it and writes dx.
  norm_conv     backward of a batch norm over 256 channels and of the 1x1
                convolution from 64 before it, 256 images of 56 x 56: the sums
                read dy, x and a bit per element; the fused kernel reads them
                again, and a, and writes da. Next to the same as kernels of
                their own (bn_backward, then PyTorch's convolution_backward).
  residual_block
                forward and backward of the first block of ResNet-50's first two
                stages, 256 images of 56 x 56 in bf16, as one node and (which moves
                other bytes) layer by layer. No bytes are given: PyTorch's 3x3
                convolutions and weight gradients are among it.
  max_pool      3x3 / stride 2 / padding 1 max pooling on the ResNet stem
                activation 256 x 64 x 112 x 112 bf16 (411 MB): forward reads x,
                writes y (1/4 of x) and half an index byte per output element
                (1/16 of x): 1.3125x; backward reads dy and the indices and
                writes dx: 1.3125x. Next to PyTorch's max_pool2d.
  fused_sgd     hvd.FusedSGD step (momentum + weight decay) over 161
                ResNet-50-shaped fp32 tensors: reads p, g, m, writes p, m
                (5x bytes). Next to torch.optim.SGD on the same tensors.

Timing is device time of the response on the communication stream (CUDA
events around the launches). Inputs are larger than L2 (126 MB) unless --mb
says otherwise. Prints one JSON line per case.
"""
import argparse
import json
import os
import statistics
import sys
import time

os.environ["HOROVOD_GPU_OP_TIMING"] = "1"
os.environ.setdefault("HOROVOD_FUSION_THRESHOLD", str(1 << 30))


def resnet50_like_sizes(total_elems):
    """161 tensor sizes with ResNet-50's skew (a few large convolutions, many
    tiny batch-norm vectors), scaled to about total_elems."""
    base = []
    for planes, blocks in ((64, 3), (128, 4), (256, 6), (512, 3)):
        for b in range(blocks):
            inp = planes * 4 if b else max(64, planes * 2)
            base += [inp * planes, planes, planes, planes * planes * 9, planes, planes,
                     planes * planes * 4, planes * 4, planes * 4]
            if b == 0:
                base += [inp * planes * 4, planes * 4, planes * 4]
    base += [64 * 3 * 49, 64, 64, 2048 * 1000, 1000]
    base = base[:161]
    scale = total_elems / float(sum(base))
    return [max(1, int(s * scale)) for s in base]


def main():
    p = argparse.ArgumentParser()
    p.add_argument("--case", default="all")
    p.add_argument("--mb", type=int, default=512, help="payload per case in MB")
    p.add_argument("--iters", type=int, default=10)
    p.add_argument("--warmup", type=int, default=3)
    args = p.parse_args()

    import torch
    import horovod_b200.torch as hvd
    from horovod_b200 import _C

    peaks = {}
    try:
        peaks = json.load(open(os.path.join(os.path.dirname(os.path.abspath(__file__)),
                                            "MEASURED_PEAKS.json")))
    except OSError:
        pass
    hbm = float(peaks.get("hbm_gbs", 6650.0))
    peak_src = "measured" if peaks else "fallback"

    hvd.init()
    torch.cuda.set_device(0)
    dev = torch.device("cuda", 0)
    nbytes = args.mb << 20

    from horovod_b200.utils.clocks import ClockLog
    clock_log = ClockLog(0)

    def run(name, fn, want_type, algorithmic_bytes):
        for _ in range(args.warmup):
            fn()
        torch.cuda.synchronize()
        _C.gpu_op_stats()
        t_begin = time.time()
        for _ in range(args.iters):
            fn()
        torch.cuda.synchronize()
        t_end = time.time()
        us = [t[3] for t in _C.gpu_op_stats() if t[0] == want_type][-args.iters:]
        med = statistics.median(us)
        gbs = algorithmic_bytes / (med * 1e-6) / 1e9
        print(json.dumps({"case": name, "payload_mb": args.mb, "device_us": round(med, 1),
                          "algorithmic_gbs": round(gbs, 1),
                          "frac_of_%s_hbm_copy" % peak_src: round(gbs / hbm, 3),
                          "hbm_gbs_peak": hbm,
                          "clocks": clock_log.window(t_begin, t_end)}), flush=True)

    cases = ["fused_local", "fused_fp16", "reducescatter", "exchange", "batch_norm", "stem_conv",
             "conv1x1", "norm_conv", "residual_block", "max_pool",
             "fused_sgd"] if args.case == "all" else [args.case]

    def timed_events(fn, reps):
        for _ in range(args.warmup):
            fn()
        torch.cuda.synchronize()
        ts = []
        for _ in range(reps):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            fn()
            e1.record()
            torch.cuda.synchronize()
            ts.append(e0.elapsed_time(e1) * 1e3)
        return statistics.median(ts)

    def report_line(name, us, algorithmic, extra=None):
        # (algorithmic is None for a path that moves other bytes.)
        rate = {}
        if algorithmic is not None:
            gbs = algorithmic / (us * 1e-6) / 1e9
            rate = {"algorithmic_gbs": round(gbs, 1),
                    "frac_of_%s_hbm_copy" % peak_src: round(gbs / hbm, 3), "hbm_gbs_peak": hbm}
        print(json.dumps({"case": name, "device_us": round(us, 1), **rate,
                          "clocks": clock_log.window(time.time() - 1.0, time.time()),
                          **(extra or {})}), flush=True)
    if "fused_local" in cases:
        xs = [torch.randn(n, device=dev) for n in resnet50_like_sizes(nbytes // 4)]
        total = sum(x.numel() * 4 for x in xs)
        run("fused_local", lambda: hvd.grouped_allreduce_(xs, op=hvd.Sum, postscale_factor=0.5,
                                                          name="k.fused"), 0, 2 * total)
    if "fused_fp16" in cases:
        xs = [torch.randn(n, device=dev).half() for n in resnet50_like_sizes(nbytes // 2)]
        total = sum(x.numel() * 2 for x in xs)
        run("fused_fp16", lambda: hvd.grouped_allreduce_(xs, op=hvd.Sum, postscale_factor=0.5,
                                                         name="k.fused16"), 0, 2 * total)
    if "reducescatter" in cases:
        n = min(nbytes, 448 << 20) // 4
        x = torch.randn(n, device=dev)
        run("reducescatter", lambda: hvd.reducescatter(x, op=hvd.Sum, name="k.rs"), 6, 2 * n * 4)
    if "exchange" in cases:
        n = min(nbytes, 192 << 20) // 4
        x = torch.randn(n, device=dev)
        run("exchange", lambda: hvd.allgather(x, name="k.ag"), 1, 2 * n * 4)
    if "batch_norm" in cases:
        import torch.nn.functional as F
        from horovod_b200.ops.batch_norm import batch_norm_act
        n = 256 if args.mb >= 512 else 64
        shape = (n, 256, 56, 56)
        x = torch.randn(shape, device=dev, dtype=torch.bfloat16) \
            .contiguous(memory_format=torch.channels_last).requires_grad_(True)
        res = torch.randn_like(x).requires_grad_(True)
        go = torch.randn_like(x)
        w = torch.ones(256, device=dev, requires_grad=True)
        b = torch.zeros(256, device=dev, requires_grad=True)
        rm, rv = torch.zeros(256, device=dev), torch.ones(256, device=dev)
        nbytes_act = x.numel() * 2

        def eager_fwd():
            return F.relu(F.batch_norm(x, rm, rv, w, b, True, 0.1, 1e-5) + res)

        def fused_fwd():
            return batch_norm_act(x, w, b, rm, rv, residual=res, training=True, relu=True)

        for name, fwd in (("batch_norm_fused", fused_fwd), ("batch_norm_eager", eager_fwd)):
            t_f = timed_events(fwd, args.iters)
            y = fwd()

            def bwd():
                torch.autograd.grad(y, (x, res, w, b), go, retain_graph=True)
            t_b = timed_events(bwd, args.iters)
            ours = name == "batch_norm_fused"
            report_line(name + "_forward", t_f, 4.0625 * nbytes_act if ours else None,
                        {"shape": list(shape)})
            report_line(name + "_backward", t_b, 6.125 * nbytes_act if ours else None,
                        {"shape": list(shape)})
            del y
    if "stem_conv" in cases:
        n = 256 if args.mb >= 512 else 64
        x = torch.randn(n, 3, 224, 224, device=dev).bfloat16() \
            .contiguous(memory_format=torch.channels_last)
        w = torch.randn(64, 3, 7, 7, device=dev).bfloat16() \
            .contiguous(memory_format=torch.channels_last)
        dy = torch.randn_like(_C.stem_conv_forward(x, w))
        moved = 2 * (x.numel() + dy.numel())

        def torch_wgrad():
            torch.ops.aten.convolution_backward(dy, x, w, None, [2, 2], [3, 3], [1, 1], False,
                                                [0, 0], 1, [False, True, False])
        for name, fwd, wgrad in (
                ("stem_conv_fused", lambda: _C.stem_conv_forward(x, w),
                 lambda: _C.stem_conv_wgrad(x, dy, w)),
                ("stem_conv_torch",
                 lambda: torch.nn.functional.conv2d(x, w, stride=2, padding=3), torch_wgrad)):
            for which, fn in (("_forward", fwd), ("_weight_gradient", wgrad)):
                us = timed_events(fn, args.iters)
                report_line(name + which, us, moved if name == "stem_conv_fused" else None,
                            {"shape": list(x.shape)})

    def activations(n, channels, size):
        return torch.randn(n, size, size, channels, device=dev).bfloat16().permute(0, 3, 1, 2)

    if "conv1x1" in cases:
        n = 256 if args.mb >= 512 else 64

        def forward(size, k, co):
            x = activations(n, k, size)
            w = torch.randn(co, k, device=dev).bfloat16()
            rows = n * size * size
            us = timed_events(lambda: _C.conv1x1(x, w), args.iters)
            report_line("conv1x1_forward", us, 2 * rows * (k + co), {"rows": rows, "k": k, "n": co})

        def gradient(size, k, co, masked):
            dy, add = activations(n, k, size), activations(n, co, size)
            w = torch.randn(k, co, device=dev).bfloat16()
            rows = n * size * size
            signs = torch.randint(0, 256, (rows, co // 8), device=dev, dtype=torch.uint8) \
                if masked else None
            us = timed_events(lambda: _C.conv1x1(dy, w, w_transposed=True, add=add, signs=signs),
                              args.iters)
            report_line("conv1x1_gradient" + ("_masked_sum" if masked else "_sum"), us,
                        2 * rows * (k + 2 * co) + (rows * co // 8 if masked else 0),
                        {"rows": rows, "k": k, "n": co})
        forward(56, 64, 256)
        gradient(56, 64, 256, True)
        gradient(14, 256, 1024, True)
        gradient(14, 256, 1024, False)
        forward(14, 256, 1024)
        forward(56, 256, 64)
    if "norm_conv" in cases:
        n = 256 if args.mb >= 512 else 64
        x, res, dy, a = (activations(n, c, 56) for c in (256, 256, 256, 64))
        w = torch.randn(256, 64, device=dev).bfloat16() / 8
        gamma = torch.ones(256, device=dev)
        _, saved, signs = _C.bn_forward(x, res, gamma, gamma, None, None, 0.1, 1e-5, True, None)
        del res
        rows = n * 56 * 56

        def apart():
            dx = _C.bn_backward(dy, x, gamma, saved, signs, True, False)[0]
            torch.ops.aten.convolution_backward(dx, a, w[:, :, None, None], None, [1, 1], [0, 0],
                                                [1, 1], False, [0, 0], 1, [True, True, False])
        moved = rows * (2 * (2 * 512 + 32) + 2 * 128)
        us = timed_events(lambda: _C.norm_conv_backward(dy, signs, x, a, w, gamma, saved),
                          args.iters)
        report_line("norm_conv_backward_fused", us, moved, {"rows": rows})
        report_line("norm_conv_backward_apart", timed_events(apart, args.iters), None,
                    {"rows": rows})
        del x, dy, a, saved, signs
    if "residual_block" in cases:
        from horovod_b200.models.resnet import ResNet
        n = 256 if args.mb >= 512 else 64
        model = ResNet().to(dev).to(memory_format=torch.channels_last)
        for which, block, channels in (("stage1", model.layer1[0], 64),
                                       ("stage2", model.layer2[0], 256)):
            x = activations(n, channels, 56).requires_grad_(True)
            wanted = [x] + list(block.parameters())

            def fwd():
                with torch.autocast("cuda", dtype=torch.bfloat16):
                    return block(x)
            dy = torch.randn_like(fwd())
            for kind, switch in (("node", "1"), ("layers", "0")):
                os.environ["HOROVOD_B200_FUSED_BLOCK"] = switch
                t_f = timed_events(fwd, args.iters)
                y = fwd()
                t_b = timed_events(lambda: torch.autograd.grad(y, wanted, dy, retain_graph=True),
                                   args.iters)
                for name, us in (("forward", t_f), ("backward", t_b)):
                    report_line("residual_block_%s_%s_%s" % (which, kind, name), us, None,
                                {"shape": list(x.shape)})
                del y
            os.environ.pop("HOROVOD_B200_FUSED_BLOCK")
    if "max_pool" in cases:
        import torch.nn.functional as F
        from horovod_b200.ops.pooling import max_pool_3x3_s2
        n = 256 if args.mb >= 512 else 32
        x = torch.relu(torch.randn(n, 64, 112, 112, device=dev)).bfloat16() \
            .contiguous(memory_format=torch.channels_last).requires_grad_(True)
        xbytes = x.numel() * 2
        for name, fwd in (("max_pool_fused", max_pool_3x3_s2),
                          ("max_pool_torch", lambda t: F.max_pool2d(t, 3, stride=2, padding=1))):
            t_f = timed_events(lambda: fwd(x), args.iters)
            y = fwd(x)
            go = torch.randn_like(y)
            t_b = timed_events(lambda: torch.autograd.grad(y, x, go, retain_graph=True), args.iters)
            moved = 1.3125 * xbytes if name == "max_pool_fused" else None
            report_line(name + "_forward", t_f, moved, {"shape": list(x.shape)})
            report_line(name + "_backward", t_b, moved, {"shape": list(x.shape)})
            del y
    if "fused_sgd" in cases:
        from horovod_b200.torch.fused_sgd import FusedSGD
        sizes = resnet50_like_sizes(min(nbytes, 256 << 20) // 4)
        total = sum(sizes) * 4
        for name, cls in (("fused_sgd", FusedSGD), ("torch_sgd", torch.optim.SGD)):
            ps = [torch.randn(n, device=dev, requires_grad=True) for n in sizes]
            for p in ps:
                p.grad = torch.randn_like(p)
            opt = cls(ps, lr=0.01, momentum=0.9, weight_decay=1e-4)
            opt.step()  # creates the momentum buffers
            us = timed_events(opt.step, args.iters)
            report_line(name + "_step_call", us, 5 * total if cls is FusedSGD else None,
                        {"tensors": len(sizes), "payload_mb": total >> 20,
                         "note": "optimizer.step() as called by a training loop: bounded by "
                                 "its Python work when the GPU is otherwise idle"})
            if cls is FusedSGD:
                # The native call alone.
                bufs = [opt.state[p]["momentum_buffer"] for p in ps]

                def kernel_only():
                    _C.sgd_step(ps, bufs, 0.01, 0.9, 0.0, 1e-4, False, False, False)
                us = timed_events(kernel_only, args.iters)
                report_line("fused_sgd_kernel", us, 5 * total,
                            {"tensors": len(sizes), "payload_mb": total >> 20})
    if "peer_copy" in cases and torch.cuda.device_count() >= 2:
        # Copy-engine copy between GPU 0 and GPU 1 over NVLink, issued on a
        # stream of the source GPU (push) or of the destination GPU (pull): the
        # link rate that the SM-driven exchange kernels are compared with.
        import ctypes
        rt = ctypes.CDLL("libcudart.so.12")
        n = min(nbytes, 256 << 20)
        a = torch.empty(n, dtype=torch.uint8, device="cuda:0").fill_(1)
        b = torch.empty(n, dtype=torch.uint8, device="cuda:1")
        b.copy_(a)  # turns peer access on
        torch.cuda.synchronize(0)
        torch.cuda.synchronize(1)
        for name, d in (("peer_copy_push", 0), ("peer_copy_pull", 1)):
            with torch.cuda.device(d):
                stream = torch.cuda.Stream(device=d)

                def copy():
                    rc = rt.cudaMemcpyAsync(ctypes.c_void_p(b.data_ptr()),
                                            ctypes.c_void_p(a.data_ptr()), ctypes.c_size_t(n),
                                            ctypes.c_int(3), ctypes.c_void_p(stream.cuda_stream))
                    assert rc == 0, rc
                for _ in range(args.warmup):
                    copy()
                stream.synchronize()
                e0 = torch.cuda.Event(enable_timing=True)
                e1 = torch.cuda.Event(enable_timing=True)
                e0.record(stream)
                for _ in range(args.iters):
                    copy()
                e1.record(stream)
                e1.synchronize()
                us = e0.elapsed_time(e1) * 1e3 / args.iters
            print(json.dumps({"case": name, "payload_mb": n >> 20, "device_us": round(us, 1),
                              "nvlink_gbs_one_direction": round(n / us / 1e3, 1)}), flush=True)
    clock_log.stop()
    hvd.shutdown()
    return 0


if __name__ == "__main__":
    sys.exit(main())
