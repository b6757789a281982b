"""``FusedSGD``: torch.optim.SGD arithmetic in one kernel launch per parameter
group (one per 256 tensors; csrc/kernels/fused_sgd.cu) instead of four to five
elementwise passes.

PyTorch's foreach SGD needs every tensor list to share strides for its
multi-tensor fast path; with channels-last convolution weights two of its
passes fall back to one launch per parameter (322 launches, 1.05 ms per step
on ResNet-50 on a B200). This optimizer walks parameters, gradients and
momentum buffers of any dense layout together, reading and writing each element
once. It is an ordinary ``torch.optim.Optimizer``: wrap it in
``hvd.DistributedOptimizer`` like any other; ``state_dict`` is compatible with
``torch.optim.SGD`` (``momentum_buffer`` per parameter). Parameters the kernel
cannot take (CPU, non-fp32, sparse gradients, mismatched layouts) are updated
with the same formulas by PyTorch ops.

The reference has no counterpart (it wraps the framework's optimizer,
horovod/torch/optimizer.py:249-325).
"""
import torch
from torch.optim.optimizer import Optimizer


def _extension():
    from horovod_b200 import _C
    return _C


def _dense(t):
    """True when the tensor's elements fill one gap-free block of memory in
    some dimension order (contiguous, channels-last, permuted...)."""
    expected = 1
    for size, stride in sorted(zip(t.shape, t.stride()), key=lambda ss: ss[1]):
        if size == 1:
            continue
        if stride != expected:
            return False
        expected *= size
    return True


class FusedSGD(Optimizer):
    def __init__(self, params, lr=1e-3, momentum=0.0, dampening=0.0, weight_decay=0.0,
                 nesterov=False, maximize=False):
        if lr < 0.0:
            raise ValueError("Invalid learning rate: %s" % lr)
        if momentum < 0.0:
            raise ValueError("Invalid momentum value: %s" % momentum)
        if weight_decay < 0.0:
            raise ValueError("Invalid weight_decay value: %s" % weight_decay)
        if nesterov and (momentum <= 0 or dampening != 0):
            raise ValueError("Nesterov momentum requires a momentum and zero dampening")
        defaults = dict(lr=lr, momentum=momentum, dampening=dampening,
                        weight_decay=weight_decay, nesterov=nesterov, maximize=maximize)
        super().__init__(params, defaults)

    @staticmethod
    def _kernel_ok(p):
        g = p.grad
        return (p.is_cuda and p.dtype == torch.float32 and not g.is_sparse and
                g.dtype == torch.float32 and g.device == p.device and
                g.shape == p.shape and g.stride() == p.stride() and _dense(p))

    def _torch_update(self, p, group):
        g = p.grad if not group["maximize"] else -p.grad
        if g.is_sparse:
            g = g.to_dense()
        if group["weight_decay"] != 0:
            g = g.add(p, alpha=group["weight_decay"])
        if group["momentum"] != 0:
            state = self.state[p]
            buf = state.get("momentum_buffer")
            if buf is None:
                buf = state["momentum_buffer"] = torch.clone(g).detach()
            else:
                buf.mul_(group["momentum"]).add_(g, alpha=1 - group["dampening"])
            g = g.add(buf, alpha=group["momentum"]) if group["nesterov"] else buf
        p.add_(g, alpha=-group["lr"])

    @torch.no_grad()
    def step(self, closure=None):
        loss = None
        if closure is not None:
            with torch.enable_grad():
                loss = closure()
        for group in self.param_groups:
            params = group["params"]
            bufs = []
            if group["momentum"] != 0:
                get, nothing = self.state.get, {}
                bufs = [get(p, nothing).get("momentum_buffer") for p in params]
            launched, rest = self._launch(params, bufs, group, first_step=False)
            if not launched:
                # A momentum buffer does not match its parameter; nothing has
                # been updated yet.
                for i in rest:
                    bufs[i] = self._matching_buffer(params[i], bufs[i])
                launched, rest = self._launch(params, bufs, group, first_step=False)
                if not launched:
                    raise RuntimeError("FusedSGD: a momentum buffer does not match its parameter")
            if rest:
                self._step_rest([params[i] for i in rest], group)
        return loss

    @staticmethod
    def _launch(params, bufs, group, first_step):
        """One native call checks, lists and updates all tensors it can; the
        positions of the others come back, or of all that it would not take if
        it has done nothing because a momentum buffer does not match."""
        return _extension().sgd_step(
            params, bufs, group["lr"], group["momentum"], group["dampening"],
            group["weight_decay"], group["nesterov"], first_step, group["maximize"])

    def _matching_buffer(self, p, buf):
        """The momentum buffer in p's memory layout (e.g. after a state_dict was
        loaded), if the kernel takes p at all."""
        if buf is not None and self._kernel_ok(p) and buf.stride() != p.stride():
            fixed = torch.empty_like(p, memory_format=torch.preserve_format)
            fixed.copy_(buf)
            buf = self.state[p]["momentum_buffer"] = fixed
        return buf

    def _step_rest(self, params, group):
        """The parameters that the kernel cannot take as they are: new ones (no
        momentum yet), and those left to PyTorch."""
        first = []
        for p in params:
            if group["momentum"] == 0 or not self._kernel_ok(p):
                self._torch_update(p, group)
                continue
            self.state[p]["momentum_buffer"] = torch.empty_like(
                p, memory_format=torch.preserve_format)
            first.append(p)
        if first:
            bufs = [self.state[p]["momentum_buffer"] for p in first]
            launched, rest = self._launch(first, bufs, group, first_step=True)
            if rest or not launched:
                raise RuntimeError("FusedSGD: the kernel does not take a parameter")
