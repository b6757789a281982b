"""The model-side and single-rank kernels at the sizes where they can go wrong:
remainders of their tiles and strips, and both sides of each dispatch rule."""
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
