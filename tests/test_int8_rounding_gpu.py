"""INT8 pre-pass: values on and beside the ties of x / scale round as the division says, on every column of a slab."""
import pytest
import torch

import miniattn
from miniattn import ops
from oracle.attention_oracle import quantize_per_block_int8

pytestmark = pytest.mark.gpu


def _prepass(q, k):
    b = ops.Int8QK(q.shape[0], q.shape[1], k.shape[1], q.shape[2], k.shape[2], q.shape[3], q.device)
    miniattn.flash_attn_fwd_int8qk(q, k, torch.zeros_like(k), buffers=b, attend=False)
    torch.cuda.synchronize()
    return b.q8.cpu(), b.k8.cpu(), b.q_scale.cpu(), b.k_scale.cpu()


def _near_ties(shape, dtype, top, seed):
    """Random n + 1/2 of either sign times top / 127, in `dtype`: its rounding leaves them on ties or a little beside.
    The rows come in pairs of opposite sign (an odd last row is zero), so that a column's sum over all rows is 0."""
    g = torch.Generator().manual_seed(seed)
    B, H, N, D = shape
    x = (torch.randint(-127, 127, (B, H, N // 2, D), generator=g) + 0.5) * (top / 127.0)
    x[:, :, ::64, 0] = top  # the largest of each slab of 128 rows
    x = torch.stack((x, -x), 3).view(B, H, N // 2 * 2, D)
    if N % 2:
        x = torch.cat((x, torch.zeros(B, H, 1, D)), 2)
    return x.to(dtype)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("N", [1, 2, 127, 129, 1025])
@pytest.mark.parametrize("top", [127.0, 127.0 / 1024, 3.0, 1.0 / 3])
def test_ties_round_as_the_division(dtype, D, N, top):
    q = _near_ties((2, 3, N, D), dtype, top, 1)
    k = _near_ties((2, 1, N, D), dtype, 127.0, 2)  # multiples of 1/2: every partial sum is exact, every mean 0
    q8, k8, q_scale, k_scale = _prepass(q.cuda(), k.cuda())
    q_ref, _ = quantize_per_block_int8(q.float())
    k_ref, ks_ref = quantize_per_block_int8(k.float())
    assert torch.equal(q8, q_ref)  # a whole number either is the division's or is not: no tolerance
    assert torch.equal(k8, k_ref)
    assert torch.equal(k_scale, ks_ref)
    assert torch.isfinite(q_scale).all()
