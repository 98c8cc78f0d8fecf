"""Row maxima that move: the exponentials of a 64-key half are taken against the maximum of the halves before
it and taken again, with O rescaled, where a row outgrew it by more than 2^8.  Scores here climb, jump and fall
at chosen keys, in all rows or in single rows of a warp.

Tolerances: the oracle bars of conftest.TOL (outputs are averages of N(0,1) values, so the bars apply as they
stand); the rows see scores of up to 600, where exp2's argument carries 2^-15 of fp32 rounding: no more."""
import pytest
import torch

import miniattn
from conftest import TOL
from oracle.attention_oracle import attention_reference, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _profile(kind, N):
    """Added score (natural-log units, after the softmax scale) of each key."""
    half = torch.arange(N) // 64
    if kind == "climb":            # every half outgrows the one before: rescaled each time
        return half * 12.0
    if kind == "creep":            # less than 2^8 per half, more over several
        return half * 3.0
    if kind == "fall":
        return -half * 12.0
    if kind == "jump_first_half":  # a jump in the first half of a 128-key tile ...
        return torch.where(torch.arange(N) >= 256, 300.0, 0.0)
    if kind == "jump_second_half":  # ... and one in the second
        return torch.where(torch.arange(N) >= 320, 300.0, 0.0)
    return torch.where(torch.arange(N) == N - 1, 600.0, 0.0)  # the very last key takes all


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("kind", ["climb", "creep", "fall", "jump_first_half", "jump_second_half", "last"])
@pytest.mark.parametrize("rows", ["all", "one"])
@pytest.mark.parametrize("kernel,Nq", [("ws", 300), ("auto", 5)])
def test_moving_maximum(kernel, Nq, rows, kind, D, dtype):
    N = 640
    q, k, v = make_inputs(1, 2, 2, Nq, N, D, dtype, seed=D)
    k[..., 0] = (_profile(kind, N) / 8.0).to(dtype)       # exact in both types
    q[..., 0] = 0.0
    amp = 8.0 * D ** 0.5
    if rows == "all":
        q[..., 0] = amp
    else:
        q[:, :, Nq // 2, 0] = amp
    for causal in (False, True):
        pos = N - Nq if causal else 0
        ref, ref_lse = attention_reference(q, k, v, causal=causal, q_pos0=pos, return_lse=True, out_dtype=torch.float32)
        out, lse = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), causal=causal, q_pos0=pos, kernel=kernel,
                                           return_lse=True)
        assert miniattn.device_status(DEV) == 0
        # a row on which few keys count is V itself, not an average of it: one rounding of values up to |V|
        tol = TOL[dtype] + v.abs().max().item() * (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8)
        assert (out.float().cpu() - ref).abs().max().item() <= tol
        assert (lse.cpu() - ref_lse).abs().max().item() <= 2e-3


def test_moving_maximum_over_a_cut_item():
    """The same through the balanced launch: pieces of one item with maxima far apart."""
    q, k, v = make_inputs(1, 1, 1, 512, 16384, 128, torch.float16, seed=9)
    k[..., 0] = (torch.arange(16384) // 2048 * 4.0).to(torch.float16)
    q[..., 0] = 30.0
    ref = attention_reference(q, k, v, out_dtype=torch.float32)
    out = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV))
    assert miniattn.device_status(DEV) == 0
    assert (out.float().cpu() - ref).abs().max().item() <= TOL[torch.float16]
