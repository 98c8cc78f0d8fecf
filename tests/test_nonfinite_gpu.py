"""Scores that are no numbers.  A NaN in one key makes the result of every row that sees the key a NaN, whatever
column of a 64-key half the key has (some columns' exponentials come from a polynomial, which would swallow it); so
does a score of +inf.  A score of -inf is a weight of 0.  Rows that do not see the key are untouched."""
import pytest
import torch

import miniattn
from conftest import TOL
from miniattn.ops import plan_info
from oracle.attention_oracle import attention_reference, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _check(out, lse, want_nan, ref, dtype):
    """want_nan: (H, Nq) rows of batch 0 whose every output is a NaN.  A causal row that sees a few keys is nearly
    one key's V, not an average of many: one rounding of values of that size on top of the bar."""
    assert miniattn.device_status(DEV) == 0
    out = out.float().cpu()
    assert bool(torch.isnan(out[0][want_nan]).all())
    assert not bool(torch.isnan(out[0][~want_nan]).any())
    if (~want_nan).any():
        tol = TOL[dtype] + ref.abs().max().item() * (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8)
        assert (out[0] - ref[0])[~want_nan].abs().max().item() <= tol
        assert bool(torch.isfinite(lse.cpu()[0][~want_nan]).all())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("half", [0, 1, 4])
@pytest.mark.parametrize("kernel,Nq", [("ws", 400), ("auto", 5)])
def test_nan_in_one_key(kernel, Nq, half, D, dtype):
    """Head h has its NaN at column h of the half."""
    q, k, v = make_inputs(1, 64, 64, Nq, 400, D, dtype, seed=half)
    key = half * 64 + torch.arange(64)
    good = k.clone()
    k[0, torch.arange(64), key, 3] = float("nan")
    for causal in (False, True):
        pos = 400 - Nq
        seen = (torch.arange(Nq)[None] + pos >= key[:, None]) if causal else torch.ones(64, Nq, dtype=torch.bool)
        ref = attention_reference(q, good, v, causal=causal, q_pos0=pos, out_dtype=torch.float32)
        out, lse = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), causal=causal, q_pos0=pos, kernel=kernel,
                                           return_lse=True)
        _check(out, lse, seen, ref, dtype)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kernel,Nq", [("ws", 300), ("auto", 8)])
def test_infinite_scores(kernel, Nq, D):
    """An infinite key channel: +inf for the rows with a 1 there, -inf for those with a -1."""
    q, k, v = make_inputs(1, 64, 64, Nq, 400, D, torch.float16, seed=D)
    q[..., 0] = torch.where(torch.arange(Nq) % 3 == 0, 1.0, -1.0).to(torch.float16)
    k[0, torch.arange(64), 128 + torch.arange(64), 0] = float("inf")
    want = (torch.arange(Nq) % 3 == 0)[None].expand(64, Nq)
    ref = torch.empty(1, 64, Nq, D)
    for h in range(64):   # without that key
        keep = torch.arange(400) != 128 + h
        ref[:, h:h + 1] = attention_reference(q[:, h:h + 1], k[:, h:h + 1, keep], v[:, h:h + 1, keep], out_dtype=torch.float32)
    out, lse = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), kernel=kernel, return_lse=True)
    _check(out, lse, want, ref, torch.float16)


COLS = torch.tensor([0, 1, 5, 10, 21, 33, 63, 8])


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("form", ["cut", "carried", "packed"])
def test_nan_in_one_key_other_forms(form, D):
    Nq, Nk, G = (330, 4096, 1) if form != "packed" else (330, 700, 2)
    if form == "cut":
        sms = torch.cuda.get_device_properties(0).multi_processor_count
        assert plan_info(1, 8, Nq, Nk, D, causal=True, q_pos0=Nk - Nq, sm_count=sms)[0].n_cut_items > 0
    q, k, v = make_inputs(1, 8 * G, 8, Nq, Nk, D, torch.float16, seed=1)
    key = Nk - 256 + COLS
    ref = attention_reference(q, k, v, causal=True, q_pos0=Nk - Nq, out_dtype=torch.float32)
    k[0, torch.arange(8), key, D - 1] = float("nan")
    seen = (torch.arange(Nq)[None] + Nk - Nq >= key[:, None]).repeat_interleave(G, 0)
    qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
    if form == "carried":
        state = miniattn.carry_state(qd)
        for a, b in ((0, 1000), (1000, 3900), (3900, Nk)):
            res = miniattn.flash_attn_fwd(qd, kd[:, :, a:b], vd[:, :, a:b], causal=True, q_pos0=Nk - Nq, k_pos0=a,
                                          carry=state, carry_in=a > 0, carry_out=b < Nk, return_lse=b == Nk)
    else:
        res = miniattn.flash_attn_fwd(qd, kd, vd, causal=True, q_pos0=Nk - Nq, kernel="ws", return_lse=True)
    _check(res[0], res[1], seen, ref, torch.float16)
