"""One key that outweighs everything its row has seen, at every column of a 64-key half, by amounts from a few to
hundreds of powers of two.  Some columns' exponentials come from a polynomial on the FMA pipe, the others from the
exp2 unit; either must notice that the row's reference no longer serves.  A warp takes a half again for all of its
rows when one of them asks, so only one row of a warp has such a key here: 64 warps, one for each column.

Tolerances: the oracle bars of conftest.TOL, and for a row whose output is one key's V the rounding of that V."""
import ctypes as C
import math

import pytest
import torch

import miniattn
from conftest import TOL
from miniattn import _lib
from miniattn.ops import plan_info
from oracle.attention_oracle import attention_reference, int8qk_reference, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
JUMPS = (20, 127, 129, 130, 150, 200, 256, 300, 400, 600)   # powers of two; one KV head each


def _inputs(tokens_per_warp, Nq, Nk, half, D, dtype, G=1):
    """Token 5 of every warp's tokens (query head 0 of a KV head) has its key at column (warp % 64) of `half`.
    A key and its row meet in one of 32 channels, with either sign; the other rows have zeros there."""
    H = len(JUMPS)
    q, k, v = make_inputs(1, H * G, H, Nq, Nk, D, dtype, seed=Nq + Nk + D)
    q[..., :32] = 0.0
    for w in range(Nq // tokens_per_warp):
        col = w % 64
        q[:, ::G, w * tokens_per_warp + 5, col // 2] = math.sqrt(D) * (1 if col % 2 else -1)
    for col in range(64):
        size = torch.tensor([j * math.log(2.0) for j in JUMPS])
        k[:, :, half * 64 + col, :32] = 0.0
        k[:, :, half * 64 + col, col // 2] = (size * (1 if col % 2 else -1)).to(dtype)
    rows = torch.arange(Nq // tokens_per_warp) * tokens_per_warp + 5
    return q, k, v, rows


def _tol(v, dtype):
    return TOL[dtype] + v.abs().max().item() * (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8)


def _check(out, lse, q, k, v, dtype, **kw):
    assert miniattn.device_status(DEV) == 0
    ref, ref_lse = attention_reference(q, k, v, return_lse=True, out_dtype=torch.float32, **kw)
    assert (out.float().cpu() - ref).abs().max().item() <= _tol(v, dtype)
    if lse is not None:
        assert (lse.cpu() - ref_lse).abs().max().item() <= 2e-3


DTYPES = [torch.float16, torch.bfloat16]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("half", [1, 4])
def test_plain(half, D, dtype):
    q, k, v, _ = _inputs(32, 2048, 400, half, D, dtype)
    out, lse = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), kernel="ws", balance=False, return_lse=True)
    _check(out, lse, q, k, v, dtype)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("D", [64, 96, 128])
def test_cut_items(D, dtype):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert plan_info(1, len(JUMPS), 2048, 3000, D, sm_count=sms)[0].n_cut_items > 0
    q, k, v, _ = _inputs(32, 2048, 3000, 23, D, dtype)
    out, lse = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), kernel="ws", return_lse=True)
    _check(out, lse, q, k, v, dtype)


@pytest.mark.parametrize("balance", [False, True])
@pytest.mark.parametrize("D", [64, 128])
def test_packed_heads(D, balance):
    Nq, Nk, G = 1090, 400, 2
    p = _lib.FwdParams()
    p.B, p.Hq, p.Hkv, p.Nq, p.Nk, p.D = 1, G * len(JUMPS), len(JUMPS), Nq, Nk, D
    info = _lib.PlanInfo()
    _lib.check(_lib.lib.miniattn_plan_fwd(C.byref(p), 148, C.byref(info), None, 0), "plan")
    assert info.split or info.n_ctas == 9 * len(JUMPS)   # 18 tiles of 64 tokens, not 9 of 128 for each head
    q, k, v, _ = _inputs(16, Nq, Nk, 3, D, torch.float16, G)
    out, lse = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), kernel="ws", balance=balance, return_lse=True)
    _check(out, lse, q, k, v, torch.float16)


@pytest.mark.parametrize("D", [96, 128])
def test_long(D):
    q, k, v, _ = _inputs(32, 2048, 8200, 77, D, torch.float16)
    out, lse = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), kernel="ws", balance=False, return_lse=True)
    _check(out, lse, q, k, v, torch.float16)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("D", [64, 96, 128])
def test_carried(D, dtype):
    q, k, v, _ = _inputs(32, 2048, 700, 5, D, dtype)
    qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
    state = miniattn.carry_state(qd)
    for a, b in ((0, 128), (128, 512), (512, 700)):
        res = miniattn.flash_attn_fwd(qd, kd[:, :, a:b], vd[:, :, a:b], carry=state, carry_in=a > 0, carry_out=b < 700,
                                      return_lse=b == 700)
    _check(res[0], res[1], q, k, v, dtype)


@pytest.mark.parametrize("balance", [False, True])
@pytest.mark.parametrize("D", [64, 128])
def test_int8qk(D, balance):
    q, k, v, rows = _inputs(32, 2048, 1500, 9, D, torch.float16)
    out = miniattn.flash_attn_fwd_int8qk(q.to(DEV), k.to(DEV), v.to(DEV), balance=balance).float().cpu()
    assert miniattn.device_status(DEV) == 0
    ref = int8qk_reference(q, k, v).float()
    # the rows with a key of their own: its V.  A step of the int8 grid of that block of keys is several units, so
    # a rounding of K to the other side moves the other rows by more than their rounding (see test_int8qk_gpu)
    assert (out[:, :, rows] - ref[:, :, rows]).abs().max().item() <= _tol(v, torch.float16)
    assert torch.nn.functional.cosine_similarity(out.flatten(), ref.flatten(), dim=0).item() >= 0.999


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("D,std,scale", [(64, 4.0, None), (128, 4.0, None), (96, 1.0, 1.0), (128, 1.0, 1.0)])
def test_queries_that_match_one_key_each(D, std, scale, causal):
    """q is a permutation of k: every row has one key about 100 nats above the rest, anywhere."""
    N = 2048
    g = torch.Generator().manual_seed(D)
    k = (torch.randn(1, 2, N, D, generator=g) * std).to(torch.float16)
    v = torch.randn(1, 2, N, D, generator=g).to(torch.float16)
    q = k[:, :, torch.randperm(N, generator=g)].contiguous()
    out, lse = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), causal=causal, softmax_scale=scale,
                                       return_lse=True)
    _check(out, lse, q, k, v, torch.float16, causal=causal, softmax_scale=scale)
