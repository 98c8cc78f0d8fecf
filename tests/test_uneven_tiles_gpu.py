"""Two Q tiles of a work item that run at different speeds.  The rows of one of them outgrow their reference in
every half of every K/V tile, so that its softmax takes each half twice and rescales O; the other tile's rows never
do and it runs ahead as far as the K/V ring lets it.  The tile that is done first folds a partial or the carried
state in through its half of that ring, and may do so only when the other tile's products no longer read it.

Tolerances: the oracle bars of conftest.TOL; a climbing row sees the last 64 keys, its output is an average of
them like any other's, and its scores of up to 800 carry 2^-14 of fp32 rounding in exp2's argument."""
import pytest
import torch

import miniattn
from conftest import TOL
from miniattn.ops import plan_info
from oracle.attention_oracle import attention_reference, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(H, Nq, Nk, D, climbing):
    """Rows of Q tile `climbing` (0 or 1) of every pair gain 12 nats per half; the others see N(0,1) keys alone."""
    q, k, v = make_inputs(1, H, H, Nq, Nk, D, torch.float16, seed=D + climbing)
    k[..., 0] = (torch.arange(Nk) // 64 * 1.5).to(torch.float16)          # exact
    q[..., 0] = ((torch.arange(Nq) // 128) % 2 == climbing).to(torch.float16) * (8.0 * D ** 0.5)
    return q, k, v


@pytest.mark.parametrize("climbing", [0, 1])
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("H,Nq,Nk", [(1, 512, 4096), (4, 2048, 2048), (3, 300, 3333)])
def test_cut_items(H, Nq, Nk, D, climbing):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert plan_info(1, H, Nq, Nk, D, sm_count=sms)[0].n_cut_items > 0
    q, k, v = _inputs(H, Nq, Nk, D, climbing)
    ref = attention_reference(q, k, v, out_dtype=torch.float32)
    qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
    outs = [miniattn.flash_attn_fwd(qd, kd, vd, kernel="ws") for _ in range(4)]
    assert miniattn.device_status(DEV) == 0
    for out in outs:
        assert (out.float().cpu() - ref).abs().max().item() <= TOL[torch.float16]


@pytest.mark.parametrize("climbing", [0, 1])
@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("Nq,cuts", [(256, (0, 1100, 1228, 2300, 3400)), (700, (0, 640, 3400))])
def test_carried_chains(Nq, cuts, D, climbing):
    q, k, v = _inputs(2, Nq, cuts[-1], D, climbing)
    ref = attention_reference(q, k, v, out_dtype=torch.float32)
    qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
    for _ in range(3):
        state = miniattn.carry_state(qd)
        for a, b in zip(cuts, cuts[1:]):
            out = miniattn.flash_attn_fwd(qd, kd[:, :, a:b], vd[:, :, a:b], carry=state, carry_in=a > 0,
                                          carry_out=b < cuts[-1])
        assert miniattn.device_status(DEV) == 0
        assert (out.float().cpu() - ref).abs().max().item() <= TOL[torch.float16]


@pytest.mark.parametrize("balance", [True, False])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Nq,Nk,pos", [(256, 256, -128), (384, 700, -192), (1024, 2000, -500)])
def test_first_tile_without_visible_keys(Nq, Nk, pos, D, balance):
    """All rows of the first Q tile lie before every key: their softmax takes each half twice, the first one too,
    and the second tile, which starts on a signal of the first, must start once and be right."""
    q, k, v = make_inputs(2, 4, 4, Nq, Nk, D, torch.float16, seed=Nq)
    ref, ref_lse = attention_reference(q, k, v, causal=True, q_pos0=pos, return_lse=True, out_dtype=torch.float32)
    qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
    for _ in range(4):
        out, lse = miniattn.flash_attn_fwd(qd, kd, vd, causal=True, q_pos0=pos, return_lse=True, kernel="ws",
                                           balance=balance)
        assert miniattn.device_status(DEV) == 0
        assert float(out[:, :, :-pos].abs().max()) == 0.0 and bool((lse[:, :, :-pos] == float("-inf")).all())
        assert (out.float().cpu() - ref).abs().max().item() <= TOL[torch.float16]
        assert (lse.cpu()[:, :, -pos:] - ref_lse[:, :, -pos:]).abs().max().item() <= 1e-3
