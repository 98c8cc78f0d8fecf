"""Query heads of a KV head that share Q tiles (PACK in csrc/fwd_ws.cu): row r of a tile is token r / G, head
r % G.  Taken where it saves K/V tiles: under a causal mask, or where the token count leaves a tile ragged.

Compared with the CPU oracle, and with the same call one KV head's query heads at a time (G = 1 each: never
packed).  Tolerances: conftest.TOL against the oracle; between the two forms, whose rows see the same scores and
differ in where a row's reference moves and in the order of cut items' folds, twice the 16-bit rounding."""
import pytest
import torch

import miniattn
from conftest import TOL
from oracle.attention_oracle import attention_reference, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


# B, Hkv, G, Nq, Nk, D, causal: token counts around 128 / G and 256 / G; groups that do not divide 128 (padding
# rows); few long items (cut over CTAs) and many short ones; more queries than keys
CASES = [
    (1, 1, 2, 130, 130, 128, True), (2, 2, 3, 127, 300, 128, True), (1, 2, 3, 85, 85, 64, True),
    (1, 1, 4, 65, 500, 96, True), (2, 1, 5, 201, 201, 128, True), (1, 2, 6, 170, 64, 64, True),
    (1, 1, 7, 300, 1000, 128, True), (1, 2, 8, 129, 4000, 128, True), (1, 1, 16, 100, 257, 128, False),
    (2, 3, 3, 140, 333, 128, False), (1, 1, 128, 66, 130, 64, True), (1, 1, 100, 70, 70, 128, True),
    (2, 8, 3, 777, 3333, 128, True), (1, 4, 4, 1024, 1024, 64, True), (16, 8, 4, 300, 300, 96, True),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["bhnd", "bnhd"])
@pytest.mark.parametrize("B,Hkv,G,Nq,Nk,D,causal", CASES)
def test_packed_heads(B, Hkv, G, Nq, Nk, D, causal, layout, dtype):
    q, k, v = make_inputs(B, Hkv * G, Hkv, Nq, Nk, D, dtype, seed=Nq + G)
    pos = Nk - Nq if causal else 0
    put = (lambda t: t.to(DEV)) if layout == "bhnd" else (lambda t: t.transpose(1, 2).contiguous().to(DEV))
    head = 1 if layout == "bhnd" else 2
    qd, kd, vd = put(q), put(k), put(v)
    kw = dict(causal=causal, q_pos0=pos, layout=layout, kernel="ws")
    wide = torch.full([s + 3 if i == 1 else s for i, s in enumerate(qd.shape)], 7.0, dtype=dtype, device=DEV)
    view = wide[:, 1:-2]  # the result goes into a view; its neighbours stay as they are
    out, lse = miniattn.flash_attn_fwd(qd, kd, vd, return_lse=True, out=view, **kw)
    plain = miniattn.flash_attn_fwd(qd, kd, vd, balance=False, **kw)
    assert bool((wide[:, 0] == 7).all()) and bool((wide[:, -2:] == 7).all())
    one, one_lse = torch.empty_like(qd), torch.empty_like(lse)
    for g in range(G):
        sel = torch.arange(Hkv, device=DEV) * G + g
        o, z = miniattn.flash_attn_fwd(qd.index_select(head, sel), kd, vd, return_lse=True, **kw)
        one.index_copy_(head, sel, o)
        one_lse.index_copy_(1, sel, z)
    assert miniattn.device_status(DEV) == 0
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    scale = max(1.0, one.abs().max().item())
    for o in (out, plain):
        assert (o.float() - one.float()).abs().max().item() <= 2 * ulp * scale
    finite = torch.isfinite(one_lse)
    assert torch.equal(torch.isfinite(lse), finite)
    assert (lse[finite] - one_lse[finite]).abs().max().item() <= 1e-4
    if B * Hkv * G * Nq * Nk <= 8_000_000:
        ref, ref_lse = attention_reference(q, k, v, causal=causal, q_pos0=pos, return_lse=True, out_dtype=torch.float32)
        back = out.float().cpu() if layout == "bhnd" else out.float().cpu().transpose(1, 2)
        assert (back - ref).abs().max().item() <= TOL[dtype]
        f = torch.isfinite(ref_lse)
        assert (lse.cpu()[f] - ref_lse[f]).abs().max().item() <= 2e-3
