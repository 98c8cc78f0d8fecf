"""Decode: a CTA finds its tiles in 32 bits where tiles x CTAs fit, in 64 bits otherwise.  Both against the general
kernel on the same inputs: the two round the same sums once, so they differ by an ulp of the result at most where
P's 16-bit rounding differs; the bound is conftest.TOL twice."""
import pytest
import torch

import miniattn
from conftest import TOL

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("B,Hkv,G,Nk,balance", [
    (2500, 8, 1, 512, False),    # 20000 items of 8 tiles, one CTA each: 3.2e9 tiles x CTAs
    (2000, 8, 1, 512, False),    # 16000: 2.05e9, just inside
    (37, 3, 2, 777, True),       # items that do not divide over the CTAs
    (1, 1, 4, 20000, True),      # one item in many pieces
])
def test_ranges_of_a_cta(B, Hkv, G, Nk, balance):
    gen = torch.Generator(device=DEV).manual_seed(B)
    q = torch.randn(B, Hkv * G, 1, 64, device=DEV, dtype=torch.float16, generator=gen)
    k, v = (torch.randn(B, Hkv, Nk, 64, device=DEV, dtype=torch.float16, generator=gen) for _ in range(2))
    kw = dict(causal=True, q_pos0=Nk - 1, return_lse=True, balance=balance)
    out, lse = miniattn.flash_attn_fwd(q, k, v, **kw)
    ref, ref_lse = miniattn.flash_attn_fwd(q, k, v, kernel="ws", **kw)
    assert miniattn.device_status(DEV) == 0
    assert (out.float() - ref.float()).abs().max().item() <= 2 * TOL[torch.float16]
    assert (lse - ref_lse).abs().max().item() <= 1e-3
