"""Every warp stores its own 32 rows of a Q tile: row counts around 32 and the tile's edges, groups of packed heads
that make a warp's box (2 to 32 heads) and that do not, each head dim, cut and whole items.  The result goes into a view
whose neighbours must stay as they are.  Tolerances: conftest.TOL against the oracle."""
import pytest
import torch

import miniattn
from conftest import TOL
from oracle.attention_oracle import attention_reference, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("Hkv,G,Nq,Nk", [
    (2, 1, 1, 40), (2, 1, 31, 70), (1, 1, 32, 32), (3, 1, 33, 200), (1, 1, 97, 130), (2, 1, 128, 128), (1, 1, 129, 3000),
    (1, 2, 65, 300), (2, 4, 33, 500), (1, 8, 17, 700), (1, 16, 9, 300), (1, 32, 5, 200), (2, 32, 70, 330), (1, 64, 7, 90),
])
def test_rows_of_a_warp(Hkv, G, Nq, Nk, D):
    dtype = torch.float16
    q, k, v = make_inputs(1, Hkv * G, Hkv, Nq, Nk, D, dtype, seed=Nq + G)
    wide = torch.full((1, Hkv * G, Nq + 2, D), 7.0, dtype=dtype, device=DEV)
    for balance in (True, False):
        out = miniattn.flash_attn_fwd(q.to(DEV), k.to(DEV), v.to(DEV), causal=True, q_pos0=Nk - Nq, kernel="ws",
                                      balance=balance, out=wide[:, :, 1:-1])
        assert miniattn.device_status(DEV) == 0
        ref = attention_reference(q, k, v, causal=True, q_pos0=Nk - Nq, out_dtype=torch.float32)
        assert (out.float().cpu() - ref).abs().max().item() <= TOL[dtype]
        assert bool((wide[:, :, 0] == 7).all() and (wide[:, :, -1] == 7).all())
