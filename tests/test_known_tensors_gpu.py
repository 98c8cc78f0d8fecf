"""A call on tensors that an earlier call was made with takes its parameter block as it is.  Tensors at the same
addresses that do not fit together any more must be refused as on a first call."""
import pytest
import torch

import miniattn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("layout", ["bhnd", "bnhd"])
def test_a_misfit_at_a_known_address_is_refused(layout):
    g = torch.Generator(device=DEV).manual_seed(1)
    shape = (1, 2, 300, 64) if layout == "bhnd" else (1, 300, 2, 64)
    tok = 2 if layout == "bhnd" else 1
    q, k, v = (torch.randn(shape, generator=g, device=DEV).to(torch.float16) for _ in range(3))
    out = torch.empty_like(q)
    short = lambda t: t.narrow(tok, 0, 200)        # noqa: E731  same address, same strides
    other = lambda t: t.view(torch.bfloat16)       # noqa: E731
    call = lambda *a, **kw: miniattn.flash_attn_fwd(*a, layout=layout, **kw)  # noqa: E731
    for kw in (dict(), dict(out=out)):
        for _ in range(2):
            call(q, k, v, **kw)
        for args in ((q, k, short(v)), (q, short(k), v), (q, k, other(v)), (q, other(k), v), (other(q), k, v)):
            with pytest.raises(RuntimeError):
                call(*args, **kw)
        call(q, short(k), short(v), **kw)
        call(other(q), other(k), other(v), **(dict(out=other(out)) if kw else {}))
    for bad in (short(out), other(out)):
        with pytest.raises(RuntimeError):
            call(q, k, v, out=bad)
    torch.cuda.synchronize()
    assert miniattn.device_status(DEV) == 0


def test_a_carry_buffer_that_shrank_is_refused():
    q = torch.randn(1, 2, 256, 64, device=DEV).to(torch.float16)
    state = miniattn.carry_state(q)
    for _ in range(2):
        miniattn.flash_attn_fwd(q, q, q, carry=state, carry_out=True)
    with pytest.raises(RuntimeError):
        miniattn.flash_attn_fwd(q, q, q, carry=state[:state.numel() // 2], carry_out=True)
    torch.cuda.synchronize()
    assert miniattn.device_status(DEV) == 0
