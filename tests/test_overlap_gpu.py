"""Launches overlap the tail of the kernel before them (programmatic dependent launch): each result must be the
one that a synchronised chain of the same calls gives.  Every call reads what the one before wrote, and writes
where the one before read, so that a load or a store ahead of its turn shows.  The two chains run the same kernels
on the same inputs; only the folds of cut items may add in another order (fp32, then one rounding to 16 bit)."""
import pytest
import torch

import miniattn

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _chain(kinds, D, sync):
    g = torch.Generator(device=DEV).manual_seed(5)
    mk = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)  # noqa: E731
    x = mk(2, 4, 512, D)
    k, v = mk(2, 2, 3000, D), mk(2, 2, 3000, D)
    few = mk(2, 4, 3, D)
    seen = []
    for i, kind in enumerate(kinds * 6):
        if kind == "prefill":
            x = miniattn.flash_attn_fwd(x, k[:, :, :512], v[:, :, :512], causal=True)
        elif kind == "cut":  # 16 items of 24 tiles on 148 SMs
            miniattn.flash_attn_fwd(x.clone() if i % 2 else x, k, v, out=x)
        elif kind == "decode":
            miniattn.flash_attn_fwd(few, k, v, causal=True, q_pos0=2997, out=few)
            k[:, :, 100 + i:103 + i] = few[:, ::2]   # an ordinary kernel between two overlapped ones
        elif kind == "int8":
            x = miniattn.flash_attn_fwd_int8qk(x, k[:, :, :512], v[:, :, :512])
        elif kind == "state":
            c = miniattn.carry_state(x)
            miniattn.flash_attn_fwd(x, k[:, :, :700], v[:, :, :700], carry=c, carry_out=True)
            x = miniattn.flash_attn_fwd(x, k[:, :, 700:], v[:, :, 700:], carry=c, carry_in=True)
        x = x * 4
        if sync:
            torch.cuda.synchronize()
        seen.append(x.clone())
        seen.append(few.clone())
    torch.cuda.synchronize()
    assert miniattn.device_status(DEV) == 0
    return seen


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kinds", [["prefill"], ["decode"], ["prefill", "decode"], ["int8", "prefill"], ["state", "decode"],
                                   ["cut", "decode", "prefill"], ["int8", "cut", "state", "decode", "prefill"]])
def test_overlapped_chain_equals_a_synchronised_one(kinds, D):
    for a, b in zip(_chain(kinds, D, False), _chain(kinds, D, True)):
        assert torch.isfinite(a.float()).all()
        # bf16 results of up to a few units, each at most one rounding apart, fed back with a gain of four
        # through averages over at least a hundred keys
        assert (a.float() - b.float()).abs().max().item() <= 2.0 ** -5 * max(1.0, b.float().abs().max().item())


def test_back_to_back_calls_are_bit_for_bit_repeatable():
    """Uncut launches, hundreds in flight, no kernel between them: output of one is the query of the next."""
    g = torch.Generator(device=DEV).manual_seed(6)
    q = torch.randn(1, 4, 256, 128, generator=g, device=DEV).to(torch.float16)
    k, v = (torch.randn(1, 4, 256, 128, generator=g, device=DEV).to(torch.float16) for _ in range(2))

    def run(sync):
        a, b = q.clone(), torch.empty_like(q)
        for _ in range(300):
            miniattn.flash_attn_fwd(a, k, v, out=b, softmax_scale=1.0)
            if sync:
                torch.cuda.synchronize()
            miniattn.flash_attn_fwd(b, k, v, out=a, softmax_scale=1.0)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return a

    assert torch.equal(run(False), run(True))
    assert miniattn.device_status(DEV) == 0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("kinds", [["decode"], ["cut"], ["cut", "cache"], ["cut", "decode", "cache"], ["int8", "int8k"],
                                   ["state"], ["prefill", "int8", "cut", "cache", "int8k", "state", "decode"]])
def test_launches_with_nothing_between_them(kinds, D):
    """This library's launches alone, dozens in flight.  Every call reads what the one before wrote, into a buffer of
    its own that holds other values before; scratch, arrival counters, INT8 buffers and the carried state are shared
    by all calls.  Afterwards each call is made again by itself, from what its input holds now: a load ahead of its
    turn read something else.  Scores are large, so that a stale row gives quite another result."""
    g = torch.Generator(device=DEV).manual_seed(7)
    mk = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)  # noqa: E731
    steps = (kinds * 28)[:28]
    bufs = [mk(2, 4, 512, D) for _ in range(len(steps) + 1)]
    k, v, few = mk(2, 2, 3000, D), mk(2, 2, 3000, D), mk(2, 4, 3, D)
    q8 = miniattn.Int8QK(2, 4, 2, 512, 512, D, torch.device(DEV))
    state = miniattn.carry_state(bufs[0])
    fwd, kw = miniattn.flash_attn_fwd, dict(softmax_scale=0.5)

    def call(kind, x, out):
        if kind == "prefill":
            fwd(x, k[:, :, :512], v[:, :, :512], causal=True, out=out, balance=False, **kw)
        elif kind == "cut":       # 16 items of 24 tiles on 148 SMs
            fwd(x, k, v, out=out, **kw)
        elif kind == "decode":    # the queries were written by the call before
            fwd(x[:, :, 5:8], k, v, out=out[:, :, 5:8], **kw)
        elif kind == "cache":     # the keys and values were
            fwd(few, x[:, :2], x[:, 2:], out=out[:, :, 5:8], **kw)
        elif kind == "int8":
            miniattn.flash_attn_fwd_int8qk(x, k[:, :, :512], v[:, :, :512], out=out, buffers=q8, **kw)
        elif kind == "int8k":
            miniattn.flash_attn_fwd_int8qk(bufs[0], x[:, :2], x[:, 2:], out=out, buffers=q8, **kw)
        else:
            fwd(x, k[:, :, :700], v[:, :, :700], carry=state, carry_out=True, **kw)
            fwd(x, k[:, :, 700:], v[:, :, 700:], carry=state, carry_in=True, out=out, **kw)

    before = [b.clone() for b in bufs]
    torch.cuda.synchronize()
    for i, kind in enumerate(steps):
        call(kind, bufs[i], bufs[i + 1])
    torch.cuda.synchronize()
    assert miniattn.device_status(DEV) == 0
    for i, kind in enumerate(steps):
        again = before[i + 1]
        call(kind, bufs[i], again)
        torch.cuda.synchronize()
        assert torch.isfinite(again.float()).all()
        # the folds of a cut item may add in another order: fp32, then one rounding to bf16
        assert (again.float() - bufs[i + 1].float()).abs().max().item() <= 2.0 ** -7 * again.float().abs().max().item()


def test_decode_into_its_own_query_repeats_bit_for_bit():
    """Hundreds of decode launches in flight, cut over CTAs, each writing the query that it read.  Pieces are folded
    in order, so nothing may differ from the synchronised chain."""
    g = torch.Generator(device=DEV).manual_seed(8)
    k, v = (torch.randn(3, 2, 5000, 128, generator=g, device=DEV).to(torch.float16) for _ in range(2))
    start = torch.randn(3, 8, 2, 128, generator=g, device=DEV).to(torch.float16)

    def run(sync):
        q = start.clone()
        for i in range(300):
            miniattn.flash_attn_fwd(q, k[:, :, i:4000 + i], v[:, :, i:4000 + i], out=q, softmax_scale=1.0)
            if sync:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        return q

    assert torch.equal(run(False), run(True))
    assert miniattn.device_status(DEV) == 0
