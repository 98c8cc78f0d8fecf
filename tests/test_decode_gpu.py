"""Calls with few query rows per KV head (csrc/fwd_decode.cu): the rows of all query heads of a KV head form
one item, and the 64-key tiles of all items are cut evenly over the CTAs of the launch.

Each case is compared with the CPU oracle and, with ``kernel="ws"``, with the general kernel.  Tolerances: the
oracle bars of conftest.TOL; between the two kernels twice the 16-bit rounding of outputs of this size (both
round the same value once, to either side), lse to fp32 summation order."""
import pytest
import torch

import miniattn
from conftest import TOL
from oracle.attention_oracle import attention_reference, make_inputs

pytestmark = pytest.mark.gpu
DEV = "cuda:0"

# B, Hq, Hkv, Nq, Nk, D: rows per KV head around 16 / 32 / 64 and past it; keys around the 64-key tile; few and
# many items; pieces that start and end inside an item; D = 96 (columns past it are zero-filled)
CASES = [
    (1, 1, 1, 1, 1, 128), (1, 1, 1, 1, 64, 64), (1, 3, 1, 5, 65, 96), (2, 16, 1, 1, 63, 128),
    (1, 17, 17, 1, 700, 64), (1, 16, 1, 1, 4099, 128), (3, 8, 2, 4, 257, 128), (3, 10, 5, 8, 1025, 64),
    (2, 24, 8, 6, 333, 96), (1, 8, 1, 4, 5000, 128), (1, 2, 1, 16, 511, 128), (1, 1, 1, 32, 130, 64),
    (1, 8, 1, 5, 40000, 128), (16, 64, 8, 5, 1030, 128), (16, 64, 8, 8, 1100, 64), (8, 64, 8, 9, 2500, 128),
    (8, 64, 8, 32, 1200, 64), (160, 4, 2, 2, 100, 64), (37, 8, 8, 1, 513, 128),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("causal,layout,balance", [(True, "bhnd", True), (True, "bnhd", True), (False, "bnhd", True),
                                                   (True, "bhnd", False)])
@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nk,D", CASES)
def test_matches_the_oracle_and_the_general_kernel(B, Hq, Hkv, Nq, Nk, D, causal, layout, balance, dtype):
    q, k, v = make_inputs(B, Hq, Hkv, Nq, Nk, D, dtype, seed=Nk + Nq)
    pos = Nk - Nq  # negative where there are more queries than keys: the first rows see nothing
    put = (lambda t: t.to(DEV)) if layout == "bhnd" else (lambda t: t.transpose(1, 2).contiguous().to(DEV))
    room = torch.full((B, Hkv, Nk + 70, D), float("nan"), dtype=dtype)  # the cache behind the filled part
    kc, vc = room.clone(), room.clone()
    kc[:, :, :Nk], vc[:, :, :Nk] = k, v
    cut = (lambda t: t[:, :, :Nk]) if layout == "bhnd" else (lambda t: t[:, :Nk])
    qd, kd, vd = put(q), cut(put(kc)), cut(put(vc))
    kw = dict(causal=causal, layout=layout, q_pos0=pos if causal else 0, return_lse=True)
    outs = [miniattn.flash_attn_fwd(qd, kd, vd, balance=balance, **kw) for _ in range(2)]
    ws, ws_lse = miniattn.flash_attn_fwd(qd, kd, vd, kernel="ws", **kw)
    assert miniattn.device_status(DEV) == 0
    back = (lambda t: t.float().cpu()) if layout == "bhnd" else (lambda t: t.float().cpu().transpose(1, 2))
    if B * Hq * Nq * Nk <= 4_000_000:
        ref, ref_lse = attention_reference(q, k, v, causal=causal, q_pos0=kw["q_pos0"], return_lse=True,
                                           out_dtype=torch.float32)
    else:
        ref, ref_lse = back(ws), ws_lse.cpu()
    finite = torch.isfinite(ref_lse)
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    for out, lse in outs:
        o, lse = back(out), lse.cpu()
        assert (o - ref).abs().max().item() <= TOL[dtype]
        assert (o - back(ws)).abs().max().item() <= 2 * ulp * max(1.0, ref.abs().max().item())
        assert torch.equal(torch.isfinite(lse), finite)
        assert float(o[~finite].abs().max() if (~finite).any() else 0.0) == 0.0
        if finite.any():
            assert (lse[finite] - ref_lse[finite]).abs().max().item() <= 1e-3


# either side of the lines in plan_decode: whole and cut items (11 / 12 tiles of 64 keys), 32 rows of either head dim
# (7 / 8 and 16 / 17 tiles whole, few / half / more items than SMs), query heads that fill a Q tile or more
EDGES = [
    (2, 2, 2, 1, 704, 128), (2, 2, 2, 1, 705, 128), (3, 8, 1, 4, 448, 64), (3, 8, 1, 4, 449, 64), (2, 24, 1, 1, 705, 64),
    (1, 8, 2, 8, 960, 128), (1, 8, 2, 8, 961, 128), (4, 40, 10, 5, 1100, 128), (19, 16, 8, 9, 700, 128),
    (1, 128, 1, 1, 9000, 128), (1, 129, 1, 1, 9500, 64), (2, 192, 1, 2, 2000, 128), (50, 129, 1, 1, 300, 64),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("balance", [True, False])
@pytest.mark.parametrize("B,Hq,Hkv,Nq,Nk,D", EDGES)
def test_either_side_of_a_line(B, Hq, Hkv, Nq, Nk, D, balance, dtype):
    test_matches_the_oracle_and_the_general_kernel(B, Hq, Hkv, Nq, Nk, D, True, "bhnd", balance, dtype)


def test_strided_views_and_output_views():
    """Heads and tokens picked out of wider tensors, the result into a view: no form is copied first."""
    g = torch.Generator().manual_seed(3)
    wide_q = torch.randn(2, 12, 7, 160, generator=g).to(torch.float16).to(DEV)
    wide_k = torch.randn(2, 4, 900, 136, generator=g).to(torch.float16).to(DEV)
    wide_v = torch.randn(2, 900, 6, 128, generator=g).to(torch.float16).to(DEV)
    q, k, v = wide_q[:, ::2, 1:6, 16:144], wide_k[:, ::2, 5:805, :128], wide_v[:, 50:850, 1:5:2].transpose(1, 2)
    big = torch.zeros(2, 6, 9, 128, dtype=torch.float16, device=DEV)
    out = big[:, :, 2:7]
    miniattn.flash_attn_fwd(q, k, v, causal=True, q_pos0=795, out=out)
    ref = attention_reference(q.cpu(), k.cpu(), v.cpu(), causal=True, q_pos0=795, out_dtype=torch.float32)
    assert (out.float().cpu() - ref).abs().max().item() <= TOL[torch.float16]
    assert float(big[:, :, :2].abs().max()) == 0.0 and float(big[:, :, 7:].abs().max()) == 0.0
    assert miniattn.device_status(DEV) == 0


def test_captured_calls_have_scratch_of_their_own():
    """Graphs captured one after the other share torch's capture stream; replayed on two streams at once, and
    beside eager calls, their partial results must not meet."""
    def make(seed):
        q, k, v = make_inputs(2, 8, 2, 1, 6000, 128, torch.float16, seed=seed)
        return q.to(DEV), k.to(DEV), v.to(DEV)
    ins = [make(s) for s in (1, 2)]
    want = [miniattn.flash_attn_fwd(*x).clone() for x in ins]
    graphs, outs = [], []
    for x in ins:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            outs.append(miniattn.flash_attn_fwd(*x))
        graphs.append(g)
    streams = [torch.cuda.Stream() for _ in ins]
    torch.cuda.synchronize()
    for _ in range(50):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        miniattn.flash_attn_fwd(*ins[0])
    torch.cuda.synchronize()
    for o, w in zip(outs, want):
        assert (o.float() - w.float()).abs().max().item() <= 2.0 ** -10  # fp32 order of the folds, one rounding
    assert miniattn.device_status(DEV) == 0


def test_scratch_too_small_for_the_pieces():
    """A caller's scratch that does for the general kernel's launch does for the call, whichever kernel the call would
    rather have: what needs no scratch there is taken with any, what needs some is refused below that."""
    import ctypes as C

    from miniattn import _lib
    from miniattn.ops import _prepare
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    buf = torch.zeros(64 << 20, dtype=torch.uint8, device=DEV)
    for B, Hq, Hkv, Nq, Nk, D in ((2, 8, 8, 1, 1200, 128), (1, 8, 1, 2, 16384, 128), (4, 16, 4, 4, 1500, 64)):
        q, k, v = make_inputs(B, Hq, Hkv, Nq, Nk, D, torch.float16, seed=Nk)
        qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
        ref = attention_reference(q, k, v, out_dtype=torch.float32)
        p, out, _ = _prepare(qd, kd, vd, False, None, "bhnd", False, None, "auto", 0, 0)
        info = _lib.PlanInfo()
        _lib.check(_lib.lib.miniattn_plan_fwd(C.byref(p), sms, C.byref(info), None, 0), "plan")
        need, general = _lib.lib.miniattn_fwd_scratch_bytes(C.byref(p), 0, 0), info.scratch_bytes
        assert need > 0
        sizes = {need, need - 1, general, 0 if general == 0 else general - 1}
        for size in sorted(sizes):
            out.zero_()
            rc = _lib.lib.miniattn_fwd_balanced(C.byref(p), C.c_void_p(buf.data_ptr()), C.c_size_t(size), stream)
            assert (rc == _lib.OK) == (size >= min(need, general)), (size, need, general)
            if rc == _lib.OK:
                torch.cuda.synchronize()
                assert (out.float().cpu() - ref).abs().max().item() <= TOL[torch.float16]
        # a misaligned pointer: the same
        rc = _lib.lib.miniattn_fwd_balanced(C.byref(p), C.c_void_p(buf.data_ptr() + 16), C.c_size_t(32 << 20), stream)
        assert (rc == _lib.OK) == (general == 0)
    torch.cuda.synchronize()
    assert int(buf[:16384].view(torch.int32).abs().sum()) == 0 and miniattn.device_status(DEV) == 0


def test_one_capture_keeps_one_scratch():
    """The calls of one capture share a buffer that the graph clears once, and on another stream of the same capture
    have another; a later capture has its own; none of them is the one that eager calls use."""
    from miniattn import ops
    q, k, v = (t.to(DEV) for t in make_inputs(2, 8, 2, 1, 6000, 128, torch.float16, seed=4))
    want = miniattn.flash_attn_fwd(q, k, v)
    dev, seen, outs = torch.device(DEV), [], []
    side = torch.cuda.Stream()

    def scratch():
        return ops._scratch_for(dev, torch.cuda.current_stream().cuda_stream, 1 << 20).data_ptr()

    graphs = []
    for _ in range(2):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            ptrs = []
            for _ in range(3):
                outs.append(miniattn.flash_attn_fwd(q, k, v))
                ptrs.append(scratch())
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                outs.append(miniattn.flash_attn_fwd(q, k, v))
                other = scratch()
            outs.append(miniattn.flash_attn_fwd(q, k, v))     # beside the one on the other stream
            torch.cuda.current_stream().wait_stream(side)
        assert len(set(ptrs)) == 1 and other != ptrs[0]
        seen += [ptrs[0], other]
        graphs.append(g)
    assert len(set(seen + [scratch()])) == 5
    for _ in range(20):
        for o in outs:
            o.zero_()
        for g in graphs:
            g.replay()
        torch.cuda.synchronize()
        for o in outs:
            assert torch.equal(o, want)      # pieces are folded in order
    assert miniattn.device_status(DEV) == 0
