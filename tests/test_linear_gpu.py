"""Linear layers that share their input in one launch (csrc/linear.cu): against the same product in fp64, and the module
path against the layers' own calls.  Both round once, from fp32 sums: a result is within half an ulp of its own size
plus the fp32 sum's error, K * 2^-24 of the terms' size."""
import ctypes as C
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

import miniattn
from miniattn import _lib, ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _launch(x, ws, bs, ys, only_if_faster=0):
    p = _lib.LinearParams()
    p.x, p.status, p.ldx, p.M, p.K = x.data_ptr(), ops._status_word(x.device).data_ptr(), x.stride(0), x.shape[0], x.shape[1]
    p.dtype, p.n_out, p.only_if_faster = ops._DTYPES[x.dtype], len(ws), only_if_faster
    for o, w, b, y in zip(p.out, ws, bs, ys):
        o.w, o.y, o.ldw, o.ldy, o.N = w.data_ptr(), y.data_ptr(), w.stride(0), y.stride(0), w.shape[0]
        o.bias = b.data_ptr() if b is not None else None
    return _lib.lib.miniattn_linear(C.byref(p), torch.cuda.current_stream().cuda_stream)


# M, K, N...: one row to several row tiles, edges of 32, 128 and 256 rows; K below, at and past a stage of 64 and past
# the ring; N of one box of 16 columns, not a multiple of 16, and several tiles; two tiles for a pair of SMs in the last
# but one
CASES = [
    (1, 8, (8,)), (31, 64, (16,)), (33, 72, (24, 40)), (128, 256, (256, 64, 8)), (129, 520, (104, 264)), (255, 448, (48,)),
    (256, 128, (512,)), (257, 1000, (72, 136)), (1000, 1024, (1024, 256)), (2300, 192, (1536, 1544)), (5000, 96, (512, 128)),
]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("M,K,N", CASES)
def test_linear_against_fp64(M, K, N, dtype):
    g = torch.Generator(device=DEV).manual_seed(M + K)
    wide = torch.randn(M, K + 8, device=DEV, generator=g).to(dtype)
    x = wide[:, :K]                                    # rows further apart than their length
    ws = [torch.randn(n, K, device=DEV, generator=g).to(dtype) for n in N]
    bs = [torch.randn(n + 1, device=DEV, generator=g).to(dtype)[1:] if i != 1 else None for i, n in enumerate(N)]  # odd base
    around = [torch.full((M + 2, n + 16), 7.0, dtype=dtype, device=DEV) for n in N]
    ys = [t[1:-1, 8:-8] for t in around]
    assert _launch(x, ws, bs, ys) == _lib.OK
    assert miniattn.device_status(DEV) == 0
    ulp = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    for w, b, y, t in zip(ws, bs, ys, around):
        ref = x.double() @ w.double().T + (b.double() if b is not None else 0.0)
        size = x.double().abs() @ w.double().abs().T + 4.0
        bound = ulp * ref.abs() + K * 2.0 ** -24 * size + 2.0 ** -24
        assert bool(((y.double() - ref).abs() <= bound).all())
        assert bool((t[0] == 7).all() and (t[-1] == 7).all() and (t[:, :8] == 7).all() and (t[:, -8:] == 7).all())


# Three and more tiles for a pair of SMs and few stages of K, so that the next accumulator is there before the copies of
# the tile before have read their buffers; boxes of a warp and tile that the buffers do not divide (1, 3, 5, 6, 7)
# and tiles cut short by the last column.  The sums' order is fixed: every launch gives the first one's result.
MANY_TILES = [
    (16384, 64, (64, 64, 64)), (32768, 64, (64, 64, 64)), (40000, 64, (64, 128)), (16384, 320, (320, 128)),
    (40000, 320, (320, 640)), (60001, 8, (16,)), (20000, 24, (352, 184)), (9000, 128, (1000, 520, 264)),
]


@pytest.mark.parametrize("M,K,N", MANY_TILES)
def test_many_tiles_of_a_pair(M, K, N):
    dtype = torch.bfloat16
    g = torch.Generator(device=DEV).manual_seed(M + K)
    x = torch.randn(M, K, device=DEV, generator=g).to(dtype)
    ws = [torch.randn(n, K, device=DEV, generator=g).to(dtype) for n in N]
    bs = [torch.randn(n, device=DEV, generator=g).to(dtype) for n in N]
    first = [torch.empty(M, n, dtype=dtype, device=DEV) for n in N]
    assert _launch(x, ws, bs, first) == _lib.OK
    for w, b, y in zip(ws, bs, first):
        ref = x.double() @ w.double().T + b.double()
        size = x.double().abs() @ w.double().abs().T + 4.0
        assert bool(((y.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + K * 2.0 ** -24 * size + 2.0 ** -24).all())
    differ = torch.zeros((), dtype=torch.int64, device=DEV)
    for _ in range(100):
        ys = [torch.full_like(y, 7.0) for y in first]
        assert _launch(x, ws, bs, ys) == _lib.OK
        for y, want in zip(ys, first):
            differ += (y.view(torch.int16) != want.view(torch.int16)).sum()
    assert int(differ) == 0 and miniattn.device_status(DEV) == 0


def test_linear_with_a_strided_row_of_one():
    x = torch.ones(1, 16, dtype=torch.float16, device=DEV)
    w = torch.ones(8, 16, dtype=torch.float16, device=DEV)
    y = torch.zeros(1, 8, dtype=torch.float16, device=DEV)
    assert _launch(x, [w], [None], [y]) == _lib.OK
    assert bool((y == 16).all())


def test_linear_refusals():
    x = torch.ones(4, 16, dtype=torch.float16, device=DEV)
    w, y = torch.ones(8, 16, dtype=torch.float16, device=DEV), torch.zeros(4, 8, dtype=torch.float16, device=DEV)
    assert _launch(x, [w[:7]], [None], [y[:, :7]]) == _lib.EINVAL           # N not a multiple of 8
    assert _launch(x[:, :12], [w[:, :12]], [None], [y]) == _lib.EINVAL      # K not a multiple of 8
    assert _launch(x[:, 4:12], [w[:, :8]], [None], [y]) == _lib.EINVAL      # not 16-byte aligned
    assert _launch(x, [w] * 3, [None] * 3, [y.clone() for _ in range(3)]) == _lib.OK


def _module(cls, *args):
    torch.manual_seed(3)
    return cls(*args).to(torch.bfloat16).to(DEV)


@pytest.mark.parametrize("cls,args,S", [(miniattn.GQA_Flash, (512, 8, 2), 700), (miniattn.MQA_Flash, (512, 4), 300),
                                        (miniattn.MHA, (256, 2, 0.0, False), 515)])
def test_modules_against_their_layers_own_calls(cls, args, S, monkeypatch):
    m = _module(cls, *args)
    x = torch.randn(2, S, args[0], device=DEV, dtype=torch.bfloat16)
    first = (lambda y: y[0] if isinstance(y, tuple) else y)
    with torch.no_grad():
        fused = first(m(x))
        monkeypatch.setattr("miniattn.variants.linear", lambda t, *layers: [layer(t) for layer in layers])
        plain = first(m(x))
    assert miniattn.device_status(DEV) == 0
    # the projections differ by their sums' order at most: an ulp of a few of the attention's inputs
    assert (fused.float() - plain.float()).norm() <= 2.0 ** -8 * plain.float().norm()


def test_calls_that_something_watches_go_through_the_layers():
    """Gradients, hooks, autocast, forward-mode tangents and modes see the layers' own calls, with the same result."""
    from torch.utils.flop_counter import FlopCounterMode
    lin = torch.nn.Linear(64, 32).half().to(DEV)
    x = torch.randn(256, 64, device=DEV, dtype=torch.float16)
    want = lin(x)
    y, = ops.linear(x, lin)
    assert y.requires_grad and torch.equal(y, want)
    y.sum().backward()
    assert lin.weight.grad is not None
    lin.requires_grad_(False)
    got, = ops.linear(x, lin)
    assert not got.requires_grad and (got - want).abs().max() <= 2.0 ** -9 * want.abs().max()
    calls = []
    handle = lin.register_forward_hook(lambda mod, args, out: calls.append(1))
    ops.linear(x, lin)
    handle.remove()
    assert calls == [1]
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert ops.linear(x, lin)[0].dtype is torch.bfloat16
    with FlopCounterMode(display=False) as counter:
        ops.linear(x, lin)
    assert counter.get_total_flops() == 2 * 256 * 64 * 32
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(x, torch.ones_like(x))
        assert torch.autograd.forward_ad.unpack_dual(ops.linear(dual, lin)[0]).tangent is not None
    batched = torch.vmap(lambda t: ops.linear(t, lin)[0])(x.view(4, 64, 64))
    assert batched.shape == (4, 64, 32)
    assert ops.linear(x.t().contiguous().t(), lin)[0].shape == (256, 32)   # not contiguous
    assert ops.linear(x[:0], lin)[0].shape == (0, 32)


@pytest.mark.parametrize("register", [True, False])
def test_a_bias_that_is_no_parameter_is_added(register):
    lin = torch.nn.Linear(64, 32).half().to(DEV).requires_grad_(False)
    bias = torch.full((32,), 100.0, dtype=torch.float16, device=DEV)
    del lin.bias
    if register:
        lin.register_buffer("bias", bias)
    else:
        lin.bias = bias
    x = torch.randn(256, 64, device=DEV, dtype=torch.float16)
    assert torch.equal(ops.linear(x, lin)[0], lin(x))


def test_more_rows_than_the_kernel_counts_go_through_the_layers(monkeypatch):
    if torch.cuda.mem_get_info()[0] < 50 << 30:
        pytest.skip("needs 34 GB of free memory")
    monkeypatch.setattr(ops, "_operands", lambda *args: pytest.fail("taken"))   # nothing is looked at
    x = torch.empty(2 ** 31 + 8, 8, dtype=torch.float16, device=DEV)
    assert ops.linear(x, lambda t: t.shape) == [x.shape]


CAPTURE = """
import torch
from miniattn import GQA_Flash
m = GQA_Flash(512, 8, 2).to(torch.bfloat16).to("cuda").requires_grad_(False)
x = torch.randn(2, 300, 512, device="cuda", dtype=torch.bfloat16)
want = m(x)
torch.cuda.synchronize()
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    y = m(x)
graph.replay()
torch.cuda.synchronize()
print(torch.equal(y, want))
"""


def test_a_captured_module_goes_the_way_of_the_calls_before_it():
    """In a process of its own, whose other calls have not set up cuBLAS: that is not possible inside a capture."""
    r = subprocess.run([sys.executable, "-c", CAPTURE], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, PYTHONPATH=str(Path(miniattn.__file__).parents[1])))
    assert r.returncode == 0 and r.stdout.strip() == "True", r.stderr[-2000:]


def test_sizes_that_are_left_to_the_layers_are_known_the_second_time(monkeypatch):
    """What is looked at for a size that does not pay: the layer once, nothing after that."""
    seen, was = [], ops._operands
    monkeypatch.setattr(ops, "_operands", lambda *args: seen.append(1) or was(*args))
    monkeypatch.setattr(ops, "_left_to_layers", set())
    lin = torch.nn.Linear(3072, 3072).half().to(DEV).requires_grad_(False)
    x = torch.randn(1554, 3072, device=DEV, dtype=torch.float16)
    for _ in range(3):
        assert torch.equal(ops.linear(x, lin)[0], lin(x))
    assert len(seen) == 1 and len(ops._left_to_layers) == 1
    small, sx = torch.nn.Linear(512, 512).half().to(DEV).requires_grad_(False), x[:, :512].contiguous()
    for _ in range(2):                                # a size that pays
        ops.linear(sx, small)
    assert len(seen) == 3 and len(ops._left_to_layers) == 1


@pytest.mark.parametrize("S,heads,names", [(300, (12, 4), ["w_q+kv", "w_o"]), (1554, (24, 8), []), (4768, (16, 4), ["w_q+kv"])])
def test_which_projections_of_a_module_are_launches(S, heads, names, monkeypatch):
    """Short ones all, ones that the library does quicker none (the output's alone neither), long ones x's."""
    m = _module(miniattn.variants.GQA_Flash, heads[0] * 128, *heads).requires_grad_(False)
    which = {(layer,): name for name, layer in m.named_children()} | {(m.w_q, m.kv): "w_q+kv"}
    was, seen = ops._one_launch, []
    def spy(x, layers, size):
        out = was(x, layers, size)
        if out is not None:
            seen.append(which[tuple(layers)])
        return out
    monkeypatch.setattr(ops, "_left_to_layers", set())
    monkeypatch.setattr(ops, "_one_launch", spy)
    m(torch.randn(1, S, heads[0] * 128, device=DEV, dtype=torch.bfloat16))
    assert seen == names
