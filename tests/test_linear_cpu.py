"""miniattn_linear's blocks have the layout of their ctypes mirrors, bad calls are refused before the GPU is looked
for, and ``ops.linear`` on CPU tensors is the layers' own calls."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest
import torch

from miniattn import _lib, ops

HEADER = Path(__file__).resolve().parent.parent / "include" / "miniattn.h"


def test_struct_layouts_match_c(tmp_path):
    pairs = [("MiniAttnLinearOut", _lib.LinearOut), ("MiniAttnLinearParams", _lib.LinearParams)]
    lines = ['#include <stdio.h>', '#include <stddef.h>', f'#include "{HEADER}"', "int main(void){"]
    for name, mirror in pairs:
        lines.append(f'printf("%zu\\n", sizeof({name}));')
        lines += [f'printf("%zu\\n", offsetof({name}, {f[0]}));' for f in mirror._fields_]
    src = tmp_path / "layout.c"
    src.write_text("\n".join(lines + ["return 0;}"]))
    subprocess.run(["gcc", "-std=c99", "-Wall", "-Werror", str(src), "-o", str(tmp_path / "layout")], check=True)
    out = iter(subprocess.run([str(tmp_path / "layout")], check=True, capture_output=True, text=True).stdout.split())
    for name, mirror in pairs:
        assert int(next(out)) == C.sizeof(mirror), name
        for f in mirror._fields_:
            assert int(next(out)) == getattr(mirror, f[0]).offset, (name, f[0])


def _call(**kw):
    p = _lib.LinearParams(0x1000, 0, 64, 32, 64, 1, 1)
    p.out[0] = (0x1000, None, 0x1000, 64, 64, 64)
    for k, v in kw.items():
        setattr(p.out[0] if hasattr(p.out[0], k) else p, k, v)
    return _lib.lib.miniattn_linear(C.byref(p), None)


def test_bad_calls_are_refused():
    for kw in (dict(K=60), dict(M=-1), dict(N=12), dict(N=0), dict(n_out=4), dict(n_out=0), dict(x=0x1008), dict(w=None),
               dict(y=0x1004), dict(ldx=60), dict(ldx=56), dict(ldw=32), dict(ldy=63), dict(bias=0x1001)):
        assert _call(**kw) == _lib.EINVAL, kw
    assert _call(dtype=2) == _lib.EUNSUPPORTED
    top = 2 ** 31 - 8
    assert _call(N=top, ldy=top) == _lib.EUNSUPPORTED  # a tile's last columns would pass 2^31
    assert _call(M=0) == _lib.OK                      # nothing to do, no device asked for


def test_cpu_tensors_go_through_the_layers():
    layers = [torch.nn.Linear(16, n) for n in (8, 24)]
    x = torch.randn(3, 5, 16)
    for y, layer in zip(ops.linear(x, *layers), layers):
        assert torch.equal(y, layer(x)) and y.requires_grad


def _layer(bias=True):
    return torch.nn.Linear(16, 8, bias=bias).half().requires_grad_(False)


def _taken(layer):
    return ops._operands(layer, 16, torch.float16, -1, True) is not None   # -1: the CPU's device index


def _bias_as(kind):
    layer = _layer()
    bias = layer.bias.detach().clone()
    if kind == "shadowed":
        layer.__dict__["bias"] = bias
        return layer
    del layer.bias
    if kind == "buffer":
        layer.register_buffer("bias", bias)
    elif kind == "attribute":
        layer.bias = bias
    return layer


def test_plain_layers_are_taken():
    layer = _layer()
    assert _taken(layer) and _taken(_layer(bias=False))
    assert ops._operands(layer, 16, torch.float16, -1, True) == (layer.weight.data_ptr(), layer.bias.data_ptr(), 8)
    assert ops._operands(_layer(bias=False), 16, torch.float16, -1, True)[1:] == (0, 8)


def test_packed_block_has_the_layout_of_the_mirror():
    one, two = (1, 2, 3, 4, 5, 6, 0), (11, 0, 13, 14, 15, 16, 0)
    p = _lib.LinearParams.from_buffer_copy(ops._pack_linear(21, 22, 23, 24, 25, 1, 2, 1, 0, *one, *two, *ops._no_output))
    assert (p.x, p.status, p.ldx, p.M, p.K, p.dtype, p.n_out, p.only_if_faster) == (21, 22, 23, 24, 25, 1, 2, 1)
    assert [(o.w, o.bias, o.y, o.ldw, o.ldy, o.N) for o in p.out] == [(1, 2, 3, 4, 5, 6), (11, None, 13, 14, 15, 16),
                                                                       (None, None, None, 0, 0, 0)]


@pytest.mark.parametrize("kind", ["buffer", "attribute", "missing", "shadowed"])
def test_a_bias_that_is_no_parameter_is_left_to_the_layer(kind):
    assert not _taken(_bias_as(kind))


@pytest.mark.parametrize("make", [
    torch.jit.script, lambda layer: torch.jit.trace(layer, torch.randn(2, 16).half()), torch.nn.Sequential,
    lambda layer: type("Own", (torch.nn.Linear,), {})(16, 8).half().requires_grad_(False), lambda layer: layer.forward,
], ids=["scripted", "traced", "wrapped", "subclass", "function"])
def test_other_callables_are_left_to_themselves(make):
    assert not _taken(make(_layer()))


@pytest.mark.parametrize("owner,name", [(torch.nn.Linear, "forward"), (torch.nn.Linear, "__call__"),
                                        (torch.nn.Module, "__call__"), (torch.nn.functional, "linear")])
def test_a_replaced_call_of_every_linear_layer_is_seen(owner, name, monkeypatch):
    assert ops._nobody_watches()
    was = getattr(owner, name)
    monkeypatch.setattr(owner, name, lambda *args, **kw: was(*args, **kw))
    assert not ops._nobody_watches()


def test_a_weight_of_more_rows_than_the_kernel_counts_is_left_to_the_layer():
    layer = torch.nn.Linear(16, 8, bias=False, device="meta", dtype=torch.float16).requires_grad_(False)
    assert _taken(layer)
    for rows in (2 ** 31 - 8, 2 ** 32 + 8):
        layer.weight = torch.nn.Parameter(torch.empty(rows, 16, device="meta", dtype=torch.float16), requires_grad=False)
        assert not _taken(layer)


# Sizes at the ends of the ranges, where sums of them do not fit 32 bits, and where the one launch pays.
TOP = 2 ** 31 - 1
ENDS = [(TOP, 64, 64), (8, 64, TOP - 7), (64, TOP - 7, 8), (1, 8, 8)]
PAYS = [
    ((64, TOP - 7, 8), 0), ((64, TOP - 7, 8, 8), 0),    # a tile of 2^31 columns of K would outlast the bounded waits
    ((2048, 2048, 2048, 1024), 1), ((512, 512, 512, 256), 1), ((2277, 1536, 1536, 1536, 1536), 1), ((700, 3072, 3072, 3072, 3072), 1),
    ((4768, 2048, 2048, 1024), 1),             # q = 1.03, 12 MB of weights
    ((4096, 4096, 4096, 2048), 0),             # q = 1.02, 50 MB
    ((1554, 3072, 3072, 2048), 0), ((804, 4096, 4096, 4096), 0),   # q = 1.09, 1.20
    ((361, 4096, 4096, 1024), 1),              # q = 1.13, 20000 clk
    ((2048, 2048, 2048), 1), ((512, 512, 512), 1), ((16384, 64, 64), 1),     # one weight: where it is short
    ((4096, 4096, 4096), 0), ((8192, 2048, 2048), 0), ((16384, 4096, 4096), 0),
]
RULE = r"""
#include <cuda_runtime.h>
#include "linear.cuh"
#include <cstdio>
int main() {
  const int shapes[][5] = {%s};
  for (auto& s : shapes) {
    int n = 1;
    while (n < 3 && s[2 + n] > 0) ++n;
    bool pays = false;
    const int w = ma::linear_tile(s[0], s[1], n, &s[2], 74, &pays);
    std::printf("%%d %%d ", w, pays ? 1 : 0);
  }
  return 0;
}
"""


def _rule(tmp_path, shapes):
    src = tmp_path / "rule.cpp"
    src.write_text(RULE % ", ".join("{%s}" % ", ".join(map(str, s)) for s in shapes))
    csrc = HEADER.parent.parent / "mini-attention_b200" / "csrc"
    subprocess.run(["g++", "-std=c++17", f"-I{csrc}", "-I/usr/local/cuda/include", str(src), "-o", str(tmp_path / "rule")],
                   check=True)
    got = subprocess.run([str(tmp_path / "rule")], check=True, capture_output=True, text=True).stdout.split()
    return [int(t) for t in got[::2]], [int(t) for t in got[1::2]]


def _width(m, k, n):
    """The same rule in whole numbers of any size."""
    clk = {w: -(-(-(-m // 256) * -(-n // w)) // 74) * (max(w // 2, 48) * -(-k // 16) + 1500) for w in range(256, 63, -16)}
    return min(clk, key=clk.get)


needs_headers = pytest.mark.skipif(not Path("/usr/local/cuda/include/cuda.h").exists(), reason="no CUDA headers")


@needs_headers
def test_tile_width_at_the_ends_of_the_ranges(tmp_path):
    assert _rule(tmp_path, ENDS)[0] == [_width(*s) for s in ENDS]


@needs_headers
def test_where_one_launch_pays(tmp_path):
    assert _rule(tmp_path, [s for s, _ in PAYS])[1] == [want for _, want in PAYS]
