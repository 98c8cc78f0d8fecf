"""Merge kernel and launchers: the merge kernel against the oracle's merge, the ring driver with
all ranks emulated on one device (same schedule, kernels and merges as the multi-process ring, no
communication), config 5 at its full size against the row-sampled oracle, shard mode run rank
after rank, and -- where the box has two GPUs or more -- the real NCCL ring and shard launchers
as one process per GPU."""
import os
import subprocess
import sys
from pathlib import Path

import pytest
import torch

import miniattn
from miniattn import parallel as par
from conftest import TOL
from oracle.attention_oracle import attention_reference, attention_reference_rows, make_inputs, merge_partials

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 128])
def test_merge_kernel_matches_oracle(dtype, D):
    g = torch.Generator().manual_seed(D)
    rows = (3, 5, 77)  # 1155 rows: not a multiple of the rows per block
    acc_o = torch.randn(*rows, D, generator=g)
    acc_lse = torch.randn(*rows, generator=g) * 4
    part_o = torch.randn(*rows, D, generator=g).to(dtype)
    part_lse = torch.randn(*rows, generator=g) * 4
    acc_lse[0, 0, :5] = float("-inf")      # empty running result
    part_lse[0, 1, :5] = float("-inf")     # empty partial
    acc_lse[0, 2, :5] = float("-inf")
    part_lse[0, 2, :5] = float("-inf")     # both empty -> zeros, -inf
    ref_o, ref_lse = merge_partials(acc_o, acc_lse, part_o, part_lse)
    a_o, a_l = acc_o.to(DEV), acc_lse.to(DEV)
    out = torch.empty(*rows, D, dtype=dtype, device=DEV)
    miniattn.merge_partials(a_o, a_l, part_o.to(DEV), part_lse.to(DEV), out=out)
    assert (a_o.cpu() - ref_o).abs().max().item() < 1e-5
    fin = torch.isfinite(ref_lse)
    assert torch.equal(torch.isfinite(a_l.cpu()), fin)
    assert (a_l.cpu()[fin] - ref_lse[fin]).abs().max().item() < 1e-5
    # `out` is the merged value rounded to the 16-bit dtype: within one rounding step of it
    rel = 2.0 ** (-10 if dtype == torch.float16 else -7)
    assert bool(((out.float().cpu() - ref_o).abs() <= rel * ref_o.abs().clamp_min(1.0)).all())
    # init=True overwrites the accumulators with the partial
    miniattn.merge_partials(a_o, a_l, part_o.to(DEV), part_lse.to(DEV), init=True)
    assert torch.equal(a_o.cpu(), part_o.float()) and torch.equal(a_l.cpu(), part_lse)


@pytest.mark.parametrize("fused", [True, False])
@pytest.mark.parametrize("world", [1, 2, 4, 8])
def test_ring_emulated_on_gpu_scaled_down_config5(world, fused):
    """Config 5 scaled to N=8192 (B=1, H=4, D=128, fp16, causal): the ring result must agree
    with the single-launch kernel and with the exact oracle on sampled rows.  fused: the running
    state is carried inside the attention kernel; otherwise 16-bit partials + the merge kernel."""
    N = 8192
    q, k, v = make_inputs(1, 4, 4, N, N, 128, torch.float16, seed=5)
    qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
    out = par.ring_forward_emulated(qd, kd, vd, world, causal=True, fused=fused).cpu()
    single = miniattn.flash_attn_fwd(qd, kd, vd, causal=True).cpu()
    assert miniattn.device_status(DEV) == 0
    assert (out.float() - single.float()).abs().max().item() <= TOL[torch.float16]
    L = N // (2 * world)
    rows = torch.tensor(sorted({0, 1, L - 1, L, L + 1, N // 2 - 1, N // 2, N - L - 1, N - L, N - 1}
                               | set(torch.randint(0, N, (64,), generator=torch.Generator().manual_seed(world)).tolist())))
    ref = attention_reference_rows(q, k, v, rows, causal=True)
    assert (out[:, :, rows].float() - ref).abs().max().item() <= TOL[torch.float16]


@pytest.mark.parametrize("fused", [True, False])
def test_ring_emulated_non_causal_bf16_gqa(fused):
    q, k, v = make_inputs(1, 4, 2, 2048, 2048, 64, torch.bfloat16, seed=8)
    out = par.ring_forward_emulated(q.to(DEV), k.to(DEV), v.to(DEV), 4, causal=False, fused=fused).cpu()
    ref = attention_reference(q, k, v, out_dtype=torch.float32)
    assert (out.float() - ref).abs().max().item() <= TOL[torch.bfloat16]


def test_config5_full_size_rows():
    """Config 5 at its stated size -- causal MHA fp16, B=1, H=32, N=131072, D=128 -- through the
    ring schedule of 8 ranks (zig-zag blocks of L=8192 tokens, every rank's steps run one after
    the other on this device).  The full oracle is out of reach on a CPU (64 GiB of scores per
    head), so 288 query rows per head are computed exactly against all their keys: row 0, every
    block boundary and its two neighbours, N-1, and seeded random rows.  Bar: 2e-3."""
    B, H, N, D, W = 1, 32, 131072, 128, 8
    L = N // (2 * W)
    g = torch.Generator().manual_seed(0)
    q = torch.randn(B, H, N, D, generator=g, dtype=torch.float32).half()
    k = torch.randn(B, H, N, D, generator=g, dtype=torch.float32).half()
    v = torch.randn(B, H, N, D, generator=g, dtype=torch.float32).half()
    out = par.ring_forward_emulated(q.to(DEV), k.to(DEV), v.to(DEV), W, causal=True)
    assert miniattn.device_status(DEV) == 0
    rows = {0, N - 1}
    for blk in range(1, 2 * W):
        rows |= {blk * L - 1, blk * L, blk * L + 1}
    extra = torch.randint(0, N, (512,), generator=torch.Generator().manual_seed(5)).tolist()
    for r in extra:
        if len(rows) >= 288:
            break
        rows.add(r)
    rows = torch.tensor(sorted(rows))
    assert rows.numel() >= 256
    got = out[:, :, rows.to(DEV)].float().cpu()
    del out
    ref = attention_reference_rows(q, k, v, rows, causal=True)
    assert (got - ref).abs().max().item() <= TOL[torch.float16]


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs or more (one process per GPU)")
def test_nccl_ring_and_shards_multi_process():
    """The real thing: one process per GPU, K/V pairs over NCCL send/recv, origin tags verified,
    ring output against the single-launch kernel and the CPU oracle, shard mode all-reduced
    against the full computation (tests/multi_gpu_ring_check.py prints a line per rank)."""
    n = min(torch.cuda.device_count(), 8)
    n = 1 << (n.bit_length() - 1)   # 2, 4 or 8 ranks
    root = Path(__file__).resolve().parent.parent
    env = dict(os.environ, NCCL_NVLS_ENABLE="0")
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={n}",
           "--master-addr", "127.0.0.1", "--master-port", "29517",
           str(root / "tests" / "multi_gpu_ring_check.py"), "--seq-len", "16384"]
    r = subprocess.run(cmd, stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=900, env=env)
    print(r.stdout[-4000:])
    assert r.returncode == 0, r.stdout[-4000:]
    assert "multi-GPU check passed" in r.stdout


def test_shard_mode_rank_by_rank():
    q, k, v = make_inputs(2, 8, 2, 512, 512, 128, torch.bfloat16, seed=2)
    qd, kd, vd = q.to(DEV), k.to(DEV), v.to(DEV)
    out = torch.zeros_like(qd)
    for r in range(4):
        par.sharded_forward(qd, kd, vd, causal=True, rank=r, world=4, out=out)
    ref = attention_reference(q, k, v, causal=True, out_dtype=torch.float32)
    assert (out.float().cpu() - ref).abs().max().item() <= TOL[torch.bfloat16]


@pytest.mark.parametrize("N,world", [(1600, 2), (3072, 4), (2560, 2)])
def test_ring_emulated_block_lengths(N, world):
    """Block lengths that are and are not multiples of the 128-row tile: with whole tiles the two
    resident blocks share one state buffer and a step's block pairs merge into one launch; without,
    every block keeps its own state and every pair its own launch.  Same result either way."""
    q, k, v = make_inputs(1, 2, 1, N, N, 128, torch.float16, seed=N)
    out = par.ring_forward_emulated(q.to(DEV), k.to(DEV), v.to(DEV), world, causal=True).cpu()
    ref = attention_reference(q, k, v, causal=True, out_dtype=torch.float32)
    assert miniattn.device_status(DEV) == 0
    assert (out.float() - ref).abs().max().item() <= TOL[torch.float16]


@pytest.mark.parametrize("causal", [False, True])
def test_ring_of_one_takes_its_own_rows_of_a_longer_kv(causal):
    """One rank whose K/V tensors go on behind its 2 L tokens: the rows see the two blocks and nothing after them,
    as on any rank."""
    q, k, v = make_inputs(1, 2, 2, 300, 364, 128, torch.float16, seed=7)
    out = par.ring_forward(q.to(DEV), k.to(DEV), v.to(DEV), causal=causal).cpu()
    ref = attention_reference(q, k[:, :, :300], v[:, :, :300], causal=causal, out_dtype=torch.float32)
    assert (out.float() - ref).abs().max().item() <= TOL[torch.float16]
    assert miniattn.device_status(DEV) == 0
