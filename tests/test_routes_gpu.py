"""Edges of the rules that pick a kernel by size: both sides give the same bits."""
import numpy as np
import pytest
import torch

import ojasx_b200
from ojasx_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,M,batch", [(512, 12288, 1), (512, 12289, 1), (640, 6144, 2), (640, 6145, 2), (512, 32768, 1)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_linear_cluster_and_persistent_kernels_meet(cuda, monkeypatch, K, M, batch, dtype):
    """A single small problem leaves the cluster kernel above 12288 rows x vectors."""
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "-1")
    layer = ops.VQLinear.from_weights(synth.make_vq_linear(M, K, M, block_dim=8, with_scales=True, with_bias=True))
    x = torch.randn(batch, K, device=cuda, generator=torch.Generator(cuda).manual_seed(M)).to(dtype)
    got = layer(x)
    monkeypatch.setenv("OJASX_B200_LINEAR_KERNEL", "persistent")
    assert torch.equal(layer(x), got)


@pytest.mark.parametrize("T,E,H,k", [
    (8, 33, 64, 4),        # one expert per warp, a ragged last block
    (37, 512, 520, 10),    # two, ragged tokens, a tile tail of eight columns
    (300, 512, 1000, 12),  # four
    (300, 500, 96, 40),    # four, ragged experts, more choices than lanes
    (3, 512, 256, 10), (1, 8, 64, 8),
])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_router_batches_against_oracle(cuda, oracle, T, E, H, k, dtype):
    """Logits by tiles of tokens and the four-warp top-k: indices and weights of the oracle, whatever the alignment of x."""
    w = synth.make_vq_moe(T + E, E, H, 64, block_dim=8, outlier_frac=0)
    x = torch.randn(T * H + 1, device=cuda, generator=torch.Generator(cuda).manual_seed(E)).to(dtype)
    moe = ops.VQMoE(w)
    for xt in (x[:-1].view(T, H), x[1:].view(T, H)):
        idx, wts = moe.route(xt, k)
        want_idx, want_w = oracle.router_topk(xt.float().cpu().numpy(), w.router, k)
        assert np.array_equal(idx.cpu().numpy(), want_idx) and np.array_equal(wts.cpu().numpy(), want_w)


@pytest.mark.parametrize("rows,hidden", [(1, 4096), (2, 4097), (3, 255)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_rmsnorm_register_limit(cuda, rows, hidden, dtype):
    """Rows at and beyond what a thread keeps in registers."""
    x = torch.randn(rows, hidden, device=cuda).to(dtype)
    add = torch.randn(rows, hidden, device=cuda).to(dtype)
    w = torch.randn(hidden, device=cuda)
    xs = x.clone()
    got = ops.rmsnorm(xs, w, 1e-6, add=add)
    s = (x.float() + add.float()).to(dtype)
    want = s.double() * torch.rsqrt(s.double().pow(2).mean(-1, keepdim=True) + 1e-6) * w.double()
    assert torch.equal(xs, s)
    # sums of up to 4097 squares in fp32 in a tree of 256 threads, one rounding to the output type
    tol = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    assert torch.all((got.double() - want).abs() <= tol * want.abs() + 1e-6)


@pytest.mark.parametrize("K,M,batch,gather", [
    (1024, 3456, 8, False), (1024, 3456, 16, False), (1024, 8192, 31, True),     # narrow: the tables win up to many vectors
    (2560, 8192, 2, True), (2560, 16384, 2, False), (2560, 16384, 16, True),     # many rows, few vectors
    (2560, 2304, 4, False), (2560, 2432, 4, True),                               # three million pairs
    (1600, 2048, 8, True),                                                       # not whole 128 dimensions
    (4096, 4096, 2, True),                                                       # against the cluster kernel
])
def test_linear_tables_and_gathered_operands_meet(cuda, monkeypatch, K, M, batch, gather):
    """The rule that gives a bf16 layer to one kernel or the other, and the bits of both."""
    layer = ops.VQLinear.from_weights(synth.make_vq_linear(K + M, K, M, block_dim=8))
    x = torch.randn(batch, K, device=cuda, generator=torch.Generator(cuda).manual_seed(M)).bfloat16()
    n0 = ojasx_b200.launch_count()
    got = layer(x)
    assert ojasx_b200.launch_count() - n0 == (2 if gather else 1)
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "-1" if gather else "0")
    assert torch.equal(layer(x), got)
