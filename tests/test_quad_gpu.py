"""The walk of four vectors at a time (fp32 linears of a batch, MoE layers that route several tokens to an expert): bit-exact
against the oracle and against the kernels of one vector, at the edges of its slices (16 groups), row blocks (32 rows on
eight warps) and groups of four vectors."""
import numpy as np
import pytest
import torch

import ojasx_b200
from ojasx_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,M,batch,dtype", [
    (64, 1, 4, "f32"),          # half a slice, one row: seven of eight warps have none
    (128, 33, 5, "f32"),        # one slice; a second block of one row; a group of one vector
    (192, 255, 6, "f32"),       # 24 groups: code rows on 8-byte boundaries, half a slice at the end
    (256, 257, 7, "f32"),       # a ninth block: the first warp has two
    (2560, 515, 33, "f32"),
    (2568, 1000, 32, "f32"),    # 321 groups do not fit: the kernels of one vector
    (2624, 3201, 4, "f32"),     # two row tiles
    (4096, 2560, 40, "f32"),
    (8256, 300, 4, "f32"),      # more activations than are staged: the kernels of one vector
    (2112, 200, 604, "f32"),    # more groups of vectors than SMs: second work items behind 17 slices
    (2048, 33, 1201, "f32"),    # third ones, 16 slices
    (1280, 700, 9, "bf16"),
])
def test_linear_batches(cuda, oracle, monkeypatch, K, M, batch, dtype):
    w = synth.make_vq_linear(K + M, K, M, block_dim=8, outlier_frac=0.01, with_scales=M % 2 == 0, with_bias=M % 3 == 0)
    x = np.random.default_rng(batch).standard_normal((batch, K)).astype(np.float32)
    if dtype == "bf16":
        x = synth.to_bf16_f32(x)
    want = oracle.linear_forward(w.codebook, w.codes, w.scales, w.bias, w.csr, x, block_dim=8)
    layer = ops.VQLinear.from_weights(w)
    xt = torch.from_numpy(x).to(cuda)
    if dtype == "bf16":
        xt = xt.bfloat16()
        want = synth.to_bf16_f32(want)
        monkeypatch.setenv("OJASX_B200_TENSOR_MIN_BATCH", "0")
        monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "-1")
    monkeypatch.setenv("OJASX_B200_QUAD_MIN_BATCH", "3")
    got = layer(xt).float().cpu().numpy()
    assert np.array_equal(got, want), np.abs(got - want).max()
    if M > 64:   # a run of rows in the middle
        assert np.array_equal(layer(xt, 31, M - 7).float().cpu().numpy(), want[:, 31:M - 7])
    assert ojasx_b200.lib().ojasx_b200_take_device_error() == 0


def test_linear_special_values(cuda, oracle, monkeypatch):
    """Infinities, NaN and sums of exactly -0 travel as they do in the kernels of one vector; a short codebook; no outliers."""
    w = synth.make_vq_linear(5, 320, 300, block_dim=8, outlier_frac=0.0)
    book, codes = w.codebook[:16].copy(), (w.codes % 16).astype(np.uint8)
    codes[7] = 3
    book[3] = 0.0
    x = np.random.default_rng(1).standard_normal((6, 320)).astype(np.float32)
    x[1] = -np.abs(x[1])           # products with +0: entries of -0
    x[2, 11], x[3, 300], x[4, 0] = np.inf, np.nan, -np.inf
    layer = ops.VQLinear(book, codes, None, None, None, block_dim=8, codebook_size=16)
    xt = torch.from_numpy(x).to(cuda)
    monkeypatch.setenv("OJASX_B200_QUAD_MIN_BATCH", "1000")
    one = layer(xt).cpu().numpy()
    monkeypatch.setenv("OJASX_B200_QUAD_MIN_BATCH", "3")
    four = layer(xt).cpu().numpy()
    assert np.array_equal(np.isnan(one), np.isnan(four))
    ok = ~np.isnan(one)
    assert np.array_equal(one.view(np.int32)[ok], four.view(np.int32)[ok])


@pytest.mark.parametrize("H,I,E,k,B,frac", [
    (256, 64, 4, 3, 9, 0.01),       # eight groups in the down codes; 128 gate/up rows
    (1280, 320, 8, 4, 30, 0.01),    # 40 groups in the down codes (8-byte boundaries), two and a half slices
    (2560, 640, 16, 10, 24, 0.0),
    (2560, 640, 16, 10, 25, 0.0038),
    (3584, 512, 6, 2, 31, 0.01),    # more hidden rows than a tile holds
    (2816, 64, 160, 2, 200, 0.01),  # more groups of pairs than SMs: whole rounds, of two tiles of hidden rows; 22 slices and one
    (1152, 320, 320, 4, 200, 0.003),   # two whole rounds and a rest; nine slices and three
])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_moe_batches(cuda, oracle, monkeypatch, H, I, E, k, B, frac, dtype):
    w = synth.make_vq_moe(H + I, E, H, I, block_dim=8, outlier_frac=frac, unit_scales=(frac == 0.0))
    rng = np.random.default_rng(E + B)
    x = rng.standard_normal((B, H)).astype(np.float32)
    idx = np.stack([rng.choice(E, size=k, replace=False) for _ in range(B)]).astype(np.int32)
    wts = rng.uniform(0.02, 0.3, size=(B, k)).astype(np.float32)
    idx[1, 0], idx[2, k - 1], wts[0, 1] = -1, E, 5e-9        # skipped pairs
    args = [torch.from_numpy(x).to(cuda), torch.from_numpy(idx).to(cuda), torch.from_numpy(wts).to(cuda)]
    if dtype == "bf16":
        args[0] = args[0].bfloat16()
        monkeypatch.setenv("OJASX_B200_MOE_GATHER_MIN_PAIRS", str(1 << 30))
    moe = ops.VQMoE(w)

    def all_ways():
        out = [moe.forward(*args), moe.forward_routed(args[0], k)]
        moe.set_gate_limit(0.05)
        out.append(moe.forward(*args))
        moe.set_gate_limit(0.0)
        return out

    monkeypatch.setenv("OJASX_B200_MOE_QUAD_MIN_PAIRS", "1")
    four = all_ways()
    shards = sum(ops.VQMoE(w, r).forward(*args).float() for r in ((0, E // 2), (E // 2, E)))
    monkeypatch.setenv("OJASX_B200_MOE_QUAD_MIN_PAIRS", str(1 << 30))
    one = all_ways()
    assert ojasx_b200.lib().ojasx_b200_take_device_error() == 0
    assert all(torch.equal(a, b) for a, b in zip(four, one))
    tol = 1e-5 if dtype == "f32" else 2 ** -7     # the halves are rounded to bf16 before they are added
    assert torch.allclose(shards, four[0].float(), rtol=tol, atol=tol * float(four[0].abs().max()))
