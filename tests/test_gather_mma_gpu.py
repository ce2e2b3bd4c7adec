"""bf16 batches below 32: weights gathered into mma.sync operands, against the fp32 oracle."""
import numpy as np
import pytest
import torch

import ojasx_b200
from ojasx_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _oracle(oracle, w, x):
    return oracle.linear_forward(w.codebook, w.codes, w.scales, w.bias, w.csr, x, block_dim=8)


def _close_once_rounded(got, want):
    """One rounding to bf16 (eight bits of significand: half an ulp is at most 2^-8 of the value) of a sum that differs
    from the oracle's by fp32 rounding: a few 1e-7 of the row's largest terms, 1e-5 where those are of order one."""
    return np.all(np.abs(got - want) <= 2.0 ** -8 * np.abs(want) + 1e-5)


@pytest.mark.parametrize("K,M,batch", [
    (512, 300, 2),
    (64, 16, 8),         # one partial chunk, one tile
    (256, 33, 9),        # one whole chunk, ragged rows
    (1088, 200, 16),     # G = 136: eight-byte code loads, an eight-group tail
    (2560, 2560, 17),
    (2560, 6912, 31),
    (6912, 2560, 16),    # K split over a cluster
    (4736, 130, 25),
])
@pytest.mark.parametrize("frac", [0.0, 0.0038])
def test_gather_mma_against_oracle(cuda, oracle, monkeypatch, K, M, batch, frac):
    w = synth.make_vq_linear(K + batch, K, M, block_dim=8, outlier_frac=frac, with_scales=True, with_bias=True)
    x = np.random.default_rng(batch).standard_normal((batch, K)).astype(np.float32)
    x *= np.float32(2.0) ** np.random.default_rng(K).integers(-20, 20, size=(batch, 1))   # every vector has its own scale
    xb = synth.to_bf16_f32(x)
    want = _oracle(oracle, w, xb)
    layer = ops.VQLinear.from_weights(w)
    xt = torch.from_numpy(xb).to(cuda).bfloat16()
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "0")
    n0 = ojasx_b200.launch_count()
    got = layer(xt).float().cpu().numpy()
    assert ojasx_b200.launch_count() - n0 == 2          # activations, rows
    size = np.abs(want).max(axis=1, keepdims=True)      # vectors of 2^-20 .. 2^20: compare at one scale
    assert _close_once_rounded(got / size, want / size)
    a, b = M // 3, M - 1                                # a row slice is the same rows
    part = layer(xt, a, b).float().cpu().numpy()
    assert _close_once_rounded(part / size, want[:, a:b] / size)
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "-1")
    table = layer(xt).float().cpu().numpy()             # the table kernels: the oracle's sums, rounded
    assert np.mean(got != table) <= 1e-5, np.mean(got != table)


def test_gather_mma_infinities_and_nan(cuda, oracle, monkeypatch):
    """A vector with an infinity or NaN is evaluated in the reference's order; its neighbours are untouched."""
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "0")
    w = synth.make_vq_linear(5, 512, 100, block_dim=8, with_scales=True)
    x = synth.to_bf16_f32(np.random.default_rng(0).standard_normal((12, 512)).astype(np.float32))
    clean = ops.VQLinear.from_weights(w)(torch.from_numpy(x).to(cuda).bfloat16()).float().cpu().numpy()
    x[1, 300], x[4, 0], x[7, 511], x[7, 3] = np.inf, np.nan, -np.inf, np.inf
    x[9] = 0.0
    got = ops.VQLinear.from_weights(w)(torch.from_numpy(x).to(cuda).bfloat16()).float().cpu().numpy()
    with np.errstate(all="ignore"):
        want = synth.to_bf16_f32(_oracle(oracle, w, x))
    for t in range(12):
        if t in (1, 4, 7):
            assert np.array_equal(got[t], want[t], equal_nan=True)
        elif t != 9:
            assert np.array_equal(got[t], clean[t])
    assert np.all(got[9] == 0)


@pytest.mark.parametrize("K,M,batch", [(2560, 6912, 16), (1088, 2112, 8), (1536, 2048, 31)])
def test_mlp_block_equals_its_layers(cuda, K, M, batch):
    ws = [synth.make_vq_linear(90 + i, *s, block_dim=8) for i, s in enumerate([(K, M), (K, M), (M, K)])]
    gate, up, down = (ops.VQLinear.from_weights(w) for w in ws)
    x = torch.randn(batch, K, device=cuda, generator=torch.Generator(cuda).manual_seed(batch)).bfloat16()
    n0 = ojasx_b200.launch_count()
    got = ops.VQMLP(gate, up, down)(x)
    assert ojasx_b200.launch_count() - n0 == 4
    want = down(ops.silu_mul(gate(x), up(x)))
    # a gate or up value whose rounding tips moves one of M terms of an output by 2^-8 of itself
    assert torch.allclose(got.float(), want.float(), rtol=2 ** -7, atol=2 ** -8 * want.float().abs().max().item() / 8)


def _table(monkeypatch, layer, x):
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "-1")
    y = layer(x).float().cpu().numpy()
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "0")
    return y


@pytest.mark.parametrize("K,M", [(64, 300), (64, 20000), (256, 300), (256, 9000), (384, 300), (384, 9000)])
@pytest.mark.parametrize("batch", [16, 31])
@pytest.mark.parametrize("fill", [0.0, float("nan")])
def test_every_listed_sum_is_stored(cuda, monkeypatch, K, M, batch, fill):
    """Narrow layers: more sums of a tile are evaluated again than the CTA has threads (all but one vector zero or NaN)."""
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "0")
    layer = ops.VQLinear.from_weights(synth.make_vq_linear(K, K, M, block_dim=8, outlier_frac=0.0))
    x = torch.full((batch, K), fill, device=cuda, dtype=torch.bfloat16)
    x[3] = torch.randn(K, device=cuda, generator=torch.Generator(cuda).manual_seed(K)).bfloat16()
    out = torch.full((batch, M), 12345.0, device=cuda, dtype=torch.bfloat16)
    n0 = ojasx_b200.launch_count()
    layer(x, out=out)
    assert ojasx_b200.launch_count() - n0 == 2
    assert np.array_equal(out.float().cpu().numpy(), _table(monkeypatch, layer, x), equal_nan=True)


def _us(f, n=20):
    for _ in range(3):
        f()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    times = []
    for _ in range(n):
        torch.cuda.synchronize()
        a.record()
        f()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) * 1e3)
    return min(times)    # the host may stall any call, but not make one faster


def test_zero_vectors_and_zero_chunks_cost_nothing_extra(cuda, monkeypatch):
    """An all-zero chunk of 256 dimensions adds nothing to a sum, so it must not widen the window in which sums are evaluated
    again.  The bits are the table kernels'; the time is that of dense vectors (a tenth of all sums evaluated again doubles it)."""
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "0")
    K, M, batch = 2560, 6912, 16
    layer = ops.VQLinear.from_weights(synth.make_vq_linear(1, K, M, block_dim=8))
    x = torch.randn(batch, K, device=cuda, generator=torch.Generator(cuda).manual_seed(1)).bfloat16()
    padded, chunk = x.clone(), x.clone()
    padded[8:] = 0
    chunk[:, 512:768] = 0
    dense = _us(lambda: layer(x))
    for v in (padded, chunk):
        took = _us(lambda: layer(v))
        assert np.array_equal(layer(v).float().cpu().numpy(), _table(monkeypatch, layer, v))
        assert took < 1.3 * dense, (took, dense)


def _kinds(rng, batch, K):
    x = rng.standard_normal((batch, K)).astype(np.float32)
    yield "gaussian", x, 0.0
    yield "one sign", np.abs(x), 1.0
    yield "constant", np.ones((batch, K), np.float32) * rng.uniform(0.5, 2, (batch, 1)).astype(np.float32), 1.0
    half = np.abs(x)
    half[:, K // 2:] *= -1
    yield "halves that cancel", half, 1.0
    yield "tiny", x * np.float32(2.0 ** -70), 0.0
    yield "tiny, one sign", np.abs(x) * np.float32(2.0 ** -90), 1.0
    yield "large", x * np.float32(2.0 ** 90), 0.0
    massive = x.copy()
    massive[:, 7] *= 3000
    yield "one massive dimension", massive, 0.0
    ramp = x * np.float32(2.0) ** np.linspace(-12, 12, K, dtype=np.float32)
    yield "chunks of different size", ramp, 0.0


@pytest.mark.parametrize("K,M,batch", [(64, 4096, 16), (2560, 4096, 16), (6912, 2560, 8)])
def test_bits_of_the_table_kernels_for_biased_data(cuda, monkeypatch, K, M, batch):
    """Sums of one sign, sums that cancel and activations of other scales: the window in which sums are formed in the table
    kernels' order has to cover what the two orders differ by."""
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "0")
    bad = {}
    for seed in range(4):
        rng = np.random.default_rng(K + seed)
        for kind, x, bias in _kinds(rng, batch, K):
            w = synth.make_vq_linear(seed, K, M, block_dim=8, outlier_frac=0.0)
            if bias:
                w.codebook[:] = np.abs(w.codebook)
            layer = ops.VQLinear.from_weights(w)
            xt = torch.from_numpy(x).to(cuda).bfloat16()
            got = layer(xt).float().cpu().numpy()
            n = int(np.count_nonzero(got != _table(monkeypatch, layer, xt)))
            bad[kind] = bad.get(kind, 0) + n
    assert not any(bad.values()), bad


@pytest.mark.parametrize("entry", [1e30, float("inf")])
def test_codebooks_of_wide_range_keep_the_table_kernels(cuda, monkeypatch, entry):
    """One entry far above the others makes every sum's window wide, so that most would be formed twice."""
    w = synth.make_vq_linear(5, 2560, 6912, block_dim=8)
    w.codes[w.codes == 255] = 3
    x = torch.randn(16, 2560, device=cuda, generator=torch.Generator(cuda).manual_seed(1)).bfloat16()
    want = ops.VQLinear.from_weights(w)(x)
    w.codebook[255] = entry                              # no code names it
    layer = ops.VQLinear.from_weights(w)
    n0 = ojasx_b200.launch_count()
    got = layer(x)
    assert ojasx_b200.launch_count() - n0 == 1           # the table kernel
    assert torch.equal(got, want)
    mlp = ops.VQMLP(layer, layer, ops.VQLinear.from_weights(synth.make_vq_linear(6, 6912, 2560, block_dim=8)))
    g = layer(x)
    assert torch.equal(mlp(x), mlp.down(ops.silu_mul(g, g)))


@pytest.mark.parametrize("K,M,batch,scratch", [(512, 512, 4, False), (2560, 6912, 2, True), (2560, 6912, 1, False)])
def test_scratch_only_where_the_gather_kernel_is_taken(cuda, monkeypatch, K, M, batch, scratch):
    """A layer too small for it launches as before, without an allocation per call; a switch set later is seen."""
    layer = ops.VQLinear.from_weights(synth.make_vq_linear(5, K, M, block_dim=8))
    x = torch.randn(batch, K, device=cuda).bfloat16()
    out = torch.empty(batch, M, device=cuda, dtype=torch.bfloat16)

    def allocations():
        n0 = torch.cuda.memory_stats()["allocation.all.allocated"]
        layer(x, out=out)
        return torch.cuda.memory_stats()["allocation.all.allocated"] - n0

    assert allocations() == int(scratch)
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "0")
    assert allocations() == int(batch > 1)
    monkeypatch.setenv("OJASX_B200_GATHER_MIN_WORK", "-1")
    assert allocations() == 0
