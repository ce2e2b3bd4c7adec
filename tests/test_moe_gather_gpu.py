"""Experts that several tokens are routed to: weights gathered into mma.sync operands (bf16), against the CPU oracle."""
import numpy as np
import pytest
import torch

import ojasx_b200
from ojasx_b200 import ops, synth

pytestmark = pytest.mark.gpu

RTOL, ATOL = 2.0 ** -8, 1e-5     # one rounding to bf16 of an fp32 sum (half an ulp is at most 2^-8 of the value)


def _oracle_moe(oracle, w, x, idx, wts):
    return np.stack([oracle.moe_forward(w.codebook, w.down_codebook, w.gate_up_codes, w.gate_up_scales, w.down_codes, w.down_scales,
                                        x[t], idx[t], wts[t], block_dim=w.block_dim, gu_csr=w.gate_up_csr, dn_csr=w.down_csr)
                     for t in range(x.shape[0])])


@pytest.fixture(autouse=True)
def gather_everywhere(monkeypatch):
    monkeypatch.setenv("OJASX_B200_MOE_GATHER_MIN_PAIRS", "1")


def _args(x, idx, wts, dtype=torch.bfloat16):
    return torch.from_numpy(x).to("cuda").to(dtype), torch.from_numpy(idx).to("cuda"), torch.from_numpy(wts).to("cuda")


@pytest.mark.parametrize("H,I,E,k,B", [
    (64, 64, 3, 2, 5),           # one partial chunk on both sides; fewer units than warps
    (256, 128, 8, 4, 33),        # items of eight, and of every smaller size
    (1088, 192, 5, 3, 20),       # G = 136, Gi = 24: eight-byte code loads, tails of eight groups
    (2560, 640, 16, 10, 12),     # benchmark geometry
    (256, 128, 2, 2, 41),        # items of sixteen pairs, the last one of nine
    (2560, 640, 4, 1, 1),        # a single pair
])
@pytest.mark.parametrize("frac", [0.0, 0.01])
def test_gather_experts_against_oracle(cuda, oracle, monkeypatch, H, I, E, k, B, frac):
    w = synth.make_vq_moe(H + B, E, H, I, block_dim=8, outlier_frac=frac, unit_scales=(frac == 0.0))
    rng = np.random.default_rng(E * B)
    x = synth.to_bf16_f32((rng.standard_normal((B, H)) * 2.0 ** rng.integers(-2, 2, (B, 1))).astype(np.float32))
    idx = np.stack([rng.choice(E, size=k, replace=False) for _ in range(B)]).astype(np.int32)
    wts = rng.uniform(0.02, 0.3, size=(B, k)).astype(np.float32)
    if B > 2:
        idx[1, 0], idx[2, k - 1], wts[0, k - 1] = -1, E, 5e-9     # skipped pairs
    moe = ops.VQMoE(w)
    args = _args(x, idx, wts)
    n0 = ojasx_b200.launch_count()
    got = moe.forward(*args)
    assert ojasx_b200.launch_count() - n0 == 6      # work list, tokens, gate/up, intermediate vectors, down, combine
    want = _oracle_moe(oracle, w, x, idx, wts)
    err = np.abs(got.float().cpu().numpy() - want)
    assert np.all(err <= ATOL + RTOL * np.abs(want)), err.max()
    assert torch.equal(moe.forward(*args), got)     # whatever order the pairs of an expert are listed in
    lo, hi = ops.VQMoE(w, (0, E // 2)), ops.VQMoE(w, (E // 2, E))
    assert np.allclose((lo.forward(*args).float() + hi.forward(*args).float()).cpu().numpy(), want, rtol=0,
                       atol=2 * RTOL * np.abs(want).max() + ATOL)     # each half rounded once
    monkeypatch.setenv("OJASX_B200_MOE_GATHER_MIN_PAIRS", "1000000")
    table = moe.forward(*args).float()              # the table kernels: another order of the sums, the same rounding
    moe.set_gate_limit(0.05)
    clamped_table = moe.forward(*args).float()
    monkeypatch.setenv("OJASX_B200_MOE_GATHER_MIN_PAIRS", "1")
    clamped = moe.forward(*args).float()
    for a, b in ((got.float(), table), (clamped, clamped_table)):
        assert torch.all((a - b).abs() <= 2.0 ** -7 * b.abs() + ATOL) and (a != b).float().mean() < 0.01
    f32 = moe.forward(*_args(x, idx, wts, torch.float32))      # fp32 keeps the table kernels, whose order is the oracle's
    moe.set_gate_limit(0.0)
    assert f32.dtype == torch.float32
    err = np.abs(moe.forward(*_args(x, idx, wts, torch.float32)).cpu().numpy() - want)
    assert np.all(err <= 1e-6 + 1e-5 * np.abs(want))


def test_gather_experts_routed_call_and_non_finite_tokens(cuda, monkeypatch):
    """The router in front, and tokens with infinities or NaN: they give what the table kernels give, others are untouched."""
    w = synth.make_vq_moe(5, 8, 512, 128, block_dim=8, outlier_frac=0.01, unit_scales=False)
    x = torch.randn(24, 512, device=cuda, generator=torch.Generator(cuda).manual_seed(1)).bfloat16()
    moe = ops.VQMoE(w)
    idx, wts = moe.route(x, 3)
    clean = moe.forward(x, idx, wts)
    assert torch.equal(moe.forward_routed(x, 3), clean)
    x[2, 7], x[9, 500], x[9, 3], x[20, 0] = float("inf"), float("-inf"), 3e38, float("nan")
    got = moe.forward(x, idx, wts)
    monkeypatch.setenv("OJASX_B200_MOE_GATHER_MIN_PAIRS", "1000000")
    table = moe.forward(x, idx, wts)
    bad = torch.zeros(24, dtype=torch.bool, device=cuda)
    bad[[2, 9, 20]] = True
    assert torch.equal(got[~bad], clean[~bad])
    assert torch.equal(torch.isnan(got[bad]), torch.isnan(table[bad])) and torch.equal(torch.isposinf(got[bad]), torch.isposinf(table[bad]))


@pytest.mark.parametrize("B", [1, 3, 5, 13])
def test_gather_experts_with_outliers_in_few_rows(cuda, oracle, B):
    """Lanes without a pair leave a unit early and lanes with a long outlier row leave it late; the warp meets again before
    the next unit's products.  Few pairs per expert and hundreds of entries in every sixteenth row, several units per warp."""
    H, I, E, k = 1024, 640, 4, 2
    w = synth.make_vq_moe(B, E, H, I, block_dim=8, outlier_frac=0.0, unit_scales=False)
    rng = np.random.default_rng(B)

    def long_rows(rows, cols):
        counts = np.where(np.arange(rows) % 16 == 5, 300, 0)
        ptr = np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)
        col = np.concatenate([np.sort(rng.choice(cols, 300, replace=False)) for _ in range(np.count_nonzero(counts))])
        return ptr, col.astype(np.int32), (rng.standard_normal(len(col)) * 0.1).astype(np.float32)

    w.gate_up_csr, w.down_csr = long_rows(E * 2 * I, H), long_rows(E * H, I)
    x = synth.to_bf16_f32(rng.standard_normal((B, H)).astype(np.float32))
    idx = np.stack([rng.choice(E, size=k, replace=False) for _ in range(B)]).astype(np.int32)
    wts = rng.uniform(0.1, 0.3, size=(B, k)).astype(np.float32)
    moe = ops.VQMoE(w)
    n0 = ojasx_b200.launch_count()
    got = moe.forward(*_args(x, idx, wts)).float().cpu().numpy()
    assert ojasx_b200.launch_count() - n0 == 6
    want = _oracle_moe(oracle, w, x, idx, wts)
    assert np.all(np.abs(got - want) <= ATOL + RTOL * np.abs(want)), np.abs(got - want).max()


@pytest.mark.parametrize("book", ["codebook", "down_codebook"])
def test_gather_experts_codebooks_of_wide_range(cuda, book):
    """A centroid that no code names, far above the others, must not cost them bits."""
    w = synth.make_vq_moe(5, 4, 512, 128, block_dim=8, outlier_frac=0.0)
    w.gate_up_codes[w.gate_up_codes == 255] = 3
    w.down_codes[w.down_codes == 255] = 3
    x = torch.randn(8, 512, device=cuda, generator=torch.Generator(cuda).manual_seed(1)).bfloat16()
    want = ops.VQMoE(w).forward_routed(x, 2).float()
    getattr(w, book)[255] = 1e30
    got = ops.VQMoE(w).forward_routed(x, 2).float()
    assert torch.all((got - want).abs() <= 2.0 ** -7 * want.abs() + ATOL)
