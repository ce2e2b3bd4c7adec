"""A handful of routed pairs: the kernels that gather first and add afterwards give the bits of the row-per-lane kernels, at the edges
of their table blocks (16 groups), pieces of work (8 groups, 32 rows), outlier passes (4096 products) and item tiles."""
import numpy as np
import pytest
import torch

import ojasx_b200
from ojasx_b200 import ops, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,I,E,k,B,frac,D", [
    (64, 8, 3, 1, 1, 0.05, 8),        # half a block of table; one down group; one output row an item
    (192, 64, 4, 3, 2, 0.0, 8),       # one and a half blocks; no outliers
    (1088, 320, 5, 4, 3, 0.01, 8),    # eight and a half blocks, 40 down groups
    (2560, 640, 12, 10, 1, 0.0038, 8),
    (2560, 640, 12, 10, 2, 0.01, 8),  # two waves of items
    (2560, 640, 3, 2, 1, 0.1, 8),     # one block of rows (18 rows), twenty table blocks; two passes of outlier products
    (2560, 256, 6, 4, 1, 0.01, 8),    # one block of rows (14), twenty table blocks
    (2560, 1280, 3, 1, 1, 0.01, 8),   # one block of rows in both passes (18), ten down blocks
    (2560, 576, 6, 4, 1, 0.0, 8),     # one block of rows, full (32)
    (1152, 256, 4, 3, 1, 0.01, 8),    # one block of rows, nine table blocks
    (4096, 128, 4, 2, 2, 0.01, 8),    # one block of rows (8), 32 table blocks, a ring of twelve
    (2560, 640, 12, 8, 8, 0.01, 8),   # the values do not fit: row-per-lane
    (1024, 256, 6, 5, 1, 0.01, 4),
    (1024, 512, 6, 5, 2, 0.01, 16),
    (2048, 1024, 6, 3, 1, 0.01, 32),
])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_few_pairs(cuda, oracle, monkeypatch, H, I, E, k, B, frac, D, dtype):
    w = synth.make_vq_moe(H + I, E, H, I, block_dim=D, outlier_frac=frac, unit_scales=(frac == 0.0))
    rng = np.random.default_rng(E + B)
    x = torch.from_numpy(rng.standard_normal((B, H)).astype(np.float32)).to(cuda)
    idx = np.stack([rng.choice(E, size=k, replace=False) for _ in range(B)]).astype(np.int32)
    wts = rng.uniform(0.02, 0.3, size=(B, k)).astype(np.float32)
    if k > 2:
        idx[0, 0], wts[B - 1, 1] = E, 5e-9        # skipped pairs
    if dtype == "bf16":
        x = x.bfloat16()
        monkeypatch.setenv("OJASX_B200_MOE_GATHER_MIN_PAIRS", str(1 << 30))
    args = [x, torch.from_numpy(idx).to(cuda), torch.from_numpy(wts).to(cuda)]
    moe = ops.VQMoE(w)
    half = ops.VQMoE(w, (E // 2, E))               # holds some of the experts only
    bad = x.clone()
    bad[0, 5], bad[0, 9], bad[B - 1, H - 1] = float("inf"), float("-inf"), float("nan")

    def all_ways():
        out = [moe.forward(*args), moe.forward_routed(x, k), half.forward(*args), moe.forward(bad, *args[1:])]
        moe.set_gate_limit(0.05)
        out.append(moe.forward(*args))
        moe.set_gate_limit(0.0)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):              # the launches' overlap, replayed back to back
            y = moe.forward_routed(x, k)
            y2 = moe.forward_routed(y, k)
        for _ in range(3):
            graph.replay()
        return out + [y.clone(), y2.clone()]

    few = all_ways()
    monkeypatch.setenv("OJASX_B200_MOE_FEW", "0")
    rows = all_ways()
    for a, b in zip(few, rows):
        assert torch.equal(torch.isnan(a), torch.isnan(b)) and torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
    assert torch.equal(few[1], few[5])
    assert ojasx_b200.lib().ojasx_b200_take_device_error() == 0
