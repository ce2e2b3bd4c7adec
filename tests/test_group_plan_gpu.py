"""Grouped launches with more layers than SMs: how the layers are cut into work items does not change a bit."""
import numpy as np
import pytest
import torch

import ojasx_b200
from ojasx_b200 import ops, synth

pytestmark = pytest.mark.gpu


def test_grouped_layers_cut_for_the_last_wave(cuda, oracle):
    """More layers than SMs: those of the last, incomplete wave are cut into tiles.  Mixed row counts, a single row range
    for all members, and a count that leaves one layer over."""
    K, D = 256, 8
    rows = [1100, 2000, 515, 1600]
    ws = [synth.make_vq_linear(800 + i, K, m, block_dim=D, outlier_frac=0.01) for i, m in enumerate(rows)]
    layers = [ops.VQLinear.from_weights(w) for w in ws]
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for count in (sms + 1, 2 * sms + 30):
        group = ops.VQLinearGroup([layers[i % 4] for i in range(count)])
        x = np.random.default_rng(count).standard_normal((count, K)).astype(np.float32)
        xt = torch.from_numpy(x).to(cuda)
        y = torch.zeros((count, max(rows)), device=cuda)
        group.forward(xt, y)
        y = y.cpu().numpy()
        for i, w in enumerate(ws):
            want = oracle.linear_forward(w.codebook, w.codes, w.scales, w.bias, w.csr, x[i::4], block_dim=D)
            assert np.array_equal(y[i::4, :rows[i]], want) and not y[i::4, rows[i]:].any()
        lib = ojasx_b200.lib()
        assert lib.ojasx_b200_linear_group_set_rows(group._g, 515, 600) == -1   # one member has no such rows: refused,
        z = torch.zeros(count, max(rows), device=cuda)
        group.forward(xt, z)                                                           # and the group is as it was
        assert np.array_equal(z.cpu().numpy(), y)
