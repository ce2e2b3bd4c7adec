"""bf16 SwiGLU blocks on the tensor cores: gate and up in one launch where their tiles fit the SMs, any number of splits along K,
rows that fill no tile, and outliers that no list exists for yet; against 64 bits, and with the bits of the layers one by one."""
import numpy as np
import pytest
import torch

import ojasx_b200
from ojasx_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _block(K, M, frac, scales):
    ws = [synth.make_vq_linear(20 + i, *s, block_dim=8, outlier_frac=frac, with_scales=scales, with_bias=scales) for i, s in enumerate([(K, M), (K, M), (M, K)])]
    if scales:
        for w in ws:
            w.scales[3] = 0.0       # a row whose outliers do not go through its scale
    return ws, ops.VQMLP(*[ops.VQLinear.from_weights(w) for w in ws])


def _dense(w):
    W = torch.from_numpy(w.codebook[w.codes].reshape(w.codes.shape[0], -1)).cuda().double()
    if w.scales is not None:
        W *= torch.from_numpy(w.scales).cuda().double()[:, None]
    if w.csr is not None and len(w.csr[2]):
        rp, ci, va = (torch.from_numpy(np.asarray(a)).cuda() for a in w.csr)
        rows = torch.repeat_interleave(torch.arange(W.shape[0], device="cuda"), (rp[1:] - rp[:-1]).long())
        W.index_put_((rows, ci.long()), va.double(), accumulate=True)
    return W, 0.0 if w.bias is None else torch.from_numpy(w.bias).cuda().double()


@pytest.mark.parametrize("K,M,batch,frac,scales", [
    (128, 128, 32, 0.0, False),       # one tile each, no split
    (1088, 6400, 70, 0.01, False),    # two sums of a tile in one CTA, the second of 7 K tiles in 17
    (1024, 192, 33, 0.01, True),      # a row tile of 64; splits of 16 K tiles
    (2560, 6912, 40, 0.0038, False),  # 108 tiles of two sums each in one launch
    (2560, 6912, 256, 0.0038, False),
    (512, 1088, 257, 0.01, True),     # a second batch tile of one vector
    (2560, 3840, 64, 0.0, False),     # four splits each: layer by layer
    (256, 12800, 64, 0.0, False),     # more tiles than SMs: layer by layer
])
def test_block(cuda, K, M, batch, frac, scales):
    ws, block = _block(K, M, frac, scales)
    x = torch.randn(batch, K, generator=torch.Generator("cuda").manual_seed(1), device=cuda).bfloat16()
    graph, y = torch.cuda.CUDAGraph(), None
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):     # before any other call: the layers' outlier lists cannot be made during a capture
        y = block(x)
    graph.replay()
    got = block(x)
    one = block.down(ops.silu_mul(block.gate(x), block.up(x)))
    (gw, gb), (uw, ub), (dw, db) = (_dense(w) for w in ws)
    xd = x.double()
    want = torch.nn.functional.silu(xd @ gw.T + gb) * (xd @ uw.T + ub) @ dw.T + db
    scale = want.norm()
    assert ojasx_b200.lib().ojasx_b200_take_device_error() == 0
    # weights, gate, up, their product and the output are rounded to 8 bits of mantissa, 2^-9 each
    assert (got.double() - want).norm() <= 5 * 2.0 ** -9 * scale
    assert torch.equal(got, one) and torch.equal(got, y)
