"""Launches that may begin while the one before them still runs: back to back, in a graph and with a synchronisation after every
call they give the same bits, also where a call's scratch is the one that the call before it still uses."""
import numpy as np
import pytest
import torch

from ojasx_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _calls(dtype):
    rng = np.random.default_rng(0)
    moe = ops.VQMoE(synth.make_vq_moe(3, 16, 256, 64, block_dim=8, outlier_frac=0.01))
    lin = ops.VQLinear.from_weights(synth.make_vq_linear(4, 256, 256, block_dim=8))
    mlp = ops.VQMLP(*[ops.VQLinear.from_weights(synth.make_vq_linear(5 + i, *s, block_dim=8)) for i, s in enumerate([(256, 512), (256, 512), (512, 256)])])
    books = [(rng.standard_normal((4, 256, 8)) / 8).astype(np.float32) for _ in range(2)]
    cache = ops.VQKVCache(1, 4, 4, 64, 8, 64, *books)

    def step(x):   # every call reads what the one before it wrote
        for t in (1, 5):
            y = moe.forward_routed(x[:t].contiguous(), 4)
            y = lin(y) if t == 1 else mlp(lin(y))
            x = torch.cat([torch.tanh(y), x[t:]])
        q = x[:1].view(1, 4, 64)
        cache.append(q, q)
        return torch.cat([cache.decode(q).view(1, 256), x[1:]])

    return step, cache, torch.from_numpy(rng.standard_normal((6, 256)).astype(np.float32)).cuda().to(dtype)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_back_to_back_equals_synchronised(cuda, dtype):
    step, cache, x0 = _calls(dtype)
    runs = []
    for wait in (True, False):
        cache.crop(0)
        x, out = x0, []
        for _ in range(20):
            x = step(x)
            out.append(x)
            if wait:
                torch.cuda.synchronize()
        runs.append(torch.stack(out))
    assert torch.equal(*runs) and torch.isfinite(runs[0]).all()


def test_captured(cuda):
    step, cache, x0 = _calls(torch.float32)
    cache.set_static_plan(True)
    want = step(step(x0))
    cache.crop(0)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(x0)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step(step(x0))
    cache.crop(0)
    graph.replay()
    assert torch.equal(got, want)
