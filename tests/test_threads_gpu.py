"""Host threads that call the same kernels at different sizes: none takes another's opt-in to shared memory away."""
from concurrent.futures import ThreadPoolExecutor

import pytest
import torch

from ojasx_b200 import ops, synth

pytestmark = pytest.mark.gpu


def _tensor(rows_of_x):
    layer = ops.VQLinear.from_weights(synth.make_vq_linear(1, 1024, 512, block_dim=8))
    x = torch.randn(rows_of_x, 1024, generator=torch.Generator("cuda").manual_seed(1), device="cuda").bfloat16()
    return lambda: layer.forward_tensor(x)


def _wide_tensor(rows_of_x):    # 256 rows a CTA
    layer = ops.VQLinear.from_weights(synth.make_vq_linear(1, 256, 32768, block_dim=8))
    x = torch.randn(rows_of_x, 256, generator=torch.Generator("cuda").manual_seed(1), device="cuda").bfloat16()
    return lambda: layer.forward_tensor(x)


def _cache(head_dim):
    g = torch.Generator("cuda").manual_seed(head_dim)
    books = [torch.randn(2, 256, 8, generator=g, device="cuda").cpu().numpy() for _ in range(2)]
    cache = ops.VQKVCache(1, 2, 8, head_dim, 8, 16, *books)
    for _ in range(3):
        cache.append(*(torch.randn(1, 2, head_dim, generator=g, device="cuda") for _ in range(2)))
    q = torch.randn(1, 8, head_dim, generator=g, device="cuda")
    return lambda: cache.decode(q)


@pytest.mark.parametrize("call,large,small", [(_tensor, 256, 32), (_wide_tensor, 256, 64), (_cache, 128, 64), (_cache, 160, 32)])
def test_a_small_call_of_another_thread_in_between(cuda, call, large, small):
    big, little = call(large), call(small)
    with ThreadPoolExecutor(1) as one, ThreadPoolExecutor(1) as other:
        first = one.submit(big).result()
        other.submit(little).result()
        again = one.submit(big).result()
    assert torch.equal(first, again) and torch.isfinite(first).all()
