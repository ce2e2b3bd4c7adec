"""fp32 decode over ranges of few tokens, which go without tables: against 64 bits around the edges of a range (64, 128, 256 tokens)
and of the plan (1024), all head shapes, ragged batches of lengths, and special values."""
import numpy as np
import pytest
import torch

from ojasx_b200 import ops

pytestmark = pytest.mark.gpu


def _books(g, Hkv, hd, D):
    return [torch.randn(Hkv, 256, D, generator=g, device="cuda") * hd ** -0.5 for _ in range(2)]


def _exact(q, kc, vc, books):
    hd, (B, Hkv, T, _) = q.shape[2], kc.shape
    out = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    R = q.shape[1] // Hkv
    for b in range(B):
        for h in range(Hkv):
            keys, values = (bk[h][c[b, h].long()].reshape(T, hd).double() for bk, c in zip(books, (kc, vc)))
            out[b, h * R:(h + 1) * R] = torch.softmax(q[b, h * R:(h + 1) * R].double() @ keys.T * hd ** -0.5, 1) @ values
    return out


@pytest.mark.parametrize("R,hd,D", [(1, 64, 8), (2, 128, 8), (4, 128, 8), (8, 128, 8), (4, 96, 8), (4, 128, 16), (2, 128, 4), (8, 64, 16), (1, 32, 16)])
def test_against_64_bits(cuda, R, hd, D):
    g = torch.Generator("cuda").manual_seed(R * hd + D)
    books = _books(g, 2, hd, D)
    for B, cap in ((1, 1200), (80, 300)):           # ranges of 64 tokens while they fit the SMs; one range per head
        for T in (1, 3, 63, 64, 65, 128, 129, 200, 256, 257, 300) + ((1023, 1024, 1025, 1200) if B == 1 else ()):
            cache = ops.VQKVCache(B, 2, 2 * R, hd, D, cap, *[b.cpu().numpy() for b in books])
            kc, vc = (torch.randint(0, 256, (B, 2, T, hd // D), generator=g, device="cuda", dtype=torch.uint8) for _ in range(2))
            cache.load(kc.cpu().numpy(), vc.cpu().numpy())
            q = torch.randn(B, 2 * R, hd, generator=g, device="cuda") * 2
            want = _exact(q, kc, vc, books)
            got = cache.decode(q).double()
            assert (got - want).norm() <= 3e-7 * want.norm(), (T, B)          # five roundings of an output


def test_static_plan_and_special_values(cuda):
    """Lengths that only the device knows, and queries with an infinity or NaN, whose heads are NaN and no others."""
    g = torch.Generator("cuda").manual_seed(1)
    books = _books(g, 8, 128, 8)
    cache = ops.VQKVCache(1, 8, 32, 128, 8, 1024, *[b.cpu().numpy() for b in books])
    cache.set_static_plan(True)
    kv = torch.randn(2, 150, 1, 8, 128, generator=g, device="cuda") * 0.1
    q = torch.randn(1, 32, 128, generator=g, device="cuda")
    bad = q.clone()
    bad[0, 3, 5], bad[0, 30, 100], bad[0, 9, 0] = np.nan, np.inf, -np.inf
    for t in range(150):
        cache.append(kv[0, t], kv[1, t])
        if t in (0, 63, 64, 149):
            codes = [torch.from_numpy(c).cuda() for c in cache.read(0, t + 1)]
            want = _exact(q, *codes, books)
            got = cache.decode(q)
            assert (got.double() - want).norm() <= 3e-7 * want.norm()
            if t == 0:      # one score may be -inf alone: it weighs nothing
                continue
            out = cache.decode(bad)
            nan = torch.isnan(out[0]).all(1)
            assert nan.nonzero().flatten().tolist() == [3, 9, 30] and torch.equal(out[0][~nan], got[0][~nan])
