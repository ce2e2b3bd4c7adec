"""fp32 prompt chunks through the prefill kernel: against 64 bits at the edges of its tiles (64 query rows, 64 tokens, runs of 512),
no further off than position by position, with special values, and the same routes for calls that it does not take."""
import numpy as np
import pytest
import torch

from ojasx_b200 import OjasxB200Error, ops

pytestmark = pytest.mark.gpu


def _cache(seed, B, Hkv, R, hd, D, T0, S):
    g = torch.Generator("cuda").manual_seed(seed)
    sig = hd ** -0.5
    books = [(torch.randn(Hkv, 256, D, generator=g, device="cuda") * sig) for _ in range(2)]
    cache = ops.VQKVCache(B, Hkv, Hkv * R, hd, D, T0 + S, *[b.cpu().numpy() for b in books])
    if T0:
        cache.load(*[torch.randint(0, 256, (B, Hkv, T0, hd // D), generator=g, device="cuda", dtype=torch.uint8).cpu().numpy() for _ in range(2)])
    k, v = (torch.randn(S, B, Hkv, hd, generator=g, device="cuda") * sig for _ in range(2))
    return books, cache, k, v, torch.randn(S, B, Hkv * R, hd, generator=g, device="cuda") * 2


def _exact(q, books, codes, T0):
    S, B, Hq, hd = q.shape
    out = torch.empty(S, B, Hq, hd, dtype=torch.float64, device="cuda")
    kc, vc = (torch.from_numpy(c).cuda().long() for c in codes)
    see = torch.arange(kc.shape[2], device="cuda")[None] <= T0 + torch.arange(S, device="cuda")[:, None]
    for b in range(B):
        for h in range(Hq):
            kv = h // (Hq // kc.shape[1])
            keys, values = (bk[kv][c[b, kv]].reshape(kc.shape[2], hd).double() for bk, c in zip(books, (kc, vc)))
            out[:, b, h] = torch.softmax((q[:, b, h].double() @ keys.T * hd ** -0.5).masked_fill(~see, -np.inf), 1) @ values
    return out


@pytest.mark.parametrize("B,Hkv,R,hd,D,T0,S", [
    (1, 2, 4, 128, 8, 0, 16),        # one tile of rows, a quarter of a tile of tokens
    (2, 1, 4, 128, 8, 0, 17),        # a second tile of one position
    (1, 2, 1, 64, 8, 0, 64), (1, 1, 1, 64, 8, 0, 65),
    (1, 1, 8, 128, 16, 0, 40),       # one CTA per SM
    (1, 2, 2, 64, 4, 60, 100),
    (1, 2, 8, 64, 8, 0, 20),         # eight positions per tile of rows
    (1, 4, 4, 128, 8, 400, 112),     # 512 tokens: one run, full
    (1, 4, 4, 128, 8, 400, 113),     # one token into the second run
    (1, 4, 4, 64, 16, 900, 200),     # three runs
])
def test_against_64_bits(cuda, B, Hkv, R, hd, D, T0, S):
    books, cache, k, v, q = _cache(T0 + S, B, Hkv, R, hd, D, T0, S)
    got = cache.prefill(k, v, q)
    want = _exact(q, books, cache.read(0, T0 + S), T0)
    many = float((got.double() - want).norm() / want.norm())
    cache.crop(T0)
    one = torch.stack([(cache.append(k[s], v[s]), cache.decode(q[s]))[1] for s in range(S)])
    single = float((one.double() - want).norm() / want.norm())
    assert many < max(1.15 * single, 1.2e-7), (many, single)       # 1.2e-7: two roundings of an output


def test_special_values(cuda):
    """A query with an infinity or NaN gives NaN for its head and leaves the others alone; scores that overflow weigh nothing."""
    books, cache, k, v, q = _cache(3, 1, 2, 4, 128, 8, 0, 40)
    clean = cache.prefill(k, v, q)
    cache.crop(0)
    q[5, 0, 2, 7], q[6, 0, 7, 0], q[7, 0, 1, 3] = np.nan, np.inf, 3e38
    got = cache.prefill(k, v, q)
    assert torch.isnan(got[5, 0, 2]).all() and torch.isnan(got[6, 0, 7]).all()
    got[5, 0, 2], got[6, 0, 7], got[7, 0, 1] = clean[5, 0, 2], clean[6, 0, 7], clean[7, 0, 1]
    assert torch.equal(got, clean)


def test_codebooks_with_infinities(cuda):
    """An infinite centroid among the values reaches only the tokens that see it."""
    books, cache, k, v, q = _cache(4, 1, 1, 4, 64, 8, 0, 48)
    inf = books[1].clone()
    inf[0, :, 3] = torch.where(torch.arange(256, device="cuda") == 255, torch.inf, inf[0, :, 3])
    other = ops.VQKVCache(1, 1, 4, 64, 8, 48, books[0].cpu().numpy(), inf.cpu().numpy())
    got = other.prefill(k, v, q)
    codes = other.read(0, 48)[1][0, 0]
    seen = np.maximum.accumulate(codes == 255, axis=0)
    finite = torch.isfinite(got[:, 0]).all(1).cpu().numpy().reshape(48, 8, 8).all(2)
    assert np.array_equal(finite, ~seen)


@pytest.mark.parametrize("R,hd,D", [(64, 64, 8), (8, 128, 4)])
def test_shapes_that_cannot_be_decoded_stay_refused(cuda, R, hd, D):
    _, cache, k, v, q = _cache(1, 1, 1, R, hd, D, 0, 20)
    with pytest.raises(OjasxB200Error):
        cache.prefill(k, v, q)
