"""The tensor-core attention kernels over the quantised cache, which take bf16, against the query-table kernel one position at a
time (itself compared with the CPU oracle and with 64 bits elsewhere)."""
import numpy as np
import pytest
import torch

from ojasx_b200 import ops

pytestmark = pytest.mark.gpu


def _make(seed, B, Hkv, R, hd, D, T0, S, scales=(1.0, 1.0, 2.0)):
    rng = np.random.default_rng(seed)
    books = [(rng.standard_normal((Hkv, 256, D)) / np.sqrt(hd) * s).astype(np.float32) for s in scales[:2]]
    codes = [rng.integers(0, 255, (B, Hkv, T0, hd // D), dtype=np.uint8) for _ in range(2)]
    k, v = (torch.from_numpy((rng.standard_normal((S, B, Hkv, hd)) / np.sqrt(hd) * s).astype(np.float32)).cuda().bfloat16() for s in scales[:2])
    q = torch.from_numpy((rng.standard_normal((S, B, Hkv * R, hd)) * scales[2]).astype(np.float32)).cuda().bfloat16()
    return books, codes, k, v, q


def _pair(books, codes, B, Hkv, R, hd, D, cap):
    caches = [ops.VQKVCache(B, Hkv, Hkv * R, hd, D, cap, *books) for _ in range(2)]
    for c in caches:
        if codes[0].shape[2]:
            c.load(*codes)
    return caches


def _one_by_one(monkeypatch, cache, k, v, q):
    monkeypatch.setenv("OJASX_B200_KV_DECODE", "table")
    out = torch.empty_like(q)
    for s in range(q.shape[0]):
        cache.append(k[s], v[s])
        cache.decode(q[s], out=out[s])
    monkeypatch.delenv("OJASX_B200_KV_DECODE")
    return out


def _same_but_for_ties(got, want, size=None):
    """Sums that differ by about 1e-7 of the largest terms, rounded to bf16: the same number or its neighbour, rarely the latter."""
    g, w = got.float(), want.float()
    size = w.abs().max().item() if size is None else size
    return bool(torch.all((g - w).abs() <= 2.0 ** -7 * w.abs() + 2e-6 * size)) and (g != w).float().mean().item() < 0.01


@pytest.mark.parametrize("B,Hkv,R,hd,D,T0,S", [
    (1, 8, 4, 128, 8, 0, 77),        # prefill kernel: ragged last tile of rows and of tokens, empty cache
    (2, 8, 4, 128, 8, 130, 33),      # a cached context, two sequences
    (1, 2, 1, 64, 4, 63, 65),        # one query head per KV head: 64 positions per tile; tile edges of the context
    (3, 2, 8, 128, 16, 5, 20),
    (1, 2, 2, 64, 16, 0, 16),
    (1, 8, 4, 128, 8, 3000, 9),      # decode kernel with a position axis, 37 positions at most
    (1, 1, 4, 64, 8, 20000, 15),     # 17 splits per position
    (1, 1, 8, 64, 8, 9000, 40),      # 40 positions on a long context: several splits each
    (16, 8, 4, 128, 8, 300, 9),      # three positions per launch
])
def test_chunk_of_positions(cuda, monkeypatch, B, Hkv, R, hd, D, T0, S):
    books, codes, k, v, q = _make(T0 + S, B, Hkv, R, hd, D, T0, S)
    many, one = _pair(books, codes, B, Hkv, R, hd, D, T0 + S)
    got, want = many.prefill(k, v, q), _one_by_one(monkeypatch, one, k, v, q)
    assert many.seq_len == many.sync_len() == T0 + S
    a, b = many.read(0, T0 + S), one.read(0, T0 + S)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
    assert _same_but_for_ties(got, want)


def test_operand_range(cuda, monkeypatch):
    """Queries and codebooks far from 1: operands are scaled per row and per codebook."""
    books, codes, k, v, q = _make(3, 1, 2, 4, 128, 8, 64, 16, (2e5, 3e-6, 2e-5))
    q[3] = 0
    many, one = _pair(books, codes, 1, 2, 4, 128, 8, 100)
    assert _same_but_for_ties(many.prefill(k, v, q), _one_by_one(monkeypatch, one, k, v, q))
    many.crop(64)
    one.crop(64)
    for s in range(3):
        many.append(k[s], v[s])
        assert _same_but_for_ties(many.decode(q[s]), _one_by_one(monkeypatch, one, k[s:s + 1], v[s:s + 1], q[s:s + 1])[0])


@pytest.mark.parametrize("which", [0, 1])
@pytest.mark.parametrize("entry", [np.inf, 1e30, 2e6])
@pytest.mark.parametrize("col", [slice(None), 3])
def test_codebooks_of_wide_range(cuda, monkeypatch, which, entry, col):
    """A centroid that no token has, far above the others, costs them nothing: such caches keep the query-table kernel."""
    books, codes, k, v, q = _make(5, 1, 2, 4, 128, 8, 500, 20)
    want = _pair(books, codes, 1, 2, 4, 128, 8, 520)[0].decode(q[0])
    books[which][1, 255, col] = entry
    many, one = _pair(books, codes, 1, 2, 4, 128, 8, 520)
    first = many.decode(q[0])
    assert _same_but_for_ties(first, want)
    assert _same_but_for_ties(many.prefill(k, v, q), _one_by_one(monkeypatch, one, k, v, q))
    many.crop(500)
    monkeypatch.setenv("OJASX_B200_KV_DECODE", "table")
    assert torch.equal(many.decode(q[0]), first)


def test_scores_that_overflow(cuda, monkeypatch):
    """Finite queries with scores of -inf over whole runs of tokens for one head: weights 0, the other heads as ever."""
    B, Hk, R, hd, T = 1, 2, 4, 128, 9000
    rng = np.random.default_rng(0)
    books = [rng.uniform(0.5, 1.5, (Hk, 256, 8)).astype(np.float32) for _ in range(2)]
    books[0][:, :128] *= 1e-3
    books[0][:, 128:] *= -1
    codes = [rng.integers(0, 128, (B, Hk, T, hd // 8), dtype=np.uint8) for _ in range(2)]
    codes[0][:, :, 100:] += 128
    cache = ops.VQKVCache(B, Hk, Hk * R, hd, 8, T, *books)
    cache.load(*codes)
    q = torch.rand(B, Hk * R, hd, device=cuda, generator=torch.Generator(cuda).manual_seed(0)) + 0.5
    q[0, 2] = 0.0
    q[0, 6] *= 1e38
    q = q.bfloat16()
    got = cache.decode(q)
    monkeypatch.setenv("OJASX_B200_KV_DECODE", "table")
    want = cache.decode(q)
    assert torch.isfinite(want).all() and _same_but_for_ties(got, want)
