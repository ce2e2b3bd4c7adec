"""Decode on mma.sync operands gathered from the codebooks against the query-table kernel and 64-bit attention."""
import numpy as np
import pytest
import torch

import ojasx_b200
from ojasx_b200 import ops

pytestmark = pytest.mark.gpu


def _cache(B, Hk, R, hd, T, cap, seed):
    rng = np.random.default_rng(seed)
    books = [(rng.standard_normal((Hk, 256, 8)) / np.sqrt(hd)).astype(np.float32) for _ in range(2)]
    codes = [rng.integers(0, 256, (B, Hk, T, hd // 8), dtype=np.uint8) for _ in range(2)]
    cache = ops.VQKVCache(B, Hk, Hk * R, hd, 8, cap, *books)
    cache.load(*codes)
    return cache, books, codes, rng


def _exact(books, codes, q, scale):
    B, Hk = codes[0].shape[:2]
    R = q.shape[1] // Hk
    out = np.zeros(q.shape, np.float64)
    for b in range(B):
        for h in range(Hk):
            k, v = (books[i][h].astype(np.float64)[codes[i][b, h]].reshape(codes[i].shape[2], -1) for i in range(2))
            s = q[b, h * R:(h + 1) * R].astype(np.float64) @ k.T * scale
            p = np.exp(s - s.max(-1, keepdims=True))
            out[b, h * R:(h + 1) * R] = p @ v / p.sum(-1, keepdims=True)
    return out


@pytest.mark.parametrize("R,hd", [(4, 64), (4, 128), (8, 64), (8, 128)])
@pytest.mark.parametrize("T", [1, 16, 17, 257, 1001, 5000])
def test_decode_against_table_kernel_and_64_bits(cuda, monkeypatch, R, hd, T):
    B, Hk = 2, 3
    cache, books, codes, rng = _cache(B, Hk, R, hd, T, T + 3, R * hd + T)
    q = rng.standard_normal((B, Hk * R, hd)).astype(np.float32) * 4       # scores of a few units: some tokens dominate
    q[0, 0] *= 1e-6                                                       # heads of other sizes
    q[1, -1] *= 1e4
    qt = torch.from_numpy(q).to(cuda)
    got = cache.decode(qt)
    half = cache.decode(qt.bfloat16())
    cache.set_static_plan(True)
    planned = cache.decode(qt)
    cache.set_static_plan(False)
    monkeypatch.setenv("OJASX_B200_KV_DECODE", "table")
    table = cache.decode(qt).cpu().numpy()
    want = _exact(books, codes, q, 1.0 / np.sqrt(hd))
    # a rounding of the scores (2^-24 of their largest terms, up to 1e4 units for the last head) is a relative error of p
    err = np.abs(got.cpu().numpy() - want).max(-1)
    ref = np.abs(table - want).max(-1)
    size = np.abs(want).max(-1)
    assert np.all(err <= 2 * ref + 1e-6 * size), (err / size, ref / size)
    assert np.allclose(planned.cpu().numpy(), got.cpu().numpy(), rtol=0, atol=float((2 * ref + 2e-6 * size).max()))
    bf = _exact(books, codes, qt.bfloat16().float().cpu().numpy(), 1.0 / np.sqrt(hd))
    assert np.all(np.abs(half.float().cpu().numpy() - bf).max(-1) <= 2.0 ** -8 * np.abs(bf).max(-1) + 4 * ref + 1e-6 * size)


def test_append_and_decode_in_one_stream_and_under_capture(cuda):
    """A decode prepares its tables while the append before it runs, and still sees the appended token."""
    cache, books, codes, rng = _cache(1, 2, 4, 128, 40, 64, 9)
    k, v = (torch.from_numpy(rng.standard_normal((20, 1, 2, 128)).astype(np.float32)).to(cuda) for _ in range(2))
    q = torch.from_numpy(rng.standard_normal((20, 1, 8, 128)).astype(np.float32)).to(cuda)
    outs = []
    for t in range(20):
        cache.append(k[t], v[t])
        outs.append(cache.decode(q[t]).cpu().numpy())
    kc, vc = cache.read(0, 60)
    for t in range(20):
        want = _exact(books, [kc[:, :, :41 + t], vc[:, :, :41 + t]], q[t].cpu().numpy(), 1.0 / np.sqrt(128))
        assert np.allclose(outs[t], want, rtol=1e-5, atol=1e-6 * np.abs(want).max())
    cache.crop(40)
    cache.set_static_plan(True)
    cache.append(k[0], v[0])
    cache.decode(q[0])
    torch.cuda.synchronize()
    cache.crop(40)
    kk, vv, qq, o = k[0].clone(), v[0].clone(), q[0].clone(), torch.empty_like(q[0])
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        cache.append(kk, vv)
        cache.decode(qq, out=o)
    for t in range(20):
        kk.copy_(k[t]); vv.copy_(v[t]); qq.copy_(q[t])
        graph.replay()
        assert np.allclose(o.cpu().numpy(), outs[t], rtol=1e-5, atol=1e-6)


def test_codebooks_with_infinities_keep_the_table_kernel(cuda, monkeypatch):
    """High and low parts of an infinity are NaN: caches whose codebooks are not finite stay on the query-table kernel."""
    rng = np.random.default_rng(0)
    books = [(rng.standard_normal((1, 256, 8)) * 0.1).astype(np.float32) for _ in range(2)]
    books[1][0, 7, 3] = np.inf
    cache = ops.VQKVCache(1, 1, 4, 64, 8, 32, *books)
    codes = rng.integers(8, 256, (1, 1, 20, 8), dtype=np.uint8)
    codes2 = codes.copy()
    codes2[0, 0, 5, 2] = 7
    q = torch.from_numpy(rng.standard_normal((1, 4, 64)).astype(np.float32)).to(cuda)
    for c in (codes, codes2):
        cache.load(codes, c)
        got = cache.decode(q).cpu().numpy()
        monkeypatch.setenv("OJASX_B200_KV_DECODE", "table")
        assert np.array_equal(got, cache.decode(q).cpu().numpy(), equal_nan=True)
        monkeypatch.delenv("OJASX_B200_KV_DECODE")
        assert np.isfinite(got).all() == (c is codes)


def test_prefill_of_a_cache_with_infinite_centroids_equals_position_by_position(cuda):
    rng = np.random.default_rng(3)
    books = [(rng.standard_normal((1, 256, 8)) * 0.1).astype(np.float32) for _ in range(2)]
    books[0][0, 9, 1] = np.inf
    k, v = (torch.from_numpy(rng.standard_normal((20, 1, 1, 64)).astype(np.float32) * 0.1).to(cuda) for _ in range(2))
    q = torch.from_numpy(rng.standard_normal((20, 1, 4, 64)).astype(np.float32)).to(cuda)
    chunk, one = (ops.VQKVCache(1, 1, 4, 64, 8, 32, *books) for _ in range(2))
    got = chunk.prefill(k, v, q)
    for s in range(20):
        one.append(k[s], v[s])
        want = one.decode(q[s])
        assert torch.allclose(got[s], want, rtol=1e-5, atol=1e-6, equal_nan=True)


@pytest.mark.parametrize("R,hd", [(4, 64), (4, 128), (8, 64), (8, 128), (1, 64), (2, 128)])
@pytest.mark.parametrize("T", [17, 700, 9000])
def test_non_finite_queries(cuda, R, hd, T):
    """An infinity or NaN in the query of one head gives NaN for that head, as attention in 64 bits does, and leaves the other
    heads as they are; the same on the query-table kernel (one or two query heads per KV head) and in chunks of 15 and of 16
    positions (the decode kernels, the prefill kernel)."""
    B, Hk = 2, 2
    cache, _, _, _ = _cache(B, Hk, R, hd, T, T + 40, T)
    q = torch.randn(B, Hk * R, hd, device=cuda, generator=torch.Generator(cuda).manual_seed(T))
    clean = cache.decode(q)
    for value in (float("inf"), -float("inf"), float("nan")):
        for dtype in (torch.float32, torch.bfloat16):
            bad = q.to(dtype)
            ok = cache.decode(bad)
            bad = bad.clone()
            bad[0, 1, 5] = value
            bad[1, R, hd - 1] = value
            got = cache.decode(bad)
            mask = torch.zeros(B, Hk * R, dtype=torch.bool, device=cuda)
            mask[0, 1] = mask[1, R] = True
            assert torch.isnan(got[mask]).all(), got[mask]
            assert torch.equal(got[~mask], ok[~mask])
    for S, dtype in ((15, torch.float32), (16, torch.float32), (15, torch.bfloat16), (16, torch.bfloat16)):
        k, v = ((torch.randn(S, B, Hk, hd, device=cuda) / hd ** 0.5).to(dtype) for _ in range(2))
        qs = torch.randn(S, B, Hk * R, hd, device=cuda).to(dtype)
        a = cache.prefill(k, v, qs)
        cache.crop(T)
        qs[S - 1, 0, 1, 5] = float("inf")
        qs[2, 1, R, 0] = float("nan")
        b = cache.prefill(k, v, qs)
        cache.crop(T)
        mask = torch.zeros(S, B, Hk * R, dtype=torch.bool, device=cuda)
        mask[S - 1, 0, 1] = mask[2, 1, R] = True
        assert torch.isnan(b[mask]).all()
        assert torch.equal(a[~mask], b[~mask])


def test_scores_that_overflow_in_one_head(cuda, monkeypatch):
    """A finite query whose scores are -inf over whole runs of tokens: weights 0 there, as in the table kernel, and the runs of
    the other heads are merged as ever."""
    B, Hk, R, hd, T = 1, 2, 4, 128, 9000
    rng = np.random.default_rng(0)
    books = [rng.uniform(0.5, 1.5, (Hk, 256, 8)).astype(np.float32) for _ in range(2)]
    books[0][:, :128] *= 1e-3
    books[0][:, 128:] *= -1
    codes = [rng.integers(0, 128, (B, Hk, T, hd // 8), dtype=np.uint8) for _ in range(2)]
    codes[0][:, :, 100:] += 128                              # 100 tokens of small scores, then large negative ones
    cache = ops.VQKVCache(B, Hk, Hk * R, hd, 8, T, *books)
    cache.load(*codes)
    q = torch.rand(B, Hk * R, hd, device=cuda, generator=torch.Generator(cuda).manual_seed(0)) + 0.5
    q[0, 2] = 0.0
    q[0, 6] *= 1e38
    got = cache.decode(q)
    monkeypatch.setenv("OJASX_B200_KV_DECODE", "table")
    want = cache.decode(q)
    assert torch.isfinite(want).all() and torch.allclose(got, want, rtol=1e-4, atol=2e-6)


@pytest.mark.parametrize("which,row,col", [(0, 255, slice(None)), (1, 255, slice(None)), (0, 255, 3), (1, slice(None), 5)])
@pytest.mark.parametrize("factor", [1e30, 2e6])
def test_codebooks_of_wide_range_keep_fp32_accuracy(cuda, oracle, which, row, col, factor):
    """Entries far above the others (a centroid that no token has, a dimension): the others keep their 24 bits."""
    rng = np.random.default_rng(0)
    B, Hk, R, hd, T, S = 1, 2, 4, 128, 500, 20
    books = [(rng.standard_normal((Hk, 256, 8)) / np.sqrt(hd)).astype(np.float32) for _ in range(2)]
    if isinstance(row, slice):
        books[which] = books[which].astype(np.float32)
        books[which][1, row, col] = np.float32(factor) * np.abs(books[which][1, row, col])
    else:
        books[which][1, row, col] = factor
    codes = [rng.integers(0, 255, (B, Hk, T, hd // 8), dtype=np.uint8) for _ in range(2)]
    cache = ops.VQKVCache(B, Hk, Hk * R, hd, 8, T + S, *books)
    cache.load(*codes)
    q = rng.standard_normal((S, B, Hk * R, hd)).astype(np.float32)
    k, v = (torch.from_numpy((rng.standard_normal((S, B, Hk, hd)) / np.sqrt(hd)).astype(np.float32)).to(cuda) for _ in range(2))
    got = [cache.decode(torch.from_numpy(q[0]).to(cuda)).cpu().numpy()]
    got += list(cache.prefill(k, v, torch.from_numpy(q).to(cuda)).cpu().numpy())
    kc, vc = cache.read(0, T + S)
    for i, (s, n) in enumerate([(0, T)] + [(s, T + s + 1) for s in range(S)]):
        want = _exact(books, [kc[:, :, :n], vc[:, :, :n]], q[s], 1.0 / np.sqrt(hd))
        for d in range(hd):     # dimensions of other sizes: each to its own
            size = np.abs(want[:, :, d]).max()
            assert np.abs(got[i][:, :, d] - want[:, :, d]).max() <= 1e-5 * size, (i, d)


def _rms(a, want):
    return np.sqrt(((a.astype(np.float64) - want) ** 2).sum() / (want ** 2).sum())


@pytest.mark.parametrize("R,hd,T", [(4, 128, 2048), (8, 128, 2048), (4, 64, 700), (8, 128, 9000)])
@pytest.mark.parametrize("positions", [0, 40])
def test_fp32_keeps_fp32_accuracy(cuda, monkeypatch, R, hd, T, positions):
    """fp32 outputs are as close to 64 bits as the query-table kernel's, in a decode and in a chunk of positions (the same
    splits; a twentieth for the order of the sums); in bf16 both round the same numbers."""
    B, Hk = 2, 4
    cache, books, codes, rng = _cache(B, Hk, R, hd, T, T + positions + 1, R + T)
    S = max(1, positions)
    k, v = (torch.from_numpy((rng.standard_normal((S, B, Hk, hd)) / np.sqrt(hd)).astype(np.float32)).to(cuda) for _ in range(2))
    q = torch.from_numpy(rng.standard_normal((S, B, Hk * R, hd)).astype(np.float32)).to(cuda)

    def outputs(dtype, table):
        if table:
            monkeypatch.setenv("OJASX_B200_KV_DECODE", "table")
        cache.crop(T)
        if positions and not table:
            out = cache.prefill(k.to(dtype), v.to(dtype), q.to(dtype))
        else:
            out = torch.empty(q.shape, dtype=dtype, device=cuda)
            for s in range(S):
                if positions:
                    cache.append(k[s].to(dtype), v[s].to(dtype))
                cache.decode(q[s].to(dtype), out=out[s])
        monkeypatch.delenv("OJASX_B200_KV_DECODE", raising=False)
        return out

    for dtype in (torch.float32, torch.bfloat16):
        got, table = (outputs(dtype, t).float().cpu().numpy() for t in (False, True))
        kc, vc = cache.read(0, T + positions) if positions else codes
        want = np.stack([_exact(books, [kc[:, :, :T + (s + 1 if positions else 0)], vc[:, :, :T + (s + 1 if positions else 0)]],
                                q[s].to(dtype).float().cpu().numpy(), 1.0 / np.sqrt(hd)) for s in range(S)])
        if dtype is torch.float32:
            assert _rms(got, want) <= 1.05 * _rms(table, want), (_rms(got, want), _rms(table, want))
        else:
            assert _rms(got, want) <= 1.0005 * _rms(table, want)



def test_chunk_whose_first_scores_overflow(cuda, monkeypatch):
    """A tile of 64 tokens whose scores are all -inf for one head, before tokens of finite scores: weights 0, as one by one."""
    B, Hk, R, hd, T, S = 1, 2, 4, 128, 200, 16
    rng = np.random.default_rng(0)
    books = [rng.uniform(0.5, 1.5, (Hk, 256, 8)).astype(np.float32) for _ in range(2)]
    books[0][:, :128] *= 1e-3
    books[0][:, 128:] *= -1
    codes = [rng.integers(0, 128, (B, Hk, T, hd // 8), dtype=np.uint8) for _ in range(2)]
    codes[0][:, :, :100] += 128
    cache = ops.VQKVCache(B, Hk, Hk * R, hd, 8, T + S, *books)
    cache.load(*codes)
    k = torch.zeros(S, B, Hk, hd, device=cuda, dtype=torch.bfloat16)
    q = torch.rand(S, B, Hk * R, hd, device=cuda, generator=torch.Generator(cuda).manual_seed(0)) + 0.5
    q[:, 0, 6] *= 1e38
    q = q.bfloat16()
    got = cache.prefill(k, k, q)
    cache.crop(T)
    monkeypatch.setenv("OJASX_B200_KV_DECODE", "table")
    for s in range(S):
        cache.append(k[s], k[s])
        want = cache.decode(q[s])
        assert torch.isfinite(want).all() and torch.allclose(got[s].float(), want.float(), rtol=2 ** -7, atol=1e-5), s
