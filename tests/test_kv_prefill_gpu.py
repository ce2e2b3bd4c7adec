"""A chunk of prompt positions through the quantised cache against the CPU oracle and against the token-by-token form."""
import numpy as np
import pytest
import torch

from ojasx_b200 import OjasxB200Error, ops

pytestmark = pytest.mark.gpu


def _make(seed, B, Hkv, Hq, hd, D, T0, S):
    rng = np.random.default_rng(seed)
    sig = 1.0 / np.sqrt(hd)
    books = [(rng.standard_normal((Hkv, 256, D)) * sig).astype(np.float32) for _ in range(2)]
    old = [rng.integers(0, 256, (B, Hkv, T0, hd // D), dtype=np.uint8) for _ in range(2)]
    k, v = ((rng.standard_normal((S, B, Hkv, hd)) * sig).astype(np.float32) for _ in range(2))
    q = (3.0 * rng.standard_normal((S, B, Hq, hd))).astype(np.float32)
    return books, old, k, v, q


@pytest.mark.parametrize("B,Hkv,Hq,hd,D,T0,S", [
    (1, 8, 32, 128, 8, 0, 77),       # ragged last tile of rows and of tokens, empty cache
    (2, 8, 32, 128, 8, 130, 33),     # a cached context, two sequences
    (1, 2, 2, 64, 4, 63, 65),        # one query head per KV head: 64 positions per tile; tile edges of the context
    (3, 2, 16, 128, 16, 5, 20),      # eight query heads per KV head
    (1, 8, 32, 128, 8, 3000, 9),     # few positions on a longer context: decode kernel with a position axis
    (1, 2, 8, 96, 8, 11, 21),        # head_dim 96: not covered by the prefill kernel, two batched decodes
])
def test_prefill_chunk(cuda, oracle, B, Hkv, Hq, hd, D, T0, S):
    books, old, k, v, q = _make(T0 + S, B, Hkv, Hq, hd, D, T0, S)
    many, one = (ops.VQKVCache(B, Hkv, Hq, hd, D, T0 + S + 3, *books) for _ in range(2))
    for c in (many, one):
        if T0:
            c.load(*old)
    kt, vt, qt = (torch.from_numpy(a).to(cuda) for a in (k, v, q))
    got = many.prefill(kt, vt, qt).cpu().numpy()
    want = np.stack([(one.append(kt[s], vt[s]), one.decode(qt[s]))[1].cpu().numpy() for s in range(S)])
    assert many.seq_len == one.seq_len == many.sync_len() == T0 + S
    a, b = many.read(0, T0 + S), one.read(0, T0 + S)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])     # codes: index-exact
    # fp32 sums in another order, over scores of magnitude ~10: the bounds of the decode tests
    assert np.allclose(got, want, rtol=1e-4, atol=2e-6), np.abs(got - want).max()
    R = Hq // Hkv
    for s, bb, h in [(0, 0, 0), (S // 2, B - 1, Hkv - 1), (S - 1, 0, Hkv - 1)]:
        ref = oracle.kvq_decode(q[s, bb, h * R:(h + 1) * R], a[0][bb, h, :T0 + s + 1], a[1][bb, h, :T0 + s + 1],
                                books[0][h], books[1][h], block_dim=D)
        assert np.allclose(got[s, bb, h * R:(h + 1) * R], ref, rtol=1e-4, atol=2e-6), (s, bb, h)
    many.crop(T0)
    bf = many.prefill(kt.bfloat16(), vt.bfloat16(), qt.bfloat16())
    assert bf.dtype == torch.bfloat16 and torch.isfinite(bf).all()
    with pytest.raises(OjasxB200Error):
        many.prefill(kt, vt, qt)                                          # does not fit: -2, nothing is appended
    assert many.seq_len == T0 + S


def test_prefill_operand_range(cuda, oracle):
    """Queries and codebooks far from 1: the operands of the prefill kernel are scaled per row and per codebook, so the
    accuracy does not depend on their magnitude."""
    books, old, k, v, q = _make(3, 1, 2, 8, 128, 8, 64, 16)
    books = [books[0] * np.float32(2e5), books[1] * np.float32(3e-6)]
    q = q * np.float32(1e-5)
    q[3] = 0
    cache = ops.VQKVCache(1, 2, 8, 128, 8, 100, *books)
    cache.load(*old)
    got = cache.prefill(*(torch.from_numpy(a).to(cuda) for a in (k, v, q))).cpu().numpy()
    kc, vc = cache.read(0, 80)
    for s in (0, 3, 15):
        ref = oracle.kvq_decode(q[s, 0, :4], kc[0, 0, :65 + s], vc[0, 0, :65 + s], books[0][0], books[1][0], block_dim=8)
        assert np.allclose(got[s, 0, :4], ref, rtol=1e-4, atol=2e-6 * 3e-6), s


def _used(f):
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    f()
    torch.cuda.synchronize()
    return free - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("cap", [8192, 16384, 32768])
@pytest.mark.parametrize("R", [2, 4])
def test_scratch_of_a_cache(cuda, cap, R):
    """Partial sums: one per 256 tokens and query head (and what fills the SMs), for positions of a prompt in one
    launch too; allocated with the cache, not in its first call."""
    rng = np.random.default_rng(0)
    B, Hk, hd = 16, 8, 128
    books = [rng.standard_normal((Hk, 256, 8)).astype(np.float32) for _ in range(2)]
    q = torch.randn(1, B, Hk * R, hd, device=cuda)
    k, v = (torch.randn(1, B, Hk, hd, device=cuda) for _ in range(2))
    first = ops.VQKVCache(B, Hk, Hk * R, hd, 8, 16, *books)  # kernels are loaded on their first launch
    first.append(k[0], v[0])
    first.decode(q[0])
    first.prefill(k, v, q)
    torch.empty(64 << 20, device=cuda)                       # outputs come from the allocator's cache
    made = []
    used = _used(lambda: made.append(ops.VQKVCache(B, Hk, Hk * R, hd, 8, cap, *books)))
    need = 2 * B * Hk * cap * (hd // 8) + 4 * B * Hk * (cap // 256) * R * (hd + 2)
    assert used <= need + (8 << 20), (used, need)            # the driver hands memory out in pieces of 2 MB
    cache = made[0]
    assert _used(lambda: (cache.append(k[0], v[0]), cache.decode(q[0]), cache.prefill(k, v, q))) == 0


@pytest.mark.parametrize("B,Hkv,R,hd,T0,S", [
    (1, 1, 4, 64, 20000, 15),        # one head: three positions of 79 splits per launch
    (16, 8, 4, 128, 300, 9),         # more heads than half the SMs: three positions per launch
    (20, 8, 2, 64, 40, 5),           # two per launch
])
def test_positions_share_the_scratch_of_one_decode(cuda, B, Hkv, R, hd, T0, S):
    books, old, k, v, q = _make(7, B, Hkv, Hkv * R, hd, 8, T0, S)
    many, one = (ops.VQKVCache(B, Hkv, Hkv * R, hd, 8, T0 + S, *books) for _ in range(2))
    for c in (many, one):
        c.load(*old)
    kt, vt, qt = (torch.from_numpy(a).to(cuda) for a in (k, v, q))
    got = many.prefill(kt, vt, qt)
    for s in range(S):
        one.append(kt[s], vt[s])
        assert torch.allclose(got[s], one.decode(qt[s]), rtol=1e-4, atol=2e-6), s
    assert many.sync_len() == T0 + S


def test_codes_of_non_finite_keys_and_values(cuda):
    """Positions in a chunk get the codes that single appends give them, also where no distance to a centroid is finite."""
    books, _, k, v, q = _make(5, 1, 2, 8, 64, 8, 1, 20)
    books[0][1, 9, 3] = np.inf
    k[3, 0, 0, 5], k[4, 0, 1, 63], v[5, 0, 0, 0], v[6], v[7] = np.nan, np.inf, -np.inf, np.nan, 3e38
    many, one = (ops.VQKVCache(1, 2, 8, 64, 8, 64, *books) for _ in range(2))
    kt, vt, qt = (torch.from_numpy(a).to(cuda) for a in (k, v, q))
    many.prefill(kt, vt, qt)
    for s in range(20):
        one.append(kt[s], vt[s])
    a, b = many.read(0, 20), one.read(0, 20)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])


def test_positions_of_many_sequences(cuda):
    """5000 sequences: 15 positions of them are more than the 65535 a grid takes in z."""
    B, S = 5000, 15
    rng = np.random.default_rng(0)
    books = [rng.standard_normal((1, 256, 16)).astype(np.float32) / 8 for _ in range(2)]
    many, one = (ops.VQKVCache(B, 1, 1, 64, 16, 20, *books) for _ in range(2))
    k, v, q = (torch.randn(S, B, 1, 64, device=cuda, generator=torch.Generator(cuda).manual_seed(i)) for i in range(3))
    got = many.prefill(k, v, q)
    for s in range(S):
        one.append(k[s], v[s])
        assert torch.allclose(got[s], one.decode(q[s]), rtol=1e-4, atol=2e-6)
