"""The work that users of this framework have it do, as cases that can be timed: VQ linears, SwiGLU blocks, groups of
layers, top-k MoE layers, the quantised KV cache and a decoder stack, all through the package's public entry points.

``listed()`` has the sizes of the benchmark configurations; ``draw(rng)`` spreads over the ranges around them.  Inputs and
weights are made on the GPU from the seed alone, with the distributions of ``synth`` (codes uniform, codebooks Gaussian,
0.38 % outliers of 15 to 36 sigma), and handed to the package as it takes them."""
import math

import numpy as np
import torch

from ojasx_b200 import inference_engine as ie
from ojasx_b200 import ops, synth

BLOCK = 8            # dimensions per code
OUTLIERS = 0.0038    # share of weight cells that are exact outliers
SIGMA = 0.02
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}


def listed():
    return [
        # One VQ linear, one token: the smallest call (an attention or output projection of a decoding model).
        {"name": "linear 2560x2560 b1", "kind": "linear", "k": 2560, "m": 2560, "batch": 1, "dtype": "f32"},
        # SwiGLU block at its three regimes: one decoding sequence, a batch of sequences, a chunk of a prompt.
        {"name": "mlp b1", "kind": "mlp", "k": 2560, "m": 6912, "batch": 1, "dtype": "bf16"},
        {"name": "mlp b16", "kind": "mlp", "k": 2560, "m": 6912, "batch": 16, "dtype": "bf16"},
        {"name": "mlp b256", "kind": "mlp", "k": 2560, "m": 6912, "batch": 256, "dtype": "bf16"},
        # Many independent layers in one launch, more code bytes than L2 holds: the headline GEMV.
        {"name": "group 222 layers", "kind": "group", "k": 2560, "m": 6912, "layers": 222, "dtype": "f32"},
        # 512-expert top-10 layer, router included: one token, a decoding batch, a chunk of a prompt.
        {"name": "moe 1", "kind": "moe", "h": 2560, "i": 640, "experts": 512, "top_k": 10, "tokens": 1, "dtype": "f32"},
        {"name": "moe 32", "kind": "moe", "h": 2560, "i": 640, "experts": 512, "top_k": 10, "tokens": 32, "dtype": "bf16"},
        {"name": "moe 256", "kind": "moe", "h": 2560, "i": 640, "experts": 512, "top_k": 10, "tokens": 256, "dtype": "f32"},
        # Attention of a decoding layer over its quantised cache: a short chat, and a batch with long contexts.
        {"name": "kv 2048 b1", "kind": "kv", "ctx": 2048, "batch": 1, "kv_heads": 8, "share": 4, "hd": 128, "steps": 32, "dtype": "bf16"},
        {"name": "kv 32768 b16", "kind": "kv", "ctx": 32768, "batch": 16, "kv_heads": 8, "share": 4, "hd": 128, "steps": 4, "dtype": "bf16"},
        # The decoder stack end to end: a prompt into the caches, and a short prompt continued token by token.
        {"name": "stack prefill 512", "kind": "stack", "layers": 2, "batch": 1, "prompt": 512, "steps": 0, "vocab": 32768, "experts": 512},
        {"name": "stack decode 32", "kind": "stack", "layers": 2, "batch": 1, "prompt": 32, "steps": 32, "vocab": 32768, "experts": 512},
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["linear", "mlp", "mlp", "group", "moe", "moe", "kv", "kv", "stack"])
    dtype = rng.choice(["f32", "bf16"])
    if kind == "linear":     # any width that is whole blocks, any number of rows
        return {"kind": kind, "k": BLOCK * _log(rng, 64, 864), "m": _log(rng, 256, 16384), "batch": _log(rng, 1, 8), "dtype": dtype}
    if kind == "mlp":        # bf16 as a model runs it; widths whole multiples of 64, batches of every size
        return {"kind": kind, "k": 64 * rng.randint(16, 40), "m": 64 * rng.randint(32, 108), "batch": _log(rng, 1, 384), "dtype": "bf16"}
    if kind == "group":
        return {"kind": kind, "k": 128 * rng.randint(8, 20), "m": rng.randint(1500, 6912), "layers": _log(rng, 24, 222), "dtype": dtype}
    if kind == "moe":
        return {"kind": kind, "h": 128 * rng.randint(8, 20), "i": 64 * rng.randint(4, 10), "experts": rng.choice([64, 128, 256, 512]),
                "top_k": rng.randint(4, 10), "tokens": _log(rng, 1, 256), "dtype": dtype}
    if kind == "kv":
        batch = _log(rng, 1, 16)
        return {"kind": kind, "ctx": _log(rng, 500, 32768 * 16 // (4 * batch)), "batch": batch, "kv_heads": rng.choice([2, 4, 8]),
                "share": rng.choice([1, 2, 4, 4, 8]), "hd": rng.choice([64, 128, 128]), "steps": 8, "dtype": dtype}
    prompt = _log(rng, 16, 384)
    return {"kind": kind, "layers": rng.randint(1, 2), "batch": rng.choice([1, 1, 2, 4]), "prompt": prompt,
            "steps": rng.choice([0, rng.randint(4, 32)]), "vocab": 1000 * rng.randint(4, 32), "experts": rng.choice([64, 128, 256])}


# ---------------------------------------------------------------------------------------------- inputs and weights

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(1000003 * int(seed) + 17)
    return g


def _randn(g, *shape, scale=1.0):
    return torch.randn(*shape, generator=g, device="cuda") * scale


def _codes(g, *shape):
    return torch.randint(0, 256, shape, generator=g, device="cuda", dtype=torch.uint8).cpu().numpy()


def _outliers(g, rows, cols):
    """CSR of distinct random cells of a [rows, cols] matrix (int32 row pointers and columns, f32 values), host arrays."""
    n = int(OUTLIERS * rows * cols)
    cells = torch.unique(torch.randint(0, rows * cols, (n,), generator=g, device="cuda", dtype=torch.int64))
    r, c = cells // cols, (cells % cols).to(torch.int32)
    ptr = torch.zeros(rows + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.cumsum(torch.bincount(r, minlength=rows), 0)
    u = torch.rand(cells.shape[0], generator=g, device="cuda") * 2 - 1
    vals = torch.sign(u) * (15.0 + 21.0 * u.abs()) * SIGMA
    return ptr.to(torch.int32).cpu().numpy(), c.cpu().numpy(), vals.cpu().numpy()


def _linear_weights(g, k, m):
    return synth.VQLinearWeights(k, m, BLOCK, _randn(g, 256, BLOCK, scale=SIGMA).cpu().numpy(), _codes(g, m, k // BLOCK), None, None,
                                 _outliers(g, m, k))


def _moe_weights(g, h, i, experts):
    cb = [_randn(g, 256, BLOCK, scale=SIGMA).cpu().numpy() for _ in range(2)]
    return synth.VQMoEWeights(experts, h, i, BLOCK, cb[0], cb[1], _codes(g, experts, 2 * i, h // BLOCK), np.ones((experts, 2 * i), np.float32),
                              _codes(g, experts, h, i // BLOCK), np.ones((experts, h), np.float32),
                              _randn(g, experts, h, scale=SIGMA).cpu().numpy(), _outliers(g, experts * 2 * i, h), _outliers(g, experts * h, i))


def _stack_config(case):
    return ie.StackConfig(layers=case["layers"], vocab=case["vocab"], experts=case["experts"], max_seq_len=1024)


def _stack_weights(g, cfg):
    h, hd = cfg.hidden, cfg.head_dim
    norm = lambda: (1.0 + 0.1 * _randn(g, h)).cpu().numpy()  # noqa: E731
    book = lambda: _randn(g, cfg.kv_heads, 256, BLOCK, scale=1.0 / math.sqrt(hd)).cpu().numpy()  # noqa: E731
    layers = [ie.LayerWeights(q=_linear_weights(g, h, cfg.q_heads * hd), k=_linear_weights(g, h, cfg.kv_heads * hd),
                              v=_linear_weights(g, h, cfg.kv_heads * hd), o=_linear_weights(g, cfg.q_heads * hd, h),
                              moe=_moe_weights(g, h, cfg.inter, cfg.experts), norm1=norm(), norm2=norm(), k_codebook=book(), v_codebook=book())
              for _ in range(cfg.layers)]
    return ie.StackWeights(layers, _randn(g, cfg.vocab, h).cpu().numpy(), norm(), _linear_weights(g, h, cfg.vocab))


def prepare(case, seed):
    g = _gen(seed)
    dtype = DTYPES[case.get("dtype", "f32")]
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "linear":
        s["layer"] = ops.VQLinear.from_weights(_linear_weights(g, case["k"], case["m"]))
        s["x"] = _randn(g, case["batch"], case["k"]).to(dtype)
    elif kind == "mlp":
        k, m = case["k"], case["m"]
        s["block"] = ops.VQMLP(*[ops.VQLinear.from_weights(_linear_weights(g, *shape)) for shape in ((k, m), (k, m), (m, k))])
        s["x"] = _randn(g, case["batch"], k).to(dtype)
    elif kind == "group":    # a few distinct sets of host arrays; every layer owns its copy on the device
        sets = [_linear_weights(g, case["k"], case["m"]) for _ in range(6)]
        s["layers"] = [ops.VQLinear.from_weights(sets[p % len(sets)]) for p in range(case["layers"])]
        s["group"] = ops.VQLinearGroup(s["layers"])
        s["x"] = _randn(g, case["layers"], case["k"]).to(dtype)
        s["y"] = torch.zeros(case["layers"], case["m"], dtype=dtype, device="cuda")
    elif kind == "moe":
        s["moe"] = ops.VQMoE(_moe_weights(g, case["h"], case["i"], case["experts"]))
        s["moe"].reserve(case["tokens"], case["top_k"])
        s["x"] = _randn(g, case["tokens"], case["h"]).to(dtype)
    elif kind == "kv":
        b, hk, hd, ctx, n = case["batch"], case["kv_heads"], case["hd"], case["ctx"], case["steps"]
        sig = 1.0 / math.sqrt(hd)
        books = [_randn(g, hk, 256, BLOCK, scale=sig).cpu().numpy() for _ in range(2)]
        s["cache"] = ops.VQKVCache(b, hk, hk * case["share"], hd, BLOCK, ctx + n, *books)
        s["cache"].load(_codes(g, b, hk, ctx, hd // BLOCK), _codes(g, b, hk, ctx, hd // BLOCK))
        s["k"], s["v"] = (_randn(g, n, b, hk, hd, scale=sig).to(dtype) for _ in range(2))
        s["q"] = _randn(g, n, b, hk * case["share"], hd).to(dtype)
        s["out"] = torch.empty_like(s["q"])
    else:
        cfg = _stack_config(case)
        stack = ie.VQDecoderStack(_stack_weights(g, cfg), cfg, case["batch"], use_graph=case["steps"] > 0)
        s["stack"] = stack
        s["prompt"] = torch.randint(0, cfg.vocab, (case["batch"], case["prompt"]), generator=g, device="cuda")
        s["next"] = torch.randint(0, cfg.vocab, (max(1, case["steps"]), case["batch"]), generator=g, device="cuda")
        if case["steps"]:    # the step is captured once, on prefilled caches, as a serving program does at start-up
            stack.prefill(s["prompt"])
            stack.decode_step(s["next"][0])
            stack.reset()
    return s


def run(s):
    kind = s["kind"]
    if kind == "linear":
        return s["layer"](s["x"])
    if kind == "mlp":
        return s["block"](s["x"])
    if kind == "group":
        return s["group"].forward(s["x"], s["y"])
    if kind == "moe":
        return s["moe"].forward_routed(s["x"], s["case"]["top_k"])
    if kind == "kv":         # a few tokens in a row; the cache is cropped back, so every pass sees the same context
        cache = s["cache"]
        cache.crop(s["case"]["ctx"])
        for t in range(s["case"]["steps"]):
            cache.append(s["k"][t], s["v"][t])
            cache.decode(s["q"][t], out=s["out"][t])
        return s["out"]
    # the stack is fed given tokens, so that a pass does the same work whatever the last bits of the logits are
    stack = s["stack"]
    stack.reset()
    logits = [stack.prefill(s["prompt"])]
    for t in range(s["case"]["steps"]):
        logits.append(stack.decode_step(s["next"][t]).clone())
    return torch.stack(logits)


# ---------------------------------------------------------------------------------------------- bounds and tolerances

def _linear_work(k, m, batch, io):
    nnz = int(OUTLIERS * k * m)
    nbytes = m * (k // BLOCK) + 1024 * BLOCK + 4 * (m + 1) + 8 * nnz + batch * (k + m) * io
    return nbytes, batch * (2 * 256 * k + m * (k // BLOCK) + 2 * nnz)   # tables, one addition per code, outliers


def work(case):
    io = 4 if case.get("dtype", "f32") == "f32" else 2
    kind = case["kind"]
    if kind == "linear":
        b, f = _linear_work(case["k"], case["m"], case["batch"], io)
    elif kind == "mlp":
        parts = [_linear_work(case["k"], case["m"], case["batch"], io)] * 2 + [_linear_work(case["m"], case["k"], case["batch"], io)]
        # gate, up and the gated vector stay on the chip
        b = sum(p[0] for p in parts) - case["batch"] * (4 * case["m"] + case["k"]) * io + case["batch"] * case["m"] * io
        f = sum(p[1] for p in parts)
    elif kind == "group":
        b, f = (case["layers"] * v for v in _linear_work(case["k"], case["m"], 1, io))
    elif kind == "moe":
        b, f = _moe_work(case["h"], case["i"], case["experts"], case["top_k"], case["tokens"], io)
    elif kind == "kv":
        g = case["hd"] // BLOCK
        heads = case["batch"] * case["kv_heads"]
        per = 2 * g * heads * case["ctx"] + heads * case["hd"] * (2 + 2 * case["share"]) * io
        f = case["steps"] * heads * case["ctx"] * case["share"] * (g + 2 * case["hd"])
        b = case["steps"] * per + 2 * case["kv_heads"] * 1024 * BLOCK
    else:
        cfg = _stack_config(case)
        h, hd = cfg.hidden, cfg.head_dim
        b = f = 0
        for rows, last in [(case["batch"] * case["prompt"], case["batch"])] + [(case["batch"], case["batch"])] * case["steps"]:
            lin = [_linear_work(h, cfg.q_heads * hd, rows, 4), _linear_work(h, cfg.kv_heads * hd, rows, 4),
                   _linear_work(h, cfg.kv_heads * hd, rows, 4), _linear_work(cfg.q_heads * hd, h, rows, 4),
                   _moe_work(h, cfg.inter, cfg.experts, cfg.top_k, rows, 4)]
            head = _linear_work(h, cfg.vocab, last, 4)
            b += cfg.layers * sum(p[0] for p in lin) + head[0]
            f += cfg.layers * sum(p[1] for p in lin) + head[1]
        pairs = case["batch"] * (case["prompt"] * (case["prompt"] + 1) // 2 + case["steps"] * (case["prompt"] + case["steps"] // 2))
        f += cfg.layers * pairs * cfg.q_heads * (hd // BLOCK + 2 * hd)
    return {"bytes": b, "flops": f}


def _moe_work(h, i, experts, top_k, tokens, io):
    hit = experts * (1.0 - (1.0 - top_k / experts) ** tokens)     # experts that at least one token is routed to
    gu, dn = 2 * i * (h // BLOCK), h * (i // BLOCK)
    nnz = OUTLIERS * 3 * h * i
    nbytes = int(hit * (gu + dn + 8 * nnz + 4 * (2 * i + h)) + 4 * experts * h + 2 * tokens * h * io)
    flops = tokens * (2 * experts * h + 2 * 256 * h + top_k * (gu + dn + 2 * 256 * i + 2 * nnz))
    return nbytes, int(flops)


def tolerance(case):
    # Measured against restatements in 64 bits: linears, groups and MoE 2e-7 to 3e-7 in fp32, the cache 1e-7; one rounding to
    # bf16 on the way out 1.7e-3; a bf16 block of three linears 3.4e-3 to 4.6e-3.
    if case["kind"] == "stack":
        # fp32, but cache codes are whole numbers: last-bit differences (3e-7 in the embeddings) move the logits by 7e-7, and
        # by 1e-4 to 4e-4 where they tip one of the hundreds of thousands of codes, as one in six such differences does
        return {"rel": 2e-3}
    if case.get("dtype", "f32") == "bf16":
        return {"rel": 1e-2 if case["kind"] == "mlp" else 7e-3}
    return {"rel": 1.5e-6}
