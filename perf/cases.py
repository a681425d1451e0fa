"""Cases that stand for what users of this framework have it do, each through its public entry points.

``kind`` says which path a case takes:

* ``gemv`` / ``swiglu``: one activation-sparse projection of one token (``teal.kernels.sparse_gemv``), the call that a
  patched model makes for every linear layer of a decode step;
* ``quantizer``: vectors into 3-bit codes and stored codes back into vectors (``TurboQuantMSE``), as a cache does that
  moves old positions into its cold store and reads the store back;
* ``decode_attention``: one query token per sequence over the packed pages of a ``PagedKVCache``;
* ``paged_prompt``: a prompt through a ``PagedKVCache`` in chunks, appended and attended to;
* ``llama_prompt`` / ``llama_decode``: ``DecodeEngine`` on a Llama / Mistral-shaped model, prompt pass and decode steps;
* ``batch_decode``: one step of ``BatchDecodeEngine``, many sequences at a long context;
* ``mixer_prompt`` / ``mixer_generate``: ``MixerDecodeEngine`` on the two mixer designs, a prompt in portions, and a prompt
  followed by single tokens.

Sizes are those of the repository's benchmark configurations or fractions of them (fewer layers, narrower widths), and
odd lengths between. Weights and inputs are random, of the scale that the benchmark's generators use.
"""

from __future__ import annotations

import math

import torch

HEAD = 128                     # head size of every TurboQuant path
VOCAB = 32768
WINDOW, POOL = 1024, 16        # mixer designs: sliding window, tokens per pooled block
KV_RANK, ROT_DIM = 512, 64     # latent layers


# ── the cases ────────────────────────────────────────────────────────────────────────────────────────────────

def listed() -> list[dict]:
    return [
        # the smallest call: one eighth of a 7B model's gate / up pair, as a tensor-parallel rank runs it per layer
        dict(name="swiglu_shard", kind="swiglu", n=1792, z=4096, sparsity=0.4, dtype="float16"),
        # the widest reduction of a 7B model's block, the benchmark's first configuration
        dict(name="gemv_down", kind="gemv", n=4096, z=14336, sparsity=0.4, dtype="float16"),
        # 8 kv heads x 8193 positions of one layer moved into the cold store, and as many read back
        dict(name="quantizer_layer", kind="quantizer", vectors=65544, bits=3, dtype="float16"),
        # one layer of a serving step: 16 sequences around 4096 tokens, not all of one length
        dict(name="decode_attention_16x4k", kind="decode_attention", batch=16, tokens=3851, more=490, longer=8, kv_heads=8),
        # one layer of a 2000-token prompt that arrives in chunks of 512
        dict(name="paged_prompt_2k", kind="paged_prompt", batch=1, tokens=2000, chunk=512, kv_heads=8),
        # the headline model: 512-token prompt, then decode steps at 40 % sparsity (tokens given, as in scoring)
        dict(name="llama_prompt_7b", kind="llama_prompt", hidden=4096, layers=32, tokens=512, chunk=512),
        dict(name="llama_decode_7b", kind="llama_decode", hidden=4096, layers=32, tokens=512, steps=4, sparsity=0.4),
        # serving at long context: 32 sequences x 4096 tokens, two layers of the 7B shape
        dict(name="batch_decode_32x4k", kind="batch_decode", hidden=4096, layers=2, batch=32, tokens=4096),
        # the mixer designs: a prompt, and an answer of single tokens behind a prompt
        dict(name="rorosun_prompt_2k", kind="mixer_prompt", design="rorosun", width=2048, layers=4, tokens=2048, chunk=2048,
             dtype="bfloat16"),
        dict(name="rorosun_generate", kind="mixer_generate", design="rorosun", width=1024, layers=6, tokens=1300, steps=48,
             dtype="bfloat16"),
        dict(name="pefitar_prompt_4k", kind="mixer_prompt", design="pefitar", width=2048, layers=4, tokens=4000, chunk=2048,
             dtype="bfloat16"),
        dict(name="pefitar_generate", kind="mixer_generate", design="pefitar", width=2048, layers=4, tokens=2048, steps=48,
             dtype="bfloat16"),
    ]


def _spread(rng, low: int, high: int) -> int:
    """A whole number between the two, evenly over the logarithm."""
    return max(low, min(high, round(math.exp(rng.uniform(math.log(low), math.log(high + 1))))))


def draw(rng) -> dict:
    kind = rng.choice(["gemv", "swiglu", "quantizer", "decode_attention", "paged_prompt", "llama_prompt", "llama_decode",
                       "batch_decode", "mixer_prompt", "mixer_generate"])
    if kind in ("gemv", "swiglu"):
        return dict(kind=kind, n=8 * _spread(rng, 64, 1792), z=_spread(rng, 512, 14336), sparsity=rng.choice([0.0, 0.25, 0.4, 0.5]),
                    dtype=rng.choice(["float16", "float16", "bfloat16", "float32"]))
    if kind == "quantizer":
        return dict(kind=kind, vectors=_spread(rng, 8, 262144), bits=rng.choice([2, 3, 3, 3, 4]),
                    dtype=rng.choice(["float16", "float16", "float32"]))
    if kind == "decode_attention":
        batch = _spread(rng, 1, 64)
        tokens = _spread(rng, 17, min(16384, 131072 // batch))
        return dict(kind=kind, batch=batch, tokens=tokens, more=rng.randint(0, max(1, tokens // 4)), longer=rng.randint(0, batch),
                    kv_heads=rng.choice([2, 4, 8, 8]))
    if kind == "paged_prompt":
        tokens = _spread(rng, 24, 4096)
        return dict(kind=kind, batch=rng.choice([1, 1, 2]), tokens=tokens, chunk=rng.choice([tokens, max(1, tokens // 2), 512, 333]),
                    kv_heads=rng.choice([2, 4, 8, 8]))
    if kind == "llama_prompt":
        tokens = _spread(rng, 2, 2048)
        return dict(kind=kind, hidden=rng.choice([1024, 2048, 4096]), layers=rng.randint(1, 6), tokens=tokens,
                    chunk=rng.choice([tokens, 512, 200]))
    if kind == "llama_decode":
        return dict(kind=kind, hidden=rng.choice([1024, 2048, 4096]), layers=rng.randint(1, 8), tokens=_spread(rng, 16, 3000),
                    steps=4, sparsity=rng.choice([0.0, 0.25, 0.4, 0.5]))
    if kind == "batch_decode":
        batch = _spread(rng, 2, 80)
        return dict(kind=kind, hidden=rng.choice([1024, 2048, 4096]), layers=rng.randint(1, 2), batch=batch,
                    tokens=_spread(rng, 64, min(4096, 65536 // batch)))
    design, dtype = rng.choice(["rorosun", "pefitar"]), rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"])
    width = rng.choice([1024, 2048]) if dtype == "bfloat16" else 1024
    if kind == "mixer_prompt":
        tokens = _spread(rng, 48, 3000 if dtype == "bfloat16" else 700)
        return dict(kind=kind, design=design, width=width, layers=2 * rng.randint(1, 2), tokens=tokens,
                    chunk=rng.choice([tokens, 1024, 600]), dtype=dtype)
    return dict(kind=kind, design=design, width=width, layers=2 * rng.randint(1, 3),
                tokens=_spread(rng, 8, 2400 if dtype == "bfloat16" else 300), steps=32, dtype=dtype)


# ── inputs ───────────────────────────────────────────────────────────────────────────────────────────────────

def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _dtype(case) -> torch.dtype:
    return getattr(torch, case["dtype"])


def _projection(case, seed: int) -> dict:
    """Weights N(0, 0.02) in fp16 and a Laplace activation with the threshold that hides its ``sparsity`` smallest."""
    gen, n, z = _gen(seed), case["n"], case["z"]
    u = torch.rand(1, 1, z, generator=gen, device="cuda") - 0.5
    x = (-torch.sign(u) * torch.log1p(-2 * u.abs().clamp(max=0.4999999))).half()
    k = int(case["sparsity"] * z)
    t = float(x.abs().flatten().float().kthvalue(k).values) if k else -1.0
    w = [(torch.randn(n, z, generator=gen, device="cuda") * 0.02).half() for _ in range(2 if case["kind"] == "swiglu" else 1)]
    return {"x": x.to(_dtype(case)), "t": t, "w": w}


def _rotation(seed: int, dtype=torch.float32) -> torch.Tensor:
    """The rotation that a quantizer with this seed uses: the Q of a seeded Gaussian matrix, R's diagonal positive."""
    q, r = torch.linalg.qr(torch.randn(HEAD, HEAD, generator=torch.Generator().manual_seed(seed)))
    return (q * torch.sign(torch.diagonal(r)).unsqueeze(0)).contiguous().to("cuda", dtype)


def _codebook(bits: int, dtype=torch.float64) -> tuple:
    """(centroids, decision boundaries): constants of the format."""
    from leankv_b200.turboquant.codebook import get_codebook_tensors

    cents, bounds = get_codebook_tensors(HEAD, bits, "cpu")
    return cents.float().to("cuda", dtype), bounds[1:-1].float().to("cuda", dtype)


def _pack(codes: torch.Tensor, bits: int) -> torch.Tensor:
    """Codes [.., 128] as the store keeps them: two (four, for 2 bits) fields a byte, the first one lowest."""
    per, width = (4, 2) if bits == 2 else (2, 4)
    c = codes.reshape(*codes.shape[:-1], -1, per).to(torch.int32)
    return sum(c[..., i] << (width * i) for i in range(per)).to(torch.uint8)


def _vectors(case, seed: int) -> dict:
    """New vectors with a few large channels, and a store of as many that were quantized earlier."""
    gen, n = _gen(seed), case["vectors"]
    x = torch.randn(n, HEAD, generator=gen, device="cuda")
    x[:, torch.randperm(HEAD, generator=gen, device="cuda")[:4]] *= 8.0
    old = torch.randn(n, HEAD, generator=gen, device="cuda")
    norms = old.norm(dim=-1)
    codes = torch.bucketize((old / norms.unsqueeze(1)) @ _rotation(42).t(), _codebook(case["bits"], torch.float32)[1])
    return {"x": x.to(_dtype(case)), "codes": codes, "norms": norms.half().float()}


def _kv(case, seed: int, tokens: int) -> dict:
    """Keys and values with a few outlier channels a head, and a query a token or one a sequence."""
    gen, b, g = _gen(seed), case["batch"], case["kv_heads"]
    out = {}
    for name in ("k", "v"):
        t = torch.randn(b, g, tokens, HEAD, generator=gen, device="cuda")
        for h in range(g):
            t[:, h, :, torch.randperm(HEAD, generator=gen, device="cuda")[:4]] *= 8.0
        out[name] = t.half()
    shape = (b, 4 * g, HEAD) if case["kind"] == "decode_attention" else (b, 4 * g, tokens, HEAD)
    out["q"] = torch.randn(shape, generator=gen, device="cuda").half()
    return out


def _lengths(case) -> list[int]:
    """``longer`` of the sequences hold ``more`` tokens than the others."""
    return [case["tokens"] + (case["more"] if b < case["longer"] else 0) for b in range(case["batch"])]


def _llama_config(case):
    from leankv_b200.engine import DecoderConfig

    h = case["hidden"]
    return DecoderConfig(vocab_size=VOCAB, hidden_size=h, intermediate_size=h * 7 // 2, num_layers=case["layers"],
                         num_q_heads=h // HEAD, num_kv_heads=h // HEAD // 4)


def _llama_weights(case, seed: int) -> dict:
    """Random weights whose stream starts at order one and takes a few per cent from every branch, as in deep trained models.
    (With branches as large as the stream, one input that a last-bit difference lifts over its threshold changes every
    later layer's choice: the outputs of two correct implementations part after a few layers.)"""
    from leankv_b200.engine import DecodeEngine

    w = DecodeEngine.random_weights(_llama_config(case), torch.device("cuda"), seed)
    w["embed"] *= 50.0
    for lw in w["layers"]:
        for n in ("wo_t", "wdown_t"):
            lw[n] *= 1.0 / 64
    return w


def _tokens(seed: int, *shape: int) -> torch.Tensor:
    return torch.randint(0, VOCAB, shape, generator=torch.Generator().manual_seed(seed))


def _thresholds(case, w: dict, seed: int):
    """A calibration's result: per projection the magnitude below which ``sparsity`` of its inputs lie over 64 tokens."""
    if not case["sparsity"]:
        return None
    seen: dict = {}
    _plain_llama(case, w, _tokens(seed + 7777, 1, 64).cuda(), [63], torch.float32, note=lambda l, n, x: seen.update({(l, n): x}))
    out: dict = {}
    names = {"qkv": ("q_proj", "k_proj", "v_proj"), "o": ("o_proj",), "gu": ("gate_proj", "up_proj"), "down": ("down_proj",)}
    for (l, n), x in seen.items():
        t = float(x.abs().flatten().kthvalue(max(1, int(case["sparsity"] * x.numel()))).values.half())
        out.setdefault(l, {}).update({p: t for p in names[n]})
    return out


def _mixer_model(case) -> dict:
    """The benchmark's layer shapes at this width."""
    w = case["width"]
    heads, ff = w // 128, w * 7 // 2
    mlp = {"kind": "dense", "ff": ff}
    if case["design"] == "rorosun":
        mixer = {"left": {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                          "mask": {"size": WINDOW, "pool": POOL}},
                 "right": {"heads": w // 64, "dim": 64}, "left_scale": 0.7, "right_scale": 0.7}
        return {"architecture": "Rorosun", "vocab": VOCAB, "width": w, "norm": {"eps": 1e-5},
                "layers": [{"type": "parallel", "mixer": mixer, "mlp": mlp}] * case["layers"]}
    rot = lambda dims: {"base": 10000.0, "dims": dims}
    attn = {"type": "attention", "mlp": mlp, "mixer": {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128,
                                                       "scale": 128 ** -0.5, "rot": rot(128)}}
    latent = {"type": "latent_attention", "mlp": mlp, "mixer": {
        "heads": heads, "dim": 128, "rot_dim": ROT_DIM, "vdim": 128, "q_rank": w // 2, "kv_rank": KV_RANK,
        "mask": {"size": WINDOW}, "scale": (128 + ROT_DIM) ** -0.5, "rot": rot(ROT_DIM)}}
    return {"architecture": "Pefitar", "vocab": VOCAB, "width": w, "norm": {"eps": 1e-5},
            "layers": [attn, latent] * (case["layers"] // 2), "residual_mult": 0.5, "logit_softcap": 30.0}


def _mixer_tensors(case, seed: int) -> dict:
    from leankv_b200.mixer_engine import MixerDecodeEngine, MixerModelConfig

    return MixerDecodeEngine.random_tensors(MixerModelConfig.from_dict(_mixer_model(case)), torch.device("cuda"), seed)


def _mixer_tokens(case, seed: int) -> tuple:
    ids = _tokens(seed, case["tokens"] + case.get("steps", 0)).tolist()
    want = [i for i in range(case["tokens"]) if i % 61 == 60 or i == case["tokens"] - 1]
    return ids, want


# ── what a user's program has before the call ────────────────────────────────────────────────────────────────

def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind in ("gemv", "swiglu"):
        from leankv_b200.teal.kernels.sparse_gemv import prepare_weight_for_sparse_gemv

        p = _projection(case, seed)
        return {"kind": kind, "x": p["x"], "t": p["t"], "w": [prepare_weight_for_sparse_gemv(w) for w in p["w"]]}
    if kind == "quantizer":
        from leankv_b200.turboquant.quantizer import MSEQuantized, TurboQuantMSE

        p = _vectors(case, seed)
        return {"kind": kind, "quantizer": TurboQuantMSE(HEAD, case["bits"], "cuda", seed=42), "x": p["x"],
                "store": MSEQuantized(_pack(p["codes"], case["bits"]), p["norms"], case["bits"])}
    if kind in ("decode_attention", "paged_prompt"):
        from leankv_b200.turboquant.paged_cache import PagedKVCache

        g = case["kv_heads"]
        n = _lengths(case) if kind == "decode_attention" else [case["tokens"]] * case["batch"]
        cache = PagedKVCache(num_layers=1, num_kv_heads=g, num_q_heads=4 * g, max_pages=sum(-(-t // 16) for t in n) + 1,
                             device="cuda")
        p = _kv(case, seed, max(n))
        if kind == "paged_prompt":
            return {"kind": kind, "cache": cache, "chunk": case["chunk"], **p}
        cache.append(0, p["k"][:, :, :n[-1]], p["v"][:, :, :n[-1]])
        if case["longer"] and max(n) > n[-1]:
            cache.append(0, p["k"][:case["longer"], :, n[-1]:], p["v"][:case["longer"], :, n[-1]:])
        return {"kind": kind, "cache": cache, "q": p["q"]}
    if kind in ("llama_prompt", "llama_decode"):
        from leankv_b200.engine import DecodeEngine

        w = _llama_weights(case, seed)
        ids = _tokens(seed, case["tokens"] + case.get("steps", 0))
        prompt, thresholds = ids[:case["tokens"]].tolist(), None
        if kind == "llama_decode":
            thresholds = _thresholds(case, w, seed)
        engine = DecodeEngine(_llama_config(case), w, "cuda", max_seq_len=case["tokens"] + 128, thresholds=thresholds)
        if kind == "llama_prompt":
            return {"kind": kind, "engine": engine, "prompt": prompt, "chunk": case["chunk"]}
        engine.prefill(prompt)
        engine.capture()
        return {"kind": kind, "engine": engine, "at": engine.state.clone(), "given": ids[case["tokens"]:].cuda().reshape(-1, 1),
                "logits": torch.empty(case["steps"], VOCAB, dtype=torch.float16, device="cuda")}
    if kind == "batch_decode":
        from leankv_b200.batch_engine import BatchDecodeEngine

        engine = BatchDecodeEngine(_llama_config(case), _llama_weights(case, seed), "cuda", case["batch"],
                                   max_seq_len=case["tokens"] + 64)
        ids = _tokens(seed, case["batch"], case["tokens"] + 1)
        engine.prefill(ids[:, :-1].contiguous(), chunk=1024)
        engine.capture()
        return {"kind": kind, "engine": engine, "pos": engine.pos.clone(), "steps": engine.steps.clone(),
                "given": ids[:, -1].cuda()}
    from leankv_b200.mixer_engine import MixerDecodeEngine, MixerModelConfig

    ids, want = _mixer_tokens(case, seed)
    n, steps = case["tokens"], case.get("steps", 0)
    engine = MixerDecodeEngine(MixerModelConfig.from_dict(_mixer_model(case)), _mixer_tensors(case, seed), "cuda",
                               max_seq_len=n + steps + 8, dtype=_dtype(case), max_chunk=min(case.get("chunk", n), 2048))
    if steps:
        engine.extend(ids[:2])
        engine.capture()
    return {"kind": kind, "engine": engine, "prompt": ids[:n], "given": ids[n:], "want": want}


# ── one pass ─────────────────────────────────────────────────────────────────────────────────────────────────

def run(state: dict):
    kind = state["kind"]
    if kind == "gemv":
        from leankv_b200.teal.kernels.sparse_gemv import sparse_gemv

        return sparse_gemv(state["x"], state["w"][0], state["t"])
    if kind == "swiglu":
        from leankv_b200.teal.kernels.sparse_gemv import sparse_swiglu

        return sparse_swiglu(state["x"], state["w"][0], state["w"][1], state["t"], state["t"])
    if kind == "quantizer":
        q = state["quantizer"].quantize(state["x"])
        return {"indices": q.indices, "norms": q.norms, "restored": state["quantizer"].dequantize(state["store"])}
    if kind == "decode_attention":
        return state["cache"].decode_attention(0, state["q"])
    if kind == "paged_prompt":
        cache, n, chunk = state["cache"], state["k"].shape[2], state["chunk"]
        cache.reset()
        out = []
        for s in range(0, n, chunk):
            cache.append(0, state["k"][:, :, s:s + chunk], state["v"][:, :, s:s + chunk])
            out.append(cache.prefill_attention(0, state["q"][:, :, s:s + chunk]))
        return out
    engine = state["engine"]
    if kind == "llama_prompt":
        engine.prefill(state["prompt"], chunk=state["chunk"])
        return engine.prefill_logits
    if kind == "llama_decode":           # score the given continuation from the end of the prompt
        engine.state.copy_(state["at"])
        for i in range(len(state["given"])):
            engine.token.copy_(state["given"][i])
            engine.step()
            state["logits"][i].copy_(engine.logits)
        return state["logits"]
    if kind == "batch_decode":           # likewise, one step
        engine.pos.copy_(state["pos"])
        engine.steps.copy_(state["steps"])
        engine.tokens.copy_(state["given"])
        engine.step()
        return engine.logits
    engine.reset()
    out = [engine.extend(state["prompt"], state["want"])]
    if state["given"]:
        out.append(torch.cat([engine.extend([t], [0]) for t in state["given"]]))
    return out


# ── what a pass cannot do without ────────────────────────────────────────────────────────────────────────────

def _llama_params(case) -> int:
    """Weights of one layer."""
    h = case["hidden"]
    return h * h + h * h // 2 + h * h + 3 * h * (h * 7 // 2)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("gemv", "swiglu"):
        m = 2 if kind == "swiglu" else 1
        live = case["z"] - int(case["sparsity"] * case["z"])
        return {"bytes": 2.0 * m * live * case["n"] + 2 * case["z"] + 2 * case["n"], "flops": 2.0 * m * live * case["n"]}
    if kind == "quantizer":
        n, size, packed = case["vectors"], 4 if case["dtype"] == "float32" else 2, 32 if case["bits"] == 2 else 64
        return {"bytes": n * (HEAD * size + packed + size + packed + 4 + 4.0 * HEAD), "flops": n * 4.0 * HEAD * HEAD}
    if kind == "decode_attention":
        keys, g = sum(_lengths(case)), case["kv_heads"]
        return {"bytes": keys * 2.0 * g * 50 + case["batch"] * 4 * g * HEAD * 4, "flops": keys * 4 * g * 4.0 * HEAD}
    if kind == "paged_prompt":
        n, g, b = case["tokens"], case["kv_heads"], case["batch"]
        return {"bytes": b * n * (2.0 * g * (2 * HEAD + 50) + 4 * g * HEAD * 4), "flops": b * n * (n + 1) / 2 * 4 * g * 4.0 * HEAD}
    if kind in ("llama_prompt", "llama_decode", "batch_decode"):
        L, h, n = case["layers"], case["hidden"], case["tokens"]
        params, head, kv, heads = _llama_params(case), VOCAB * h, 2 * (h // HEAD // 4) * 50, h // HEAD
        if kind == "llama_prompt":
            return {"bytes": 2.0 * (L * params + head) + L * n * kv, "flops": 2.0 * (n * L * params + head) + L * n * (n + 1) / 2 * heads * 4 * HEAD}
        if kind == "llama_decode":
            live = (1 - case["sparsity"]) * L * params + head
            return {"bytes": case["steps"] * (2.0 * live + L * n * kv), "flops": case["steps"] * (2.0 * live + L * n * heads * 4 * HEAD)}
        b = case["batch"]
        return {"bytes": 2.0 * (L * params + head) + b * L * n * kv + 2 * b * VOCAB, "flops": b * (2.0 * (L * params + head) + L * n * heads * 4 * HEAD)}
    size, w, L, n = (4 if case["dtype"] == "float32" else 2), case["width"], case["layers"], case["tokens"]
    heads, ff, mlp = w // 128, w * 7 // 2, 3 * w * (w * 7 // 2)
    window = sum(min(i + 1, WINDOW) for i in range(n))
    if case["design"] == "rorosun":
        params = L * (w * w * 3 // 2 + 4 * w * w + 2 * 64 * w + 2 * w * w + mlp)
        pooled = sum(max(0, i - WINDOW + 1) // POOL for i in range(n))
        math_ = L * ((window + pooled) * heads * 2.0 * (256 + heads) + n * w * 64 * 6.0)
        step = L * (min(n, WINDOW) * heads // 4 * 256 * size + 2 * w * 64 * 4)
    else:
        full = L // 2
        params = full * (w * w * 7 // 2 + mlp) + full * (w * (w // 2 + KV_RANK + ROT_DIM) + w // 2 * heads * (128 + ROT_DIM)
                                                        + KV_RANK * heads * 256 + w * w + mlp)
        math_ = full * heads * 2.0 * (n * (n + 1) / 2 * 256 + window * (256 + ROT_DIM))
        step = full * size * (n * heads // 4 * 256 + min(n, WINDOW) * (KV_RANK + ROT_DIM))
    steps, rows = case.get("steps", 0), len(_mixer_tokens(case, 0)[1])
    return {"bytes": float(size * (params + VOCAB * w) + steps * (size * (params + VOCAB * w) + step) + 4 * VOCAB * (rows + steps)),
            "flops": 2.0 * (n + steps) * params + math_ + 2.0 * (rows + steps) * VOCAB * w}


def tolerance(case: dict):
    kind = case["kind"]
    if kind in ("gemv", "swiglu"):       # fp16 (or bf16) results of 32-bit sums; swiglu rounds both factors first
        return {"rel": 8e-3 if case["dtype"] == "bfloat16" else 1.5e-3, "max": 0.02}
    if kind == "quantizer":              # codes and fp16 norms are the same bits, the rotation is a 32-bit sum
        return {"rel": 2e-6, "max": 1e-4, "differ": 0.0}
    if kind in ("decode_attention", "paged_prompt"):
        return {"rel": 1.5e-3, "max": 0.03}
    # Whole models: a last-bit difference moves a few 3-bit codes and thresholded inputs of later layers, which come back
    # as the quantization's own noise on a few coordinates. Off the 64-bit result: 2e-3, 1.1e-2 (with thresholds) and 5e-4.
    if kind in ("llama_prompt", "llama_decode", "batch_decode"):
        return {"llama_prompt": {"rel": 8e-3, "max": 0.1}, "llama_decode": {"rel": 0.03, "max": 0.3},
                "batch_decode": {"rel": 3e-3, "max": 0.05}}[kind]
    return {"rel": 1e-4, "max": 1e-3} if case["dtype"] == "float32" else {"rel": 0.02, "max": 0.2}


# ── the same in 64 bits, plain torch ─────────────────────────────────────────────────────────────────────────

F64 = torch.float64


def _masked(x: torch.Tensor, t) -> torch.Tensor:
    return x if t is None or t <= 0 else x * (x.abs() > t)


def _quantized(x: torch.Tensor, rotation: torch.Tensor, book: tuple, fp16_norms: bool = True) -> torch.Tensor:
    """x [.., 128] through the store: rotated, each coordinate to its centroid, rotated back, times the stored norm."""
    cents, bounds = book
    norm = x.norm(dim=-1, keepdim=True)
    codes = torch.bucketize((x / (norm + 1e-10)) @ rotation.t(), bounds)
    return (cents[codes] @ rotation) * (norm.half().to(x.dtype) if fp16_norms else norm)


def _attend(q, k, v, scale, hidden=None, pooled=0):
    """q [T, H, d], k / v [S, G, d] -> [T, H, dv], one kv head at a time; ``hidden`` [T, S]: what a query does not see."""
    T, H = q.shape[:2]
    G = k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    for g in range(G):
        for h in range(g * (H // G), (g + 1) * (H // G)):
            s = (q[:, h] @ k[:, g].t()) * scale
            out[:, h] = torch.softmax(s if hidden is None else s.masked_fill(hidden, -math.inf), dim=-1) @ v[:, g]
    return out


def _rms(x, gain, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * gain


def _silu(x):
    return x * torch.sigmoid(x)


def _plain_llama(case, w, ids, rows, dtype, thresholds=None, sparse_from=None, note=None, quantize=True):
    """Logits [B, len(rows), vocab] of ids [B, T] at the places ``rows``. Keys and values go through the 3-bit store; from
    ``sparse_from`` on the inputs of the projections lose what lies under their thresholds."""
    cfg = _llama_config(case)
    B, T = ids.shape
    nq, nkv = cfg.num_q_heads, cfg.num_kv_heads
    book = _codebook(3, dtype)
    rate = 1.0 / cfg.rope_theta ** (torch.arange(0, HEAD, 2, dtype=dtype, device="cuda") / HEAD)
    angle = torch.arange(T, dtype=dtype, device="cuda").reshape(T, 1, 1) * torch.cat([rate, rate])
    cos, sin = torch.cos(angle), torch.sin(angle)
    turn = lambda x: x * cos + torch.cat([-x[..., HEAD // 2:], x[..., :HEAD // 2]], -1) * sin
    hidden = torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1)
    x = w["embed"][ids].to(dtype)

    def sparse(l, name, a, first):
        if note:
            note(l, name, a)
        t = (thresholds or {}).get(l, {}).get({"qkv": "q_proj", "o": "o_proj", "gu": "up_proj", "down": "down_proj"}[name])
        if t is None or first >= a.shape[0]:
            return a
        return torch.cat([a[:first], _masked(a[first:], t)])

    for l in range(cfg.num_layers):
        lw = {n: t.to(dtype) for n, t in w["layers"][l].items() if n != "wgu_t"}
        pk, pv = _rotation(42 + 2 * l, dtype), _rotation(43 + 2 * l, dtype)
        last = l + 1 == cfg.num_layers and note is None
        parts = []
        for b in range(B):
            first = T if sparse_from is None else sparse_from
            qkv = sparse(l, "qkv", _rms(x[b], lw["ln1"], cfg.rms_eps), first) @ lw["wqkv_t"]
            q = turn(qkv[:, :nq * HEAD].reshape(T, nq, HEAD))
            k = turn(qkv[:, nq * HEAD:(nq + nkv) * HEAD].reshape(T, nkv, HEAD))
            v = qkv[:, (nq + nkv) * HEAD:].reshape(T, nkv, HEAD)
            k, v = _quantized(k, pk, book), _quantized(v, pv, book)
            h, see = x[b], hidden
            if last:
                q, h, see, first = q[rows], h[rows], hidden[rows], 0 if rows[0] >= first else len(rows)
            a = _attend(q, k, v, HEAD ** -0.5, see).reshape(q.shape[0], nq * HEAD)
            h = h + sparse(l, "o", a, first) @ lw["wo_t"]
            m = sparse(l, "gu", _rms(h, lw["ln2"], cfg.rms_eps), first)
            m = _silu(m @ lw["wgate_t"]) * (m @ lw["wup_t"])
            parts.append(h + sparse(l, "down", m, first) @ lw["wdown_t"])
        x = torch.stack(parts)
    if note is not None:
        return None
    return _rms(x, w["final_norm"].to(dtype), cfg.rms_eps) @ w["lm_head_t"].to(dtype)


def _turned(x, base, dims):
    """x [T, heads, d]: coordinates 2i, 2i + 1 of the first ``dims`` turn by position * base^(-2i / dims)."""
    rate = float(base) ** (-torch.arange(0, dims, 2, dtype=F64, device="cuda") / dims)
    angle = torch.arange(x.shape[0], dtype=F64, device="cuda").reshape(-1, 1, 1) * rate
    c, s, e, o = torch.cos(angle), torch.sin(angle), x[..., 0:dims:2], x[..., 1:dims:2]
    out = x.clone()
    out[..., 0:dims:2], out[..., 1:dims:2] = e * c - o * s, o * c + e * s
    return out


def _plain_pefitar(model, t, ids):
    """The fp64 stream [T, width] after the last layer."""
    eps, mult, T = model["norm"]["eps"], model["residual_mult"], len(ids)
    gap = torch.arange(T, device="cuda").reshape(T, 1) - torch.arange(T, device="cuda").reshape(1, T)
    x = t["embed"][ids].to(F64)
    for i, layer in enumerate(model["layers"]):
        w = {n[len(f"l{i}."):]: a.to(F64) for n, a in t.items() if n.startswith(f"l{i}.")}
        m, h = layer["mixer"], _rms(x, w["norm1"], eps)
        H, d, dv = m["heads"], m["dim"], m["vdim"]
        if layer["type"] == "attention":
            G = m["kv_heads"]
            q = _turned((h @ w["mix.q"].t()).reshape(T, H, d), m["rot"]["base"], m["rot"]["dims"])
            k = _turned((h @ w["mix.k"].t()).reshape(T, G, d), m["rot"]["base"], m["rot"]["dims"])
            a = _attend(q, k, (h @ w["mix.v"].t()).reshape(T, G, dv), m["scale"], gap < 0).reshape(T, H * dv)
            a = a * torch.sigmoid(h @ w["mix.g"].t())
        else:
            r, n = m["rot_dim"], m["kv_rank"]
            q = (_rms(h @ w["mix.dq"].t(), w["mix.dq.norm"], eps) @ w["mix.uq"].t()).reshape(T, H, d + r)
            q = torch.cat([q[..., :d], _turned(q[..., d:], m["rot"]["base"], r)], -1)
            low = h @ w["mix.dkv"].t()
            c, part = _rms(low[:, :n], w["mix.dkv.norm"], eps), _turned(low[:, None, n:], m["rot"]["base"], r)
            k = torch.cat([(c @ w["mix.uk"].t()).reshape(T, H, d), part.expand(T, H, r)], -1)
            v = (c @ w["mix.uv"].t()).reshape(T, H, dv)
            a = _attend(q, k, v, m["scale"], (gap < 0) | (gap >= m["mask"]["size"])).reshape(T, H * dv)
        x = x + mult * _rms(a @ w["mix.o"].t(), w["norm1b"], eps)
        h = _rms(x, w["norm2"], eps)
        f = (_silu(h @ w["mlp.gate"].t()) * (h @ w["mlp.up"].t())) @ w["mlp.down"].t()
        x = x + mult * _rms(f, w["norm2b"], eps)
    return x


def _plain_rorosun(model, t, ids):
    """The fp64 stream [T, width] after the last layer."""
    eps, T = model["norm"]["eps"], len(ids)
    i, j = torch.arange(T, device="cuda").reshape(T, 1), torch.arange(T, device="cuda").reshape(1, T)
    blocks = T // POOL
    ends = torch.arange(blocks, device="cuda").reshape(1, -1) * POOL + POOL - 1
    hidden = torch.cat([(j > i) | (i - j >= WINDOW), ends > i - WINDOW], 1)
    pooled = lambda a: torch.cat([a, a[:blocks * POOL].reshape(blocks, POOL, *a.shape[1:]).mean(1)])
    one = lambda g: g.reshape(())
    x = t["embed"][ids].to(F64)
    for n, layer in enumerate(model["layers"]):
        w = {k[len(f"l{n}."):]: a.to(F64) for k, a in t.items() if k.startswith(f"l{n}.")}
        m, left, right = layer["mixer"], layer["mixer"]["left"], layer["mixer"]["right"]
        h = _rms(x, one(w["norm1"]), eps)
        H, G, d = left["heads"], left["kv_heads"], left["dim"]
        q, k, v = (h @ w[f"mix.left.{s}"].t() + w[f"mix.left.{s}.b"] for s in "qkv")
        q = _rms(q, w["mix.left.q.norm"], eps).reshape(T, H, d)
        k, v = pooled(_rms(k, w["mix.left.k.norm"], eps).reshape(T, G, d)), pooled(v.reshape(T, G, left["vdim"]))
        weights = torch.stack([torch.softmax((q[:, a] @ k[:, a // (H // G)].t() * left["scale"]).masked_fill(hidden, -math.inf), -1)
                               for a in range(H)])
        weights = torch.einsum("hg,gij->hij", w["mix.left.talk"], weights)
        out = torch.stack([weights[a] @ v[:, a // (H // G)] for a in range(H)], 1).reshape(T, -1)
        x1 = m["left_scale"] * (out @ w["mix.left.o"].t())
        del weights

        H, d = right["heads"], right["dim"]
        before = torch.cat([torch.zeros_like(h[:1]), h[:-1]])
        mixed = {s: h + (before - h) * w["mix.right.mu." + s] for s in "rkvgw"}
        r, k, v = ((mixed[s] @ w["mix.right." + s].t()).reshape(T, H, d) for s in "rkv")
        keep = torch.exp(-torch.exp(torch.tanh(mixed["w"] @ w["mix.right.w1"].t()) @ w["mix.right.w2"].t() + w["mix.right.w0"]))
        keep, S, out = keep.reshape(T, H, d, 1), torch.zeros(H, d, d, dtype=F64, device="cuda"), torch.empty_like(r)
        kv, bonus, r4 = k.unsqueeze(-1), w["mix.right.u"].unsqueeze(-1), r.unsqueeze(-2)
        for a in range(T):
            new = kv[a] * v[a].unsqueeze(-2)
            out[a] = (r4[a] @ (S + bonus * new)).squeeze(-2)
            S = keep[a] * S + new
        out = _rms(out, 1.0, eps).reshape(T, H * d) * w["mix.right.norm"] * _silu(mixed["g"] @ w["mix.right.g"].t())
        x = x + (x1 + m["right_scale"] * (out @ w["mix.right.o"].t())) * w["ls1"]
        h = _rms(x, one(w["norm2"]), eps)
        x = x + ((_silu(h @ w["mlp.gate"].t()) * (h @ w["mlp.up"].t())) @ w["mlp.down"].t()) * w["ls2"]
    return x


@torch.no_grad()
def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind in ("gemv", "swiglu"):
        p = _projection(case, seed)
        x = p["x"].half().to(F64)
        y = [_masked(x, p["t"]) @ w.to(F64).t() for w in p["w"]]
        return _silu(y[0]) * y[1] if kind == "swiglu" else y[0]
    if kind == "quantizer":
        p = _vectors(case, seed)
        restored = _codebook(case["bits"])[0][p["codes"]] @ _rotation(42, F64) * p["norms"].to(F64).unsqueeze(1)
        return {"indices": None, "norms": p["x"].to(F64).norm(dim=-1), "restored": restored}
    if kind in ("decode_attention", "paged_prompt"):
        n = _lengths(case) if kind == "decode_attention" else [case["tokens"]] * case["batch"]
        p, book = _kv(case, seed, max(n)), _codebook(3)
        k, v = _quantized(p["k"].to(F64), _rotation(42, F64), book), _quantized(p["v"].to(F64), _rotation(43, F64), book)
        if kind == "decode_attention":
            return torch.stack([_attend(p["q"][b].to(F64).unsqueeze(0), k[b, :, :t].transpose(0, 1), v[b, :, :t].transpose(0, 1),
                                        HEAD ** -0.5)[0] for b, t in enumerate(n)])
        hidden = torch.ones(n[0], n[0], dtype=torch.bool, device="cuda").triu(1)
        out = torch.stack([_attend(p["q"][b].to(F64).transpose(0, 1), k[b].transpose(0, 1), v[b].transpose(0, 1), HEAD ** -0.5,
                                   hidden).transpose(0, 1) for b in range(case["batch"])])
        return [out[:, :, s:s + case["chunk"]] for s in range(0, n[0], case["chunk"])]
    if kind in ("llama_prompt", "llama_decode"):
        w = _llama_weights(case, seed)
        ids = _tokens(seed, case["tokens"] + case.get("steps", 0)).reshape(1, -1).cuda()
        if kind == "llama_prompt":
            return _plain_llama(case, w, ids, [case["tokens"] - 1], F64)[0, 0]
        rows = list(range(case["tokens"], ids.shape[1]))
        return _plain_llama(case, w, ids, rows, F64, _thresholds(case, w, seed), case["tokens"])[0]
    if kind == "batch_decode":
        ids = _tokens(seed, case["batch"], case["tokens"] + 1).cuda()
        return _plain_llama(case, _llama_weights(case, seed), ids, [case["tokens"]], F64)[:, 0]
    model, t = _mixer_model(case), _mixer_tensors(case, seed)
    ids, want = _mixer_tokens(case, seed)
    gain, n = t["final.norm"].to(F64), case["tokens"]
    x = (_plain_rorosun if case["design"] == "rorosun" else _plain_pefitar)(model, t, torch.tensor(ids, device="cuda"))
    rows = x[want + list(range(n, len(ids)))]
    if case["design"] == "rorosun":
        z = _rms(rows, gain.reshape(()), model["norm"]["eps"]) @ t["head"].to(F64).t()
    else:
        cap = model["logit_softcap"]
        z = cap * torch.tanh(_rms(rows, gain, model["norm"]["eps"]) @ t["embed"].to(F64).t() / cap)
    return [z[:len(want)], z[len(want):]] if len(ids) > n else [z]
