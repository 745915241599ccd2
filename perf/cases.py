"""The workloads that the attention path is timed on: one token step or one prompt chunk, over all the layers of a
small model, through the public calls of `AttnContext`.

A case is one call pattern of an inference engine: `decode` (one token of each of B sequences), `prefill` (a chunk of
one prompt behind an already cached prefix), `layer_decode` and `layer_prefill` (the same with the q / k / v and output
projections on the device). One pass runs the call once per layer, as the engine's layer loop does. Model shapes are
those of gguf_runner_b200.presets; the cache formats are the five that the library stores.
"""
from __future__ import annotations

import numpy as np
import torch

import gguf_runner_b200 as g
from gguf_runner_b200.binding import (KV_BF16, KV_FORMATS, KV_TURBO, ROPE_ADJACENT, ROPE_NEOX, SCALE_Q_PRESCALED, W_BF16,
                                      W_F32, W_Q4_K, W_Q6_K, W_Q8_0, AttnConfig, RawCuda, Weights, gemma_layer_windows)

# name: (query heads, KV heads, head_dim, hidden size, RoPE style, theta, has QK-norm)
SHAPES = {
    "qwen3_0p6b": (16, 8, 128, 1024, ROPE_NEOX, 1e6, True),
    "llama3_8b": (32, 8, 128, 4096, ROPE_ADJACENT, 5e5, False),
    "qwen3_30b_a3b": (32, 4, 128, 2048, ROPE_NEOX, 1e6, True),
    "gemma3_4b": (8, 4, 256, 2560, ROPE_NEOX, 1e6, True),
    "qwen25_14b": (40, 8, 128, 5120, ROPE_NEOX, 1e6, False),
}
# bytes of cache per element of K or V (codes, and scales where they are per block)
KV_BYTES = {"f32": 4.0, "bf16": 2.0, "q8_row": 1.0, "q8_block32": 1.125, "turbo": 0.4375}
# bytes per weight as the model file has them
W_BYTES = {"f32": 4.0, "bf16": 2.0, "q8_0": 34 / 32, "q4_k_m": 144 / 256}
GEMMA_WINDOW = 1024


def listed():
    return [
        # The smallest model, one conversation, f32 cache: a token costs 28 short launches.
        dict(name="decode_f32_b1", kind="decode", shape="qwen3_0p6b", kv="f32", layers=28, batch=1, ctx=2048, ragged=False,
             host=False, norm=False),
        # The unmodified engine: its q / k / v rows and the result are in host memory; the default q8 cache.
        dict(name="decode_q8_host_b1", kind="decode", shape="llama3_8b", kv="q8_row", layers=32, batch=1, ctx=1501,
             ragged=False, host=True, norm=False),
        # The engine's own default cache format, one long conversation, QK-norm on the device.
        dict(name="decode_turbo_b1", kind="decode", shape="qwen3_30b_a3b", kv="turbo", layers=12, batch=1, ctx=7777,
             ragged=False, host=False, norm=True),
        # Eight long conversations in step: reading the cache is all that counts.
        dict(name="decode_bf16_b8_long", kind="decode", shape="qwen3_30b_a3b", kv="bf16", layers=6, batch=8, ctx=32768,
             ragged=False, host=False, norm=False),
        # A server's batch: every sequence at a position of its own, from just begun to long.
        dict(name="decode_bf16_ragged", kind="decode", shape="qwen25_14b", kv="bf16", layers=8, batch=16, ctx=6000,
             ragged=True, host=False, norm=False),
        # A whole prompt at once.
        dict(name="prefill_bf16_4096", kind="prefill", shape="llama3_8b", kv="bf16", layers=4, m=4096, base=0, bf16_in=True,
             norm=False),
        # The next user turn of a conversation: a short chunk behind a prefix, f32 rows.
        dict(name="prefill_bf16_turn", kind="prefill", shape="llama3_8b", kv="bf16", layers=8, m=333, base=1700,
             bf16_in=False, norm=False),
        # Chunked prefill with five sliding-window layers to one global layer.
        dict(name="prefill_gemma_chunk", kind="prefill", shape="gemma3_4b", kv="bf16", layers=6, m=2048, base=14336,
             bf16_in=True, norm=False),
        # A prompt on the default q8 cache.
        dict(name="prefill_q8_prompt", kind="prefill", shape="llama3_8b", kv="q8_row", layers=3, m=1000, base=0,
             bf16_in=False, norm=False),
        # A chunk on the engine's default cache format behind a prefix.
        dict(name="prefill_turbo_chunk", kind="prefill", shape="qwen3_0p6b", kv="turbo", layers=3, m=512, base=700,
             bf16_in=False, norm=False),
        # The attention half of a token step of a 4-bit model file, one conversation.
        dict(name="layer_decode_q4k_b1", kind="layer_decode", shape="llama3_8b", kv="bf16", layers=4, batch=1, ctx=2000,
             ragged=False, weights="q4_k_m"),
        # The attention half of a prompt chunk of an 8-bit model file.
        dict(name="layer_prefill_q8_0", kind="layer_prefill", shape="llama3_8b", kv="bf16", layers=3, m=500, base=256,
             weights="q8_0", norm=False),
    ]


def _log_int(rng, lo, hi):
    """A whole number of lo .. hi, evenly spread over its logarithm."""
    return max(lo, min(hi, round(lo * (hi / lo) ** rng.random())))


def draw(rng):
    """Another case of the same kinds: one of twelve patterns, with sizes from its range."""
    pattern = rng.randrange(12)
    any_shape = ("qwen3_0p6b", "llama3_8b", "qwen3_30b_a3b", "qwen25_14b")
    if pattern < 5:
        shape, kv = rng.choice(any_shape), ("f32", rng.choice(("q8_row", "q8_block32", "f32")), "turbo", "bf16", "bf16")[pattern]
        host = pattern == 1
        batch = 1 if host else (_log_int(rng, 1, 4) if pattern in (0, 2) else _log_int(rng, 1, 48))
        ctx = _log_int(rng, 64, 4096 if pattern in (0, 1) else 32768)
        per_layer = 2 * batch * ctx * SHAPES[shape][1] * SHAPES[shape][2] * KV_BYTES[kv]
        ctx = max(64, int(ctx * min(1.0, 1e9 / per_layer)))
        layers = max(2, min(28 if pattern < 2 else 8, int(2.5e9 / per_layer)))
        return dict(kind="decode", shape=shape, kv=kv, layers=layers, batch=batch, ctx=ctx,
                    ragged=batch > 1 and rng.random() < 0.6, host=host, norm=SHAPES[shape][6] and rng.random() < 0.5)
    if pattern < 10:
        shape = "gemma3_4b" if pattern == 7 else rng.choice(any_shape)
        kv = ("bf16", "bf16", "bf16", rng.choice(("q8_row", "q8_row", "q8_block32")), "turbo")[pattern - 5]
        m = _log_int(rng, 33, 4096 if kv == "bf16" else 1024)
        base = rng.choice((0, _log_int(rng, 16, 16384 if kv == "bf16" else 1500)))
        if kv != "bf16" and m > 600:
            base = min(base, 300)
        layers = 6 if shape == "gemma3_4b" else (3 if kv != "bf16" or m > 1500 else 6)
        if shape != "gemma3_4b" and kv == "bf16":
            base = min(base, max(0, 12_000_000 // m - m // 2))
        return dict(kind="prefill", shape=shape, kv=kv, layers=layers, m=m, base=base,
                    bf16_in=kv == "bf16" and rng.random() < 0.5, norm=SHAPES[shape][6] and rng.random() < 0.3)
    shape, weights = rng.choice(any_shape), rng.choice(("q8_0", "q4_k_m", "q4_k_m", "bf16"))
    if pattern == 10:
        batch = rng.choice((1, 1, _log_int(rng, 2, 32)))
        return dict(kind="layer_decode", shape=shape, kv="bf16", layers=4, batch=batch, ctx=_log_int(rng, 64, 8192),
                    ragged=batch > 1, weights=weights)
    return dict(kind="layer_prefill", shape=shape, kv="bf16", layers=3, m=_log_int(rng, 17, 1024),
                base=rng.choice((0, _log_int(rng, 16, 2048))), weights=weights, norm=SHAPES[shape][6] and rng.random() < 0.3)


def _positions(case, seed):
    """Position of the new token of every sequence; a ragged batch has them spread from ctx / 32 to ctx - 1."""
    if not case["ragged"]:
        return np.full(case["batch"], case["ctx"] - 1, np.int32)
    r = np.random.default_rng(case["ctx"] * 97 + case["batch"])  # the lengths belong to the case, not to the seed
    pos = np.exp(r.uniform(np.log(case["ctx"] / 32), np.log(case["ctx"]), case["batch"])).astype(np.int32)
    pos = np.clip(pos, 1, case["ctx"] - 1)
    pos[0] = case["ctx"] - 1
    return pos


def _config(case, seq_len):
    heads, kv_heads, dim, _, style, theta, _ = SHAPES[case["shape"]]
    more = {}
    if case["shape"] == "gemma3_4b":
        more = dict(rope_theta_swa=1e4, swa_theta_on_window_layers=1, scale_mode=SCALE_Q_PRESCALED,
                    layer_windows=gemma_layer_windows(case["layers"], GEMMA_WINDOW, 6))
    return AttnConfig(n_layers=case["layers"], n_heads=heads, n_kv_heads=kv_heads, head_dim=dim, seq_len=seq_len,
                      max_batch=case.get("batch", 1), rope_theta=theta, rope_style=style,
                      kv_format=KV_FORMATS[case["kv"]], **more)


def _cache_views(ctx):
    """The library's K and V arrays (codes for the quantised formats) and its scales as tensors
    [sequence][layer][position][...]."""
    cfg = ctx.config
    k, v, ks, vs, nbytes = ctx.kv_device_ptrs()
    dt = {"f32": torch.float32, "bf16": torch.bfloat16, "turbo": torch.uint8}.get(
        next(n for n, f in KV_FORMATS.items() if f == cfg.kv_format), torch.int8)
    lead = (cfg.max_batch, cfg.n_layers, cfg.seq_len)

    def tensor(ptr, size, dtype):
        raw = RawCuda(ptr, size)
        raw.owner = ctx  # the tensor keeps `raw`, and so the cache behind it, alive
        return torch.as_tensor(raw, device="cuda").view(dtype)

    views = [tensor(p, nbytes, dt).view(*lead, -1) for p in (k, v)]
    if ks:
        n = {KV_FORMATS["q8_row"]: 1, KV_FORMATS["q8_block32"]: cfg.kv_dim // 32, KV_TURBO: cfg.n_kv_heads}[cfg.kv_format]
        rows = cfg.max_batch * cfg.n_layers * cfg.seq_len
        views += [tensor(p, rows * n * 4, torch.float32).view(*lead, n) for p in (ks, vs)]
    return views


def _fill_cache(ctx, views, rows, gen, rng):
    """Rows 0 .. rows - 1 of every layer and sequence as appended N(0, 1) rows would leave them."""
    cfg = ctx.config
    if rows <= 0:
        return
    if cfg.kv_format == KV_TURBO:
        levels = np.array([0.163, 0.337, 0.337, 0.163])  # N(0, 1) mass of the four code intervals
        table = rng.choice(4, size=(1 << 18, 4), p=levels).astype(np.uint8)
        table = table[:, 0] | table[:, 1] << 2 | table[:, 2] << 4 | table[:, 3] << 6
        kd, h = cfg.kv_dim, cfg.n_kv_heads
        for seq in range(cfg.max_batch):
            for layer in range(cfg.n_layers):
                codes = table[rng.integers(0, 1 << 18, (2, rows, kd // 4), dtype=np.int32)]
                signs = np.frombuffer(rng.bytes(2 * rows * kd // 8), np.uint8).reshape(2, rows, kd // 8)
                sigma = rng.uniform(0.85, 1.15, (2, rows, h)).astype(np.float32)
                rnorm = (sigma * rng.uniform(3.6, 4.2, (2, rows, h))).astype(np.float32)
                ctx.kv_import_turbo(layer, 0, dict(k_base=codes[0], v_base=codes[1], k_sign=signs[0], v_sign=signs[1],
                                                   k_scale=sigma[0], v_scale=sigma[1], k_rnorm=rnorm[0],
                                                   v_rnorm=rnorm[1]), seq=seq)
        return
    for a in views[:2]:
        for seq in range(cfg.max_batch):
            x = torch.randn(a.shape[1], rows, a.shape[3], generator=gen, device="cuda")
            a[seq, :, :rows] = x if a.dtype.is_floating_point else (x * 35.0).round_().clamp_(-127, 127)
    for s in views[2:]:
        s[:, :, :rows] = torch.rand(*s[:, :, :rows].shape, generator=gen, device="cuda") * 0.01 + 0.025


def _set_norms(ctx, case, gen):
    """QK-norm weights per layer, or an empty list."""
    norms = []
    for layer in range(case["layers"] if case.get("norm") else 0):
        qn, kn = (1.0 + 0.2 * torch.randn(2, ctx.config.head_dim, generator=gen, device="cuda")).cpu().numpy()
        ctx.set_layer_fixups(layer, q_norm=qn, k_norm=kn, eps=1e-6)
        norms.append((qn, kn))
    return norms


def _weights(kind, rows, cols, rng):
    """A projection matrix of N(0, 0.02)-like weights in the row layout of the model file: (type, rows, cols, data)."""
    n = rows * cols
    if kind in ("f32", "bf16"):
        w = (rng.standard_normal((rows, cols), dtype=np.float32) * 0.02)
        return (W_F32, rows, cols, w) if kind == "f32" else (W_BF16, rows, cols, (w.view(np.uint32) >> 16).astype(np.uint16))
    if kind == "q8_0":
        blocks = np.frombuffer(rng.bytes(n // 32 * 34), np.uint8).reshape(-1, 34).copy()
        blocks[:, :2] = (rng.uniform(0.8, 1.2, n // 32) * 0.02 / 74).astype(np.float16).view(np.uint8).reshape(-1, 2)
        return W_Q8_0, rows, cols, blocks
    if kind == "q4_k":
        blocks = np.frombuffer(rng.bytes(n // 256 * 144), np.uint8).reshape(-1, 144).copy()
        d = rng.uniform(0.8, 1.2, (n // 256, 2)) * np.array([1.0, 7.5]) * 0.02 / 250
        blocks[:, :4] = d.astype(np.float16).view(np.uint8).reshape(-1, 4)
        return W_Q4_K, rows, cols, blocks
    blocks = np.frombuffer(rng.bytes(n // 256 * 210), np.uint8).reshape(-1, 210).copy()
    blocks[:, 208:] = (rng.uniform(0.8, 1.2, n // 256) * 0.02 / 1360).astype(np.float16).view(np.uint8).reshape(-1, 2)
    return W_Q6_K, rows, cols, blocks


def _layer_weights(case, layer, rng):
    """wq, wk, wv, wo of a layer; a Q4_K_M file keeps every other layer's v projection in Q6_K."""
    heads, kv_heads, dim, hidden, *_ = SHAPES[case["shape"]]
    kind = case["weights"]
    kinds = ["q4_k", "q4_k", "q6_k" if layer % 2 == 0 else "q4_k", "q4_k"] if kind == "q4_k_m" else [kind] * 4
    sizes = [(heads * dim, hidden), (kv_heads * dim, hidden), (kv_heads * dim, hidden), (hidden, heads * dim)]
    return [_weights(k, r, c, rng) for k, (r, c) in zip(kinds, sizes)]


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    heads, kv_heads, dim, hidden, *_ = SHAPES[case["shape"]]
    decode = case["kind"] in ("decode", "layer_decode")
    layers, rows = case["layers"], case["batch"] if decode else case["m"]
    first = case["ctx"] - 1 if decode else case["base"]
    ctx = g.AttnContext(_config(case, case["ctx"] if decode else case["base"] + case["m"]))
    views = _cache_views(ctx)
    _fill_cache(ctx, views, first, gen, rng)
    norms = _set_norms(ctx, case, gen)
    state = {"case": case, "ctx": ctx, "layers": range(layers), "views": views, "norms": norms}

    def randn(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")

    if case["kind"] in ("layer_decode", "layer_prefill"):
        state["w"] = [[Weights(*w) for w in _layer_weights(case, layer, rng)] for layer in range(layers)]
        state["x"] = list(randn(layers, rows, hidden))
        out = torch.empty(layers, rows, hidden, device="cuda")
    else:
        qkv = [randn(layers, rows, n * dim) for n in (heads, kv_heads, kv_heads)]
        out = torch.empty(layers, rows, heads * dim, device="cuda")
        if case.get("bf16_in"):
            qkv = [t.bfloat16() for t in qkv]
        if case.get("host"):
            qkv, out = [t.cpu().numpy() for t in qkv], out.cpu().numpy()
        state["q"], state["k"], state["v"] = (list(t) for t in qkv)
    state["out"] = list(out)
    # what the step leaves: the result, and the cache rows it appended
    appended = [view[:, :, first:first + (1 if decode else case["m"])] for view in views]
    if decode:
        state["pos"] = _positions(case, seed)
        if case["ragged"]:  # K rows of sixteen sequences at their own positions
            appended = [views[0][b, :, p] for b, p in list(enumerate(state["pos"]))[:16]]
    state["result"] = {"out": out, "appended": appended}
    torch.cuda.synchronize()
    return state


def run(state):
    ctx, out, kind = state["ctx"], state["out"], state["case"]["kind"]
    if kind == "decode":
        pos, q, k, v = state["pos"], state["q"], state["k"], state["v"]
        for layer in state["layers"]:
            ctx.decode(layer, pos, q[layer], k[layer], v[layer], out=out[layer])
    elif kind == "prefill":
        base, q, k, v = state["case"]["base"], state["q"], state["k"], state["v"]
        for layer in state["layers"]:
            ctx.prefill(layer, base, q[layer], k[layer], v[layer], out=out[layer])
    elif kind == "layer_decode":
        pos, x, w = state["pos"], state["x"], state["w"]
        for layer in state["layers"]:
            ctx.layer_decode(layer, pos, x[layer], *w[layer], out=out[layer])
    else:
        base, x, w = state["case"]["base"], state["x"], state["w"]
        for layer in state["layers"]:
            ctx.layer_prefill(layer, base, x[layer], *w[layer], out=out[layer])
    return state["result"]


def _visible(case):
    """(query, key) pairs and cached keys read, summed over the layers."""
    if case["kind"] in ("decode", "layer_decode"):
        keys = int((_positions(case, 0).astype(np.int64) + 1).sum())
        return keys * case["layers"], keys * case["layers"]
    m, base = case["m"], case["base"]
    windows = (gemma_layer_windows(case["layers"], GEMMA_WINDOW, 6) if case["shape"] == "gemma3_4b"
               else [0] * case["layers"])
    pairs = keys = 0
    for w in windows:
        ends = np.arange(base + 1, base + m + 1, dtype=np.int64)
        pairs += int(np.minimum(ends, w).sum() if w else ends.sum())
        keys += min(base, w - 1) if w else base
    return pairs, keys


def work(case):
    heads, kv_heads, dim, hidden, *_ = SHAPES[case["shape"]]
    q_dim, kv_dim, layers = heads * dim, kv_heads * dim, case["layers"]
    rows = (case["batch"] if "batch" in case else case["m"]) * layers
    pairs, keys = _visible(case)
    e = 2.0 if case.get("bf16_in") else 4.0
    flops = 4.0 * q_dim * pairs
    bytes_ = 2.0 * kv_dim * KV_BYTES[case["kv"]] * (keys + rows)  # prefix read, new rows written
    if "weights" in case:
        params = hidden * (2 * q_dim + 2 * kv_dim)
        flops += 2.0 * rows * params
        bytes_ += layers * params * W_BYTES[case["weights"]] + rows * 2 * hidden * 4.0
    else:
        bytes_ += rows * ((q_dim + 2 * kv_dim) * e + q_dim * 4.0)
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """Caches and arithmetic in f32: 1e-5. bf16 operands (bf16 caches; the tensor-core TurboQuant decode): 1e-2. Codes of
    appended rows may fall to the other side of a rounding boundary."""
    if case["kv"] == "bf16" or (case["kv"] == "turbo" and case["kind"] == "decode"):
        return {"rel": 1e-2, "differ": 5e-3}
    return {"rel": 1e-5, "differ": 5e-3}


def _dense(w):
    """A projection matrix in 64 bits from its model-file bytes (the GGML block layouts)."""
    wtype, rows, cols, data = w
    if wtype in (W_F32, W_BF16):
        d = data if wtype == W_F32 else (data.astype(np.uint32) << 16).view(np.float32)
        return torch.from_numpy(d).cuda().double()
    b = torch.from_numpy(data).cuda()

    def halves(cols_):
        return b[:, cols_].contiguous().view(torch.float16).double()

    if wtype == W_Q8_0:
        out = halves(slice(0, 2)) * b[:, 2:].contiguous().view(torch.int8).double()
    elif wtype == W_Q4_K:  # d, dmin, twelve bytes of eight 6-bit (scale, min) pairs, nibbles in groups of 64
        sc, qs = b[:, 4:16].int(), b[:, 16:].reshape(-1, 4, 32)
        scale = torch.cat([sc[:, :4] & 63, (sc[:, 8:] & 15) | (sc[:, :4] >> 6 << 4)], 1)
        low = torch.cat([sc[:, 4:8] & 63, (sc[:, 8:] >> 4) | (sc[:, 4:8] >> 6 << 4)], 1)
        q = torch.stack([qs & 15, qs >> 4], 2).reshape(-1, 8, 32).double()
        out = (halves(slice(0, 2)) * scale)[..., None] * q - (halves(slice(2, 4)) * low)[..., None]
    else:  # Q6_K: low nibbles, high bit pairs, sixteen int8 scales, d
        lo, hi = b[:, :128].reshape(-1, 2, 64).int(), b[:, 128:192].reshape(-1, 2, 32).int()
        q = torch.stack([(lo[..., :32] & 15) | (hi & 3) << 4, (lo[..., 32:] & 15) | (hi >> 2 & 3) << 4,
                         (lo[..., :32] >> 4) | (hi >> 4 & 3) << 4, (lo[..., 32:] >> 4) | (hi >> 6 & 3) << 4], 2)
        scale = halves(slice(208, 210)) * b[:, 192:208].contiguous().view(torch.int8).double()
        out = scale[..., None] * (q.reshape(-1, 16, 16) - 32).double()
    return out.reshape(rows, cols)


def _rotate(x, pos, theta, style):
    """RoPE of x [rows][heads][dim] in 64 bits; frequencies and angles are f32, as the models define them."""
    dim = x.shape[-1]
    power = (float(theta) ** (np.arange(0, dim, 2, dtype=np.float32) / np.float32(dim)).astype(np.float64)).astype(np.float32)
    freq = np.float32(1.0) / power
    angle = torch.from_numpy(np.asarray(pos, np.float32)[:, None] * freq).cuda().double()[:, None]
    c, s = angle.cos(), angle.sin()
    a, b = (x[..., :dim // 2], x[..., dim // 2:]) if style == ROPE_NEOX else (x[..., ::2], x[..., 1::2])
    pair = a * c - b * s, a * s + b * c
    return torch.cat(pair, -1) if style == ROPE_NEOX else torch.stack(pair, -1).flatten(-2)


def _stored(x, kv):
    """Rows [n][elements] as the cache holds them: values in 64 bits, and the scales of a q8 cache."""
    if kv in ("f32", "bf16"):
        return (x.float().double() if kv == "f32" else x.float().bfloat16().double()), None
    blocks = x.float().reshape(x.shape[0], -1, 32 if kv == "q8_block32" else x.shape[1])
    top = blocks.abs().amax(-1, keepdim=True)
    codes = (blocks * (127.0 / top)).double()
    codes = torch.sign(codes) * torch.floor(codes.abs() + 0.5)
    return (codes * (top / 127.0)).reshape(x.shape), (top / 127.0)[..., 0]


def _attend(q, k, v, ends, window):
    """q [rows][heads][dim] over k, v [keys][kv_heads][dim]; row i sees keys max(0, ends[i] - window) .. ends[i] - 1."""
    group, at = q.shape[1] // k.shape[1], torch.arange(k.shape[0], device="cuda")
    out = torch.empty_like(q)
    hide = (at >= ends[:, None]) | (at < ends[:, None] - window if window else torch.zeros_like(at, dtype=torch.bool))
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // group].T) * q.shape[-1] ** -0.5
        out[:, h] = torch.softmax(s.masked_fill_(hide, -torch.inf), -1) @ v[:, h // group]
    return out


def exact(case, seed):
    """What a pass leaves, in 64 bits from the stored cache rows. Codes of quantised caches have no such value, and the
    TurboQuant cache none that is not made of the same transforms."""
    if case["kv"] == "turbo":
        return None
    heads, kv_heads, dim, _, style, theta, _ = SHAPES[case["shape"]]
    state = prepare(case, seed)
    views, layers = state["views"], case["layers"]
    decode = case["kind"] in ("decode", "layer_decode")
    pos = state["pos"] if decode else np.arange(case["base"], case["base"] + case["m"])
    windows = (gemma_layer_windows(layers, GEMMA_WINDOW, 6) if case["shape"] == "gemma3_4b" else [0] * layers)
    rng, outs, rows_k, rows_v, scales = np.random.default_rng(seed), [], [], [], []
    for layer in range(layers):
        if "weights" in case:
            w = [_dense(x) for x in _layer_weights(case, layer, rng)]
            q, k, v = (state["x"][layer].double() @ m.T for m in w[:3])
        else:
            q, k, v = (torch.as_tensor(state[n][layer]).cuda().double() for n in "qkv")
        n = q.shape[0]
        q, k = q.reshape(n, heads, dim), k.reshape(n, kv_heads, dim)
        if state["norms"]:
            q, k = (x * (x.square().mean(-1, keepdim=True) + 1e-6).rsqrt() * torch.from_numpy(g_).cuda().double()
                    for x, g_ in zip((q, k), state["norms"][layer]))
        th = 1e4 if windows[layer] else theta
        q, k = _rotate(q, pos, th, style), _rotate(k, pos, th, style).reshape(n, -1)
        (k_kept, k_scale), (v_kept, v_scale) = _stored(k, case["kv"]), _stored(v, case["kv"])
        rows_k.append(k)
        rows_v.append(v)
        scales.append((k_scale, v_scale))
        out = torch.empty_like(q)
        for b in range(n if decode else 1):
            first = int(pos[b]) if decode else case["base"]
            old = [a[b, layer, :first].double() for a in views[:2]]
            for i, s in enumerate(views[2:]):
                s = s[b, layer, :first].double()
                old[i] = (old[i].reshape(first, s.shape[1], old[i].shape[1] // s.shape[1]) * s[..., None]).flatten(1)
            sel = slice(b, b + 1) if decode else slice(None)
            kk, vv = (torch.cat([o, r[sel]]).reshape(-1, kv_heads, dim) for o, r in zip(old, (k_kept, v_kept)))
            out[sel] = _attend(q[sel], kk, vv, torch.as_tensor(pos[sel], device="cuda") + 1, windows[layer])
        out = out.reshape(n, -1)
        outs.append(out @ w[3].T if "weights" in case else out)

    def as_appended(rows):  # [sequence][layer][position][...]
        x = torch.stack(rows)
        return x.transpose(0, 1)[:, :, None] if decode else x[None]

    if decode and case["ragged"]:
        coded = case["kv"].startswith("q8")
        appended = [None if coded else as_appended(rows_k)[b, :, 0] for b in range(min(16, case["batch"]))]
    elif scales[0][0] is not None:
        appended = [None, None, as_appended([s[0] for s in scales]), as_appended([s[1] for s in scales])]
    else:
        appended = [as_appended(rows_k), as_appended(rows_v)]
    return {"out": torch.stack(outs), "appended": appended}
