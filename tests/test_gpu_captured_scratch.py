"""Captured launches keep the addresses of their scratch: calls made between capture and replay must not move it.

A replayed launch runs on the same rows as an eager one in front of it and gives the same bits.
"""
import numpy as np
import pytest
import torch

import gguf_runner_b200 as g
from gguf_runner_b200.binding import AttnConfig, KV_BF16, KV_Q8_BLOCK32, KV_Q8_ROW, KV_TURBO, ROPE_NEOX, W_F32, Weights

pytestmark = pytest.mark.gpu
SEQ = 6000


def context(fmt, **more):
    return g.AttnContext(AttnConfig(n_layers=2, n_heads=32, n_kv_heads=8, head_dim=128, seq_len=SEQ, rope_theta=1e6,
                                    rope_style=ROPE_NEOX, kv_format=fmt, **more))


def rows(cfg, m, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(m, d, generator=gen, device="cuda") for d in (cfg.q_dim, cfg.kv_dim, cfg.kv_dim)]


def captured(call):
    """`call` on a side stream: eagerly once, then captured. Returns the stream and the graph."""
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        call()
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            call()
    return side, graph


@pytest.mark.parametrize("fmt,norm", [(KV_BF16, False), (KV_Q8_ROW, False), (KV_Q8_BLOCK32, False), (KV_BF16, True), (KV_TURBO, True)])
def test_decode_graph_survives_a_prompt(fmt, norm):
    ctx = context(fmt)
    cfg, pos = ctx.config, np.array([1700], np.int32)
    if norm:  # rows on their way through the fix-ups, rotated queries of a TurboQuant cache
        for layer in range(2):
            ctx.set_layer_fixups(layer, q_norm=np.full(128, 1.1, np.float32), k_norm=np.full(128, 0.9, np.float32))
    ctx.prefill(1, 0, *rows(cfg, 1700, 1))
    step, out = rows(cfg, 1, 2), torch.empty(1, cfg.q_dim, device="cuda")
    torch.cuda.synchronize()
    side, graph = captured(lambda: ctx.decode(1, pos, *step, out=out))
    eager, splits = out.clone(), ctx.last_split_count
    with torch.cuda.stream(side):
        for m in (333, 40, 2000):  # chunks that split their keys and chunks that need longer buffers
            ctx.prefill(0, 1700, *rows(cfg, m, 3))
        junk = [torch.full((1 << 20,), float("nan"), device="cuda") for _ in range(8)]  # whoever reuses freed memory
        out.zero_()
        for _ in range(3):
            graph.replay()
        side.synchronize()
        assert torch.equal(out, eager)
        assert all(bool(t.isnan().all()) for t in junk)
        ctx.decode(1, pos, *step, out=out)  # and the split count does not depend on the prompts before
        side.synchronize()
        assert torch.equal(out, eager) and ctx.last_split_count == splits > 1
    del graph
    ctx.close()


def test_half_layer_graph_survives_a_prompt():
    ctx = context(KV_BF16)
    cfg, pos, rng = ctx.config, np.array([40], np.int32), np.random.default_rng(3)
    w = [Weights(W_F32, r, c, rng.standard_normal((r, c)).astype(np.float32) * 0.03)
         for r, c in ((cfg.q_dim, 512), (cfg.kv_dim, 512), (cfg.kv_dim, 512), (512, cfg.q_dim))]
    prompt = torch.randn(700, 512, device="cuda")
    x, out = torch.randn(1, 512, device="cuda"), torch.empty(1, 512, device="cuda")
    ctx.layer_prefill(1, 0, prompt[:40], *w)
    torch.cuda.synchronize()
    side, graph = captured(lambda: ctx.layer_decode(1, pos, x, *w, out=out))
    eager = out.clone()
    with torch.cuda.stream(side):
        for m in (200, 700):
            ctx.layer_prefill(0, 0, prompt[:m], *w)
        out.zero_()
        graph.replay()
        side.synchronize()
    assert torch.equal(out, eager)
    del graph
    ctx.close()


@pytest.mark.parametrize("fmt", [KV_BF16, KV_Q8_ROW])
def test_prefill_graph_survives_longer_prefixes(fmt):
    """A captured chunk whose keys are split, then the same chunk behind a longer prefix (more splits), then the replay."""
    ctx = context(fmt)
    cfg = ctx.config
    ctx.prefill(1, 0, *rows(cfg, 5600, 1))
    chunk, out = rows(cfg, 40, 2), torch.empty(40, cfg.q_dim, device="cuda")
    torch.cuda.synchronize()
    side, graph = captured(lambda: ctx.prefill(1, 1700, *chunk, out=out))
    eager = out.clone()
    with torch.cuda.stream(side):
        ctx.prefill(1, 5600, *rows(cfg, 40, 3))
        out.zero_()
        graph.replay()
        side.synchronize()
    assert torch.equal(out, eager)
    del graph
    ctx.close()
