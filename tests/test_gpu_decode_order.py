"""Decode launches overlap their first loads with the end of the decode launch in front. Rows that something else wrote in
between have to be seen all the same: a kernel or copy of the host's through kv_device_ptrs, a replayed graph, an import.
Every scenario runs once with the stream left to itself and once with a synchronisation after every piece of work; the two
give the same bits, since both run the same launches.
"""
import numpy as np
import pytest
import torch

import gguf_runner_b200 as g
from gguf_runner_b200.binding import AttnConfig, KV_BF16, KV_F32, KV_Q8_ROW, RawCuda, ROPE_NEOX

pytestmark = pytest.mark.gpu
N, STEPS = 2500, 10
DTYPES = {KV_F32: torch.float32, KV_BF16: torch.bfloat16, KV_Q8_ROW: torch.int8}


def context(fmt, batch, **more):
    return g.AttnContext(AttnConfig(n_layers=2, n_heads=16, n_kv_heads=4, head_dim=128, seq_len=N + STEPS, max_batch=batch,
                                    rope_theta=1e6, rope_style=ROPE_NEOX, kv_format=fmt, **more))


def views(ctx):
    """K and V as [sequence][layer][position][kv_dim], and the scales of a q8 cache [sequence][layer][position]."""
    cfg = ctx.config
    k, v, ks, vs, nbytes = ctx.kv_device_ptrs()
    lead = (cfg.max_batch, cfg.n_layers, cfg.seq_len)

    def tensor(ptr, size, dtype):
        raw = RawCuda(ptr, size)
        raw.owner = ctx
        return torch.as_tensor(raw, device="cuda").view(dtype).view(*lead, -1)

    out = [tensor(p, nbytes, DTYPES[cfg.kv_format]) for p in (k, v)]
    return out + ([tensor(p, 4 * lead[0] * lead[1] * lead[2], torch.float32) for p in (ks, vs)] if ks else [])


def fill(view, rows, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(*rows, generator=gen, device="cuda")
    if view.dtype == torch.int8:
        return (x * 35).round().clamp(-127, 127).to(torch.int8)
    return (x.abs() * 0.02 if view.shape[-1] == 1 else x).to(view.dtype)


def inputs(cfg):
    gen = torch.Generator(device="cuda").manual_seed(1)
    return [torch.randn(STEPS, 2, cfg.max_batch, d, generator=gen, device="cuda") for d in (cfg.q_dim, cfg.kv_dim, cfg.kv_dim)]


def run(fmt, batch, between, sync, **more):
    """STEPS token steps over layers 1 and 0; `between(ctx, views, step, call)` enqueues foreign work before each decode."""
    ctx = context(fmt, batch, **more)
    vw = views(ctx)
    for i, w in enumerate(vw):
        w.copy_(fill(w, w.shape, 50 + i))
    qkv, pos = inputs(ctx.config), N - 1 - 300 * (np.arange(batch, dtype=np.int32) % 2)
    out = torch.empty(STEPS, 2, batch, ctx.config.q_dim, device="cuda")
    torch.cuda.synchronize()
    for step in range(STEPS):
        for layer in (1, 0):
            def call(layer=layer):
                ctx.decode(layer, pos + step, *(t[step, layer] for t in qkv), out=out[step, layer])
            between(ctx, vw, step, layer, call)
            if sync:
                torch.cuda.synchronize()
    torch.cuda.synchronize()
    ctx.close()
    return out.cpu()


def foreign_kernel(ctx, vw, step, layer, call):
    """Fresh rows for the layer that is read next, by a kernel per array, right in front of the decode."""
    fresh = [fill(w, w[:, layer, :N - 400].shape, 7 * step + i) for i, w in enumerate(vw)]
    for w, x in zip(vw, fresh):
        w[:, layer, :N - 400].copy_(x)
    call()


def foreign_copy(ctx, vw, step, layer, call):
    """The same as one flat device-to-device copy of a sequence's prefix (a forked conversation)."""
    for w in vw:
        w[-1, layer, :N - 400].copy_(w[0, layer, 17:N - 383].clone())
    call()


@pytest.mark.parametrize("fmt,batch", [(KV_F32, 1), (KV_Q8_ROW, 1), (KV_BF16, 1), (KV_BF16, 3), (KV_Q8_ROW, 4)])
@pytest.mark.parametrize("between", [foreign_kernel, foreign_copy])
def test_rows_written_by_the_host(fmt, batch, between):
    assert torch.equal(run(fmt, batch, between, False), run(fmt, batch, between, True))


@pytest.mark.parametrize("fmt", [KV_F32, KV_BF16])
def test_replayed_graph_between_eager_calls(fmt):
    """A graph of one decode of layer 0 appends a row that the eager decode of the same layer reads next; what the host last
    launched itself was layer 1."""

    def steps(sync):
        ctx = context(fmt, 1)
        for i, w in enumerate(views(ctx)):
            w.copy_(fill(w, w.shape, 50 + i))
        (q, k, v), pos = inputs(ctx.config), np.array([N - 1], np.int32)
        out = torch.empty(STEPS, 3, 1, ctx.config.q_dim, device="cuda")
        rows = [t.clone() for t in (q[0, 0], k[0, 0], v[0, 0])]
        got = torch.empty_like(out[0, 0])
        side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            ctx.decode(0, pos, *rows, out=got)
            side.synchronize()
            with torch.cuda.graph(graph, stream=side):
                ctx.decode(0, pos, *rows, out=got)
            for step in range(STEPS):
                ctx.decode(1, pos, q[step, 1], k[step, 1], v[step, 1], out=out[step, 0])
                if sync:
                    side.synchronize()
                for r, t in zip(rows, (q, k, v)):
                    r.copy_(t[step, 0])
                graph.replay()
                if sync:
                    side.synchronize()
                out[step, 1].copy_(got)
                ctx.decode(0, pos + 1, q[step, 1], k[step, 0], v[step, 0], out=out[step, 2])
                if sync:
                    side.synchronize()
            side.synchronize()
        del graph
        ctx.close()
        return out.cpu()

    assert torch.equal(steps(False), steps(True))


def test_imported_rows():
    def imported(ctx, vw, step, layer, call):
        rng = np.random.default_rng(step)
        codes = rng.integers(-127, 128, (2, 900, ctx.config.kv_dim)).astype(np.int8)
        ctx.kv_import(layer, 100, *codes, *rng.uniform(0.01, 0.03, (2, 900)).astype(np.float32))
        call()

    assert torch.equal(run(KV_Q8_ROW, 1, imported, False), run(KV_Q8_ROW, 1, imported, True))
