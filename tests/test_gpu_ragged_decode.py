"""Decode of sequences of different lengths: pieces of one size per sequence, numbered over all sequences, against the
per-warp CUDA-core kernel (decode_impl = SIMT), which splits every sequence the same number of ways. Two layers, so that the
second launch of a step requests its first tiles while the first one merges.

Tolerance: f32 arithmetic on both sides as in test_gpu_prefill_split.py (7e-5); bf16 queries and probabilities on the
tensor-core side: 2^-9 relative on each, on outputs of a few units, 2e-2.
"""
import numpy as np
import pytest
import torch

import gguf_runner_b200 as g
from gguf_runner_b200.binding import AttnConfig, IMPL_SIMT, KV_BF16, KV_F32, KV_Q8_BLOCK32, KV_Q8_ROW, KV_TURBO, ROPE_NEOX

pytestmark = pytest.mark.gpu
SHAPES = [(KV_F32, 16, 8, 128), (KV_Q8_ROW, 12, 2, 64), (KV_BF16, 40, 8, 128), (KV_BF16, 4, 4, 128), (KV_BF16, 8, 2, 64),
          (KV_TURBO, 16, 4, 128)]


@pytest.mark.parametrize("fmt,heads,kv_heads,head_dim", SHAPES)
@pytest.mark.parametrize("window,max_splits,batch", [(0, 0, 9), (0, 3, 9), (100, 0, 9), (0, 0, 2), (0, 0, 40)])
def test_ragged_lengths(fmt, heads, kv_heads, head_dim, window, max_splits, batch):
    base = dict(n_layers=2, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, seq_len=3000, max_batch=batch, rope_theta=1e6,
                rope_style=ROPE_NEOX, kv_format=fmt, layer_windows=[window] * 2 if window else [])
    ctx = g.AttnContext(AttnConfig(max_splits=max_splits, **base))
    ref = g.AttnContext(AttnConfig(decode_impl=IMPL_SIMT, **base))
    cfg, rng = ctx.config, np.random.default_rng(batch)
    pos = np.array(([2990, 0, 1, 63, 64, 255, 256, 257, 1100] * 5)[:batch], np.int32)
    for seq in range(min(batch, 9)):
        m = int(pos[seq])
        if m:
            for layer in range(2):
                rows = [rng.standard_normal((m, d)).astype(np.float32) for d in (cfg.q_dim, cfg.kv_dim, cfg.kv_dim)]
                for c in (ctx, ref):
                    c.prefill(layer, 0, *rows, seq=seq)
    rows = [torch.randn(6, batch, d, device="cuda") for d in (cfg.q_dim, cfg.kv_dim, cfg.kv_dim)]
    got, want = (torch.empty(6, batch, cfg.q_dim, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    for c, out in ((ctx, got), (ref, want)):
        for call in range(6):  # back to back: three steps over two layers, each step one position further
            c.decode(call % 2, pos + call // 2, *(r[call] for r in rows), out=out[call])
    torch.cuda.synchronize()
    assert float((got - want).abs().max()) <= (2e-2 if fmt in (KV_BF16, KV_TURBO) else 7e-5)
    ctx.close()
    ref.close()


# format, query heads, KV heads, head_dim, sequences, longest, others
LONG_AND_SHORT = [(KV_BF16, 24, 8, 64, 20, 6000, 100), (KV_BF16, 32, 8, 128, 20, 4000, 100), (KV_BF16, 16, 8, 128, 8, 3000, 100),
                  (KV_F32, 16, 8, 128, 6, 3000, 150), (KV_Q8_ROW, 24, 8, 64, 16, 3000, 60), (KV_Q8_BLOCK32, 8, 4, 128, 9, 3000, 100),
                  (KV_TURBO, 16, 4, 128, 9, 3000, 100)]


@pytest.mark.parametrize("fmt,heads,kv_heads,head_dim,batch,longest,others", LONG_AND_SHORT)
def test_one_long_sequence_among_short_ones(fmt, heads, kv_heads, head_dim, batch, longest, others):
    """The ragged launch of every kernel family. The split count says that it was taken: it is the one of the longest sequence,
    which a batch of that length throughout would not be split into."""
    base = dict(n_layers=1, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, seq_len=longest + 8, max_batch=batch,
                rope_theta=1e6, rope_style=ROPE_NEOX, kv_format=fmt)
    ctx, ref = g.AttnContext(AttnConfig(**base)), g.AttnContext(AttnConfig(decode_impl=IMPL_SIMT, **base))
    cfg, rng = ctx.config, np.random.default_rng(batch)
    pos = others + np.arange(batch, dtype=np.int32) % 3 - 1
    pos[batch // 2] = longest - 1
    for seq in range(batch):
        rows = [rng.standard_normal((int(pos[seq]), d)).astype(np.float32) for d in (cfg.q_dim, cfg.kv_dim, cfg.kv_dim)]
        for c in (ctx, ref):
            c.prefill(0, 0, *rows, seq=seq)
    rows = [torch.randn(batch, d, device="cuda") for d in (cfg.q_dim, cfg.kv_dim, cfg.kv_dim)]
    got, want = (torch.empty(batch, cfg.q_dim, device="cuda") for _ in range(2))
    torch.cuda.synchronize()
    ctx.decode(0, pos, *rows, out=got)
    ragged = ctx.last_split_count
    ref.decode(0, pos, *rows, out=want)
    torch.cuda.synchronize()
    assert float((got - want).abs().max()) <= (2e-2 if fmt in (KV_BF16, KV_TURBO) else 7e-5)
    ctx.decode(0, np.full(batch, longest - 1, np.int32), *rows, out=got)
    torch.cuda.synchronize()
    assert ragged > ctx.last_split_count
    ctx.close()
    ref.close()


@pytest.mark.parametrize("batch,length,heads,kv_heads", [(8, 32768, 32, 4), (16, 4000, 32, 8), (16, 1000, 40, 8), (2, 6000, 32, 4)])
def test_nearly_equal_lengths_go_with_equal_ones(batch, length, heads, kv_heads):
    """One position of difference does not change the launch (its split count is another one for ragged pieces)."""
    with g.AttnContext(AttnConfig(n_layers=1, n_heads=heads, n_kv_heads=kv_heads, head_dim=128, seq_len=length, max_batch=batch,
                                  rope_theta=1e6, rope_style=ROPE_NEOX, kv_format=KV_BF16)) as ctx:
        rows = [torch.zeros(batch, d, device="cuda") for d in (ctx.config.q_dim, ctx.config.kv_dim, ctx.config.kv_dim)]
        counts = []
        for less in (0, 1, length // 50):
            ctx.decode(0, length - 1 - less * (np.arange(batch, dtype=np.int32) % 2), *rows)
            counts.append(ctx.last_split_count)
        torch.cuda.synchronize()
    assert counts[0] == counts[1] == counts[2]
