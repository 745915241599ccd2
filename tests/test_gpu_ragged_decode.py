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
from gguf_runner_b200.binding import AttnConfig, IMPL_SIMT, KV_BF16, KV_F32, KV_Q8_ROW, KV_TURBO, ROPE_NEOX

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
