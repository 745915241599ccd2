"""bf16 prefill chunks whose key tiles are split over CTAs (few query tiles behind a long prefix) against the unsplit launch
(max_splits = 1), at chunk sizes around the 128- and 256-row tiles.

Tolerance: the two differ in the reference maximum of each softmax row, so every probability is rounded to bf16 at another
scale: 2^-9 relative on probabilities, on outputs of up to about 4.5 units, 1e-2.
"""
import numpy as np
import pytest

import gguf_runner_b200 as g
from gguf_runner_b200.binding import AttnConfig, KV_BF16, ROPE_NEOX

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim,heads,kv_heads", [(64, 4, 2), (128, 5, 1), (128, 32, 8)])
@pytest.mark.parametrize("window", [0, 1500])
def test_splits_match_the_unsplit_launch(head_dim, heads, kv_heads, window):
    base = dict(n_layers=1, n_heads=heads, n_kv_heads=kv_heads, head_dim=head_dim, seq_len=6000, rope_theta=1e6,
                rope_style=ROPE_NEOX, kv_format=KV_BF16, layer_windows=[window] if window else [])
    ctxs = [g.AttnContext(AttnConfig(max_splits=n, **base)) for n in (0, 1)]
    cfg, rng, pos = ctxs[0].config, np.random.default_rng(heads), 0
    for m in (3000, 1, 17, 128, 129, 255, 256, 257, 333):
        q, k, v, gate = (rng.standard_normal((m, d)).astype(np.float32) for d in (cfg.q_dim, cfg.kv_dim, cfg.kv_dim, cfg.q_dim))
        got, want = (c.prefill(0, pos, q, k, v) for c in ctxs)
        assert np.max(np.abs(got - want)) <= 1e-2, m
        got, want = (c.prefill_gated(0, pos, q, k, v, gate) for c in ctxs)
        assert np.max(np.abs(got - want)) <= 1e-2, m
        if pos:  # at least 12 visible key tiles and at most 64 query tiles x heads: two splits and more
            assert ctxs[0].last_split_count > 1 and ctxs[1].last_split_count == 1, m
        pos += m


def test_merge_launches_are_counted_and_timed():
    import torch
    counts = []
    for max_splits in (0, 1):
        ctx = g.AttnContext(AttnConfig(n_layers=1, n_heads=8, n_kv_heads=2, head_dim=128, seq_len=3000, rope_theta=1e6,
                                       rope_style=ROPE_NEOX, kv_format=KV_BF16, max_splits=max_splits))
        rows = [torch.randn(40, d, device="cuda") for d in (ctx.config.q_dim, ctx.config.kv_dim, ctx.config.kv_dim)]
        before = ctx.launch_count
        ctx.prefill(0, 2900, *rows)
        ctx.set_kernel_timing(True)
        after = ctx.launch_count
        ctx.prefill(0, 2900, *rows)
        counts.append((after - before, ctx.kernel_time(0)[1], ctx.kernel_time(1)[1], ctx.kernel_time(2)[1]))
        ctx.close()
    assert counts == [(3, 1, 1, 1), (2, 1, 1, 0)]


def test_image_blocks_with_splits():
    base = dict(n_layers=1, n_heads=4, n_kv_heads=2, head_dim=128, seq_len=3000, rope_theta=1e6, rope_style=ROPE_NEOX,
                kv_format=KV_BF16, image_mode=1, layer_windows=[1200])
    ctxs = [g.AttnContext(AttnConfig(max_splits=n, **base)) for n in (0, 1)]
    cfg, rng = ctxs[0].config, np.random.default_rng(1)
    for c in ctxs:
        c.set_media_blocks([(2100, 200)], 3000)
    for pos, m, call in ((0, 2000, "prefill"), (2000, 400, "prefill_block")):
        rows = [rng.standard_normal((m, d)).astype(np.float32) for d in (cfg.q_dim, cfg.kv_dim, cfg.kv_dim)]
        got, want = (getattr(c, call)(0, pos, *rows) for c in ctxs)
        assert np.max(np.abs(got - want)) <= 1e-2
        assert ctxs[0].last_split_count > 1 and ctxs[1].last_split_count == 1
