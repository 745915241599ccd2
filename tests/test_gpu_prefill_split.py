"""Prefill over the quantised caches: the tensor-core kernel with two-way f16 splits against the f32 CUDA-core kernel
(prefill_impl = SIMT) on the same rows, at the edges of its 64-row and 64-key tiles.

Tolerance: both kernels round every product and sum to f32. A score of head_dim N(0, 1) products carries an error of
about sqrt(128) * 2^-24 * |q| |k| / sqrt(128) = 2^-24 * 11.3 * 11.3 = 7.6e-6 (the two f16 parts of an operand leave out up to
2^-23 of it, but independently per element: they add less than half of that), which is the relative error of its softmax
weight; outputs are weighted means of values up to ~4.5, so two such evaluations differ by less than 7e-5.
"""
import numpy as np
import pytest

import gguf_runner_b200 as g
from gguf_runner_b200.binding import (AttnConfig, IMPL_SIMT, KV_Q8_BLOCK32, KV_Q8_ROW, KV_TURBO, ROPE_NEOX)

pytestmark = pytest.mark.gpu
TOL = 7e-5
FORMATS = [(KV_Q8_ROW, 128), (KV_Q8_ROW, 64), (KV_Q8_BLOCK32, 128), (KV_Q8_BLOCK32, 64), (KV_TURBO, 128)]


def pair(fmt, head_dim, n_heads, n_kv_heads, seq_len, **more):
    base = dict(n_layers=1, n_heads=n_heads, n_kv_heads=n_kv_heads, head_dim=head_dim, seq_len=seq_len, rope_theta=1e6,
                rope_style=ROPE_NEOX, kv_format=fmt, **more)
    return g.AttnContext(AttnConfig(**base)), g.AttnContext(AttnConfig(prefill_impl=IMPL_SIMT, **{**base, "max_splits": 0}))


def rows(rng, cfg, m):
    return [rng.standard_normal((m, d)).astype(np.float32) for d in (cfg.q_dim, cfg.kv_dim, cfg.kv_dim)]


def both(ctxs, pos, q, k, v, call="prefill"):
    got, want = (getattr(c, call)(0, pos, q, k, v) for c in ctxs)
    return float(np.max(np.abs(got - want)))


@pytest.mark.parametrize("fmt,head_dim", FORMATS)
@pytest.mark.parametrize("heads,kv_heads", [(1, 1), (6, 2), (5, 1), (32, 4)])
@pytest.mark.parametrize("window", [0, 70])
def test_tile_edges(fmt, head_dim, heads, kv_heads, window):
    """Chunks whose rows and keys end on, before and behind the tile edges, behind prefixes of every residue."""
    ctxs = pair(fmt, head_dim, heads, kv_heads, 700, layer_windows=[window] if window else [])
    rng, pos = np.random.default_rng(heads + window), 0
    for m in (1, 63, 1, 64, 2, 129, 300, 33):
        q, k, v = rows(rng, ctxs[0].config, m)
        assert both(ctxs, pos, q, k, v) <= TOL, (m, pos)
        pos += m


@pytest.mark.parametrize("fmt,head_dim", FORMATS)
@pytest.mark.parametrize("max_splits", [1, 3, 0])
def test_split_keys(fmt, head_dim, max_splits):
    ctxs = pair(fmt, head_dim, 8, 2, 4000, max_splits=max_splits)
    rng = np.random.default_rng(3)
    for pos, m in ((0, 3001), (3001, 40), (3041, 7)):
        q, k, v = rows(rng, ctxs[0].config, m)
        assert both(ctxs, pos, q, k, v) <= TOL, (m, pos)
    assert ctxs[0].last_split_count > 1 or max_splits == 1


@pytest.mark.parametrize("fmt,head_dim", FORMATS)
def test_image_blocks_and_gate(fmt, head_dim):
    ctxs = pair(fmt, head_dim, 6, 2, 400, image_mode=1, layer_windows=[50])
    for c in ctxs:
        c.set_media_blocks([(10, 100), (200, 70)], 400)
    q, k, v = rows(np.random.default_rng(4), ctxs[0].config, 400)
    assert both(ctxs, 0, q, k, v, "prefill_block") <= TOL
    ctxs = pair(fmt, head_dim, 6, 2, 400)
    gate = np.random.default_rng(5).standard_normal((400, ctxs[0].config.q_dim)).astype(np.float32)
    got, want = (c.prefill_gated(0, 0, q, k, v, gate) for c in ctxs)
    assert np.max(np.abs(got - want)) <= TOL


@pytest.mark.parametrize("fmt", [KV_Q8_ROW, KV_Q8_BLOCK32])
def test_scales_far_apart(fmt):
    """Value scales over forty orders of magnitude and query rows over twelve: no product leaves f16's range unseen."""
    ctxs = pair(fmt, 128, 4, 1, 400)
    rng, cfg = np.random.default_rng(6), ctxs[0].config
    n, shape = 300, (300,) if fmt == KV_Q8_ROW else (300, 4)
    codes = rng.integers(-127, 128, (2, n, cfg.kv_dim)).astype(np.int8)
    ks = np.full(shape, 1e-2, np.float32)
    vs = (10.0 ** rng.uniform(-30, 10, shape)).astype(np.float32)
    for c in ctxs:
        c.kv_import(0, 0, codes[0], codes[1], ks, vs)
    q, k, v = rows(rng, cfg, 66)
    q *= 10.0 ** rng.uniform(-12, 0, (66, 1)).astype(np.float32)
    q[5] = 0.0
    got, want = (c.prefill(0, n, q, k, v) for c in ctxs)
    # relative to each row: weights differ by 7.6e-6, and the largest value dominates the row's sum
    err = np.linalg.norm(got - want, axis=1) / np.linalg.norm(want, axis=1)
    assert np.all(np.isfinite(got)) and np.max(err) <= 3e-5


@pytest.mark.parametrize("fmt,head_dim", [(KV_Q8_ROW, 32), (KV_Q8_ROW, 256), (KV_TURBO, 64)])
def test_other_head_dims_stay_on_the_general_kernel(fmt, head_dim):
    ctxs = pair(fmt, head_dim, 4, 2, 200)
    q, k, v = rows(np.random.default_rng(7), ctxs[0].config, 130)
    assert both(ctxs, 0, q, k, v) == 0.0
