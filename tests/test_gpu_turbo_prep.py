"""The TurboQuant preparation kernel (biases, QK-norm, RoPE, quantising append in one launch, heads of 128) against the separate
kernels: the rows of an f32 cache are what bias, norm and RoPE make of the keys, and the granular write quantises them.
Rows are compared bit for bit, since both sides do the same rounded operations; outputs with the oracle (bf16 class, 2e-2).
"""
import numpy as np
import pytest

import gguf_runner_b200 as g
from gguf_runner_b200.binding import (AttnConfig, KV_F32, KV_TURBO, ROPE_ADJACENT, ROPE_INTERLEAVED, ROPE_NEOX,
                                      SCALE_Q_PRESCALED)
from tests.oracle_binding import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads", [(1, 1), (6, 2), (32, 4)])
@pytest.mark.parametrize("style,plan,prescaled", [(ROPE_NEOX, False, False), (ROPE_ADJACENT, False, True), (ROPE_NEOX, True, False)])
@pytest.mark.parametrize("bias,norm", [(False, False), (True, False), (True, True), (False, True)])
def test_rows_equal_the_separate_kernels(heads, kv_heads, style, plan, prescaled, bias, norm):
    base = dict(n_layers=2, n_heads=heads, n_kv_heads=kv_heads, head_dim=128, seq_len=64, rope_theta=1e6, rope_style=style)
    if plan:
        base.update(rope_sections=[24, 20, 20, 0], rope_layout=ROPE_INTERLEAVED)
    if prescaled:
        base.update(scale_mode=SCALE_Q_PRESCALED)
    cfg = AttnConfig(kv_format=KV_TURBO, **base)
    fused, plain, f32, ora = (g.AttnContext(cfg), g.AttnContext(cfg), g.AttnContext(AttnConfig(kv_format=KV_F32, **base)),
                              Oracle(cfg, threads=4))
    rng = np.random.default_rng(heads)

    def rand(*shape):
        return rng.standard_normal(shape).astype(np.float32)

    kw = {}
    if bias:
        kw.update(q_bias=rand(cfg.q_dim), k_bias=rand(cfg.kv_dim), v_bias=rand(cfg.kv_dim))
    if norm:
        kw.update(q_norm=1 + 0.1 * rand(128), k_norm=1 + 0.1 * rand(128))
    position_plan = g.RopePositionPlan()
    position_plan.append_text(3)
    position_plan.append_grid([1, 3, 4], 12)
    position_plan.append_text(4)
    for c in (fused, f32, ora):
        if kw:
            c.set_layer_fixups(1, eps=1e-6, **kw)
        if plan and c is ora:
            c.set_position_plan(position_plan.positions, position_plan.next_text_position)
        elif plan:
            c.set_position_plan(position_plan)
    m = 21
    q, k, v = rand(m, cfg.q_dim), rand(m, cfg.kv_dim), rand(m, cfg.kv_dim)
    k[3] = 0.0
    for c in (fused, f32, ora):
        out = c.prefill(1, 0, q[:-1], k[:-1], v[:-1])
        last = c.decode(1, [m - 1], q[-1:], k[-1:], v[-1:])
        if c is fused:
            got = out, last
    assert max(float(np.max(np.abs(a - b))) for a, b in zip(got, (out, last))) <= 2e-2
    for pos in range(m):
        plain.kv_write_token(1, pos, *f32.kv_read_row(1, pos))
        a, b = fused.kv_read_turbo(1, pos), plain.kv_read_turbo(1, pos)
        for name in b:
            assert np.array_equal(a[name], b[name]), (pos, name)
