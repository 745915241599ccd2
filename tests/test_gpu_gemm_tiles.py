"""Every column-tile width of the projection GEMM (64, 128, 192 and 256 columns, chosen by the number of waves) against
64-bit products of the same bf16 operands.

Tolerance: sums of k <= 1024 products of N(0, 1) values in f32: k * 2^-24 * sqrt(k) * 0.3 = 6e-4 at the largest k.
"""
import numpy as np
import pytest

import gguf_runner_b200 as g
from gguf_runner_b200.binding import AttnConfig, W_F32, Weights
from tests.oracle_binding import bf16_round

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k", [(17, 1000, 256), (100, 256, 512), (130, 2048, 1024), (500, 4096, 512), (500, 6144, 256),
                                   (700, 12288, 192)])
def test_gemm_tile_widths(m, n, k):
    rng = np.random.default_rng(n + m)
    x, w = (bf16_round(rng.standard_normal(s).astype(np.float32)) for s in ((m, k), (n, k)))
    with g.AttnContext(AttnConfig(n_layers=1, n_heads=1, n_kv_heads=1, head_dim=64, seq_len=8)) as ctx:
        got = ctx.proj_matmul(Weights(W_F32, n, k, w), x)
    assert np.max(np.abs(got - x.astype(np.float64) @ w.astype(np.float64).T)) <= 6e-4
