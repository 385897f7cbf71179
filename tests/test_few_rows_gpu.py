"""Q4_0 products of a few rows with float32 operands (fewer than 16 rows): every slicing of K the
kernel can take (one to eight CTAs along K, one to three block pairs per warp, ragged last slices),
ragged row tiles, one to fifteen rows, the three stores, and the experts form."""

import numpy as np
import pytest

from bobcat_b200 import ACCUMULATE, OVERWRITE, Q4_0, SWIGLU
from conftest import random_q4_0
from oracle import oracle

pytestmark = pytest.mark.gpu

# Per unit of sum |w x|: products are exact, what is left is the order of float32 sums.
TOLERANCE = 1e-6


def matrix(rng, n_rows, n_cols):
    raw = random_q4_0(rng, n_rows, n_cols)
    return raw, oracle.dequantize(2, raw, n_rows * n_cols).reshape(n_rows, n_cols).astype(np.float64)


@pytest.mark.parametrize("n_rows,n_cols,n_tokens", [(16, 64, 1), (17, 128, 2), (100, 1024, 8), (64, 1088, 9), (2064, 2048, 5), (48, 3072, 15), (33, 3136, 3),
                                                    (2048, 10752, 7), (80, 6144, 13), (16, 24576, 2), (5000, 2048, 11)])
def test_few_rows_with_float_operands(cuda, n_rows, n_cols, n_tokens):
    rng = np.random.default_rng(n_rows + n_cols + n_tokens)
    raw, w = matrix(rng, n_rows, n_cols)
    # Magnitudes over many orders: what a rounded operand would lose.
    x = (rng.uniform(-1, 1, (n_tokens, n_cols)) * 10.0 ** rng.integers(-6, 4, (n_tokens, n_cols))).astype(np.float32)
    y0 = rng.uniform(-1, 1, (n_tokens + 1, n_rows)).astype(np.float32)
    wb, xb, yb = cuda.upload_matrix(Q4_0, raw, n_rows, n_cols), cuda.buffer_from(x), cuda.buffer_from(y0)
    product, budget = x.astype(np.float64) @ w.T, np.abs(x.astype(np.float64)) @ np.abs(w).T
    old = y0[:n_tokens].astype(np.float64)
    for store, want, room in ((OVERWRITE, product, budget), (ACCUMULATE, old + product, budget + np.abs(old)),
                              (SWIGLU, old / (1 + np.exp(-old)) * product, budget)):
        cuda.write(yb, y0)
        cuda.begin(); cuda.matmul(Q4_0, wb, n_rows, n_cols, xb, yb, n_tokens, store); cuda.end()
        out = cuda.read(yb, np.zeros_like(y0))
        assert float((np.abs(out[:n_tokens] - want) / np.maximum(room, 1e-30)).max()) < TOLERANCE
        assert np.array_equal(out[n_tokens], y0[n_tokens])


@pytest.mark.parametrize("n_tokens,n_ff,n_embd", [(1, 64, 128), (3, 1792, 2048), (15, 192, 1024), (12, 128, 4096)])
def test_experts_of_a_few_rows(cuda, n_tokens, n_ff, n_embd):
    """All tokens on one expert (two groups of 8 rows), and spread picks."""
    rng = np.random.default_rng(n_tokens)
    n_experts, n_used = 6, 2
    gate_raw, gate = matrix(rng, n_experts * n_ff, n_embd)
    up_raw, up = matrix(rng, n_experts * n_ff, n_embd)
    down_raw, down = matrix(rng, n_experts * n_embd, n_ff)
    x = rng.uniform(-1, 1, (n_tokens, n_embd)).astype(np.float32)
    route = np.zeros((n_tokens, 2 * n_used), dtype=np.uint32)
    for t in range(n_tokens):
        route[t, :n_used] = (4, rng.choice([0, 1, 3]))
        route[t, n_used:] = np.float32(0.5).view(np.uint32)
    gb, ub, db = (cuda.upload_matrix(Q4_0, raw, rows, cols) for raw, rows, cols in
                  ((gate_raw, n_experts * n_ff, n_embd), (up_raw, n_experts * n_ff, n_embd), (down_raw, n_experts * n_embd, n_ff)))
    xb, rb, ob, eb = cuda.buffer_from(x), cuda.buffer_from(route), cuda.new_buffer((n_experts + 1) * 4), cuda.new_buffer(n_tokens * n_used * 4)
    ffn, out = cuda.new_buffer(n_tokens * n_used * n_ff * 4), cuda.new_buffer(n_tokens * n_used * n_embd * 4)
    cuda.begin()
    cuda.moe_group(rb, ob, eb, n_experts, n_used, n_tokens)
    cuda.matmul_experts(Q4_0, gb, ub, n_ff, n_embd, n_experts, xb, True, ob, eb, n_used, ffn, n_tokens)
    cuda.matmul_experts(Q4_0, db, None, n_embd, n_ff, n_experts, ffn, False, ob, eb, n_used, out, n_tokens)
    cuda.end()
    hidden = cuda.read(ffn, np.zeros((n_tokens, n_used, n_ff), dtype=np.float32))
    got = cuda.read(out, np.zeros((n_tokens, n_used, n_embd), dtype=np.float32))
    for t in range(n_tokens):
        for s in range(n_used):
            e = int(route[t, s])
            g, u = gate[e * n_ff:(e + 1) * n_ff] @ x[t], up[e * n_ff:(e + 1) * n_ff] @ x[t]
            want = g / (1 + np.exp(-g)) * u
            assert float(np.abs(hidden[t, s] - want).max()) < 1e-5 * max(1.0, float(np.abs(want).max()))
            d = down[e * n_embd:(e + 1) * n_embd]
            room = np.abs(d) @ np.abs(hidden[t, s].astype(np.float64))
            assert float((np.abs(got[t, s] - d @ hidden[t, s].astype(np.float64)) / np.maximum(room, 1e-30)).max()) < TOLERANCE
