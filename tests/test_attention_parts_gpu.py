"""Prefill attention with the keys cut into parts: ragged batches, groups of query heads, parts that lie past some rows."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_heads,n_kv,hd,first_pos,n_q", [(8, 2, 256, 0, 64), (8, 2, 256, 1500, 33), (4, 4, 128, 700, 40), (6, 2, 64, 333, 50), (8, 1, 64, 1, 63),
                                                           (2, 2, 256, 62, 66), (16, 4, 128, 0, 130)])
def test_parts_join_to_the_whole(cuda, n_heads, n_kv, hd, first_pos, n_q):
    rng = np.random.default_rng(n_heads * hd + first_pos + n_q)
    n = first_pos + n_q
    q = rng.uniform(-2, 2, (n_q, n_heads, hd)).astype(np.float32)
    k, v = (rng.uniform(-2, 2, (n, n_kv, hd)).astype(np.float16) for _ in range(2))
    n_ctx = n + 40
    qb, kb, vb, ob = cuda.buffer_from(q), cuda.buffer_from(k), cuda.buffer_from(v), cuda.new_buffer(q.nbytes)
    sb = cuda.new_buffer(cuda.attention_scratch_floats(n_heads, hd, n_ctx, n_q) * 4)
    cuda.begin(); cuda.attention(qb, kb, vb, True, sb, ob, n_heads, n_kv, hd, first_pos, n_q, n_ctx); cuda.end()
    got = cuda.read(ob, np.zeros_like(q))
    for h in range(n_heads):
        kv = h // (n_heads // n_kv)
        scores = q[:, h].astype(np.float64) @ k[:, kv].astype(np.float64).T / np.sqrt(hd)
        scores[np.arange(n)[None] > first_pos + np.arange(n_q)[:, None]] = -np.inf
        p = np.exp(scores - scores.max(axis=1, keepdims=True))
        want = p / p.sum(axis=1, keepdims=True) @ v[:, kv].astype(np.float64)
        assert np.abs(got[:, h] - want).max() < 1e-5
