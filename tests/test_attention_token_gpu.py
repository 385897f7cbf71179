"""One query over a short context takes one launch, a cluster of CTAs per KV head. Positions around the ends of a
chunk (16), of a cluster's round (32 chunks) and of the range (2048); head sizes, groups, both caches."""

import numpy as np
import pytest

from bobcat_b200 import Cuda

pytestmark = pytest.mark.gpu


def float64(q, k, v, group):
    out = np.empty(q.shape)
    for h in range(q.shape[0]):
        s = k[:, h // group].astype(np.float64) @ q[h].astype(np.float64) / np.sqrt(q.shape[1])
        w = np.exp(s - s.max())
        out[h] = (w / w.sum()) @ v[:, h // group].astype(np.float64)
    return out


@pytest.mark.parametrize("kv_half", [True, False])
@pytest.mark.parametrize("heads, kv_heads, hd", [(8, 8, 64), (16, 8, 64), (32, 8, 64), (12, 4, 128), (8, 2, 256)])
@pytest.mark.parametrize("pos, n_ctx", [(0, 1), (15, 40), (16, 40), (511, 512), (512, 700), (700, 1024), (1500, 1600), (2047, 2048), (2047, 2049)])
def test_one_query(kv_half, heads, kv_heads, hd, pos, n_ctx):
    cuda = Cuda.open(0)
    rng = np.random.default_rng(pos + hd + heads)
    q = rng.uniform(-1, 1, (heads, hd)).astype(np.float32)
    dtype = np.float16 if kv_half else np.float32
    k, v = (rng.uniform(-1, 1, (n_ctx, kv_heads, hd)).astype(dtype) for _ in range(2))
    out = cuda.new_buffer(q.nbytes)
    scratch = cuda.new_buffer(cuda.attention_scratch_floats(heads, hd, n_ctx, 1) * 4)
    qb, kb, vb = cuda.buffer_from(q), cuda.buffer_from(k), cuda.buffer_from(v)
    cuda.begin()
    cuda.attention(qb, kb, vb, kv_half, scratch, out, heads, kv_heads, hd, pos, 1, n_ctx)
    cuda.end()
    got = cuda.read(out, np.zeros_like(q))
    want = float64(q, k[: pos + 1], v[: pos + 1], heads // kv_heads)
    # The bound of the other float32 attention kernels on inputs of this size (test_ops_gpu.py).
    assert np.abs(got - want).max() < 2e-6
    cuda.close()


@pytest.mark.parametrize("kv_half", [True, False])
@pytest.mark.parametrize("heads, kv_heads, hd", [(14, 14, 64), (30, 15, 64), (64, 16, 64), (24, 24, 128), (32, 32, 64), (8, 2, 64)])
@pytest.mark.parametrize("pos, n_ctx", [(100, 512), (512, 513), (1000, 1024), (1000, 1025)])
def test_either_side_of_the_lines(kv_half, heads, kv_heads, hd, pos, n_ctx):
    """Many KV heads, whose clusters do not run at once, and contexts of 33 to 64 chunks of a half cache take two launches."""
    test_one_query(kv_half, heads, kv_heads, hd, pos, n_ctx)
