"""The convolutions over a batch at the edges of their runs of tokens, taps and channel groups, the
history carried across batches, against f64."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BATCHES = (1, 3, 5, 8, 9, 2, 33)


@pytest.mark.parametrize("n_embd,kernel", [(70, 3), (70, 9), (132, 4), (132, 5)])
def test_short_conv_runs(cuda, n_embd, kernel):
    rng = np.random.default_rng(n_embd + kernel)
    taps = rng.uniform(-1, 1, (n_embd, kernel)).astype(np.float32)
    past = np.zeros((kernel - 1, n_embd))
    tb, hb = cuda.buffer_from(taps), cuda.buffer_from(past.astype(np.float32))
    for n in BATCHES:
        bcx = rng.uniform(-1, 1, (n, 3, n_embd)).astype(np.float32)
        bb, ob = cuda.buffer_from(bcx), cuda.new_buffer(n * n_embd * 4)
        cuda.begin(); cuda.short_conv(bb, tb, hb, ob, n_embd, kernel, n); cuda.end()
        bx = np.concatenate([past, (bcx[:, 0] * bcx[:, 2]).astype(np.float64)])
        want = bcx[:, 1] * sum(taps[:, kk] * bx[kk:kk + n] for kk in range(kernel))
        past = bx[-(kernel - 1):]
        assert np.abs(cuda.read(ob, np.zeros((n, n_embd), dtype=np.float32)) - want).max() < 1e-5
        assert np.abs(cuda.read(hb, np.zeros((kernel - 1, n_embd), dtype=np.float32)) - past).max() < 1e-6


@pytest.mark.parametrize("conv_dim,kernel", [(40, 2), (128, 4), (200, 5), (8192, 4), (300, 8)])
def test_gdn_conv_runs(cuda, conv_dim, kernel):
    rng = np.random.default_rng(conv_dim + kernel)
    taps = rng.uniform(-1, 1, (conv_dim, kernel)).astype(np.float32)
    past = np.zeros((kernel - 1, conv_dim))
    tb, hb = cuda.buffer_from(taps), cuda.buffer_from(np.zeros((conv_dim, kernel - 1), dtype=np.float32))
    for n in BATCHES + (300,):
        x = rng.uniform(-1, 1, (n, conv_dim)).astype(np.float32)
        xb, ob = cuda.buffer_from(x), cuda.new_buffer(n * conv_dim * 4)
        cuda.begin(); cuda.gdn_conv(xb, tb, hb, ob, conv_dim, kernel, n); cuda.end()
        rows = np.concatenate([past, x.astype(np.float64)])
        s = sum(taps[:, i] * rows[i:i + n] for i in range(kernel))
        past = rows[-(kernel - 1):]
        assert np.abs(cuda.read(ob, np.zeros((n, conv_dim), dtype=np.float32)) - s / (1 + np.exp(-s))).max() < 1e-5
        assert np.abs(cuda.read(hb, np.zeros((conv_dim, kernel - 1), dtype=np.float32)) - past.T).max() == 0
