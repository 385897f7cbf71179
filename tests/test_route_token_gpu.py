"""The router of a few tokens: one cluster of CTAs per token up to 32 experts, 2048 columns and nine tokens, and
what lies just past each of these. Ids exactly the checker's; ragged columns leave threads without any."""

import numpy as np
import pytest

from bobcat_b200 import Cuda, Norm
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused_norm", [False, True])
@pytest.mark.parametrize("n_cols, n_experts, n_tokens", [(4, 1, 1), (1020, 17, 1), (1024, 16, 2), (1028, 31, 3), (2048, 32, 1), (2048, 32, 9),
                                                         (2048, 32, 10), (2052, 32, 1), (2048, 33, 1), (66, 8, 2)])
def test_route_of_a_few_tokens(n_cols, n_experts, n_tokens, fused_norm):
    cuda = Cuda.open(0)
    rng = np.random.default_rng(n_cols + n_experts)
    n_used = min(4, n_experts)
    x = rng.standard_normal((n_tokens, n_cols)).astype(np.float32)
    nw = rng.uniform(0.5, 1.5, n_cols).astype(np.float32)
    router = (rng.standard_normal((n_experts, n_cols)) * 0.05).astype(np.float32)
    bias = (rng.standard_normal(n_experts) * 0.02).astype(np.float32)
    xb, nb, rb, bb = cuda.buffer_from(x), cuda.buffer_from(nw), cuda.buffer_from(router), cuda.buffer_from(bias)
    normed, route = cuda.new_buffer(x.nbytes), cuda.new_buffer(cuda.route_bytes(n_used, n_tokens))
    cuda.begin()
    cuda.moe_route(xb, (Norm(nb.at(0), 1e-5), normed.at(0)) if fused_norm else None, rb, bb, route, n_cols, n_experts, n_used, n_tokens)
    cuda.end()
    got = cuda.read(route, np.zeros((n_tokens, 2 * n_used), dtype=np.uint32))
    rows = cuda.read(normed, np.zeros_like(x)) if fused_norm else x
    if fused_norm:
        scale = (1 / np.sqrt((x.astype(np.float64) ** 2).mean(1, keepdims=True) + 1e-5)).astype(np.float32)
        assert np.abs(rows - nw * (x * scale)).max() <= 2 ** -22 * np.abs(rows).max()  # the scale may round the other way
    for t in range(n_tokens):
        experts, scores = oracle.lfm2_route(oracle.matvec(0, router, rows[t], n_experts, threads=1), bias, n_used)
        assert got[t, :n_used].tolist() == experts[:n_used].tolist()
        assert np.abs(got[t, n_used:].view(np.float32) - scores[experts[:n_used]]).max() < 1e-6  # the bound of test_moe_gpu.py
    cuda.close()
