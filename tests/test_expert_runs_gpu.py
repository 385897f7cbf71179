"""Products over experts whose jobs are cut into equal runs across all groups of rows: more experts than a
warp has lanes, experts without rows between others, an expert with every token (several groups), one
cluster per run (wide matrices), fewer jobs than the device has SMs; float32 and half operands."""

import numpy as np
import pytest

from bobcat_b200 import Q4_0
from conftest import random_q4_0
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_tokens,n_rows,n_cols,n_experts", [(1, 16, 64, 33), (15, 48, 1024, 40), (9, 1792, 256, 70), (7, 32, 4096, 5), (16, 16, 64, 33),
                                                              (70, 64, 1024, 40), (33, 400, 256, 70), (97, 32, 4096, 36), (203, 208, 512, 32)])
def test_runs_across_experts(cuda, n_tokens, n_rows, n_cols, n_experts):
    rng = np.random.default_rng(n_tokens + n_rows)
    n_used = 2
    raw = random_q4_0(rng, n_experts * n_rows, n_cols)
    w = oracle.dequantize(2, raw, n_experts * n_rows * n_cols).reshape(n_experts, n_rows, n_cols).astype(np.float64)
    x = rng.uniform(-1, 1, (n_tokens, n_cols)).astype(np.float32)
    route = np.zeros((n_tokens, 2 * n_used), dtype=np.uint32)
    others = [e for e in range(n_experts) if e != 2 and e % 3 != 1]  # a third of the experts get nothing
    for t in range(n_tokens):
        route[t, :n_used] = (2, rng.choice(others))
    wb, xb, rb = cuda.upload_matrix(Q4_0, raw, n_experts * n_rows, n_cols), cuda.buffer_from(x), cuda.buffer_from(route)
    ob, eb = cuda.new_buffer((n_experts + 1) * 4), cuda.new_buffer(n_tokens * n_used * 4)
    out = cuda.buffer_from(np.full((n_tokens + 1, n_used, n_rows), 7, dtype=np.float32))
    cuda.begin()
    cuda.moe_group(rb, ob, eb, n_experts, n_used, n_tokens)
    cuda.matmul_experts(Q4_0, wb, None, n_rows, n_cols, n_experts, xb, True, ob, eb, n_used, out, n_tokens)
    cuda.end()
    got = cuda.read(out, np.zeros((n_tokens + 1, n_used, n_rows), dtype=np.float32))
    picked = w[route[:, :n_used]]
    want = np.einsum("tsrc,tc->tsr", picked, x.astype(np.float64))
    room = np.einsum("tsrc,tc->tsr", np.abs(picked), np.abs(x.astype(np.float64)))
    assert float((np.abs(got[:n_tokens] - want) / np.maximum(room, 1e-30)).max()) < (1e-6 if n_tokens < 16 else 1e-3)
    assert (got[n_tokens] == 7).all()
