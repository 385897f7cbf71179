"""Experts of a batch on the kernel that unpacks weights into tensor memory: one matrix and gate with up; groups of
32, 64 and 128 rows and an expert with several of them; columns that leave a stage or a copy short; rows that leave a tile short."""

import numpy as np
import pytest

from bobcat_b200 import Q4_0
from conftest import random_q4_0
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dual", [False, True])
@pytest.mark.parametrize("n_tokens,n_rows,n_cols,n_experts", [(16, 16, 64, 5), (40, 144, 192, 9), (150, 80, 320, 6), (170, 128, 1088, 4), (300, 64, 512, 3), (64, 208, 2048, 12)])
def test_experts_of_a_batch(cuda, n_tokens, n_rows, n_cols, n_experts, dual):
    rng = np.random.default_rng(n_tokens + n_cols)
    n_used = 2
    raws = [random_q4_0(rng, n_experts * n_rows, n_cols) for _ in range(1 + dual)]
    ws = [oracle.dequantize(2, raw, n_experts * n_rows * n_cols).reshape(n_experts, n_rows, n_cols).astype(np.float64) for raw in raws]
    x = rng.uniform(-1, 1, (n_tokens, n_cols)).astype(np.float32)
    route = np.zeros((n_tokens, 2 * n_used), dtype=np.uint32)
    for t in range(n_tokens):  # the last expert gets every token
        route[t, :n_used] = (n_experts - 1, rng.integers(0, n_experts - 1))
    mats = [cuda.upload_matrix(Q4_0, raw, n_experts * n_rows, n_cols) for raw in raws]
    xb, rb = cuda.buffer_from(x), cuda.buffer_from(route)
    ob, eb = cuda.new_buffer((n_experts + 1) * 4), cuda.new_buffer(n_tokens * n_used * 4)
    out = cuda.buffer_from(np.full((n_tokens + 1, n_used, n_rows), 7, dtype=np.float32))
    cuda.begin()
    cuda.moe_group(rb, ob, eb, n_experts, n_used, n_tokens)
    cuda.matmul_experts(Q4_0, mats[0], mats[1] if dual else None, n_rows, n_cols, n_experts, xb, True, ob, eb, n_used, out, n_tokens)
    cuda.end()
    got = cuda.read(out, np.zeros((n_tokens + 1, n_used, n_rows), dtype=np.float32))
    sums, rooms = [], []
    for w in ws:
        picked = w[route[:, :n_used]]
        sums.append(np.einsum("tsrc,tc->tsr", picked, x.astype(np.float64)))
        rooms.append(np.einsum("tsrc,tc->tsr", np.abs(picked), np.abs(x.astype(np.float64))) + 1e-30)
    # A product is off by at most 2^-11 for each rounded operand and the f32 sums: 1e-3 of the sum of its terms' sizes (room).
    if dual:
        g, u = sums
        want = g / (1 + np.exp(-g)) * u
        room = 1.1 * rooms[0] * np.abs(u) + np.abs(g) * rooms[1] + 1e-3 * rooms[0] * rooms[1]  # |silu'| <= 1.1, |silu(g)| <= |g|
    else:
        want, room = sums[0], rooms[0]
    assert float((np.abs(got[:n_tokens] - want) / room).max()) < 1e-3
    assert (got[n_tokens] == 7).all()


# Fewer jobs than fill the device leave a batch to the few-row kernel (up to 64 rows an expert on the average) or to the kernel that unpacks
# into shared memory (more, of narrow matrices; and rows that are no multiple of 16, which have no tiles of their own): the first four
# stay on the kernel with weights in tensor memory (groups of 32 and 64 rows, both lengths of its parts of K, more than a stretch of K; of
# 128, summing all of K), the others are on either side of the lines.
@pytest.mark.parametrize("dual", [False, True])
@pytest.mark.parametrize("n_tokens,n_rows,n_cols,n_experts", [(200, 272, 192, 100), (240, 656, 1088, 12), (240, 528, 2112, 24), (1100, 272, 320, 16),
                                                              (96, 1184, 576, 3), (97, 1184, 576, 3), (64, 208, 2048, 12), (300, 64, 512, 3), (300, 64, 576, 3),
                                                              (40, 24, 192, 9), (300, 200, 320, 4), (170, 136, 1088, 3)])
def test_batches_on_either_side_of_the_lines(cuda, n_tokens, n_rows, n_cols, n_experts, dual):
    rng = np.random.default_rng(n_tokens + n_cols)
    n_used = 2
    raws = [random_q4_0(rng, n_experts * n_rows, n_cols) for _ in range(1 + dual)]
    ws = [oracle.dequantize(2, raw, n_experts * n_rows * n_cols).reshape(n_experts, n_rows, n_cols).astype(np.float16).astype(np.float64) for raw in raws]
    x = rng.standard_normal((n_tokens, n_cols)).astype(np.float32)
    route = np.zeros((n_tokens, 2 * n_used), dtype=np.uint32)
    route[:, :n_used] = np.argsort(rng.random((n_tokens, n_experts)), axis=1)[:, :n_used]
    mats = [cuda.upload_matrix(Q4_0, raw, n_experts * n_rows, n_cols) for raw in raws]
    xb, rb = cuda.buffer_from(x), cuda.buffer_from(route)
    ob, eb = cuda.new_buffer((n_experts + 1) * 4), cuda.new_buffer(n_tokens * n_used * 4)
    out = cuda.buffer_from(np.full((n_tokens + 1, n_used, n_rows), 7, dtype=np.float32))
    cuda.begin()
    cuda.moe_group(rb, ob, eb, n_experts, n_used, n_tokens)
    cuda.matmul_experts(Q4_0, mats[0], mats[1] if dual else None, n_rows, n_cols, n_experts, xb, True, ob, eb, n_used, out, n_tokens)
    cuda.end()
    got = cuda.read(out, np.zeros((n_tokens + 1, n_used, n_rows), dtype=np.float32))
    assert (got[n_tokens] == 7).all()
    halves = x.astype(np.float16).astype(np.float64)
    want = np.empty((n_tokens, n_used, n_rows))
    for e in range(n_experts):
        t, s = np.nonzero(route[:, :n_used] == e)
        g = halves[t] @ ws[0][e].T
        want[t, s] = g / (1 + np.exp(-g)) * (halves[t] @ ws[1][e].T) if dual else g
    # Against float64 of the same fp16 operands, in the 2-norm: half as much again as sums in parts lose (2.0e-7, a SwiGLU of two 3.7e-7), and,
    # where one accumulator sums all of K, as much again of its 1.2e-9 (2.4e-9) a column.
    bound = 5.6e-7 if dual else 3e-7
    if 2 * n_tokens > 64 * n_experts or n_rows % 16:
        bound += 1.5 * (2.4e-9 if dual else 1.2e-9) * n_cols
    assert np.linalg.norm(got[:n_tokens] - want) / np.linalg.norm(want) < bound
