"""The SwiGLU of a batch in one launch, every kernel that may serve it: tiles of 128 rows of both matrices and of 64
rows of either (weights expanded to fp16), the dequantising kernel, the few-row kernel with half and with
float operands; ragged row and token counts, and the result as the packed operand of the next product."""

import ctypes as C
import os

import numpy as np
import pytest

from bobcat_b200 import Q4_0
from conftest import random_q4_0
from oracle import oracle

pytestmark = pytest.mark.gpu

DEQUANT, FEW, WHOLE, HALVES, EXACT = range(5)
# (n_rows, n_cols, n_tokens): one to several row tiles of 128 and halves of 64, short of them, one token
# short of and past 16, 32, a tile's 128 and 256 tokens; few and many chunks of 64 columns.
SHAPES = [(64, 64, 33), (100, 64, 47), (128, 256, 128), (130, 1024, 129), (192, 2048, 64), (300, 128, 257), (704, 256, 100), (2816, 1024, 65), (2816, 1024, 255),
          (4608, 1024, 127), (6144, 2048, 200), (10752, 2048, 96), (10752, 2048, 512), (10752, 2048, 48), (12288, 4096, 33), (1000, 192, 513),
          (128, 128, 16), (100, 1088, 17), (4608, 1024, 31), (2048, 2048, 32), (48, 1024, 1), (1000, 2048, 15)]


def no_expanded_weights():
    return os.environ.get("BOBCAT_NO_HALF_MATMUL") == "1"


def form_of(cuda, gate, up, n_rows, n_cols, x, y, n_tokens, packed=False):
    form = C.c_int32(-1)
    cuda._check(cuda._L.bc_test_matmul_swiglu(cuda._h, gate._h, up._h, n_rows, n_cols, x._h if x else None, y._h if y else None, n_tokens, int(packed), C.byref(form)))
    return form.value


def unpacked(operand, n_rows, n_tokens):
    """The rows of a packed operand (packed_operand_index, device_utils.cuh), tokens rounded up to 16."""
    groups = (n_tokens + 15) // 16 * 2
    tok, col = np.arange(groups * 8)[:, None], np.arange(n_rows)[None, :]
    c, w, e = col & 63, col & 31, col & 3
    core, at = (c >> 5) * 4 + ((w & 15) >> 2), (w >> 4) * 4 + (e & 1) * 2 + (e >> 1)
    return operand[((((col >> 6) * groups + (tok >> 3)) * 8 + core) * 8 + (tok & 7)) * 8 + at]


@pytest.mark.parametrize("n_rows,n_cols,n_tokens", SHAPES)
def test_swiglu_of_a_batch(cuda, n_rows, n_cols, n_tokens):
    rng = np.random.default_rng(n_rows + n_cols + n_tokens)
    half = n_tokens >= 16
    raws = [random_q4_0(rng, n_rows, n_cols) for _ in range(2)]
    weights = [oracle.dequantize(2, raw, n_rows * n_cols).reshape(n_rows, n_cols) for raw in raws]
    x = rng.uniform(-1, 1, (n_tokens, n_cols)).astype(np.float32)
    if half:  # the tensor cores' operands, rounded once
        operands = [w.astype(np.float16).astype(np.float64) for w in weights]
        rows = x.astype(np.float16).astype(np.float64)
    else:
        operands, rows = [w.astype(np.float64) for w in weights], x.astype(np.float64)
    g, u = (rows @ w.T for w in operands)
    silu = g / (1 + np.exp(-g))
    want = silu * u
    # Float32 sums: 2e-5 of sum |w x| with half operands, 1e-6 with exact ones (tests of the single products); silu's slope is
    # at most 1.1. The activation itself adds a few units in the last place.
    sums = 2e-5 if half else 1e-6
    budget = [np.abs(rows) @ np.abs(w).T for w in operands]
    room = sums * (1.1 * budget[0] * np.abs(u) + budget[1] * np.abs(silu)) + 1e-6 * np.abs(want) + 1e-30
    gate, up = (cuda.upload_matrix(Q4_0, raw, n_rows, n_cols) for raw in raws)
    xb = cuda.buffer_from(x)
    guard = np.full((n_tokens + 1, n_rows), 7.5, dtype=np.float32)
    yb = cuda.buffer_from(guard)
    cuda.begin(); form_of(cuda, gate, up, n_rows, n_cols, xb, yb, n_tokens); cuda.end()
    got = cuda.read(yb, np.zeros_like(guard))
    assert float((np.abs(got[:n_tokens] - want) / room).max()) < 1
    assert (got[n_tokens] == 7.5).all()
    buffers = [gate, up, xb, yb]
    if half and n_rows % 64 == 0:
        tokens = (n_tokens + 15) // 16 * 16
        guard = np.full(tokens * n_rows + 64, 7.5, dtype=np.float16)
        pb = cuda.buffer_from(guard)
        buffers.append(pb)
        cuda.begin(); form_of(cuda, gate, up, n_rows, n_cols, xb, pb, n_tokens, packed=True); cuda.end()
        operand = cuda.read(pb, np.zeros_like(guard))
        assert (operand[tokens * n_rows:] == 7.5).all()
        out = unpacked(operand, n_rows, n_tokens).astype(np.float64)
        # Rounded to fp16 once more: half a unit in the last of 11 bits, or of the subnormal step 2^-24.
        assert float((np.abs(out[:n_tokens] - want) / (room + 2.0 ** -11 * np.abs(want) + 2.0 ** -25)).max()) < 1.01
        assert (out[n_tokens:] == 0).all()  # the operand's rows past the tokens
    for buffer in buffers:
        buffer.free()


def test_the_shapes_reach_every_kernel(cuda):
    rng = np.random.default_rng(0)
    seen = {}
    cuda.begin()
    for n_rows, n_cols, n_tokens in SHAPES:
        gate, up = (cuda.upload_matrix(Q4_0, random_q4_0(rng, n_rows, n_cols), n_rows, n_cols) for _ in range(2))
        seen.setdefault(form_of(cuda, gate, up, n_rows, n_cols, None, None, n_tokens), []).append((n_rows, n_cols, n_tokens))
        gate.free(), up.free()
    cuda.end()
    assert sorted(seen) == ([DEQUANT, FEW, EXACT] if no_expanded_weights() else [FEW, WHOLE, HALVES, EXACT]), seen
