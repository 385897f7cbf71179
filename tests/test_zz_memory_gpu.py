"""The copies of weights expanded for products of many tokens are optional: when the library cannot allocate what a
call needs, it gives them back and goes on with the kernels that read the Q4_0 layouts. Checked for a sequence's state
(contiguous and paged), for the scratch of a pass that is under way, for buffers, and with another thread prefilling
meanwhile. The device is filled up to a known rest with plain allocations. Collected late on purpose."""

import threading

import numpy as np
import pytest

from bobcat_b200 import OVERWRITE, Q4_0, Cuda, Model, SeqCuda, errors
from conftest import random_q4_0, rel_error

pytestmark = pytest.mark.gpu

MB = 1 << 20
# 287 M weights of lfm2-350m, two bytes each.
COPIES = 574 * MB
# The two kernels multiply the same rounded operands and add in another order, which now and then rounds a later
# fp16 activation the other way: the class of a half-precision prefill against exact operands.
TOLERANCE = 5e-3


class Filled:
    """All of the device's free memory but `rest` bytes, taken."""

    def __init__(self, rest):
        self.rest = rest

    def __enter__(self):
        import torch

        torch.cuda.empty_cache()
        self.blocks = []
        while True:
            left = torch.cuda.mem_get_info()[0] - self.rest
            if left < 2 * MB:
                break
            try:
                self.blocks.append(torch.empty(min(left, 8 << 30) // (2 * MB) * (2 * MB), dtype=torch.uint8, device="cuda"))
            except torch.OutOfMemoryError:  # the last few megabytes may lie apart
                break
        return self

    def __exit__(self, *_):
        import torch

        self.blocks = []
        torch.cuda.empty_cache()


def prompt_of(model, n, seed):
    return np.random.default_rng(seed).integers(0, model.hp.n_vocab, size=n).astype(np.uint32)


def logits_of(seq, prompt):
    seq.reset()
    out = np.zeros(seq.model.hp.n_vocab, dtype=np.float32)
    seq.prefill(prompt, out)
    return out


@pytest.mark.parametrize("paged", [False, True])
def test_a_sequence_takes_the_place_of_the_copies(model_path, paged):
    model, cuda, other = Model.load(model_path("lfm2-350m")), Cuda.open(0), Cuda.open(0)
    prompt = prompt_of(model, 100, 1)
    first, busy = SeqCuda(model, cuda, 128, True), SeqCuda(model, other, 128, True)
    want = logits_of(first, prompt)
    assert rel_error(logits_of(busy, prompt), want) == 0.0
    stop, seen = threading.Event(), []

    def keep_prefilling():
        try:
            while not stop.is_set():
                seen.append(rel_error(logits_of(busy, prompt), want))
        except Exception as e:  # told to the test below
            seen.append(e)

    thread = threading.Thread(target=keep_prefilling)
    with Filled(256 * MB):
        thread.start()
        try:
            # 12 KB of cache per position: 400 MB, more than is free, less than what is free and the copies.
            second = SeqCuda(model, cuda, 34000, True, paged=paged)
        finally:
            stop.set()
            thread.join()
        assert seen and all(isinstance(e, float) and e < TOLERANCE for e in seen), seen[-1]
        for seq in (second, first, busy):
            assert rel_error(logits_of(seq, prompt), want) < TOLERANCE
        assert len(second.generate(4)) == 4
    for handle in (second, busy, first, other, cuda, model):
        handle.close()


def test_a_pass_that_lacks_scratch_gives_its_own_copies_back(model_path):
    model, warm, cuda = Model.load(model_path("lfm2-350m")), Cuda.open(0), Cuda.open(0)
    prompt = prompt_of(model, 512, 2)
    first = SeqCuda(model, warm, 512, True)
    want = logits_of(first, prompt)  # loads the kernels
    seq = SeqCuda(model, cuda, 512, True)  # whose backend has no scratch yet
    with Filled(4 * MB):
        assert rel_error(logits_of(seq, prompt), want) < TOLERANCE
    for handle in (seq, first, cuda, warm, model):
        handle.close()


def test_a_buffer_takes_the_place_of_a_matrix_copy():
    cuda = Cuda.open(0)
    rng = np.random.default_rng(3)
    n_rows, n_cols, n_tokens = 16384, 2048, 64  # 64 MB expanded
    wb = cuda.upload_matrix(Q4_0, random_q4_0(rng, n_rows, n_cols), n_rows, n_cols)
    xb, yb = cuda.buffer_from(rng.uniform(-1, 1, (n_tokens, n_cols)).astype(np.float32)), cuda.new_buffer(n_tokens * n_rows * 4)

    def product():
        cuda.begin(); cuda.matmul(Q4_0, wb, n_rows, n_cols, xb, yb, n_tokens, OVERWRITE); cuda.end()
        return cuda.read(yb, np.zeros((n_tokens, n_rows), dtype=np.float32))

    want = product()
    with Filled(24 * MB):
        room = cuda.new_buffer(60 * MB)
        assert rel_error(product(), want) < 1e-5  # the same operands, another order of float32 sums
    for buffer in (room, yb, xb, wb):
        buffer.free()
    cuda.close()


def test_a_copy_in_a_callers_graph_stays():
    """A product recorded into a graph of the caller's keeps its matrix's copy for good, and a matrix first met there is
    multiplied without one (nothing may be allocated during a capture)."""
    import torch

    stream = torch.cuda.Stream()
    cuda = Cuda.open(0, stream.cuda_stream)
    rng = np.random.default_rng(4)
    n_rows, n_cols, n_tokens = 16384, 2048, 64
    raw = random_q4_0(rng, n_rows, n_cols)
    known, unmet = (cuda.upload_matrix(Q4_0, raw, n_rows, n_cols) for _ in range(2))
    xb = cuda.buffer_from(rng.uniform(-1, 1, (n_tokens, n_cols)).astype(np.float32))
    ya, yb = (cuda.new_buffer(n_tokens * n_rows * 4) for _ in range(2))
    zeros = np.zeros((n_tokens, n_rows), dtype=np.float32)
    cuda.begin(); cuda.matmul(Q4_0, known, n_rows, n_cols, xb, ya, n_tokens, OVERWRITE); cuda.end()
    want = cuda.read(ya, zeros.copy())
    graph = torch.cuda.CUDAGraph()
    cuda.begin()
    with torch.cuda.graph(graph, stream=stream):
        cuda.matmul(Q4_0, known, n_rows, n_cols, xb, ya, n_tokens, OVERWRITE)
        cuda.matmul(Q4_0, unmet, n_rows, n_cols, xb, yb, n_tokens, OVERWRITE)
    cuda.end()
    cuda.write(ya, zeros)
    with Filled(24 * MB):
        rooms = []
        with pytest.raises(errors.Allocation):  # whatever else holds copies gives them up first
            for _ in range(4000):
                rooms.append(cuda.new_buffer(60 * MB))
        with torch.cuda.stream(stream):
            graph.replay()
        assert np.array_equal(cuda.read(ya, zeros.copy()), want)
        assert rel_error(cuda.read(yb, zeros.copy()), want) < 1e-5
    del graph
    for buffer in (*rooms, yb, ya, xb, unmet, known):
        buffer.free()
    cuda.close()
