"""A decoded token's attention on each of its kernels: a sequence opened for a short context takes one launch, a longer one a
chunk pass and a combine pass. The same tokens through sequences that differ only in what they can hold,
against the CPU checker, at the ends of a chunk (16), of a cluster's round (32 chunks) and behind it."""

import numpy as np
import pytest

from bobcat_b200 import Lfm2Cuda, Model, Qwen35Cuda, synth
from conftest import rel_error
from oracle import oracle

pytestmark = pytest.mark.gpu

# The reference's bounds (crates/bobcat/tests/lfm2_reference.rs:19-25): f32 cache 1e-4, half cache 5e-3.
TOLERANCE = {False: 1e-4, True: 5e-3}
CHECKS = (0, 15, 16, 63, 64, 255, 511, 512, 539)
FEW = (0, 15, 16, 63, 64, 255)


def lfm2(heads, kv_heads, head_dim):
    return dict(arch="lfm2", vocab=512, hidden=heads * head_dim, layers=3, attention=[1, 2], heads=heads, kv_heads=kv_heads, ff=256,
                conv_kernel=3, theta=1e6, eps=1e-5)


def qwen(heads, kv_heads):
    return dict(arch="qwen35", vocab=512, hidden=128, layers=4, heads=heads, kv_heads=kv_heads, head_dim=256, n_rot=64, ff=256, k_heads=2,
                v_heads=4, k_dim=32, v_dim=32, conv_kernel=4, theta=1e7, eps=1e-6)


# Contexts: up to 2048 positions of heads of 64 elements (1024 of 128, 512 of 256) one launch; beyond, chunks of 16 up to 4096, then of 64.
@pytest.mark.parametrize("config, contexts, checks", [
    (lfm2(4, 2, 64), (640, 4096, 5000), CHECKS),
    (lfm2(8, 2, 64), (2048, 2049), CHECKS),
    (lfm2(3, 3, 64), (640, 40000), FEW),
    (lfm2(4, 1, 128), (1024, 1025), CHECKS),
    (lfm2(2, 1, 256), (512, 513, 1000), CHECKS),
    (qwen(2, 1), (512, 513, 1000), CHECKS),
    (qwen(4, 1), (300, 5000), FEW),
], ids=["64x2", "64x4", "64x1", "128x4", "256x2", "gated-256x2", "gated-256x4"])
def test_contexts_of_every_length(tmp_path, cuda, config, contexts, checks):
    path = synth.write_model(str(tmp_path / "model.gguf"), config, 3)
    model, ref = Model.load(path), oracle.Model(path)
    seq_class = Qwen35Cuda if config["arch"] == "qwen35" else Lfm2Cuda
    tokens = np.random.default_rng(9).integers(0, 512, size=max(checks) + 1).astype(np.uint32)
    st = ref.state(len(tokens))
    want = {}
    for pos, token in enumerate(tokens):
        step = st.step(int(token), want_logits=pos in checks)
        if pos in checks:
            want[pos] = step["logits"]
    for kv_half in (True, False):
        got = []
        for n_ctx in contexts:
            seq = seq_class(model, cuda, n_ctx, kv_half)
            logits = np.zeros(512, dtype=np.float32)
            here = {}
            for pos, token in enumerate(tokens[:n_ctx]):
                seq.step(int(token), logits)
                if pos in checks:
                    here[pos] = logits.copy()
                    assert rel_error(logits, want[pos]) < TOLERANCE[kv_half], (kv_half, n_ctx, pos)
            got.append(here)
        # Over a half cache both forms add the same chunks of 16 in the same order.
        for n_ctx, here in zip(contexts[1:], got[1:]):
            for pos in set(here) & set(got[0]):
                if kv_half and n_ctx <= 4096:
                    assert np.array_equal(here[pos], got[0][pos]), (n_ctx, pos)
                else:
                    assert rel_error(here[pos], got[0][pos]) < TOLERANCE[False], (kv_half, n_ctx, pos)
