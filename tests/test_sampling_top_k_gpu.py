"""Top-k draws at the edges of what one CTA sorts, with the other cuts after it, and equal logits among the candidates."""

import numpy as np
import pytest

from oracle import sampler as ref
from test_sampling_gpu import gpu_sample, settings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("top_k,top_p,min_p", [(1, 1.0, 0.0), (2, 0.9, 0.0), (32, 1.0, 0.02), (33, 0.8, 0.0), (700, 0.99, 0.0), (1024, 1.0, 0.0), (1025, 0.999, 0.001)])
def test_top_k_draws(cuda, top_k, top_p, min_p):
    rng = np.random.default_rng(top_k)
    logits = (rng.permutation(70001).astype(np.float32) / 70001 * 12 - 6).astype(np.float32)  # all different
    case = dict(temperature=1.3, top_k=top_k, top_p=top_p, min_p=min_p, repeat_penalty=1.0)
    _, probs = ref.candidates(logits, [], **case)
    edges = np.cumsum(probs.astype(np.float64))
    for uniform in np.linspace(0.003, 0.997, 25):
        if np.min(np.abs(edges - uniform)) < 2e-6 * top_k ** 0.5 + 1e-6:
            continue
        token, _ = gpu_sample(cuda, logits, [], settings(**case), float(uniform))
        assert token == ref.sample(logits, [], float(uniform), **case), uniform


def test_equal_logits_among_the_candidates(cuda):
    logits = np.full(65536, -5.0, dtype=np.float32)
    tied = np.array([7, 900, 8191, 8192, 40000, 65535])
    logits[tied] = 2.0
    for i, uniform in enumerate((np.arange(6) + 0.5) / 6):
        assert gpu_sample(cuda, logits, [], settings(1.0, top_k=6), float(uniform))[0] == tied[i]
        assert gpu_sample(cuda, logits, [], settings(1.0, top_k=3), float(uniform))[0] == tied[i]  # all equal to the cut value stay
