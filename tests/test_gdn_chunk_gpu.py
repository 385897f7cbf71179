"""The delta rule in chunks of 64 tokens against the rule token by token in float64: batches that end
inside a chunk, on its edges and on the edges of its 16-row blocks, every key width, and decays down
to zero."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rule(q, k, v, beta, decay, state):
    """q, k [n][k_heads][kd], v [n][v_heads][vd], gates [n][v_heads], state [v_heads][kd][vd]."""
    S, out = state.astype(np.float64).copy(), np.zeros(v.shape)
    n_k = q.shape[1]
    for t in range(q.shape[0]):
        for h in range(v.shape[1]):
            kk, qq = k[t, h % n_k].astype(np.float64), q[t, h % n_k].astype(np.float64)
            S[h] *= decay[t, h]
            S[h] += np.outer(kk, (v[t, h] - kk @ S[h]) * beta[t, h])
            out[t, h] = qq @ S[h]
    return out, S


@pytest.mark.parametrize("n,kd,vd,n_k,n_v", [(12, 128, 128, 2, 4), (16, 32, 32, 1, 2), (33, 64, 64, 2, 2), (63, 96, 32, 1, 1), (64, 128, 128, 2, 4),
                                              (65, 128, 32, 1, 3), (130, 128, 256, 1, 2), (512, 128, 128, 1, 2)])
def test_chunks_follow_the_rule(cuda, n, kd, vd, n_k, n_v):
    rng = np.random.default_rng(n + kd)
    q, k = (rng.standard_normal((n, n_k, kd)) for _ in range(2))
    q, k = q / np.linalg.norm(q, axis=2, keepdims=True) / np.sqrt(kd), k / np.linalg.norm(k, axis=2, keepdims=True)
    k[1::3] = 0.9 * k[1::3] + 0.1 * k[::3][: len(k[1::3])]  # neighbours that overlap: the system is not close to the identity
    v = rng.standard_normal((n, n_v, vd))
    beta, decay = rng.uniform(0, 1, (n, n_v)), rng.uniform(0.7, 1, (n, n_v)) ** rng.integers(0, 40, (n, n_v))
    decay[5] = 0.0
    state = rng.standard_normal((n_v, kd, vd))
    qkv = np.concatenate([q.reshape(n, -1), k.reshape(n, -1), v.reshape(n, -1)], axis=1).astype(np.float32)
    beta, decay, state = (a.astype(np.float32) for a in (beta, decay, state))
    q, k, v = qkv[:, :n_k * kd].reshape(n, n_k, kd), qkv[:, n_k * kd:2 * n_k * kd].reshape(n, n_k, kd), qkv[:, 2 * n_k * kd:].reshape(n, n_v, vd)
    want, want_state = rule(q, k, v, beta, decay, state)
    qb, bb, db, sb, ob = (cuda.buffer_from(a) for a in (qkv, beta, decay, state, np.zeros((n, n_v, vd), dtype=np.float32)))
    cuda.begin()
    cuda.gdn_recurrence(qb, bb, db, sb, ob, n_k, n_v, kd, vd, n, normalize=False)
    cuda.end()
    out, after = cuda.read(ob, np.zeros((n, n_v, vd), dtype=np.float32)), cuda.read(sb, np.zeros((n_v, kd, vd), dtype=np.float32))
    assert float(np.abs(out - want).max()) < 5e-6 * float(np.abs(want).max())
    assert float(np.abs(after - want_state).max()) < 5e-6 * max(1.0, float(np.abs(want_state).max()))
