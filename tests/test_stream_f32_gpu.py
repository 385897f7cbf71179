"""The f32 stream products at the edges of their row groups, steps of 128 columns and row counts."""

import numpy as np
import pytest

from bobcat_b200 import F32, OVERWRITE, Norm

pytestmark = pytest.mark.gpu


def products(w, x):
    return x.astype(np.float64) @ w.astype(np.float64).T, np.abs(x).astype(np.float64) @ np.abs(w).astype(np.float64).T


@pytest.mark.parametrize("n_rows,n_cols", [(4736, 32), (4739, 160), (9001, 1024), (30001, 288)])
def test_one_row_and_several_agree_with_f64_and_each_other(cuda, n_rows, n_cols):
    rng = np.random.default_rng(n_rows + n_cols)
    w = (rng.standard_normal((n_rows, n_cols)) / 16).astype(np.float32)
    x = rng.uniform(-1, 1, (16, n_cols)).astype(np.float32)
    nw = rng.uniform(0.5, 1.5, n_cols).astype(np.float32)
    wb, xb, nb = cuda.upload_matrix(F32, w.view(np.uint8), n_rows, n_cols), cuda.buffer_from(x), cuda.buffer_from(nw)
    yb = cuda.new_buffer(16 * n_rows * 4)
    cuda.begin(); cuda.matvec(F32, wb, n_rows, n_cols, xb, yb); cuda.end()
    one = cuda.read(yb, np.zeros(n_rows, dtype=np.float32))
    for n in (2, 4, 5, 8, 11, 16):
        cuda.begin(); cuda.matmul(F32, wb, n_rows, n_cols, xb, yb, n, OVERWRITE); cuda.end()
        got = cuda.read(yb, np.zeros((n, n_rows), dtype=np.float32))
        want, budget = products(w, x[:n])
        assert (np.abs(got - want) / budget).max() < 1e-6
        assert np.array_equal(got[0], one)
    cuda.begin(); cuda.matvec(F32, wb, n_rows, n_cols, xb, yb, norm=Norm(nb.at(0), 1e-5)); cuda.end()
    x0 = x[0].astype(np.float64)
    want, budget = products(w, (x0 / np.sqrt((x0 ** 2).mean() + 1e-5) * nw)[None])
    assert (np.abs(cuda.read(yb, np.zeros(n_rows, dtype=np.float32)) - want[0]) / budget[0]).max() < 1e-6
