"""The vocabulary's argmax, by one CTA up to 8192 values and cut over a cluster's CTAs beyond: every place a share or a 16-byte load ends, rows that do not
start on 16 bytes, ties in different shares, -inf everywhere."""

import numpy as np
import pytest

from bobcat_b200 import Cuda

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 31, 33, 4096, 8191, 8192, 8193, 65536, 65539, 100003])
@pytest.mark.parametrize("shift", [0, 1])
def test_argmax(n, shift):
    cuda = Cuda.open(0)
    rng = np.random.default_rng(n)
    out = cuda.new_buffer(4)
    places = sorted({0, n // 8, n // 2, n - 1})
    for first in places:
        x = rng.uniform(-1, 1, n + shift).astype(np.float32)
        x[[shift + i for i in places if i >= first]] = 2.0  # equal maxima from `first` on
        xb = cuda.buffer_from(x)
        cuda.begin(); cuda.argmax(xb.at(4 * shift), out, n); cuda.end()
        assert int(cuda.read(out, np.zeros(1, dtype=np.uint32))[0]) == first
    x = np.full(n + shift, -np.inf, dtype=np.float32)
    xb = cuda.buffer_from(x)
    cuda.begin(); cuda.argmax(xb.at(4 * shift), out, n); cuda.end()
    assert int(cuda.read(out, np.zeros(1, dtype=np.uint32))[0]) == 0
    cuda.close()
