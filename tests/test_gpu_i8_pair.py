"""The SP2 step by CTA pairs (256 x 128 tiles, two passes over K) on the integer tensor cores.

Sizes: the first order that takes this path on 148 SMs, whole tiles, a ragged row and column
edge with an odd number of K blocks, and one with more tiles than pairs (a CTA then finishes a
tile beside the next one's products). Checked against the fp64 product: the bound of the step's
own error (2e-17 n of the largest element, times 4) plus that of the fp64 product (n eps / 4 of
its row sums of |x_ik x_kj| <= 1).
"""
import numpy as np
import pytest

from pm7b200 import api

pytestmark = pytest.mark.gpu


def _iterate(n, seed):
    rng = np.random.default_rng(seed)
    v = rng.normal(size=(n, n // 2)) / np.sqrt(n)
    x = 0.3 * (v @ v.T)  # spectrum in [0, 1)
    x[np.arange(n), np.arange(n)] += rng.uniform(0.0, 0.1, size=n)
    return 0.5 * (x + x.T)


@pytest.mark.parametrize("n", [1409, 1536, 1761, 2306])
@pytest.mark.parametrize("square", [True, False])
def test_pair_step_matches_fp64_product(n, square):
    x = _iterate(n, n)
    y, norms = api.sp2_step_i8(x, square)
    ref = x @ x if square else 2 * x - x @ x
    assert float(np.max(np.abs(y - ref))) < 8e-17 * n + n * 2.2e-16 / 4
    np.testing.assert_array_equal(y, y.T)
    assert abs(norms[0] - np.trace(y)) < 1e-12 * n
    assert abs(norms[1] - np.sum(y * y)) < 1e-12 * n
