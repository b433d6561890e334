"""An expired wait of the integer tensor-core squaring: status, tensor memory and context.

Each CTA's copies stop after two stages (a phase that nothing completes), so the pipeline's waits run
out; the kernels wait for the copies and MMAs that did start, free their tensor memory and return.
Single CTAs (300, 1,000 orbitals) and CTA pairs (1,500, 2,048); tensor memory that was not given back
would leave the next squaring without any.
"""
import time

import numpy as np
import pytest

from pm7b200 import api

pytestmark = pytest.mark.gpu

PM7_ERR_TIMEOUT = 10


@pytest.mark.parametrize("n", [300, 1000, 1500, 2048])
def test_expired_waits_report_timeout_and_the_next_squaring_is_right(n):
    t = time.perf_counter()
    assert api.i8_wait_drill(n) == PM7_ERR_TIMEOUT
    assert time.perf_counter() - t < 30.0
    rng = np.random.default_rng(n)
    v = rng.normal(size=(n, n // 2)) / np.sqrt(n)
    x = 0.3 * (v @ v.T)
    x = 0.5 * (x + x.T)
    y, _ = api.sp2_step_i8(x, True)
    assert float(np.max(np.abs(y - x @ x))) < 8e-17 * n + n * 2.2e-16 / 4
