"""Purifications of the orders that take the spectral bounds another way.

Above 5,333 orbitals the one-launch purification leaves the Lanczos vectors to the bounds kernel, above
9,400 both paths take them from the launched form. The matrix is banded with an open gap, so no
eigensolve is needed: the projector commutes with it, is idempotent and has the trace. Bounds as for
a known spectrum: the stopping rule 1e-13 n_occ and the roundings of up to 40 squarings seen through the gap
(interval / gap < 11), relative to the vectors that the products are applied to.
"""
import os

import numpy as np
import pytest

from pm7b200 import api

pytestmark = pytest.mark.gpu


def _banded(n):
    rng = np.random.default_rng(n)
    occ = 2 * n // 3
    d = np.concatenate([np.linspace(-40.0, -6.0, occ), np.linspace(1.0, 10.0, n - occ)])
    rng.shuffle(d)
    f = np.diag(d)
    for k in range(1, 9):
        i = np.arange(n - k)
        f[i, i + k] = f[i + k, i] = rng.normal(size=n - k) * 0.25
    return f, occ


@pytest.mark.parametrize("n,gemm", [(5400, "dmma"), (9500, "i8")])
def test_projector_of_a_banded_matrix(n, gemm):
    f, occ = _banded(n)
    old = os.environ.get("PM7_SP2_GEMM")
    os.environ["PM7_SP2_GEMM"] = gemm
    try:
        p, info = api.sp2(f, occ)
    finally:
        if old is None:
            del os.environ["PM7_SP2_GEMM"]
        else:
            os.environ["PM7_SP2_GEMM"] = old
    assert info["settled"] and info["retries"] == 0 and info["i8"] == (gemm == "i8")
    tol = 2.0 * (1.0e-13 * occ + 40 * n * 1.1e-16 * 11.0)
    v = np.random.default_rng(0).normal(size=(n, 4))
    pv = p @ v
    assert abs(np.trace(p) - 2 * occ) < tol * occ
    assert np.abs(p @ pv - 2.0 * pv).max() < tol * np.abs(pv).max()
    assert np.abs(f @ pv - p @ (f @ v)).max() < tol * np.abs(f @ pv).max()
