"""The whole-GPU reduction alone: scales, exact multiplicities, uncoupled rows, and its grid.

Where a row lies (registers or shared memory, which block) depends on the grid, which follows the
device's SM count; the values may not. Against numpy the bound is that of the cluster kernel's tests:
1e-12 sqrt(n) of the largest level.
"""
import numpy as np
import pytest

from pm7b200 import api

pytestmark = pytest.mark.gpu


def _random(n, seed=0):
    a = np.random.default_rng(n + seed).standard_normal((n, n))
    return 0.5 * (a + a.T)


# (order, grids): registers alone, rows in shared memory, the 512-column boundaries of a thread
GRIDS = [(2, (1, 2)), (9, (1, 3, 9)), (40, (4, 7, 40)), (300, (0, 33, 75, 148)), (512, (0, 43, 100, 148)),
         (513, (0, 37, 74, 148)), (700, (0, 70, 83, 148)), (1300, (0, 100, 120, 148)), (2048, (0, 140, 147, 148))]


@pytest.mark.parametrize("n,grids", GRIDS)
def test_values_do_not_depend_on_the_grid(n, grids):
    a = _random(n)
    got = [api.levels(a, ctas=g) for g in grids]
    for w in got[1:]:
        np.testing.assert_array_equal(w, got[0])
    ref = np.linalg.eigvalsh(a)
    assert np.max(np.abs(got[0] - ref)) < 1e-12 * np.sqrt(n) * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("scale", [1e-180, 1e-30, 1e30, 1e120])
@pytest.mark.parametrize("n", [2, 40, 161, 700])
def test_values_at_the_ends_of_the_exponent_range(n, scale):
    a = _random(n, 1)
    ref = np.linalg.eigvalsh(a)
    assert np.max(np.abs(api.levels(a * scale) / scale - ref)) < 1e-12 * np.sqrt(n) * max(1.0, np.abs(ref).max())


def test_degenerate_uncoupled_and_zero_matrices():
    d = np.diag(np.repeat([1.0, -2.0, 0.0, 1.0], 30))
    np.testing.assert_allclose(api.levels(d), np.sort(np.diag(d)), rtol=0, atol=1e-12)
    block = np.zeros((600, 600))  # two coupled blocks with uncoupled zero rows between them
    block[:200, :200] = _random(200)
    block[400:, 400:] = _random(200)
    np.testing.assert_allclose(api.levels(block), np.linalg.eigvalsh(block), rtol=0, atol=1e-12 * np.sqrt(600) * 30)
    np.testing.assert_allclose(api.levels(np.zeros((64, 64))), 0.0, rtol=0, atol=1e-300)


@pytest.mark.parametrize("n,ctas", [(1, 0), (2049, 0), (700, 40), (2048, 100), (40, 41), (700, -1), (700, 149)])
def test_what_no_grid_can_hold_is_refused(n, ctas):
    with pytest.raises(api.Pm7Error) as e:
        api.levels(np.eye(n), ctas=ctas)
    assert e.value.code == 1
